"""tci_dots on the caller's stream: vector lengths at the edges of its blocks, row counts at the edges of its row groups,
odd leading dimensions, two streams sharing a context's scratch, and a call inside a graph capture followed by calls
outside it."""
import numpy as np
import pytest

import tigerci_b200 as T
from tigerci_b200.synthetic import synthetic_operator

pytestmark = pytest.mark.gpu


def _builder():
    h, L = synthetic_operator(9, 8, seed=2, scale=0.1)
    return T.SigmaBuilder(T.Deck(9, 3, 0, 6, 1, ["222"]), T.Operator(h, L))


def test_lengths_rows_and_streams(need_gpu):
    import torch

    sb = _builder()
    g = torch.Generator(device="cuda").manual_seed(3)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    todo = []
    for k, n in enumerate((1, 31, 1023, 1024, 1025, 4097, 40539, 606209)):
        for m in (1, 3, 4, 5, 29):
            lda = n + (k % 3)
            A = torch.randn(m, lda, generator=g, device="cuda", dtype=torch.float64)
            x = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
            out = torch.full((m,), float("nan"), device="cuda", dtype=torch.float64)
            torch.cuda.synchronize()
            sb.dots(A.data_ptr(), lda, m, x.data_ptr(), n, out.data_ptr(), streams[len(todo) % 2].cuda_stream)
            todo.append((A, x, out, n))
    torch.cuda.synchronize()
    for A, x, out, n in todo:
        ref = A[:, :n] @ x
        # n products and sums on either side, |a||x| summed
        bound = 2 * (n + 2) * 2.0 ** -53 * (A[:, :n].abs() @ x.abs())
        assert ((out - ref).abs() <= bound).all()
    sb.close()


def test_capture_then_plain_calls(need_gpu):
    import torch

    sb = _builder()
    m, n = 5, 5000
    A = torch.randn(m, n, device="cuda", dtype=torch.float64)
    x = torch.randn(n, device="cuda", dtype=torch.float64)
    out, out2 = torch.zeros(m, device="cuda", dtype=torch.float64), torch.zeros(m, device="cuda", dtype=torch.float64)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    sb.dots(A.data_ptr(), n, m, x.data_ptr(), n, out.data_ptr(), s.cuda_stream)
    s.synchronize()
    ref = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
        sb.dots(A.data_ptr(), n, m, x.data_ptr(), n, out2.data_ptr(), s.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out2, ref)
    out.zero_()
    sb.dots(A.data_ptr(), n, m, x.data_ptr(), n, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
    del graph
    sb.close()
