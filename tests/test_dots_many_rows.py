"""tci_dots with more row groups than one launch's grid takes in y (4 x 65535 rows)."""
import pytest

import tigerci_b200 as T
from tigerci_b200.synthetic import synthetic_operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [4 * 65535, 4 * 65535 + 1, 2 * 4 * 65535 + 7])
def test_many_rows(m, need_gpu):
    import torch

    h, L = synthetic_operator(9, 8, seed=2, scale=0.1)
    sb = T.SigmaBuilder(T.Deck(9, 3, 0, 6, 1, ["222"]), T.Operator(h, L))
    n, lda = 3, 5
    g = torch.Generator(device="cuda").manual_seed(m)
    A = torch.randn(m, lda, generator=g, device="cuda", dtype=torch.float64)
    x = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    out = torch.full((m,), float("nan"), device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    sb.dots(A.data_ptr(), lda, m, x.data_ptr(), n, out.data_ptr())
    torch.cuda.synchronize()
    # n products and sums on either side, |a||x| summed
    ref, mag = (A[:, :n] * x).sum(1), (A[:, :n] * x).abs().sum(1)
    assert ((out - ref).abs() <= 2 * (n + 2) * 2.0 ** -53 * mag).all()
    sb.close()
