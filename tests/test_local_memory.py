"""The device bytes the FP64 pair-domain operator gives to the packed integrals: a caller's bound holds whatever its size,
an allocation that fails falls back to the Cholesky form, and a local deck's context keeps room for what it allocates
afterwards."""
import numpy as np
import pytest

import tigerci_b200 as T
from tigerci_b200 import local
from tigerci_b200._lib import TciError, lib
from tigerci_b200.synthetic import random_civec, synthetic_operator

pytestmark = pytest.mark.gpu


def test_bound_default_and_fallback(need_gpu):
    n_virt, n_int = 320, 17
    heads, dom, total = local.pair_domain_problem(150, n_int, n_virt, 20, 150, seed=5)
    _, L = synthetic_operator(n_int + n_virt, 1000, seed=4, scale=0.5)
    x_bytes = 8 * (n_virt * (n_virt + 1) // 2) ** 2
    assert x_bytes > 20e9
    c = random_civec(total, 3)

    def run(expect, **kw):
        op = local.LocalAllExternal(n_int, n_virt, L, heads, dom, total, autotune=False, **kw)
        assert op.stats()["form"] == expect
        assert (op.stats()["device_bytes"] > x_bytes) == (expect == "integral")
        s = op.apply(c)
        op.close()
        return s

    ref = run("integral")
    # FP64 sums of at most 150^2 products of 1000-term integrals: far inside the repository's 1e-10
    tol = 1e-12 * np.abs(ref).max()
    assert np.abs(run("cholesky", chunk_bytes=20e9) - ref).max() <= tol
    assert np.array_equal(run("integral", chunk_bytes=30e9), ref)
    lib().tci_selftest_local_alloc_limit(x_bytes - 1)
    try:
        assert np.abs(run("cholesky") - ref).max() <= tol
        with pytest.raises(TciError) as e:
            run("integral", form="integral")
        assert e.value.code == 5
    finally:
        lib().tci_selftest_local_alloc_limit(0)
    assert np.array_equal(run("integral"), ref)


def test_context_keeps_room_for_its_later_allocations(need_gpu):
    import torch

    n_int, n_ext = 3, 200
    rng = np.random.default_rng(8)
    pick = lambda: np.sort(rng.choice(n_ext, size=int(rng.integers(140, 180)), replace=False)).tolist()
    args = (n_int + n_ext, n_int, 0, 2 * n_int, 1, ["2" * n_int])
    base = T.CsfSpace(T.Deck(*args)).counts()
    deck = T.Deck(*args, nm1_domains=[pick() for _ in range(base["paths_nm1"])],
                  nm2_domains=[pick() for _ in range(base["paths_nm2"])])
    h, L = synthetic_operator(deck.num_orbitals, 300, seed=3, scale=0.05, diag_range=(-2.0, 1.0), offdiag_sigma=0.02)
    op = T.Operator(h, L)
    x_bytes = 8 * (n_ext * (n_ext + 1) // 2) ** 2  # 3.2 GB

    def build(leave):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        hold = None
        if leave:
            hold = torch.empty(int(torch.cuda.mem_get_info()[0] - leave), dtype=torch.uint8, device="cuda")
        free = torch.cuda.mem_get_info()[0]
        sb = T.SigmaBuilder(deck, op)
        used = free - torch.cuda.mem_get_info()[0]
        s = sb.sigma(random_civec(sb.n, 1))
        sb.close()
        del hold
        torch.cuda.empty_cache()
        return s, used

    ref, used = build(0)
    assert used > x_bytes  # room enough: the integrals are there
    # 10 GB: the operator alone would fit them (0.6 of the free memory), but not beside the 8 GB the context keeps
    got, used = build(10e9)
    assert used < x_bytes
    assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()  # the repository's FP64 sigma tolerance
