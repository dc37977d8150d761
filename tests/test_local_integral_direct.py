"""The integral form of the pair-domain all-external term as "auto" takes it, at sizes whose row tiles fill the chip
without copies of sigma (and just not), with one and two batches of accumulator columns: against the Cholesky form."""
import numpy as np
import pytest

from tigerci_b200 import local
from tigerci_b200.synthetic import random_civec, synthetic_operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_virt,dmin,dmax,parts", [(300, 20, 150, 2), (320, 20, 150, 1), (250, 120, 200, 1)])
def test_auto_takes_the_integrals(n_virt, dmin, dmax, parts, need_gpu):
    n_int = 17
    heads, dom, total = local.pair_domain_problem(150, n_int, n_virt, dmin, dmax, seed=n_virt)
    _, L = synthetic_operator(n_int + n_virt, 1000, seed=4, scale=0.5)
    c = random_civec(total, 3)
    op = local.LocalAllExternal(n_int, n_virt, L, heads, dom, total)
    st = op.stats()
    assert st["form"] == "integral" and st["integral_parts"] == parts
    assert 0 < st["integral_flops"] < st["flops"]
    got = op.apply(c)
    assert np.array_equal(got, op.apply(c))
    op.close()
    ch = local.LocalAllExternal(n_int, n_virt, L, heads, dom, total, form="cholesky")
    ref = ch.apply(c)
    assert ch.stats()["form"] == "cholesky" and ch.stats()["integral_parts"] == 0
    ch.close()
    # FP64 sums of at most 200^2 products of 1000-term integrals: far inside the repository's 1e-10
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
