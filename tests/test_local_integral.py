"""The pair-domain all-external term from the integrals on the domains (form "integral") against the oracle's
integral form: domains of one external up to all of them, more externals than one column chunk, heads with several
64-wide pieces, several heads per external and heads with a singlet block only."""
import numpy as np
import pytest

from oracle import dense
from tigerci_b200 import local
from tigerci_b200.synthetic import random_civec, synthetic_operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pairs,n_int,n_virt,dmin,dmax", [(15, 5, 9, 1, 9), (10, 5, 33, 1, 33), (21, 6, 64, 63, 64),
                                                            (12, 5, 70, 5, 70), (6, 3, 131, 60, 131)])
def test_integral_form_matches_oracle(n_pairs, n_int, n_virt, dmin, dmax, need_gpu):
    heads, dom, total = local.pair_domain_problem(n_pairs, n_int, n_virt, dmin, dmax, seed=n_virt)
    _, L = synthetic_operator(n_int + n_virt, 40, seed=4, scale=0.5)
    c = random_civec(total, 3)
    ref = dense.allext_local_sigma(n_int, L, heads, dom, c)
    op = local.LocalAllExternal(n_int, n_virt, L, heads, dom, total, form="integral")
    assert op.stats()["form"] == "integral"
    got = op.apply(c)
    # FP64 sums of at most 131^2 products of 40-term integrals: far inside the repository's 1e-10
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.array_equal(got, op.apply(c))
    op.close()
    ch = local.LocalAllExternal(n_int, n_virt, L, heads, dom, total, form="cholesky")
    assert np.abs(ch.apply(c) - got).max() <= 1e-12 * np.abs(ref).max()
    ch.close()


def test_integral_form_refused_in_mixed_precision(need_gpu):
    heads, dom, total = local.pair_domain_problem(5, 3, 12, 2, 12, seed=1)
    _, L = synthetic_operator(15, 10, seed=4)
    with pytest.raises(Exception):
        local.LocalAllExternal(3, 12, L, heads, dom, total, precision="tf32x3", form="integral")


def test_integral_form_more_columns_than_a_block_holds(need_gpu):
    """91 pairs whose domains nearly all hold every external: up to 182 columns for one a, in batches, jobs of several
    passes and of single columns."""
    heads, dom, total = local.pair_domain_problem(91, 13, 20, 17, 20, seed=2)
    _, L = synthetic_operator(33, 30, seed=4, scale=0.5)
    c = random_civec(total, 3)
    ref = dense.allext_local_sigma(13, L, heads, dom, c)
    op = local.LocalAllExternal(13, 20, L, heads, dom, total, form="integral")
    got = op.apply(c)
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.array_equal(got, op.apply(c))
    op.close()
