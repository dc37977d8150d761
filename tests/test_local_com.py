"""The two-external products of a local deck on the common virtuals (local_com.cu) in every row-tile class (domains
up to 126, 280 and above), with more than 48 common columns per term, and with the integral operands gathered instead of compacted (a
device without room for the copies): against the non-local FP64 sigma of the same deck on the padded vector."""
import numpy as np
import pytest
import torch

import tigerci_b200 as T
from local_helpers import injection
from oracle import sgga
from tigerci_b200.synthetic import random_civec, synthetic_operator

pytestmark = pytest.mark.gpu


def _check(n_int, n_ext, sizes1, sizes2, gathered):
    rng = np.random.default_rng(n_ext)
    nm1 = [np.sort(rng.choice(n_ext, size=m, replace=False)).tolist() for m in sizes1]
    nm2 = [np.sort(rng.choice(n_ext, size=m, replace=False)).tolist() for m in sizes2]
    args = (n_int + n_ext, n_int, 0, 2 * n_int, 1, ["2" * n_int])
    base, loc = T.Deck(*args), T.Deck(*args, nm1_domains=nm1, nm2_domains=nm2)
    h, L = synthetic_operator(base.num_orbitals, 24, seed=3, scale=0.05, diag_range=(-2.0, 1.0), offdiag_sigma=0.02)
    P = injection(loc, nm1, nm2, sgga.build_space(sgga.Deck(*args)), n_ext)
    op = T.Operator(h, L)
    nl = T.SigmaBuilder(base, op)
    x = random_civec(len(P), 1)
    full = np.zeros(nl.n)
    full[P] = x
    ref = nl.sigma(full)[P]
    nl.close()
    hold = None
    if gathered:  # leave less than the margin the compact copies need
        torch.cuda.empty_cache()
        hold = torch.empty(int(torch.cuda.mem_get_info()[0] - 6e9), dtype=torch.uint8, device="cuda")
    lc = T.SigmaBuilder(loc, op)
    got = lc.sigma(x)
    assert np.array_equal(got, lc.sigma(x))
    lc.close()
    del hold
    torch.cuda.empty_cache()
    assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()  # the repository's FP64 sigma tolerance


def test_row_tile_classes(need_gpu):
    _check(2, 290, [290, 283], [281, 127, 290], gathered=False)


@pytest.mark.parametrize("gathered", [False, True])
def test_common_columns_and_gathered_operands(gathered, need_gpu):
    _check(4, 140, [1, 17, 64, 140], [1, 2, 15, 16, 17, 63, 64, 65, 126, 140], gathered)
