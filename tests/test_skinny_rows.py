"""The products of few rows (gemm_skinny_f64: two output columns per warp) at an odd and an even number of externals,
one external, and one, two and several rows per integral matrix, against the numpy interpreter of the same plan."""
import numpy as np
import pytest

import tigerci_b200 as T
from plan_exec import PlanInterpreter
from tigerci_b200.synthetic import random_civec, synthetic_operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ext", [1, 2, 7, 32, 33, 64])
@pytest.mark.parametrize("ni,na,ne,mult,ref", [(2, 0, 4, 1, "22"), (1, 2, 4, 3, "211"), (2, 3, 7, 2, "22210")])
def test_against_plan_interpreter(n_ext, ni, na, ne, mult, ref, need_gpu, tmp_path):
    d = T.Deck(ni + na + n_ext, ni, na, ne, mult, [ref])
    h, L = synthetic_operator(d.num_orbitals, 14, seed=n_ext, scale=0.1, diag_range=(-2.0, 1.0), offdiag_sigma=0.02)
    op = T.Operator(h, L)
    sb = T.SigmaBuilder(d, op)
    x = random_civec(sb.n, 2)
    got = sb.sigma(x)
    sb.close()
    path = str(tmp_path / "p.plan")
    T.Plan(d, op).export(path)
    ref_s = PlanInterpreter(path, h, L).sigma(x)
    assert np.abs(got - ref_s).max() <= 1e-10 * np.abs(ref_s).max()  # the repository's FP64 sigma tolerance
