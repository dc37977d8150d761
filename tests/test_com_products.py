"""The two-external products of a local deck on the common virtuals (tci_selftest_com) against numpy at the edges of the
row-tile classes and of the column windows (domains of 126, 280, 1200 and 2100 externals), compact and gathered."""
import numpy as np
import pytest

from tigerci_b200._lib import lib, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 126, 127, 281, 1200, 1201, 2100, 2101, 2407])
@pytest.mark.parametrize("compact", [1, 0])
def test_against_numpy(m, compact, need_gpu):
    rng = np.random.default_rng(m)
    n = m + 9
    pick = lambda k: np.sort(rng.choice(n, size=k, replace=False)).astype(np.int64)
    dom = pick(m)
    src = [pick(k) for k in (n, max(1, m // 3), 5)]
    alpha = np.array([1.0, -0.5, 2.0 ** 0.5])
    A, D = (rng.uniform(-0.5, 0.5, (3, n, n)) for _ in range(2))
    R = rng.uniform(-0.5, 0.5, (n, n))
    got = R.copy()
    ms = np.array([len(s) for s in src], dtype=np.int64)
    rc = lib().tci_selftest_com(0, n, m, ptr(dom), 3, ptr(ms), ptr(np.concatenate(src)), ptr(alpha), ptr(A), ptr(D), compact,
                                ptr(got))
    assert rc == 0
    ref, mag = R.copy(), np.abs(R)
    for s, d in enumerate(src):
        both = np.intersect1d(dom, d)
        a, x = A[s][np.ix_(dom, d)], D[s][np.ix_(d, both)]
        ref[np.ix_(dom, both)] += alpha[s] * (a @ x)
        mag[np.ix_(dom, both)] += abs(alpha[s]) * (np.abs(a) @ np.abs(x))
    # sum_s (m_s products) + alpha and the sums: that many roundings of at most mag on either side
    assert (np.abs(got - ref) <= 2 * (int(ms.sum()) + 8) * 2.0 ** -53 * mag).all()
    out = np.ones(n, dtype=bool)
    out[dom] = False
    assert (got[out] == R[out]).all() and (got[:, out] == R[:, out]).all()
