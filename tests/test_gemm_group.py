"""Launches of the FP64 matrix-instruction GEMM with problems of many heights (tci_selftest_gemm_f64_group): one launch for
all of them where the heights' own launches would leave the chip idle, one each where they fill it; results against
numpy in every pair of operand modes and height."""
import numpy as np
import pytest

from tigerci_b200._lib import lib, ptr

ROW_CLASSES = 96


def _run(device, M, N, K, tA=0, tB=0, pad=0, A=None, B=None, C=None):
    M, N, K = (np.asarray(x, dtype=np.int64) for x in (M, N, K))
    tiles = np.zeros(ROW_CLASSES + 6, dtype=np.int64)
    rc = lib().tci_selftest_gemm_f64_group(device, len(M), ptr(M), ptr(N), ptr(K), tA, tB, pad, ptr(A) if A is not None else None,
                                           0 if A is None else A.size, ptr(B) if B is not None else None, 0 if B is None else B.size,
                                           ptr(C) if C is not None else None, 0 if C is None else C.size, ptr(tiles))
    assert rc == 0
    return tiles


def test_few_tiles_of_many_heights_run_together():
    # the second product of 30 pair domains: n x n with a long k, heights of 5 to 8 blocks
    n = [60, 61, 69, 72, 76, 79, 80, 82, 85, 88, 91, 92, 94, 98, 101, 106, 111, 122, 123, 124, 124, 125, 126, 128, 133, 147, 147,
         148, 149, 150]
    t = _run(-1, n + n, n + n, [400 * x for x in n + n])
    assert (t[:ROW_CLASSES] > 0).sum() == 0 and (t[ROW_CLASSES:] > 0).sum() == 1


def test_launches_that_fill_the_chip_stay_apart():
    # twenty thousand columns: hundreds of tiles of either height
    t = _run(-1, [28, 36], [20000, 20000], [500, 500])
    assert t[ROW_CLASSES:].sum() == 0 and (t > 0).sum() == 2


@pytest.mark.gpu
@pytest.mark.parametrize("tA", [0, 1])
@pytest.mark.parametrize("tB", [0, 1])
@pytest.mark.parametrize("pad", [0, 1])
def test_against_numpy(tA, tB, pad, need_gpu):
    rng = np.random.default_rng(4 * tA + 2 * tB + pad)
    # heights of one to eight blocks, one and two tiles high, whole and ragged, up to four column blocks a warp; even, so that
    # pad 0 takes the 16-byte modes
    M = 4 * [2, 8, 10, 16, 24, 30, 32, 38, 40, 46, 48, 54, 56, 62, 64, 66, 80, 94, 110, 126, 128]
    N = 4 * [128, 126, 128, 120, 128, 66, 128, 128, 34, 128, 100, 128, 98, 128, 128, 96, 128, 128, 112, 128, 120]
    K = [400 + 2 * (i % 21) for i in range(len(M))]
    assert _run(-1, M, N, K, tA, tB, pad)[ROW_CLASSES:].sum() > 80  # most of its tiles, of every height
    ea = [((k if tA else m) * ((m if tA else k) + pad) + 1) // 2 * 2 for m, k in zip(M, K)]
    eb = [((n if tB else k) * ((k if tB else n) + pad) + 1) // 2 * 2 for n, k in zip(N, K)]
    ec = [(m * n + 1) // 2 * 2 for m, n in zip(M, N)]
    A, B, C = (rng.uniform(-0.5, 0.5, sum(e)) for e in (ea, eb, ec))
    got = C.copy()
    _run(0, M, N, K, tA, tB, pad, A, B, got)
    oa, ob, oc = (np.concatenate([[0], np.cumsum(e)]) for e in (ea, eb, ec))
    for p, (m, n, k) in enumerate(zip(M, N, K)):
        ra, ca, rb, cb = (k, m, n, k) if tA and tB else (k, m, k, n) if tA else (m, k, n, k) if tB else (m, k, k, n)
        a = A[oa[p]:][: ra * (ca + pad)].reshape(ra, ca + pad)[:, :ca]
        b = B[ob[p]:][: rb * (cb + pad)].reshape(rb, cb + pad)[:, :cb]
        a, b = (a.T if tA else a), (b.T if tB else b)
        c = got[oc[p]:][: m * n].reshape(m, n)
        # K products and sums on either side, of at most |a||b|
        assert (np.abs(c - a @ b) <= 2 * (k + 4) * 2.0 ** -53 * (np.abs(a) @ np.abs(b))).all(), (p, m, n, k)


@pytest.mark.gpu
@pytest.mark.parametrize("tA", [0, 1])
@pytest.mark.parametrize("tB", [0, 1])
@pytest.mark.parametrize("M,N,K", [(35, 35, 35), (53, 57, 130), (64, 128, 200), (33, 129, 500), (128, 40, 67), (40, 24, 1000), (30, 48, 63)])
def test_sums_do_not_depend_on_the_launch(tA, tB, M, N, K, need_gpu):
    """One product alone, on few tiles, and six hundred copies of it, which fill the chip: the same sums bit for bit."""
    rng = np.random.default_rng(M + N)
    one, many = [], 600
    for rows, cols in ((K, M) if tA else (M, K), (N, K) if tB else (K, N)):
        x = np.zeros((rows * cols + 1) // 2 * 2)
        x[: rows * cols] = rng.uniform(-0.5, 0.5, rows * cols)
        one.append(x)
    ec = (M * N + 1) // 2 * 2
    alone, filled = np.zeros(ec), np.zeros(many * ec)
    ta = _run(0, [M], [N], [K], tA, tB, 0, one[0], one[1], alone)
    tm = _run(0, many * [M], many * [N], many * [K], tA, tB, 0, np.tile(one[0], many), np.tile(one[1], many), filled)
    assert (np.flatnonzero(ta)[0] % 16 >= 8) and (np.flatnonzero(tm)[0] % 16 < 8)  # both work splits
    assert (filled.reshape(many, ec) == alone).all()
