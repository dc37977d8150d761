"""The FP64 matrix-instruction GEMM (tci_selftest_gemm_f64) against numpy at the edges of its tiles: every operand
orientation, odd and even leading dimensions and starts, several segments, remainders in M, N and K, the shapes that
take the k-sharing, the transposed and the several-row-tile forms."""
import numpy as np
import pytest

from tigerci_b200._lib import lib, ptr

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (5, 3, 2), (8, 8, 8), (9, 17, 5), (36, 300, 40), (63, 65, 16), (64, 128, 33), (65, 129, 47),
          (173, 101, 31), (30, 1000, 9), (1000, 3, 20), (128, 120, 15), (20, 20000, 21), (40, 20011, 17),
          (260, 2200, 18), (700, 1990, 35), (33, 16, 3000)]


@pytest.mark.parametrize("tA", [0, 1])
@pytest.mark.parametrize("tB", [0, 1])
@pytest.mark.parametrize("pad,off", [(0, 0), (1, 0), (2, 1), (3, 3)])
def test_gemm_against_numpy(tA, tB, pad, off, need_gpu):
    rng = np.random.default_rng(100 * pad + 10 * off + 2 * tA + tB)
    for i, (M, N, K) in enumerate(SHAPES):
        for nseg, alpha, beta in ((1, 1.0, 0.0), (3, -0.7, 1.0), (0, 1.0, -0.5))[: 3 if i < 8 else 2]:
            lda, ldb, ldc = (M if tA else K) + pad, (K if tB else N) + pad, N + (i & 1)
            ra, rb = (K if tA else M), (N if tB else K)
            A = rng.uniform(-0.5, 0.5, off + max(nseg, 1) * ra * lda)
            B = rng.uniform(-0.5, 0.5, off + max(nseg, 1) * rb * ldb)
            C = rng.uniform(-0.5, 0.5, M * ldc)
            got = C.copy()
            rc = lib().tci_selftest_gemm_f64(0, M, N, K, nseg, tA, tB, lda, ldb, ldc, off, off, ra * lda, rb * ldb, alpha,
                                             beta, ptr(A), A.size, ptr(B), B.size, ptr(got))
            assert rc == 0
            C2, got = C.reshape(M, ldc), got.reshape(M, ldc)
            ref = beta * C2[:, :N]
            mag = np.abs(ref)
            for s in range(nseg):
                a = A[off + s * ra * lda:][: ra * lda].reshape(ra, lda)[:, : (M if tA else K)]
                b = B[off + s * rb * ldb:][: rb * ldb].reshape(rb, ldb)[:, : (K if tB else N)]
                a, b = (a.T if tA else a), (b.T if tB else b)
                ref = ref + alpha * (a @ b)
                mag = mag + abs(alpha) * (np.abs(a) @ np.abs(b))
            # nseg K products, alpha on one factor, the sums and beta: nseg K + 4 roundings of at most mag on
            # either side
            assert (np.abs(got[:, :N] - ref) <= 2 * (nseg * K + 4) * 2.0 ** -53 * mag).all(), (M, N, K, nseg)
            assert (got[:, N:] == C2[:, N:]).all()


@pytest.mark.parametrize("K", [3, 16, 70])
def test_many_segments(K, need_gpu):
    """Segment counts around the 16 records a block holds at a time and around twice that, tiles of 2 x 2 to 8 x 16
    blocks."""
    rng = np.random.default_rng(K)
    for M, N in ((16, 16), (35, 33), (53, 57), (64, 128), (200, 300)):
        for nseg in (2, 15, 16, 17, 31, 32, 33, 50):
            A, B, C = (rng.uniform(-0.5, 0.5, s) for s in (nseg * M * K, nseg * K * N, M * N))
            got = C.copy()
            rc = lib().tci_selftest_gemm_f64(0, M, N, K, nseg, 0, 0, K, N, N, 0, 0, M * K, K * N, 0.5, 1.0, ptr(A), A.size,
                                             ptr(B), B.size, ptr(got))
            assert rc == 0
            A3, B3 = A.reshape(nseg, M, K), B.reshape(nseg, K, N)
            ref = C.reshape(M, N) + 0.5 * np.einsum("smk,skn->mn", A3, B3, optimize=True)
            mag = np.abs(C.reshape(M, N)) + 0.5 * np.einsum("smk,skn->mn", np.abs(A3), np.abs(B3), optimize=True)
            assert (np.abs(got.reshape(M, N) - ref) <= 2 * (nseg * K + 4) * 2.0 ** -53 * mag).all(), (M, N, nseg)
