"""The asynchronous copies of the FP64 matrix-instruction GEMM, address by address on the host
(tci_selftest_gemm_f64_copies): each is aligned to its instruction's size, those of no bytes too, and stays inside the
operand's allocation and the shared-memory slice, in every tile class, for ragged tiles and k, odd and even starts
and leading dimensions."""
import numpy as np
import pytest

from tigerci_b200._lib import lib, ptr

# operand modes of a class (row operand, column operand): K16 / K8 rows of contiguous k in 16 / 8-byte copies, RT8 / R16
# rows of k with contiguous tile rows in 8 / 16-byte copies
PAIRS = [("K16", "K16"), ("K16", "R16"), ("K8", "K8"), ("K8", "R16"), ("RT8", "K8"), ("RT8", "R16")]


def _copies(cls, which, nr, K, ld, off, length):
    out = np.zeros(3, dtype=np.int64)
    assert lib().tci_selftest_gemm_f64_copies(cls, which, nr, K, ld, off, length, ptr(out)) == 0
    return out.tolist()


@pytest.mark.parametrize("pair", range(6))
@pytest.mark.parametrize("shared_k", [0, 1])
@pytest.mark.parametrize("which", [0, 1])
def test_every_copy_aligned_and_inside(pair, shared_k, which):
    mode = PAIRS[pair][which]
    for mb in range(1, 9):
        cls = 16 * pair + 8 * shared_k + mb - 1
        widest = 8 * mb if which == 0 else (32 if shared_k else 128)
        for K in (1, 2, 7, 15, 16, 17, 31, 33, 63, 64, 65, 129):
            for pad in (0, 1, 2, 3):
                for off in (0, 1, 2, 5):
                    for nr in sorted({1, 2, 7, widest - 1, widest}):
                        rows, cols = (nr, K) if mode[0] == "K" else (K, nr)  # as stored
                        ld = cols + pad
                        if mode == "K16" and (ld % 2 or off % 2):
                            continue  # such an operand takes K8
                        if mode == "R16" and (ld % 2 or off % 2) and nr > 120 and not shared_k:
                            continue  # at most 15 column blocks: a row may start one place in
                        n, bad, out = _copies(cls, which, nr, K, ld, off, off + (rows - 1) * ld + cols)
                        assert n > 0 and bad == 0 and out == 0, (mode, mb, nr, K, ld, off, bad, out)
