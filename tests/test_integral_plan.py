"""The tables of the integral form of the pair-domain all-external term, on the host (tci_selftest_integral_plan): the
lists' lengths, the copies of sigma by the number of row tiles, and block sets whose lists outgrow 32-bit indexes."""
import numpy as np
import pytest

from tigerci_b200._lib import lib, ptr


def _plan(nv, off, length, dom, sms=148):
    out = np.zeros(5, dtype=np.int64)
    off, length, dom = (np.asarray(x, dtype=np.int64) for x in (off, length, dom))
    assert lib().tci_selftest_integral_plan(nv, len(off), ptr(off), ptr(length), ptr(dom), len(dom), sms, ptr(out)) == 0
    return dict(zip(("fits", "parts", "tasks", "jobs", "entries"), out.tolist()))


@pytest.mark.parametrize("nv,nblk,parts", [(20, 7, 8), (131, 11, 8), (300, 12, 2), (310, 12, 1)])
def test_lists_and_copies(nv, nblk, parts):
    rng = np.random.default_rng(nv)
    size = [nv] + rng.integers(1, nv + 1, nblk - 1).tolist()
    doms = [np.sort(rng.choice(nv, size=k, replace=False)) for k in size]
    p = _plan(nv, np.cumsum([0] + size[:-1]), size, np.concatenate(doms))
    assert p["fits"] == 1 and p["entries"] == sum(k * k for k in size)
    # one block on every external: at most 128 columns for each a, a job per (a, c), row tiles of at most 64 rows
    assert p["jobs"] == nv * nv
    # tiles x copies fill six blocks per multiprocessor, or there are eight copies
    tiles = sum((a + 64) // 64 for a in range(nv))
    assert p["parts"] == parts and (parts == 8 or tiles * parts >= 6 * 148)
    assert tiles <= p["tasks"] <= tiles * parts


def test_lists_beyond_32_bits():
    # 9721 blocks of 470 externals: 2,147,368,900 entries; one more: 2^31 + 106,152
    dom = np.arange(470)
    assert 9721 * 470 ** 2 < 2 ** 31 < 9722 * 470 ** 2
    assert _plan(470, np.zeros(9722), np.full(9722, 470), dom) == dict(fits=0, parts=0, tasks=0, jobs=0, entries=0)
