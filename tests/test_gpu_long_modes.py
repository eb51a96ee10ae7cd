"""Reads whose best alignment is far from the best one of their first rows.

A read joined from two copies of a sequence that lie next to each other in the haplotype:
its first rows match one copy, the others the second.  The path that wins crosses the
copies' differences in the first rows and is by then hundreds of binary orders below the
one along the first copy, which loses as much later.  A tier that scales a whole row of
the matrix by one power of two drops it there; the likelihood is then wrong by tens of
orders of magnitude.  The bound is the one the mixed mode keeps everywhere (1e-4 log10 of
the FP64 oracle).
"""
import numpy as np
import pytest

from conftest import LN10
from oracle import oracle as O
from vardepth_b200 import native
from vardepth_b200 import synthetic as S

pytestmark = pytest.mark.gpu

MIXED_ATOL_LOG10 = 1e-4


def _copies(rng, n, split, first, per_256):
    """(haplotype, read) of n-base copies that differ at `first` bases before `split` and at
    `per_256` in every 256 after it; the read follows the first copy, then the second."""
    x = S._random_hap(rng, n)
    y = x.copy()
    pos = list(rng.choice(np.arange(5, split - 5), first, replace=False))
    for a in range(split, n, 256):
        pos += list(rng.choice(np.arange(a, min(n, a + 256)), min(per_256, min(n, a + 256) - a), replace=False))
    for p in pos:
        y[p] = S.ALPHABET[S.ALPHABET != y[p]][rng.integers(0, 3)]
    return np.concatenate([x, y]), np.concatenate([x[:split], y[split:]])


def joined_reads(seed, levels):
    rng = np.random.default_rng(seed)
    regions = []
    for n, split, first, per_256 in ((1200, 250, 30, 12), (1200, 250, 27, 6), (1200, 256, 25, 10),
                                     (1200, 500, 30, 3), (700, 120, 24, 8)):
        hap, read = _copies(rng, n, split, first, per_256)
        reads = [read, read[:-40]]
        regions.append(([hap, hap[:-7]], reads, [np.resize(np.array(levels, np.uint8), len(r)) for r in reads]))
    return regions


def oracle_of(regions, gap, ext, anchored=False):
    return np.array([O.forward(bytes(r).decode(), q, bytes(h).decode(), gap, ext, anchored)
                     for haps, reads, quals in regions for r, q in zip(reads, quals) for h in haps])


def packed(w):
    return native.Packed(w.read_bases, w.read_quals, w.read_off, w.hap_bases, w.hap_off,
                         region_read_off=w.region_read_off, region_hap_off=w.region_hap_off)


@pytest.mark.parametrize("levels", [[30], [20, 30, 40]])
@pytest.mark.parametrize("mode,rows", [("warp", 256), ("warp", 128), ("block", 256), ("block", 128)])
def test_joined_long_reads(mode, rows, levels):
    regions = joined_reads(5, levels)
    want = oracle_of(regions, S.GAP_Q45, S.EXT_Q10)
    w = S._assemble("joined", regions, S.GAP_Q45, S.EXT_Q10, {})
    eng = native.Engine(0, 2048)
    eng.set_tuning(long_read_rows=rows, long_mode={"warp": native.VD_LONG_WARP, "block": native.VD_LONG_BLOCK}[mode])
    params, _ = native.make_params(S.GAP_Q45, S.EXT_Q10, False, native.VD_PRECISION_MIXED)
    got, st = eng.forward(packed(w), params)
    assert st.long_strips > 0
    assert np.max(np.abs(got - want)) / LN10 <= MIXED_ATOL_LOG10
    eng.close()
