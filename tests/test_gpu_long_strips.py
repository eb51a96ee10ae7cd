"""The long-read kernel's strips at the edges of its layout.

Reads just below, at and above a change of rows per lane or of the strip count
(32 R rows per strip, R = 5..8), haplotypes shorter than a window of 32 columns
and around its multiples, halves of very unequal length, one haplotype alone in
its pair, and gap parameters that change how fast a path falls off a row.  The
bound is the one the mixed mode keeps everywhere (1e-4 log10 of the FP64
oracle); the plain schedule runs the same strips and must agree bit for bit.
"""
import numpy as np
import pytest

from conftest import LN10
from oracle import oracle as O
from vardepth_b200 import native
from vardepth_b200 import synthetic as S

pytestmark = pytest.mark.gpu

MIXED_ATOL_LOG10 = 1e-4


def _region(rng, n, hap_lengths, err, quals):
    """One region: two reads of n bases drawn (with errors) from a sequence the haplotypes are
    cut from, so short haplotypes hold a part of the read only."""
    base = S._random_hap(rng, max(max(hap_lengths), n) + 40)
    haps = [base[:m].copy() for m in hap_lengths]
    reads, qs = [], []
    for k in range(2):
        a = int(rng.integers(0, len(base) - n + 1))
        r = base[a:a + n].copy()
        sub = rng.random(n) < err
        r[sub] = rng.choice(S.ALPHABET, int(sub.sum()))
        reads.append(r)
        qs.append(rng.choice(quals, n).astype(np.uint8))
    return haps, reads, qs


@pytest.mark.parametrize("gap,ext", [(10 ** -4.5, 0.1), (0.02, 0.6), (1e-4, 0.02), (1e-4, 0.005), (0.001, 0.0)])
@pytest.mark.parametrize("n", [257, 288, 320, 321, 384, 385, 512, 513, 577, 768, 769, 1025])
def test_strip_and_window_edges(n, gap, ext):
    rng = np.random.default_rng([n, int(gap * 1e6), int(ext * 1000)])
    levels = np.array([10, 20, 30, 40], np.uint8)
    low = np.array([2, 3, 8, 60], np.uint8)
    regions = [_region(rng, n, [n + 100, n + 131], 0.02, levels),
               _region(rng, n, [n + 33, 1, n + 64], 0.08, levels),
               _region(rng, n, [31, 32, 33, 64, 65, 2, n, n - 1, n + 1], 0.05, low),
               _region(rng, n, [n + 7], 0.01, low)]
    w = S._assemble("strips", regions, gap, ext, {})
    pk = native.Packed(w.read_bases, w.read_quals, w.read_off, w.hap_bases, w.hap_off,
                       region_read_off=w.region_read_off, region_hap_off=w.region_hap_off)
    eng = native.Engine(0, 4096)
    batched, _ = native.make_params(gap, ext, False, native.VD_PRECISION_MIXED)
    plain, _ = native.make_params(gap, ext, False, native.VD_PRECISION_MIXED, schedule=native.VD_SCHEDULE_PLAIN)
    got, st = eng.forward(pk, batched)
    want = []
    for g, (haps, reads, qs) in enumerate(regions):
        want += [O.forward(bytes(r).decode(), q, bytes(h).decode(), gap, ext, False) for r, q in zip(reads, qs)
                 for h in haps]
    want = np.array(want)
    finite = np.isfinite(want)  # ext 0: a read longer than its haplotype by two bases or more has no path
    assert np.array_equal(np.isneginf(got), np.isneginf(want))
    assert np.max(np.abs(got[finite] - want[finite])) / LN10 <= MIXED_ATOL_LOG10
    pairs_of = lambda h: -(-min(h, 8) // 2) + (-(-(h - 8) // 2) if h > 8 else 0)
    assert st.long_strips == sum(2 * pairs_of(len(h)) * -(-n // 256) for h, _, _ in regions)
    np.testing.assert_array_equal(eng.forward(pk, plain)[0], got)
    eng.close()
