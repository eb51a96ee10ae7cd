"""FP64 mode on long reads that hang off their haplotype by a quarter of their length or more.

Every placement of the inserted run along the alignment carries as much of the final sum,
and the cells of one row that belong to them lie hundreds of binary orders apart, more the
smaller the gap continuation.  A strip's boundary has to keep them as far down as rows
divided by their maximum do (the FP64 oracle).  The values come from the long double oracle;
pairs on which the FP64 oracle itself departs from it are left out.  FP64 rounding over
1,100 rows leaves less than 1e-11 of the likelihood and 1e-11 of a logarithm of 7,000;
the bound is 1e-9.
"""
import numpy as np
import pytest

from conftest import LN10
from oracle import oracle as O
from test_gpu_long_strips import _region
from vardepth_b200 import native
from vardepth_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def hanging_regions(rng):
    low, levels = np.array([2, 3, 8, 60], np.uint8), np.array([10, 20, 30, 40], np.uint8)
    out = []
    for n in (257, 300, 385, 513, 769, 1025):
        out += [_region(rng, n, [n // 4, n // 3, n // 2, 2 * n // 3, n - 50, n // 2 + 5], 0.02, low),
                _region(rng, n, [n // 4, n // 3, n // 2, 2 * n // 3, n - 50], 0.2, np.array([5, 30], np.uint8)),
                _region(rng, n, [n - 20, n - 60, n - 120, n // 2, n + 300], 0.03, levels),
                _region(rng, n, [n - 30, n + 5], 0.01, np.array([30], np.uint8))]
    return out


def oracle_values(regions, gap, ext):
    """(long double values, pairs on which the FP64 oracle agrees with them)"""
    f = lambda fn: np.array([fn(bytes(r).decode(), q, bytes(h).decode(), gap, ext, False)
                             for haps, reads, quals in regions for r, q in zip(reads, quals) for h in haps])
    exact, f64 = f(O.forward_ld), f(O.forward)
    with np.errstate(invalid="ignore"):
        holds = (exact == f64) | (np.abs(exact - f64) <= 1e-9)
    return exact, holds


def packed(regions, gap, ext):
    w = S._assemble("regions", regions, gap, ext, {})
    return native.Packed(w.read_bases, w.read_quals, w.read_off, w.hap_bases, w.hap_off,
                         region_read_off=w.region_read_off, region_hap_off=w.region_hap_off)


def worst_log10(got, exact, holds):
    finite = holds & np.isfinite(exact)
    assert np.array_equal(np.isneginf(got[holds]), np.isneginf(exact[holds]))
    assert finite.sum() > 0.8 * len(exact)
    return np.max(np.abs(got[finite] - exact[finite])) / LN10


@pytest.mark.parametrize("gap,ext", [(1e-4, 0.075), (1e-4, 0.04), (1e-4, 0.02), (1e-4, 0.01)])
@pytest.mark.parametrize("rows", [256, 128])
def test_hanging_long_reads(rows, gap, ext):
    eng = native.Engine(0, 4096)
    eng.set_tuning(long_read_rows=rows)
    params, _ = native.make_params(gap, ext, False, native.VD_PRECISION_FLOAT64)
    for seed in (1, 2):
        regions = hanging_regions(np.random.default_rng([seed, 99]))
        got, _ = eng.forward(packed(regions, gap, ext), params)
        assert worst_log10(got, *oracle_values(regions, gap, ext)) <= 1e-9
    eng.close()
