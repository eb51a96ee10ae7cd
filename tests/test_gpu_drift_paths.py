"""The drift tier on pairs whose winning path is not the best one of the first rows.

Reads of one strip joined from two copies of a sequence (each path crosses 15-40 Phred-40
differences, so the pair leaves the primary tier's range), reads that hang off their
haplotype, unrelated reads, and reads of several strips that reach the tier through the
single-read path at every strip height.  The bound is the one the mixed mode keeps
everywhere (1e-4 log10 of the FP64 oracle); the plain schedule must agree bit for bit.
"""
import numpy as np
import pytest

from conftest import LN10
from oracle import oracle as O
from test_gpu_long_strips import _region
from vardepth_b200 import native
from vardepth_b200 import synthetic as S

pytestmark = pytest.mark.gpu

MIXED_ATOL_LOG10 = 1e-4
PARAMETERS = [(10 ** -4.5, 0.1), (0.02, 0.6)]


def joined(rng, n, first, second, apart):
    """A haplotype with two copies of an n-base sequence, `apart` bases between them, that
    differ at `first` bases of the first half and `second` of the other; a read of the
    first copy's first half and the second copy's other half."""
    x = S._random_hap(rng, n + 60)
    y, h = x.copy(), n // 2
    for p in list(rng.choice(np.arange(2, h - 2), first, replace=False)) + \
            list(rng.choice(np.arange(h + 2, n - 2), second, replace=False)):
        y[p] = S.ALPHABET[S.ALPHABET != y[p]][rng.integers(0, 3)]
    hap = np.concatenate([x, S._random_hap(rng, apart), y])
    return [hap], [np.concatenate([x[:h], y[h:n]])], [np.full(n, 40, np.uint8)]


def regions_of(kind, rng):
    low, high = np.array([2, 3, 8, 60], np.uint8), np.array([20, 30, 40], np.uint8)
    if kind == "joined":
        return [joined(rng, n, f, s, a) for n in (100, 200, 250) for f, s in ((15, 18), (20, 22), (25, 30), (18, 40))
                for a in (0, 40, 200)]
    if kind == "hanging":
        return [_region(rng, n, [31, 32, 33, 64, 65, n, n - 1, n + 1, n // 2, n // 3], 0.05, low if k % 2 else high)
                for n in (33, 64, 97, 128, 150, 200, 256) for k in range(4)]
    if kind == "unrelated":
        return [([S._random_hap(rng, int(m)) for m in rng.integers(30, 600, 6)], [S._random_hap(rng, n) for _ in range(4)],
                 [rng.choice(high, n).astype(np.uint8) for _ in range(4)]) for n in (40, 100, 150, 200, 256)]
    if kind == "phred01":  # two-sided emission
        out = regions_of("hanging", rng)[::3] + regions_of("joined", rng)[::3]
        for _, _, quals in out:
            for q in quals:
                q[::17] = 0
                q[5::31] = 1
        return out
    return [r for n in (257, 320, 513, 769, 1025)  # several strips
            for r in (_region(rng, n, [n + 33, 1, n + 64], 0.08, np.array([10, 20, 30, 40], np.uint8)),
                      _region(rng, n, [31, 64, 65, 2, n, n - 1, n // 2], 0.05, low))]


def check(eng, regions, gap, ext):
    want = np.array([O.forward(bytes(r).decode(), q, bytes(h).decode(), gap, ext, False)
                     for haps, reads, quals in regions for r, q in zip(reads, quals) for h in haps])
    w = S._assemble("drift", regions, gap, ext, {})
    pk = native.Packed(w.read_bases, w.read_quals, w.read_off, w.hap_bases, w.hap_off,
                       region_read_off=w.region_read_off, region_hap_off=w.region_hap_off)
    batched, _ = native.make_params(gap, ext, False, native.VD_PRECISION_MIXED)
    plain, _ = native.make_params(gap, ext, False, native.VD_PRECISION_MIXED, schedule=native.VD_SCHEDULE_PLAIN)
    got, st = eng.forward(pk, batched)
    assert st.rescued_fp32 + st.rescued_fp64 > 0  # the rescue tiers saw pairs
    finite = np.isfinite(want)
    assert np.array_equal(np.isneginf(got), np.isneginf(want))
    assert np.max(np.abs(got[finite] - want[finite])) / LN10 <= MIXED_ATOL_LOG10
    np.testing.assert_array_equal(eng.forward(pk, plain)[0], got)
    return st


@pytest.mark.parametrize("kind,gap,ext", [(k, *p) for k in ("joined", "hanging", "unrelated", "phred01") for p in PARAMETERS] +
                         [("joined", 1e-4, 0.02), ("joined", 1e-4, 0.005), ("joined", 0.001, 0.0)])
def test_reads_of_one_strip(kind, gap, ext):
    eng = native.Engine(0, 1024)
    check(eng, regions_of(kind, np.random.default_rng(9)), gap, ext)
    eng.close()


@pytest.mark.parametrize("gap,ext", PARAMETERS)
@pytest.mark.parametrize("rows", [256, 128, 64])
def test_reads_of_several_strips(rows, gap, ext):
    eng = native.Engine(0, 1024)
    eng.set_tuning(long_mode=native.VD_LONG_SINGLE, long_read_rows=rows)
    check(eng, regions_of("long", np.random.default_rng(10)), gap, ext)
    eng.close()
