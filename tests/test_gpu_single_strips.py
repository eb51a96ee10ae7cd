"""Long reads in the single-read kernel's FP32 strips: pairs in list form, VD_LONG_SINGLE and
reads with Phred 0 and 1 bases.

The joined reads of test_gpu_long_modes: at a strip's boundary the path that wins lies
hundreds of binary orders below the best one, while no strip loses enough to leave the
range by itself.  Anchored mode goes through the same strips.  The bound is the one the
mixed mode keeps everywhere (1e-4 log10 of the FP64 oracle).
"""
import numpy as np
import pytest

from conftest import LN10
from test_gpu_float64_strips import hanging_regions, oracle_values, worst_log10
from test_gpu_long_modes import joined_reads, oracle_of, packed
from vardepth_b200 import native
from vardepth_b200 import synthetic as S

pytestmark = pytest.mark.gpu

MIXED_ATOL_LOG10 = 1e-4


def pair_form(w):
    pr, ph = w.explicit_pairs()
    return native.Packed(w.read_bases, w.read_quals, w.read_off, w.hap_bases, w.hap_off, pair_read=pr, pair_hap=ph)


@pytest.mark.parametrize("levels", [[30], [20, 30, 40], [0] + [30] * 11, [1] + [40] * 40])
@pytest.mark.parametrize("form,rows", [("region", 256), ("region", 128), ("region", 64), ("pairs", 256)])
def test_joined_reads(form, rows, levels):
    regions = joined_reads(5, levels)
    w = S._assemble("joined", regions, S.GAP_Q45, S.EXT_Q10, {})
    pk = packed(w) if form == "region" else pair_form(w)
    eng = native.Engine(0, 2048)
    eng.set_tuning(long_read_rows=rows, long_mode=native.VD_LONG_SINGLE)
    for anchored in (False, True):
        want = oracle_of(regions, S.GAP_Q45, S.EXT_Q10, anchored)
        batched, _ = native.make_params(S.GAP_Q45, S.EXT_Q10, anchored, native.VD_PRECISION_MIXED)
        plain, _ = native.make_params(S.GAP_Q45, S.EXT_Q10, anchored, native.VD_PRECISION_MIXED,
                                      schedule=native.VD_SCHEDULE_PLAIN)
        got, _ = eng.forward(pk, batched)
        assert np.max(np.abs(got - want)) / LN10 <= MIXED_ATOL_LOG10
        np.testing.assert_array_equal(eng.forward(pk, plain)[0], got)
    eng.close()


def test_reads_without_errors_stay_in_the_primary_tier():
    """200 bits hold a read of several strips with a dozen Phred-30 errors."""
    rng = np.random.default_rng(3)
    hap = S._random_hap(rng, 1500)
    reads = []
    for n, errors in ((300, 3), (700, 8), (1200, 12)):
        r = hap[100:100 + n].copy()
        for p in rng.choice(n, errors, replace=False):
            r[p] = S.ALPHABET[S.ALPHABET != r[p]][rng.integers(0, 3)]
        reads.append(r)
    regions = [([hap], reads, [np.full(len(r), 30, np.uint8) for r in reads])]
    w = S._assemble("clean", regions, S.GAP_Q45, S.EXT_Q10, {})
    eng = native.Engine(0, 1024)
    params, _ = native.make_params(S.GAP_Q45, S.EXT_Q10, False, native.VD_PRECISION_MIXED)
    got, st = eng.forward(pair_form(w), params)
    assert st.rescued_fp32 + st.rescued_fp64 == 0
    assert np.max(np.abs(got - oracle_of(regions, S.GAP_Q45, S.EXT_Q10))) / LN10 <= MIXED_ATOL_LOG10
    eng.close()


@pytest.mark.parametrize("gap,ext", [(0.02, 0.6), (10 ** -4.5, 0.1), (1e-4, 0.02)])
@pytest.mark.parametrize("rows", [256, 64])
def test_hanging_reads(rows, gap, ext):
    eng = native.Engine(0, 4096)
    eng.set_tuning(long_read_rows=rows, long_mode=native.VD_LONG_SINGLE)
    params, _ = native.make_params(gap, ext, False, native.VD_PRECISION_MIXED)
    for seed in (1, 2, 3):
        regions = hanging_regions(np.random.default_rng([seed, 99]))
        exact, holds = oracle_values(regions, gap, ext)
        got, _ = eng.forward(packed(S._assemble("hanging", regions, gap, ext, {})), params)
        assert worst_log10(got, exact, holds) <= MIXED_ATOL_LOG10
    eng.close()
