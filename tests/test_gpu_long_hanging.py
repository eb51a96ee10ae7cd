"""The long-read kernel and the drift tier on reads that hang off their haplotype by 20 bases to three quarters
of their length.

Every placement of the inserted run along the alignment carries as much of the final sum,
so the lanes' exponents have to keep cells of one lane that lie (steps + 2 rows) insertions
apart.  Values from the long double oracle, pairs on which the FP64 oracle departs from it
left out; the bound is the one the mixed mode keeps everywhere (1e-4 log10).
"""
import numpy as np
import pytest

from test_gpu_drift_paths import regions_of
from test_gpu_float64_strips import hanging_regions, oracle_values, packed, worst_log10
from vardepth_b200 import native

pytestmark = pytest.mark.gpu

MIXED_ATOL_LOG10 = 1e-4


@pytest.mark.parametrize("gap,ext", [(0.02, 0.6), (10 ** -4.5, 0.2), (10 ** -4.5, 0.1), (1e-6, 0.1), (10 ** -4.5, 0.08),
                                     (1e-4, 0.04), (1e-4, 0.02), (1e-4, 0.01)])
def test_hanging_long_reads(gap, ext):
    eng = native.Engine(0, 4096)
    mixed, _ = native.make_params(gap, ext, False, native.VD_PRECISION_MIXED)
    plain, _ = native.make_params(gap, ext, False, native.VD_PRECISION_MIXED, schedule=native.VD_SCHEDULE_PLAIN)
    for seed in (1, 2, 3):
        regions = hanging_regions(np.random.default_rng([seed, 99]))
        exact, holds = oracle_values(regions, gap, ext)
        pk = packed(regions, gap, ext)
        for rows in (256, 128):
            eng.set_tuning(long_read_rows=rows)
            got, st = eng.forward(pk, mixed)
            assert st.long_strips > 0
            assert worst_log10(got, exact, holds) <= MIXED_ATOL_LOG10
            np.testing.assert_array_equal(eng.forward(pk, plain)[0], got)
    eng.close()


@pytest.mark.parametrize("gap,ext", [(1e-4, 0.04), (1e-4, 0.02), (1e-4, 0.01), (1e-4, 0.005)])
@pytest.mark.parametrize("kind", ["hanging", "unrelated", "phred01"])
def test_reads_of_one_strip_at_small_gap_continuations(kind, gap, ext):
    eng = native.Engine(0, 1024)
    params, _ = native.make_params(gap, ext, False, native.VD_PRECISION_MIXED)
    regions = regions_of(kind, np.random.default_rng(9))
    exact, holds = oracle_values(regions, gap, ext)
    got, st = eng.forward(packed(regions, gap, ext), params)
    assert st.rescued_fp32 + st.rescued_fp64 > 0
    assert worst_log10(got, exact, holds) <= MIXED_ATOL_LOG10
    eng.close()
