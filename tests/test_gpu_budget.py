"""The memory budget of vd_forward.

What a chunk allocates stays inside memory_mb: long reads with Phred 0 and 1 bases beside
ordinary long ones (the single-read kernel then strip-mines beside the long-read kernel,
and both keep strip boundaries), many strip tasks, short reads on a small budget, and the
plain schedule.  A batch over the budget is cut into chunks; two of them are in flight
at a time.  The likelihoods do not depend on any of it.
"""
import numpy as np
import pytest

from vardepth_b200 import native
from vardepth_b200 import synthetic as S

pytestmark = pytest.mark.gpu

MB = 1 << 20


def long_regions(rng, n_regions, n_reads, n_haps, n, hap_len, phred01):
    """Reads of n bases from (or, where it is shorter, around) haplotypes of about hap_len."""
    regions = []
    for _ in range(n_regions):
        hap0 = S._random_hap(rng, hap_len)
        haps = [hap0] + [S._mutate(rng, hap0, 2, 3) for _ in range(n_haps - 1)]
        reads, quals = [], []
        for k in range(n_reads):
            a = int(rng.integers(0, max(1, hap_len - n)))
            r = np.concatenate([hap0[a:a + n], S._random_hap(rng, max(0, n - hap_len))])[:n]
            q = S._q_standard(rng)(n)
            if phred01 and k % 2:
                q[7::50] = 0
            reads.append(r)
            quals.append(q)
        regions.append((haps, reads, quals))
    return regions


def run(regions, memory_mb, schedule=native.VD_SCHEDULE_BATCHED):
    w = S._assemble("budget", regions, S.GAP_Q45, S.EXT_Q10, {})
    pk = native.Packed(w.read_bases, w.read_quals, w.read_off, w.hap_bases, w.hap_off,
                       region_read_off=w.region_read_off, region_hap_off=w.region_hap_off)
    params, _ = native.make_params(S.GAP_Q45, S.EXT_Q10, False, native.VD_PRECISION_MIXED, schedule=schedule)
    eng = native.Engine(0, memory_mb)
    got, st = eng.forward(pk, params)
    eng.close()
    return got, st


def test_two_kernels_with_strips():
    regions = long_regions(np.random.default_rng(1), 3, 4, 4, 700, 1500, True)
    wide, st = run(regions, 4096)
    assert st.batches == 1
    # room for the larger of the two kernels' boundaries, not for both
    room = -(-max(1501 * 2960, 2 * (1540 + 2 * 52) * 1776) * 16 // MB) + 2
    tight, st = run(regions, room)
    assert st.live_bytes <= min(st.batches, 2) * room * MB
    np.testing.assert_array_equal(tight, wide)


@pytest.mark.parametrize("schedule", [native.VD_SCHEDULE_BATCHED, native.VD_SCHEDULE_PLAIN])
def test_many_strip_tasks(schedule):
    regions = long_regions(np.random.default_rng(2), 24, 60, 30, 1100, 120, False)
    wide, _ = run(regions, 4096, schedule)
    tight, st = run(regions, 9, schedule)
    assert st.batches > 1 and st.live_bytes <= 2 * 9 * MB
    np.testing.assert_array_equal(tight, wide)


def test_short_reads_on_a_small_budget():
    rng = np.random.default_rng(3)
    regions = []
    for _ in range(12):
        hap0 = S._random_hap(rng, 900)
        haps = [hap0] + [S._mutate(rng, hap0, 2, 3) for _ in range(3)]
        reads, quals = S._sim_reads(rng, haps, 30, rng.integers(80, 250, 30), 0.01, 0.001, S._q_standard(rng))
        regions.append((haps, reads, quals))
    wide, _ = run(regions, 4096)
    tight, st = run(regions, 8)
    assert st.live_bytes <= min(st.batches, 2) * 8 * MB
    np.testing.assert_array_equal(tight, wide)
