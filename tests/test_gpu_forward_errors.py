"""An engine after a call that ended with an error between two chunks.

The call's first chunk is in flight when the second one is found to exceed the memory
budget.  What the engine scores next -- in either form, with fewer outputs, or region
genotypes -- must be its own: nothing of the abandoned chunk may reach a later call's
output, the memory behind it or its counters.
"""
import ctypes

import numpy as np
import pytest

from vardepth_b200 import native
from vardepth_b200 import synthetic as S

pytestmark = pytest.mark.gpu

GUARD = -12345.0


def _forward(eng, packed, params, room):
    """(return code, outputs, memory behind them, counters)"""
    n = packed.n_outputs()
    buf = np.full(max(n, room), GUARD)
    st = native.VdStats()
    rc = native.library().vd_forward(eng.handle, ctypes.byref(packed.batch), ctypes.byref(params),
                                     buf.ctypes.data_as(native.c_dp), ctypes.byref(st))
    return rc, buf[:n].copy(), buf[n:], st


def _pairs(rng, reads, haps, pr, ph):
    off = lambda x: np.concatenate([[0], np.cumsum([len(v) for v in x])])
    return native.Packed(np.concatenate(reads), np.concatenate([np.full(len(r), 30, np.uint8) for r in reads]), off(reads),
                         np.concatenate(haps), off(haps), pair_read=pr, pair_hap=ph)


def test_calls_after_a_chunk_over_the_budget():
    rng = np.random.default_rng(11)
    haps = [S._random_hap(rng, 120) for _ in range(40)]
    reads = [haps[0][10:90].copy(), haps[1][5:100].copy()]
    # read 0: 400 pairs, the first chunk; read 1: more pairs than 16 MiB hold
    big = 500_000
    over = _pairs(rng, reads, haps, np.concatenate([np.zeros(400, np.int32), np.ones(big, np.int32)]),
                  np.concatenate([np.arange(400) % 40, np.zeros(big, np.int64)]))
    small = _pairs(rng, reads, haps, [0, 1, 1], [0, 1, 2])
    wl = S._assemble("one", [(haps[:3], reads, [np.full(len(r), 30, np.uint8) for r in reads])], S.GAP_Q45, S.EXT_Q10, {})
    region = native.Packed(wl.read_bases, wl.read_quals, wl.read_off, wl.hap_bases, wl.hap_off,
                           region_read_off=wl.region_read_off, region_hap_off=wl.region_hap_off)
    params, _ = native.make_params(S.GAP_Q45, S.EXT_Q10, False, native.VD_PRECISION_MIXED)

    clean = native.Engine(0, 16)
    want_pairs, st_pairs = clean.forward(small, params)
    want_region, st_region = clean.forward(region, params)
    want_geno = clean.region_genotypes(region, params)
    clean.close()

    eng = native.Engine(0, 16)
    for nxt in ("pairs", "region", "genotypes"):
        rc, *_ = _forward(eng, over, params, 0)
        assert rc == native.VD_ENOMEM
        if nxt == "genotypes":
            got = eng.region_genotypes(region, params)
            np.testing.assert_array_equal(got["ln"], want_geno["ln"])
            for a, b in zip(got["gl"], want_geno["gl"]):
                np.testing.assert_array_equal(a, b)
        if nxt in ("pairs", "genotypes"):
            rc, got, behind, st = _forward(eng, small, params, 2000)
            assert rc == native.VD_OK
            np.testing.assert_array_equal(got, want_pairs)
            assert np.all(behind == GUARD)
            assert st.d2h_bytes == st_pairs.d2h_bytes
        if nxt == "region":
            rc, got, behind, st = _forward(eng, region, params, 2000)
            assert rc == native.VD_OK
            np.testing.assert_array_equal(got, want_region)
            assert np.all(behind == GUARD)
            assert st.d2h_bytes == st_region.d2h_bytes
    eng.close()
