"""vd_region_genotypes counts the kernels it launches: a haplotype without bases adds the fill
of its outputs and nothing else."""
import numpy as np
import pytest

from vardepth_b200 import native
from vardepth_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def test_the_fill_is_counted():
    rng = np.random.default_rng(4)
    hap = S._random_hap(rng, 200)
    haps = [hap, S._mutate(rng, hap, 2, 3)]
    reads, quals = S._sim_reads(rng, haps, 6, np.full(6, 100), 0.01, 0.001, S._q_standard(rng))
    params, _ = native.make_params(S.GAP_Q45, S.EXT_Q10, False, native.VD_PRECISION_MIXED)
    eng = native.Engine(0, 1024)
    launches = []
    for hs in (haps, haps + [hap[:0]]):
        w = S._assemble("launches", [(hs, reads, quals)], S.GAP_Q45, S.EXT_Q10, {})
        pk = native.Packed(w.read_bases, w.read_quals, w.read_off, w.hap_bases, w.hap_off,
                           region_read_off=w.region_read_off, region_hap_off=w.region_hap_off)
        launches.append(eng.region_genotypes(pk, params)["stats"].kernel_launches)
    assert launches[1] == launches[0] + 1
    eng.close()
