"""Region genotype sums at the edges of the runs a region's rows are cut into.

Few haplotypes and many reads (many runs), one read, numbers of reads around the
8-row minimum of a run, and enough haplotypes that a region has one run only.  The
sums are recomputed in numpy from the likelihoods the same call returns: FP64
sums of at most 500 logarithms in another order, |terms| below 700, so 1e-10 leaves
two orders of magnitude over 500 * 700 * 2^-53 per rounding.
"""
import numpy as np
import pytest

from vardepth_b200 import native
from vardepth_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prior", [None, 0.0, 0.01])
def test_rows_in_runs(prior):
    rng = np.random.default_rng(88)
    qf = S._q_standard(rng)
    regions = []
    for H, nr in ((1, 1), (1, 500), (2, 7), (2, 8), (2, 9), (3, 300), (5, 64), (16, 17), (24, 40)):
        hap0 = S._random_hap(rng, 90)
        haps = [hap0] + [S._mutate(rng, hap0, 2, 3) for _ in range(H - 1)]
        reads, quals = S._sim_reads(rng, haps, nr, rng.integers(30, 80, nr), 0.01, 0.001, qf)
        regions.append((haps, reads, quals))
    w = S._assemble("runs", regions, S.GAP_Q45, S.EXT_Q10, {})
    pk = native.Packed(w.read_bases, w.read_quals, w.read_off, w.hap_bases, w.hap_off,
                       region_read_off=w.region_read_off, region_hap_off=w.region_hap_off)
    eng = native.Engine(0, 4096)
    params, _ = native.make_params(w.gap, w.ext, False, native.VD_PRECISION_MIXED)
    got = eng.region_genotypes(pk, params, artifact_prior=prior)
    again = eng.region_genotypes(pk, params, artifact_prior=prior)
    weights = np.array([.025, .1, .225, .3, .225, .1, .025])
    balance = np.array([.2, .3, .4, .5, .6, .7, .8])
    theta, theta_w = np.array([.02, .1, .2, .3]), np.array([.4, .35, .2, .05])
    o = 0
    for g, (haps, reads, _) in enumerate(regions):
        H, nr = len(haps), len(reads)
        v = got["values"][o:o + nr * H].reshape(nr, H)
        o += nr * H
        ln = lambda x: np.log(np.maximum(1e-300, x)).sum(0)
        want = []
        for b in range(H):
            for a in range(b + 1):
                if prior is None:
                    want.append(ln((v[:, a] + v[:, b]) / 2))
                    continue
                clean = np.logaddexp.reduce([ln(x * v[:, a] + (1 - x) * v[:, b]) + np.log(y)
                                             for x, y in zip(balance, weights)])
                if prior > 0:
                    art = np.logaddexp.reduce([ln((1 - x) * (v[:, a] + v[:, b]) / 2 + x * v[:, c]) + np.log(y / H)
                                               for x, y in zip(theta, theta_w) for c in range(H)])
                    clean = np.logaddexp(np.log1p(-prior) + clean, np.log(prior) + art)
                want.append(clean)
        np.testing.assert_allclose(got["gl"][g], want, rtol=0, atol=1e-10 * max(1.0, np.abs(want).max()))
        np.testing.assert_array_equal(got["gl"][g], again["gl"][g])
    eng.close()
