"""The two-pair gradient kernels at the edges of their items.

Odd numbers of pairs per rows-per-lane class (the last one runs beside a copy of
itself), halves of very unequal haplotype length, haplotypes shorter than the
wavefront's ramp and around multiples of the sub-segment, and a half that leaves the
FP32 range beside one that does not.  VD_CHECKPOINT_ALL runs the one-pair kernel with
the same operations in the same order, so the two agree bit for bit; the summed
gradient is held to the oracle as everywhere (1e-6 relative).
"""
import numpy as np
import pytest

from oracle import oracle as O
from vardepth_b200 import native
from vardepth_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 100, 128, 129, 160, 161, 200, 224, 225, 256])
def test_two_pair_items(n):
    rng = np.random.default_rng(n)
    qf = S._q_standard(rng)
    rb, rq, hb, ro, ho, pr, ph = [], [], [], [0], [0], [], []
    for k, m in enumerate((1, 2, 5, 31, 32, 33, 37, 64, 300, n + 9, 7, 301, n + 40)):
        hap = S._random_hap(rng, m)
        src = np.resize(hap, n).copy()
        sub = rng.random(n) < (0.5 if k == 8 else 0.03)
        src[sub] = rng.choice(S.ALPHABET, int(sub.sum()))
        rb.append(src)
        rq.append(qf(n))
        hb.append(hap)
        ro.append(ro[-1] + n)
        ho.append(ho[-1] + m)
        pr.append(k)
        ph.append(k)
    pk = native.Packed(np.concatenate(rb), np.concatenate(rq), ro, np.concatenate(hb), ho, pair_read=pr, pair_hap=ph)
    eng = native.Engine(0, 4096)
    params, _ = native.make_params(S.GAP_Q45, S.EXT_Q10, False, native.VD_PRECISION_MIXED)
    ln, jac, st = eng.forward_backward(pk, params)
    one_ln, one_jac, _ = eng.forward_backward(pk, params, native.VD_CHECKPOINT_ALL)
    np.testing.assert_array_equal(ln, one_ln)
    np.testing.assert_array_equal(jac, one_jac)
    assert st.failed_pairs == 0
    p64, _ = native.make_params(S.GAP_Q45, S.EXT_Q10, False, native.VD_PRECISION_FLOAT64)
    _, jac64, _ = eng.forward_backward(pk, p64)
    np.testing.assert_allclose(jac.sum(0), jac64.sum(0), rtol=1e-6, atol=1e-6 * np.abs(jac64).max())
    want = [O.forward(bytes(r).decode(), q, bytes(h).decode(), S.GAP_Q45, S.EXT_Q10, False)
            for r, q, h in zip(rb, rq, hb)]
    assert np.max(np.abs(ln - np.array(want))) / np.log(10.0) <= 1e-4
    eng.close()
