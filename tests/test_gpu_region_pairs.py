"""vd_forward_region_noalloc with two reads per warp.

From eight (read, haplotype) pairs per SM on, the FP32 semiglobal call packs two reads of
one class (rows per lane, one-sided emission) into a warp; below it every read runs alone.
Both run the same arithmetic per pair, so a region gives the same bits scored whole and
scored in slices of reads too small to be packed; every pair is also within the library's
bound of the FP64 oracle.
"""
import numpy as np
import pytest

from test_zz_no_alloc import assert_agree, call_noalloc, oracle_region
from vardepth_b200 import native

pytestmark = pytest.mark.gpu

BASES = np.frombuffer(b"ACGT", dtype=np.uint8)


def region(seed, lengths, n_haps, hap_len):
    """Reads of the given lengths from mutated copies of one haplotype; every 11th read has a
    Phred-0 base, every 13th is unrelated (it leaves the FP32 range)."""
    rng = np.random.default_rng(seed)
    base = rng.choice(BASES, hap_len)
    haps = [base]
    for _ in range(n_haps - 1):
        h = base[:hap_len - int(rng.integers(0, 5))].copy()
        h[rng.integers(0, len(h), 3)] = rng.choice(BASES, 3)
        haps.append(h)
    if n_haps > 2:
        haps[1] = haps[1][:0]
    reads, quals = [], []
    for i, n in enumerate(lengths):
        src = np.concatenate([haps[0]] * (1 + n // hap_len))
        o = int(rng.integers(0, len(src) - n + 1))
        s = src[o:o + n].copy()
        q = rng.integers(8, 41, n).astype(np.uint8)
        if n and i % 11 == 7:
            q[rng.integers(0, n)] = 0
        if i % 13 == 5:
            s = rng.choice(BASES, n)
        reads.append(s)
        quals.append(q)
    off = lambda x: np.concatenate([[0], np.cumsum([len(v) for v in x])]).astype(np.int64)
    return (np.concatenate(reads).astype(np.uint8), np.concatenate(quals).astype(np.uint8), off(reads),
            np.concatenate(haps).astype(np.uint8), off(haps))


def slices(reg, step):
    rb, rq, ro, hb, ho = reg
    parts = []
    for a in range(0, len(ro) - 1, step):
        b = min(len(ro) - 1, a + step)
        lo, hi = ro[a], ro[b]
        rc, got = call_noalloc((rb[lo:hi] if hi > lo else rb[:1], rq[lo:hi] if hi > lo else rq[:1], ro[a:b + 1] - lo, hb, ho),
                               False, native.VD_PRECISION_MIXED)
        assert rc == native.VD_OK, native.last_error()
        parts.append(got)
    return np.concatenate(parts)


CASES = {
    # every class odd and even in number, reads at the edges of the classes, an empty one
    "classes": (list(range(1, 256, 2)) + [32, 33, 64, 65, 96, 97, 128, 129, 224, 225, 255, 255, 0], 9, 301),
    # one class, an even and an odd number of reads
    "even": ([150] * 600, 2, 200),
    "odd": ([150] * 601, 2, 97),
    # one read per class, and a class of one
    "one_each": ([20, 40, 70, 100, 130, 170, 200, 250], 300, 120),
    # more haplotypes than pieces, streams of many haplotypes
    "many_haps": ([101] * 33 + [250], 700, 40),
    # as many pairs as the line and one fewer on a GPU of 148 SMs
    "line": ([90] * 1184, 1, 150),
    "below": ([90] * 1183, 1, 150),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_packed_region_matches_reads_alone_and_the_oracle(name):
    lengths, n_haps, hap_len = CASES[name]
    reg = region(5, lengths, n_haps, hap_len)
    rc, got = call_noalloc(reg, False, native.VD_PRECISION_MIXED)
    assert rc == native.VD_OK, native.last_error()
    alone = slices(reg, max(1, 600 // n_haps))
    assert np.array_equal(got, alone)
    assert_agree(got, oracle_region(reg, False), native.VD_PRECISION_MIXED)
