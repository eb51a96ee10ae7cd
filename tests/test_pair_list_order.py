"""Pair lists that go haplotype by haplotype, so that every read comes back after thousands of
others: the regrouping is that of the same pairs read by read, bad input is reported as
there, and what is kept of the objects seen does not grow with the number of pairs."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from vardepth_b200 import native

ROOT = Path(__file__).resolve().parents[1]


def strings(rng, n, length):
    return ["".join(s) for s in rng.choice(list("ACGT"), (n, length))]


def test_regrouping_is_that_of_the_other_order():
    rng = np.random.default_rng(1)
    reads, haps = strings(rng, 9000, 12), strings(rng, 40, 30)  # 360,000 pairs
    quals = [rng.integers(2, 41, 12).astype(np.uint8) for _ in reads]
    by_hap = native.pair_list_plan([(s, q, h) for h in haps for s, q in zip(reads, quals)])
    by_read = native.pair_list_plan([(s, q, h) for s, q in zip(reads, quals) for h in haps])
    for name in ("read", "hap", "region", "slot"):
        a = by_hap[name].reshape(len(haps), len(reads)).T
        np.testing.assert_array_equal(a, by_read[name].reshape(len(reads), len(haps)))
    for name in ("n_reads", "n_haps", "n_regions", "n_slots"):
        assert by_hap[name] == by_read[name]


def test_the_first_bad_pair_is_reported():
    rng = np.random.default_rng(2)
    reads, haps = strings(rng, 9000, 8), strings(rng, 40, 20)
    quals = [np.full(8, 30, np.uint8) for _ in reads]
    pairs = [(s, q, h) for h in haps for s, q in zip(reads, quals)]
    pairs[5] = ("acgtacgt", quals[0], haps[0])
    with pytest.raises(ValueError, match="Uppercase DNA required"):
        native.pair_list_plan(pairs)
    pairs[5] = pairs[4]
    pairs[-1] = (reads[0], quals[0], "ACGX")
    with pytest.raises(ValueError, match="Uppercase DNA required"):
        native.pair_list_plan(pairs)


PROGRAM = """
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from vardepth_b200 import native
rng = np.random.default_rng(3)
reads = ["".join(s) for s in rng.choice(list("ACGT"), (20000, 8))]
quals = [np.full(8, 30, np.uint8) for _ in reads]
haps = ["".join(s) for s in rng.choice(list("ACGT"), (100, 20))]
pl = native.PairList([(s, q, h) for h in haps for s, q in zip(reads, quals)])
warm = native.pair_list_plan(native.PairList([(reads[0], quals[0], haps[0])]))
kb = lambda key: next(int(line.split()[1]) for line in open("/proc/self/status") if line.startswith(key))
before = kb("VmRSS")
native.pair_list_plan(pl)
print((kb("VmHWM") - before) // 1024)  # (ru_maxrss would count what the process it was forked from held)
"""


def test_memory_does_not_grow_with_the_pairs():
    """2,000,000 pairs of 20,000 reads: 28 bytes a pair of regrouping and 20 of results are 92 MB
    (a 40-byte object per pair, in a vector that doubles, is 80 to 200 more)."""
    out = subprocess.run([sys.executable, "-c", PROGRAM, str(ROOT)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert int(out.stdout) < 130, out.stdout
