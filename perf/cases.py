"""The work users have this framework do, as measurable cases.

Every case goes through a public entry point (vardepth_b200.accelerator and
vardepth_b200.native) on inputs of the shapes the synthetic workloads, the tests
and the benchmark use: regions of reads x candidate haplotypes, pair lists of
strings, anchored refinement windows, 1-10 kb reads, the gradient of the error
model and region genotypes.  The entry points take host buffers, so ``run`` of
those cases is the whole call (work list, copies, kernels, results); the resident
plan and the device-buffer region start from inputs already on the GPU.

Sizes (reads, haplotypes, lengths) depend on the case alone and the contents on
the seed, so two seeds of a case are the same amount of work.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from vardepth_b200 import native
from vardepth_b200 import synthetic as S
from vardepth_b200.accelerator import CudaPairHMM

MEMORY_MB = 8192


# ---- cases ------------------------------------------------------------------------

def listed():
    return [
        # one active region as a caller scores it while it walks the genome: launch and
        # host latency (the single-region workload: 64 reads of 150 bp, 2 haplotypes)
        {"name": "one_region", "kind": "host", "shape": "short", "regions": 1, "reads": 64, "read_lo": 150,
         "read_hi": 150, "haps_lo": 2, "haps_hi": 2, "hap_lo": 300, "hap_hi": 300, "sizes": 1},
        # the same with the inputs already in the caller's device memory and no allocation allowed
        {"name": "device_region", "kind": "device", "shape": "short", "regions": 1, "reads": 301, "read_lo": 100,
         "read_hi": 250, "haps_lo": 13, "haps_hi": 13, "hap_lo": 421, "hap_hi": 421, "anchored": False, "sizes": 2},
        # indel refinement: read spans against left + allele + right windows of about their
        # length, anchored (global) mode, a list of Python strings
        {"name": "anchored_windows", "kind": "list", "shape": "windows", "regions": 1500, "reads": 9, "read_lo": 20,
         "read_hi": 180, "haps_lo": 2, "haps_hi": 5, "hap_lo": 0, "hap_hi": 0, "anchored": True, "sizes": 3},
        # the reference's call signature: a list of (read, qualities, haplotype) of 60 regions
        {"name": "pair_list", "kind": "list", "shape": "short", "regions": 60, "reads": 60, "read_lo": 100,
         "read_hi": 250, "haps_lo": 2, "haps_hi": 16, "hap_lo": 100, "hap_hi": 1000, "anchored": False, "sizes": 4},
        # a batch of ordinary regions kept on the device and scored again
        {"name": "regions_resident", "kind": "plan", "shape": "short", "regions": 500, "reads": 60, "read_lo": 100,
         "read_hi": 250, "haps_lo": 2, "haps_hi": 16, "hap_lo": 100, "hap_hi": 1000, "sizes": 5},
        # the throughput workload: a large batch of regions from host buffers
        {"name": "regions_large", "kind": "host", "shape": "short", "regions": 2500, "reads": 60, "read_lo": 100,
         "read_hi": 250, "haps_lo": 2, "haps_hi": 16, "hap_lo": 100, "hap_hi": 1000, "sizes": 6},
        # the FP64 mode callers use for ties and for checking
        {"name": "regions_float64", "kind": "host", "shape": "short", "regions": 40, "reads": 60, "read_lo": 100,
         "read_hi": 250, "haps_lo": 2, "haps_hi": 16, "hap_lo": 100, "hap_hi": 1000, "float64": True, "sizes": 7},
        # 1-5 kb haplotypes, reads of 150-300 bases, a fifth of them of poor quality
        {"name": "long_haplotypes", "kind": "host", "shape": "stress", "regions": 120, "reads": 50, "read_lo": 150,
         "read_hi": 300, "haps_lo": 4, "haps_hi": 4, "hap_lo": 1000, "hap_hi": 5000, "sizes": 8},
        # 1-10 kb reads at 8% error: the few long-read regions of a small batch
        {"name": "long_reads", "kind": "host", "shape": "long", "regions": 6, "reads": 5, "read_lo": 1000,
         "read_hi": 10000, "haps_lo": 2, "haps_hi": 32, "hap_lo": 0, "hap_hi": 0, "sizes": 9},
        # regions of 150 bp reads with 2% of them long-read regions, in one batch
        {"name": "mixed_lengths", "kind": "host", "shape": "mixed", "regions": 400, "reads": 40, "read_lo": 150,
         "read_hi": 150, "haps_lo": 2, "haps_hi": 32, "hap_lo": 80, "hap_hi": 8000, "sizes": 10},
        # one evaluation of the error-model fit: ln L and its six derivatives per pair
        {"name": "gradient", "kind": "gradient", "shape": "short", "regions": 40, "reads": 60, "read_lo": 100,
         "read_hi": 250, "haps_lo": 2, "haps_hi": 16, "hap_lo": 100, "hap_hi": 1000, "anchored": False,
         "float64": False, "sizes": 11},
        # forward pass, normalised rows and diploid genotype likelihoods with the near-tie guard
        {"name": "genotypes", "kind": "genotypes", "shape": "short", "regions": 150, "reads": 60, "read_lo": 100,
         "read_hi": 250, "haps_lo": 2, "haps_hi": 16, "hap_lo": 100, "hap_hi": 1000, "prior": -1.0, "sizes": 12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    base = dict(rng.choice(listed()))
    del base["name"]
    base["sizes"] = rng.randrange(1000, 1 << 30)
    kind, shape = base["kind"], base["shape"]
    if kind == "device":
        base["reads"] = _log_int(rng, 8, 700)
        base["haps_lo"] = base["haps_hi"] = rng.randint(1, 24)
        base["hap_lo"] = base["hap_hi"] = _log_int(rng, 90, 1000)
        base["read_lo"] = rng.randint(20, 150)
        base["read_hi"] = rng.randint(150, 255)
        return base
    if shape == "windows":
        base["regions"] = _log_int(rng, 20, 2500)
        base["reads"] = rng.randint(2, 15)
        base["read_hi"] = rng.randint(60, 250)
        return base
    if shape == "long":
        base["regions"] = rng.randint(1, 6)
        base["reads"] = rng.randint(1, 5)
        base["read_lo"] = rng.randint(300, 2000)
        base["read_hi"] = rng.randint(2500, 9000)
        return base
    if shape == "stress":
        base["regions"] = _log_int(rng, 4, 120)
        base["haps_lo"], base["haps_hi"] = 2, rng.randint(2, 6)
        base["read_hi"] = rng.randint(200, 300)
        return base
    if shape == "mixed":
        base["regions"] = _log_int(rng, 40, 400)
        base["haps_hi"] = rng.randint(4, 32)
        return base
    # short reads: a single region up to the listed batch
    top = max(base["regions"], 8)
    base["regions"] = _log_int(rng, 1, top)
    base["reads"] = _log_int(rng, 10, 90)
    a, b = sorted((rng.randint(25, 250), rng.randint(25, 256)))
    if kind == "gradient":
        b = min(b, 255)
        base["anchored"] = rng.random() < 0.2
        base["float64"] = rng.random() < 0.2
        if base["float64"]:
            base["regions"] = max(1, base["regions"] // 4)
    base["read_lo"], base["read_hi"] = a, b
    base["haps_lo"] = rng.randint(1, 6)
    base["haps_hi"] = rng.randint(base["haps_lo"], 16)
    base["hap_lo"] = rng.randint(60, 400)
    base["hap_hi"] = rng.randint(base["hap_lo"], 1000)
    if kind == "genotypes":
        base["prior"] = rng.choice([-1.0, 0.0, 0.01])
    return base


# ---- inputs -----------------------------------------------------------------------

def _is_long(case, sizes_rng):
    return case["shape"] == "long" or (case["shape"] == "mixed" and sizes_rng.random() < 0.02)


def _region_sizes(case):
    """Per region: (first haplotype's length, haplotypes, read lengths, long-read region),
    from the case alone."""
    rng = np.random.default_rng([case["sizes"], 77])
    out = []
    for g in range(case["regions"]):
        H = int(rng.integers(case["haps_lo"], case["haps_hi"] + 1))
        long_region = _is_long(case, rng) or (case["shape"] == "mixed" and g == 0)
        if long_region:
            lo, hi = (case["read_lo"], case["read_hi"]) if case["shape"] == "long" else (1000, 10000)
            nr = case["reads"] if case["shape"] == "long" else int(rng.integers(2, 9))
            lengths = rng.integers(lo, hi + 1, nr)
            m0 = int(lengths.max() + rng.integers(100, 1000))
        elif case["shape"] == "windows":
            nr = case["reads"]
            span = int(rng.integers(case["read_lo"], case["read_hi"] + 1))
            lengths = np.clip(span + rng.integers(-3, 4, nr), 4, None)
            m0 = span
        else:
            if case["kind"] == "device" or case["regions"] == 1 and case["shape"] == "short":
                nr = case["reads"]
            elif case["shape"] == "stress":
                nr = case["reads"]
            else:
                nr = int(np.clip(round(rng.lognormal(np.log(case["reads"]), 1.0)), 4, 500))
            lengths = rng.integers(case["read_lo"], case["read_hi"] + 1, nr)
            if case["shape"] == "mixed":
                m0 = int(np.clip(round(rng.lognormal(np.log(400), 0.6)), case["hap_lo"], case["hap_hi"]))
            else:
                m0 = int(rng.integers(case["hap_lo"], case["hap_hi"] + 1))
        out.append((m0, H, lengths.astype(np.int64), long_region))
    return out


def _workload(case, seed) -> S.Workload:
    rng = np.random.default_rng([seed, case["sizes"]])
    good = S._q_standard(rng)
    poor = lambda n: rng.integers(2, 16, n).astype(np.uint8)
    regions = []
    for m0, H, lengths, long_region in _region_sizes(case):
        hap0 = S._random_hap(rng, m0)
        nr = len(lengths)
        if case["shape"] == "windows":
            # left + allele + right windows: the alleles differ by a short indel or an SNV
            haps = [hap0]
            for _ in range(H - 1):
                haps.append(S._mutate(rng, hap0, int(rng.integers(0, 2)), int(rng.integers(1, 5))))
            reads, quals = S._sim_reads(rng, haps, nr, lengths, 0.01, 0.001, good)
        else:
            haps = [hap0]
            cap = 1023 if case["kind"] == "device" else 1 << 30  # the device-buffer call's haplotype limit
            while len(haps) < H:
                h = S._mutate(rng, hap0, int(rng.integers(1, 5)), int(rng.integers(1, 11)))
                haps.append(h[:cap])
            if long_region:
                reads, quals = S._sim_reads(rng, haps, nr, lengths, 0.06, 0.02, good)
            elif case["shape"] == "stress":
                bad = np.arange(nr) % 5 == 0
                reads, quals = S._sim_reads(rng, haps, int((~bad).sum()), lengths[~bad], 0.01, 0.001, good)
                r2, q2 = S._sim_reads(rng, haps, int(bad.sum()), lengths[bad], 0.05, 0.0, poor)
                reads, quals = reads + r2, quals + q2
            else:
                reads, quals = S._sim_reads(rng, haps, nr, lengths, 0.01, 0.001, good)
        regions.append((haps, reads, quals))
    return S._assemble("case", regions, S.GAP_Q45, S.EXT_Q10, {})


def _packed(w):
    return native.Packed(w.read_bases, w.read_quals, w.read_off, w.hap_bases, w.hap_off,
                         region_read_off=w.region_read_off, region_hap_off=w.region_hap_off)


def _strings(w):
    """The workload as the reference's list of (read, qualities, haplotype) triples, region by
    region, reads x haplotypes."""
    pairs = []
    reads, quals, haps = w.read_bases.tobytes(), w.read_quals.tobytes(), w.hap_bases.tobytes()
    for g in range(w.n_regions):
        hs = [haps[w.hap_off[h]:w.hap_off[h + 1]].decode()
              for h in range(w.region_hap_off[g], w.region_hap_off[g + 1])]
        for r in range(w.region_read_off[g], w.region_read_off[g + 1]):
            a, b = w.read_off[r], w.read_off[r + 1]
            s, q = reads[a:b].decode(), quals[a:b]
            pairs.extend((s, q, h) for h in hs)
    return pairs


def prepare(case, seed):
    w = _workload(case, seed)
    state = {"case": case}
    kind = case["kind"]
    f64 = bool(case.get("float64", False))
    if kind == "device":
        dev = torch.device("cuda", torch.cuda.current_device())
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
        state["bufs"] = [put(a) for a in (w.read_bases, w.read_quals, w.read_off, w.hap_bases, w.hap_off)]
        state["n"] = (len(w.read_off) - 1, len(w.hap_off) - 1)
        state["out"] = torch.empty(w.pairs(), dtype=torch.float64, device=dev)
        state["params"] = native.make_params(w.gap, w.ext, case["anchored"], native.VD_PRECISION_MIXED)
        return state
    state["engine"] = CudaPairHMM(memory_mb=MEMORY_MB, precision="float64" if f64 else "mixed", gap=w.gap, ext=w.ext)
    if kind == "list":
        state["pairs"] = _strings(w)
        return state
    state["packed"] = _packed(w)
    precision = native.VD_PRECISION_FLOAT64 if f64 else native.VD_PRECISION_MIXED
    state["params"] = native.make_params(w.gap, w.ext, bool(case.get("anchored", False)), precision)
    if kind == "plan":
        state["plan"] = state["engine"].engine.plan(state["packed"], state["params"][0])
    if kind == "genotypes":
        state["mq"] = np.random.default_rng([seed, 5]).integers(20, 61, len(w.read_off) - 1).astype(np.uint8)
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "host":
        return state["engine"].score_packed(state["packed"])
    if kind == "list":
        return state["engine"].score(state["pairs"], state["case"]["anchored"])
    if kind == "plan":
        state["plan"].run()
        return state["plan"].fetch()
    if kind == "gradient":
        ln, jac, _ = state["engine"].engine.forward_backward(state["packed"], state["params"][0])
        return ln, jac
    if kind == "genotypes":
        prior = state["case"]["prior"]
        g = state["engine"].engine.region_genotypes(state["packed"], state["params"][0], mapping_quality=state["mq"],
                                                    artifact_prior=None if prior < 0 else prior, near_tie_guard=True)
        return g["ln"], g["values"], g["certainty"], np.concatenate(g["gl"]), g["guarded"]
    # device: one region from the caller's device buffers, on the current stream
    rb, rq, ro, hb, ho = (t.data_ptr() for t in state["bufs"])
    nr, nh = state["n"]
    out = state["out"]
    native.check(native.library().vd_forward_region_noalloc(
        out.device.index, rb, rq, ro, nr, hb, ho, nh, ctypes.byref(state["params"][0]), out.data_ptr(),
        torch.cuda.current_stream().cuda_stream), "vd_forward_region_noalloc")
    return out


def work(case):
    """Cells of the recurrence (one multiply and four multiply-adds each; the gradient adds a
    reverse sweep of twice that) and the input and output bytes."""
    cells = in_bytes = outs = gls = reads = 0
    for m0, H, lengths, _ in _region_sizes(case):
        n = int(np.minimum(lengths, m0).sum())
        cells += n * m0 * H
        in_bytes += 2 * n + m0 * H
        outs += len(lengths) * H
        gls += H * (H + 1) // 2
        reads += len(lengths)
    per_cell, out_bytes = 9, 8 * outs
    if case["kind"] == "gradient":
        per_cell, out_bytes = 27, 56 * outs
    if case["kind"] == "genotypes":
        out_bytes = 16 * outs + 8 * gls + 8 * reads
    return {"bytes": in_bytes + out_bytes, "flops": per_cell * cells}


# ---- values in 64 bits ----------------------------------------------------------------

EXACT_CELLS = 6e10
_BLOCK = 1 << 24  # cells of one DP row over the pairs done together


def _pair_index(w):
    pr, ph = w.explicit_pairs()
    return pr.astype(np.int64), ph.astype(np.int64)


def _forward64(w, gap, ext, anchored, phred, device, dtype=torch.float64):
    """Likelihoods of every pair of the workload as (mantissa, ln scale): row by row over the
    reads, the deletions of a row by doubling, rows divided by their maximum.  ``phred`` maps
    the 256 quality bytes to their Phred values; gap, ext and phred may carry an imaginary
    part (complex-step differentiation)."""
    pr, ph = _pair_index(w)
    rl, hl = w.read_lengths(), w.hap_lengths()
    err = (10.0 ** (-torch.as_tensor(phred, dtype=dtype, device=device) / 10.0))
    p_hit, p_miss = 1.0 - err, err / 3.0
    rb = torch.from_numpy(w.read_bases).to(device)
    rq = torch.from_numpy(w.read_quals.astype(np.int64)).to(device)
    hb = torch.from_numpy(w.hap_bases).to(device)
    mant = torch.zeros(len(pr), dtype=dtype, device=device)
    scale = torch.zeros(len(pr), dtype=torch.float64, device=device)
    order = np.lexsort((rl[pr], hl[ph]))
    a, b = 1.0 - 2.0 * gap, 1.0 - ext
    lo = 0
    while lo < len(order):
        hi = lo
        while hi < len(order) and (hi - lo + 1) * (hl[ph[order[hi]]] + 1) <= _BLOCK:
            hi += 1
        hi = max(hi, lo + 1)
        idx = order[lo:hi]
        idx = idx[np.argsort(-rl[pr[idx]], kind="stable")]  # longest reads first: finished pairs drop off the end
        lo = hi
        n, m = rl[pr[idx]], hl[ph[idx]]
        N, Mx = int(n.max()), int(m.max())
        P = len(idx)
        tn = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(device)
        mt = tn(m)
        cols = torch.arange(Mx, device=device)
        haps = hb[torch.clamp(tn(w.hap_off[ph[idx]])[:, None] + cols, max=len(hb) - 1)]
        M = torch.zeros((P, Mx + 1), dtype=dtype, device=device)
        D = torch.zeros_like(M)
        if anchored:
            M[:, 0] = 1.0
            D[:, 1:] = gap * torch.as_tensor(ext, dtype=dtype, device=device) ** cols
        else:
            M += (1.0 / (mt + 1).to(torch.float64))[:, None]
        I = torch.zeros_like(M)
        ln = torch.zeros(P, dtype=torch.float64, device=device)
        row0 = tn(w.read_off[pr[idx]])
        for i in range(N):
            live = int(np.searchsorted(-n, -i, side="left"))  # pairs with n > i
            if live < len(M):
                M, I, D, haps, ln, mt, row0 = M[:live], I[:live], D[:live], haps[:live], ln[:live], mt[:live], row0[:live]
            base, q = rb[row0 + i], rq[row0 + i]
            em = torch.where(haps == base[:, None], p_hit[q][:, None], p_miss[q][:, None])
            Mn = torch.zeros_like(M)
            Mn[:, 1:] = em * (a * M[:, :-1] + b * (I[:, :-1] + D[:, :-1]))
            I = (gap * M + ext * I) * 0.25
            D = torch.zeros_like(M)
            D[:, 1:] = gap * Mn[:, :-1]
            s = 1
            while s <= Mx and abs(ext) ** s > 1e-300:
                prev = D.clone()
                D[:, s:] += (ext ** s) * prev[:, :-s]
                s *= 2
            M = Mn
            done_hi = live
            done_lo = int(np.searchsorted(-n, -(i + 1), side="left"))  # pairs with n == i + 1: [done_lo, live)
            if i % 4 == 3 or done_lo < done_hi:
                top = torch.maximum(torch.maximum(M.real if M.is_complex() else M, I.real if I.is_complex() else I),
                                    D.real if D.is_complex() else D).amax(1)
                inv = (1.0 / top)[:, None]
                M, I, D = M * inv, I * inv, D * inv
                ln = ln + torch.log(top)
            if done_lo < done_hi:
                sl = slice(done_lo, done_hi)
                at = mt[sl]
                if anchored:
                    row = M[sl] + I[sl] + D[sl]
                    z = row.gather(1, at[:, None])[:, 0]
                else:
                    inside = torch.arange(Mx + 1, device=device) <= at[:, None]
                    z = torch.where(inside, M[sl] + I[sl], torch.zeros((), dtype=dtype, device=device)).sum(1)
                where = tn(idx[done_lo:done_hi])
                mant[where] = z
                scale[where] = ln[sl]
    return mant, scale


def _phred():
    return np.minimum(np.arange(256), 60).astype(np.float64)


def _exact_ln(w, anchored, device):
    mant, scale = _forward64(w, w.gap, w.ext, anchored, _phred(), device)
    return (torch.log(mant) + scale).cpu().numpy()


def _exact_jacobian(w, anchored, device):
    """d ln L / d (Qg, Qx, o0..o3) by the complex step."""
    h = 1e-40
    bins = np.searchsorted(np.array([15, 25, 35]), np.arange(256), side="right")
    ln10 = math.log(10.0) / 10.0
    cols = []
    for k in range(6):
        gap = w.gap * complex(1.0, -ln10 * h) if k == 0 else complex(w.gap)
        ext = w.ext * complex(1.0, -ln10 * h) if k == 1 else complex(w.ext)
        ph = _phred().astype(np.complex128)
        if k >= 2:
            ph = ph + 1j * h * (bins == k - 2)
        mant, _ = _forward64(w, gap, ext, anchored, ph, device, torch.complex128)
        cols.append((mant.imag / mant.real / h).cpu().numpy())
    return np.stack(cols, 1)


def exact(case, seed):
    total = work(case)["flops"] / (27 if case["kind"] == "gradient" else 9)
    limit = EXACT_CELLS / 12 if case["kind"] == "gradient" else EXACT_CELLS
    if total > limit:
        return None
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    w = _workload(case, seed)
    anchored = bool(case.get("anchored", False))
    ln = _exact_ln(w, anchored, device)
    if case["kind"] == "gradient":
        return ln, _exact_jacobian(w, anchored, device)
    if case["kind"] == "device":
        return torch.from_numpy(ln)
    if case["kind"] != "genotypes":
        return ln
    mq = np.random.default_rng([seed, 5]).integers(20, 61, len(w.read_off) - 1).astype(np.uint8)
    values, certainty, gls = np.empty_like(ln), np.full(len(mq), np.nan), []
    o = 0
    for g in range(w.n_regions):
        r0, r1 = w.region_read_off[g], w.region_read_off[g + 1]
        H = int(w.region_hap_off[g + 1] - w.region_hap_off[g])
        ll = ln[o:o + (r1 - r0) * H].reshape(r1 - r0, H)
        e = (10.0 ** (-np.minimum(mq[r0:r1], 60).astype(np.float64) / 10.0))[:, None]
        v = np.exp(ll - ll.max(1, keepdims=True))
        v = (1.0 - e) * v + e * v.mean(1, keepdims=True)
        values[o:o + v.size] = v.ravel()
        lv = np.log(np.maximum(v, 1e-300))
        certainty[r0:r1] = lv.max(1) - lv.min(1)
        b_, a_ = np.tril_indices(H)  # b = 0..H-1, a = 0..b
        gls.append(np.log(np.maximum(1e-300, 0.5 * (v[:, a_] + v[:, b_]))).sum(0))
        o += v.size
    return ln, values, certainty, np.concatenate(gls) if case["prior"] < 0 else None, None
