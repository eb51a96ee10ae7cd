// Long reads (more rows than one strip), FP32, semiglobal: a read against TWO
// haplotypes of its region at a time, strip by strip, the strips of a pair
// running side by side on different warps of the GPU.
//
// The read's rows are packed as float2 over the two haplotypes of a pair (x:
// the first, y: the second), so every FMA serves both (fma.rn.f32x2) and the
// read's per-row constants and its strip count are shared: the halves always
// have the same number of strips, which two reads of different lengths would
// not.  A region's haplotypes differ by a few small edits, so their lengths
// nearly agree and the shorter one idles for a few columns at most.
//
// Tasks.  A strip of a pair is one task; an item (a read against up to
// kLongGroupMax haplotypes) holds its pairs' strips in order, and warps pull
// tasks from one counter.  Strip s+1 follows strip s at a distance of about
// three windows of 32 columns, reading the boundary rows s has published so
// far, so a pair takes about one strip's time plus that distance per strip
// instead of its strips one after another.  Every wait is for a task with a
// smaller number, which some resident warp has already pulled, so the lowest
// unfinished task can always go on; the waits are bounded all the same.
//
// Range.  An error-rich read (8% errors at reported Q30) loses about one bit
// per row along its best path, far more over a strip than FP32 holds, and
// along a row the cells away from the path lie thousands of binary orders
// lower.  So every lane keeps its rows' state scaled by its own power of two
// 2^e, chosen anew every 16 steps: a value never grows along a path, so what a
// lane can reach in the next 16 steps is bounded by the state of its own rows
// and of the lanes (and the boundary) above it, and e puts that bound at 2^100.
// The factor between a lane and the one above is folded into the lane's row 0,
// so the step itself carries no scaling; all factors are exact powers of two,
// undone in the exponent of the final sum.  What falls below 2^-126 lies more
// than 200 binary orders below the best cell near it.
//
// Nothing depends on which warp runs a task or when: a pair's result is a
// function of the read and its two haplotypes.  The final log is taken as
// ln f + (e + E) ln 2 with the sum z = f 2^e, so the bits do not depend on the
// powers of two either.  The plain schedule forms the same pairs and gives the
// same bits.
//
// What bounds it: alone, the chain of a strip's steps; in a full batch, issue
// slots and latency at 12 warps per SM (119 warp instructions a step for 256 x 2
// cells, 72 of them the rows; a quarter of the stalls are boundary words from
// L2).  Measured against a warp per item (its strips one after another, re-run
// with measured boosts when they left the FP32 range: 1.11 runs per strip): 30
// reads of 1-10 kb, 375 pairs, 388 -> 9.5 ms; 400 mixed-length regions 390 -> 28 ms;
// 16,000 of them (2.5e12 cells) 804 -> 782 ms, their long reads alone 557 -> 486 ms
// (2,586 GCUPS).  Exponents every 16 steps cost 12% against every 32, which a
// 40-base insertion run would defeat; letting a waiting strip fall 1 or 3 blocks
// further back, to meet the one above less often, cost 3% and 8%.
#pragma once
#include "pairhmm_kernel.cuh"
#include "pairhmm_wait.h"

namespace vd {

// A pair that has decayed by more than this many bits over its read's first
// `rows` rows goes to the drift and FP64 tiers: an error-rich read takes about one
// bit per row; a random read against a random haplotype takes four to five, and
// there alignment families that trade places across rows lie hundreds of bits
// apart (restated on the CPU with a looser bound of the lanes' exponents than
// rescale's: exact to FP32 rounding below 4.0 bits per row, off by up to 0.2 log10 at
// 4.0 to 4.4; with rescale's, 1,344 pairs of hanging reads were within 1.3e-5 without
// this line too, so it decides who scores such a pair, not whether FP32 could).
__host__ __device__ constexpr int long_max_bits(int rows) { return rows * 15 / 4; }
constexpr int kLongTop = 100;             // a lane's bound for the coming steps, binary orders
constexpr int kLongNone = -(1 << 28);     // exponent of "nothing there"

template <int R, bool GEN = false>
struct LongRows {
  uint32_t rb[R];        // read bases (kNeverBase for rows past the read)
  float miss[R];         // mismatch factor of rows 1 .. R-1 (the same for both halves)
  float hit[GEN ? R : 1];  // match factor (only where some row has P0 > P1; else 1)
  float2 hit0, miss0;    // row 0's match and mismatch factors times the lane's scale against the lane above, per half
  float2 K[R], X[R];     // k1 f_i and (x/4) f_i (alpha f_n on the last row), both halves
                         // (row 0's times that scale)
  float2 W[R], s[R];     // om of the next column and s of the column finished last
};

template <int R, bool GEN>
__device__ __forceinline__ void column_long(LongRows<R, GEN>& w, uint32_t hbx, uint32_t hby, float2 s_top, float2 u_top,
                                            float2 k2, float2 x, float2& u_bot) {
  float2 s_above = s_top;
  float2 nu = u_top;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float2 mu_new;
    if (r == 0) {
      const float fx = w.rb[0] == hbx ? w.hit0.x : w.miss0.x;
      const float fy = w.rb[0] == hby ? w.hit0.y : w.miss0.y;
      mu_new = __fmul2_rn(s_above, make_float2(fx, fy));
    } else if (GEN) {
      mu_new = __fmul2_rn(s_above, make_float2(w.rb[r] == hbx ? w.hit[r] : w.miss[r],
                                               w.rb[r] == hby ? w.hit[r] : w.miss[r]));
    } else {
      mu_new = s_above;
      mul_if_ne(mu_new.x, w.rb[r], hbx, w.miss[r]);
      mul_if_ne(mu_new.y, w.rb[r], hby, w.miss[r]);
    }
    const float2 om_new = w.W[r];
    const float2 u_new = __ffma2_rn(w.X[r], nu, mu_new);
    const float2 s_new = __ffma2_rn(k2, om_new, __ffma2_rn(w.K[r], nu, mu_new));
    s_above = w.s[r];
    w.W[r] = __ffma2_rn(x, om_new, mu_new);
    w.s[r] = s_new;
    nu = u_new;
  }
  u_bot = nu;
}

// Steps between two choices of the lanes' exponents.  A lane's bound takes every
// match at its full value, so in a path that inserts instead the lane's last cells lie
// up to (span + 2 R) log2(4/x) bits and a gap opening below it: at x = 0.1 185 bits for
// 16 steps of 8 rows, of the 226 between the bound and 2^-126, at 0.08 196; smaller x
// needs 8 steps (200 bits at 0.02).  Below kLongMinExt (pairhmm_kernel.cuh) the pair
// goes to the FP64 tier.  Measured against the long double oracle on 2,688 pairs of
// reads that hang off their haplotype by 20 bases to three quarters of their length,
// where every placement of the inserted run weighs the same: within 1e-5 log10 from
// x = 0.007 up, off by 6e-5 at 0.005 and 4e-2 at 0.003.  (With a bound that let a path
// come down by span / R + 1 lanes of matches after any number of insertions, and with
// the inputs of the whole window in it, up to 0.3 at 0.1 and 1 at 0.08; the closer bound
// costs 4% on error-rich 1-10 kb reads.)
constexpr int kLongSpan = 16, kLongSpanShort = 8;

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Waits until the task behind `p` has published `need` blocks; returns its word
// (wait_word; the same in every lane).
struct TaskWarp {
  const unsigned long long* word;
  int* error_flag;
  __device__ __forceinline__ unsigned long long load() const { return ld_acquire(word); }
  __device__ __forceinline__ bool stopped() const { return *(volatile int*)error_flag != 0; }
  __device__ __forceinline__ void give_up() const { atomicExch(error_flag, 2); }
  __device__ __forceinline__ void pause() const { __nanosleep(64); }
  __device__ __forceinline__ unsigned long long from_leader(unsigned long long v) const {
    v = __shfl_sync(0xffffffffu, v, 0);
    __syncwarp();  // (the other lanes' reads of the boundary come after the leader's acquire)
    return v;
  }
};
__device__ __forceinline__ unsigned long long wait_task(const unsigned long long* p, int need, int* error_flag,
                                                        bool& ok) {
  return wait_word(TaskWarp{p, error_flag}, need, ok);
}

// exponent of a non-negative float, kLongNone below the normal range
__device__ __forceinline__ int state_exponent(float v) {
  const int e = (int)((unsigned)__float_as_int(v) >> 23);
  return e == 0 ? kLongNone : e - 127;
}
__device__ __forceinline__ float normal_or_0(float v) { return v < 1.17549435e-38f ? 0.f : v; }
// v 2^k for any k: two exact factors (0 or inf past the range)
__device__ __forceinline__ float scale2(float v, int k) {
  k = max(-252, min(252, k));
  const int a = max(-126, min(126, k));
  return (v * pow2T(a, 0.f)) * pow2T(k - a, 0.f);
}

// One task: strip `strip` of item w's pair g (haplotypes g, g+1 of the item).
// `task` is its number; `half` the records of one boundary buffer (the block
// exponents follow at record exp_off); `bufs` the first buffer, `mine` the
// buffer this task writes.  `ring` and `oring` (32 float4 each) and `oexp` (4
// int2) are the warp's shared memory: the boundary read, the boundary written
// and lane 31's exponents of its four groups of 8 columns.  Returns
// false when a wait gave up.
// ALONE: the drift tier (pairhmm_drift.cu).  The warp runs the strips of its pair
// one after another, alternating between its two buffers, so nothing is waited for or
// published; `failed` carries the halves that left the range from strip to strip.
template <int R, int SPAN, bool GEN = false, bool ALONE = false>
__device__ __forceinline__ bool long_task(const BatchView& bv, const QueueView& qv, const WorkItem& w, const int g,
                                          const int strip, const int nstrips, const long long task,
                                          const Tables<float>* __restrict__ tb, const Scalars<float>& sc,
                                          const int lane, float4* const bufs, const long long half, const int mine,
                                          float4* __restrict__ ring, float4* __restrict__ oring,
                                          int2* __restrict__ oexp, unsigned& failed) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr double kLn2 = 0.6931471805599453094;
  constexpr int SR = kWarp * R;
  const int64_t roff = bv.read_off[w.read];
  const int n = (int)(bv.read_off[w.read + 1] - roff);
  const uint8_t* __restrict__ rbase = bv.read_bases + roff;
  const uint8_t* __restrict__ rqual = bv.read_quals + roff;
  const bool two = g + 1 < w.nhap;
  const int64_t h1 = w.hap_begin + g, h2 = two ? h1 + 1 : h1;
  const int64_t ho1 = bv.hap_off[h1], ho2 = bv.hap_off[h2];
  const int m1 = (int)(bv.hap_off[h1 + 1] - ho1), m2 = (int)(bv.hap_off[h2 + 1] - ho2);
  const uint8_t* __restrict__ hp1 = bv.hap_bases + ho1 - 1;  // hp[j] = base of column j >= 1
  const uint8_t* __restrict__ hp2 = bv.hap_bases + ho2 - 1;
  const int M = max(m1, m2);
  const bool first = strip == 0, last = strip == nstrips - 1;
  if (!ALONE && sc.x < kLongMinExt) {  // the whole pair to the next tiers
    if (last && lane < (two ? 2 : 1)) {
      const int64_t o = w.out_begin + g + lane;
      bv.out[o] = __longlong_as_double(0x7ff8000000000000LL);
      spill_pair<float>(qv, w.read, h1 + lane, o);
    }
    if (lane == 0) {
      st_release(qv.long_words + task, 0x3fffffffull);
      if (qv.strip_runs != nullptr) {
        atomicAdd(qv.strip_runs, 1ull);
        atomicAdd(qv.strip_runs + 1, 1ull);
      }
    }
    return true;
  }
  // windows of 32 steps; lane 31 finishes columns 32 (w-1) + 1 .. 32 w in window w (block w)
  const int nwin = (M + kWarp - 1) / kWarp + 1;
  unsigned long long* const word = qv.long_words + task;
  const unsigned long long* const above = word - 1;
  int* const err = qv.error_flag;
  bool ok = true;

  LongRows<R, GEN> rw;
  const int i0 = strip * SR;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = i0 + lane * R + r;
    if (i < n) {
      const unsigned q = rqual[i];
      rw.rb[r] = rbase[i];
      rw.miss[r] = tb->miss[q];
      if (GEN) rw.hit[r] = tb->hit[q];
      const float K = tb->K[q], X = (i == n - 1) ? tb->A[q] : tb->X[q];
      rw.K[r] = make_float2(K, K);
      rw.X[r] = make_float2(X, X);
    } else {  // past the read: pass u down the column
      rw.rb[r] = kNeverBase;
      rw.miss[r] = 0.f;
      if (GEN) rw.hit[r] = 0.f;
      rw.K[r] = make_float2(0.f, 0.f);
      rw.X[r] = make_float2(1.f, 1.f);
    }
    rw.W[r] = make_float2(0.f, 0.f);
    rw.s[r] = make_float2(0.f, 0.f);
  }
  const float K0 = rw.K[0].x, X0 = rw.X[0].x;  // row 0's own factors (those in rw carry the lane factor)
  // bits a path loses when it crosses this lane by insertions, one run of them
  // (X per row) or single ones (K), summed over the lanes down to this one (the
  // lanes past the read lose nothing, and no path to a lane of the read crosses its
  // last one)
  const int used = (min(SR, n - i0) + R - 1) / R;  // lanes holding read rows
  constexpr int near = (SPAN + R) / (R + 1);       // lanes a path can come down by matches alone (rescale)
  int cross = 0, far_off = 0, row_min = 30, row_max = 0;
  {
    float b = 0.f, top = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float c = -log2f(fmaxf(rw.X[r].x, rw.K[r].x));
      b += c;
      top = fmaxf(top, fminf(96.f, c));
      if (i0 + lane * R + r < n) row_min = min(row_min, (int)floorf(fminf(30.f, c - 0.01f)));
    }
    row_min = max(0, __reduce_min_sync(FULL, row_min));  // bits per row, at least
    row_max = __reduce_max_sync(FULL, lane < used - 1 ? (int)ceilf(top + 0.01f) : 0);  // and at most
    // (at most 96, so that neighbours' exponents differ by less than a float's range)
    const int own = lane < used - 1 ? max(0, (int)floorf(fminf(96.f, b - 0.01f))) : 0;
    cross = own;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
      const int v = __shfl_up_sync(FULL, cross, o);
      if (lane >= o) cross += v;
    }
    far_off = row_max * (SPAN - lane) - (cross - own);
  }

  // boundary above: lane i of window w holds column 32 w + i, raw, with the
  // exponents of the block it came in
  const float4* src = nullptr;
  const int2* src_exp = nullptr;
  float4 nxt = make_float4(0.f, 0.f, 0.f, 0.f);
  int2 nexp = make_int2(0, 0);
  int published = 0;  // blocks of the strip above known to be published
  if (ALONE && !first) {
    src = bufs + (long long)(mine ^ 1) * half;
    src_exp = reinterpret_cast<const int2*>(src + qv.long_exp_off);
  }
  auto load_window = [&](int wn) {
    if (!ALONE && published < min(wn + 2, nwin)) {
      const unsigned long long v = wait_task(above, min(wn + 2, nwin), err, ok);
      published = task_blocks(v);
      if (src == nullptr) {
        src = bufs + (long long)task_buffer(v) * half;
        src_exp = reinterpret_cast<const int2*>(src + qv.long_exp_off);
      }
    }
    const int p = wn * kWarp + lane;
    if (ok && p <= M) {
      nxt = __ldcg(src + p);
      // (denormals would count for nothing in the bound and still be scaled up)
      nxt = make_float4(normal_or_0(nxt.x), normal_or_0(nxt.y), normal_or_0(nxt.z), normal_or_0(nxt.w));
      nexp = __ldcg(src_exp + ((p + kWarp - 1) >> 3));
    } else {
      nxt = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  if (first) {
    nxt = make_float4(sc.c, sc.c, sc.c, sc.c);  // row 0: c at every column
  } else {
    load_window(0);
    if (!ok) return false;
  }
  float4* const dst = bufs + (long long)mine * half;
  int2* const dst_exp = reinterpret_cast<int2*>(dst + qv.long_exp_off);
  const unsigned long long tag = (unsigned long long)(unsigned)mine << 32;

  int ex = 0, ey = 0;  // the lane's state is scaled by 2^-e
  float2 s_top = make_float2(0.f, 0.f), u_bot = make_float2(0.f, 0.f), acc32 = make_float2(0.f, 0.f);
  double accx = 0.0, accy = 0.0;            // row sums of the window (scale of e)
  double totx = 0.0, toty = 0.0;            // row sums so far, times 2^-E
  int Ex = kLongNone, Ey = kLongNone;
  int bmx = kLongNone, bmy = kLongNone;     // exponents of the bottom row's maxima (this lane's columns)
  const bool lane0 = lane == 0;

  auto add_total = [&](double& acc, int e, double& tot, int& E) {
    if (acc > 0.0) {
      if (E == kLongNone) {
        tot = acc;
        E = e;
      } else if (e > E) {
        tot = ldexp(tot, max(-2000, E - e)) + acc;
        E = e;
      } else {
        tot += ldexp(acc, max(-2000, e - E));
      }
    } else if (acc != acc) {
      tot = acc;
    }
    acc = 0.0;
  };

  // new exponents for the steps from t on, from the state, the lanes above and
  // the inputs of these steps; `stage`: a window starts, its inputs go into the ring.
  // (Inputs of later steps do not count: along a run of insertions the boundary
  // rises by log2(4/x) bits a column, and every column of it carries as much of the
  // final sum.  They may leave the range in the ring, which is filled again then.)
  // INNER: no lane comes to a haplotype's end in these steps.
  auto rescale = [&](auto inner_tag, const int t, const bool stage) {
    constexpr bool INNER = decltype(inner_tag)::value;
    if (last) {
      add_total(accx, ex, totx, Ex);
      add_total(accy, ey, toty, Ey);
    }
    // the lane below still holds this lane's last diagonal, in this lane's scale
    float mx = __shfl_down_sync(FULL, s_top.x, 1), my = __shfl_down_sync(FULL, s_top.y, 1);
    if (lane == kWarp - 1) mx = my = 0.f;
    mx = fmaxf(mx, lane0 ? fmaxf(u_bot.x, s_top.x) : u_bot.x);
    my = fmaxf(my, lane0 ? fmaxf(u_bot.y, s_top.y) : u_bot.y);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      mx = fmaxf(mx, fmaxf(rw.s[r].x, rw.W[r].x));
      my = fmaxf(my, fmaxf(rw.s[r].y, rw.W[r].y));
    }
    // records past a haplotype's end do not count (nor do they lead anywhere)
    const int p = (t & ~(kWarp - 1)) + lane;
    const bool soon = (unsigned)(p - t) < (unsigned)SPAN;
    const int in_x = __reduce_max_sync(FULL, soon && (INNER || p <= m1) ? state_exponent(fmaxf(nxt.x, nxt.y)) + nexp.x : kLongNone);
    const int in_y = __reduce_max_sync(FULL, soon && (INNER || p <= m2) ? state_exponent(fmaxf(nxt.z, nxt.w)) + nexp.y : kLongNone);
    const int ox = state_exponent(mx), oy = state_exponent(my);
    // Largest exponent the lane can reach in the coming steps, from its own state,
    // the lanes above and the inputs (a lane above lane 0).  A path that comes down d
    // lanes takes a step for each, and one for each row it takes by a match (what
    // lies on the diagonal into the lane below is a match ahead): of the (d-1) R + 1
    // rows to the lane's first, at most SPAN - d + 1 are matches, which may lose
    // nothing, and the others cost insertions.  That leaves the lanes d <= near at
    // their full value, and the others less the bits of the lanes crossed, row_max
    // back for each match.  Near the haplotype's end the columns left bound the
    // matches too.  A lane that has gone past the last column feeds nothing any more.
    // (A shuffle from above lane 0 returns the lane's own value.)
    auto bound = [&](int o, int e, int in, int mh) -> int {
      int v = o + e;  // (far below every real one when there is nothing)
      if (!INNER && t - 1 - lane > mh) v = kLongNone;
      if (!INNER && t > mh) in = kLongNone;
      const int cols = INNER ? SPAN : max(0, min(SPAN, mh - (t - 1 - lane)));  // columns left
      int h = v;
      if (INNER) {
        int left = near;
#pragma unroll
        for (int o2 = 1; o2 < kWarp; o2 <<= 1) {
          if (left > 0) h = max(h, __shfl_up_sync(FULL, h, min(o2, left)));
          left -= min(o2, left);
        }
      } else {
#pragma unroll
        for (int d = 1; d <= near; ++d)
          h = max(h, __shfl_up_sync(FULL, v - row_min * max(0, R * (d - 1) + 1 - min(SPAN - d + 1, cols + 1)), d));
      }
      if (lane < near) h = max(h, in);
      int a = v + cross + row_max * lane;
#pragma unroll
      for (int o2 = 1; o2 < kWarp; o2 <<= 1) a = max(a, __shfl_up_sync(FULL, a, o2));
      a = __shfl_up_sync(FULL, a, near + 1);
      a = max(lane > near ? a : kLongNone, in - row_max) + far_off;
      if (!INNER) {
        int b = v + cross + row_max * cols;
#pragma unroll
        for (int o2 = 1; o2 < kWarp; o2 <<= 1) b = max(b, __shfl_up_sync(FULL, b, o2));
        b = __shfl_up_sync(FULL, b, near + 1);
        a = min(a, max(lane > near ? b : kLongNone, in + row_max * SPAN) + far_off - row_max * (SPAN - lane));
      }
      if (lane >= near) h = max(h, a);
      if (used < kWarp) {
        // the lanes past the read pass u down the column unchanged
        const int pad = __reduce_max_sync(FULL, lane >= used ? v : kLongNone);
        const int end = __shfl_sync(FULL, h, used - 1);
        if (lane >= used) h = max(pad, end);
      }
      return h;
    };
    const int Px = bound(ox, ex, in_x, m1), Py = bound(oy, ey, in_y, m2);
    const int nx = Px > kLongNone / 2 ? Px - kLongTop : ex, ny = Py > kLongNone / 2 ? Py - kLongTop : ey;
    int kx = ex - nx, ky = ey - ny;
    float2 f;
    // (nothing but denormals: they go to zero, whatever the new exponent)
    const bool none_x = ox == kLongNone, none_y = oy == kLongNone;
    const bool wide = __any_sync(FULL, (!none_x && abs(kx) > 126) || (!none_y && abs(ky) > 126));
    f = make_float2(none_x ? 0.f : pow2T(kx, 0.f), none_y ? 0.f : pow2T(ky, 0.f));
    if (wide) {
      // a shift beyond one factor: halve it (what needs more than 2^252 is zero)
      kx = none_x ? -252 : max(-252, min(252, kx));
      ky = none_y ? -252 : max(-252, min(252, ky));
      f = make_float2(pow2T(kx / 2, 0.f), pow2T(ky / 2, 0.f));
      const float2 f2 = make_float2(pow2T(kx - kx / 2, 0.f), pow2T(ky - ky / 2, 0.f));
      float2 g2 = make_float2(__shfl_up_sync(FULL, f2.x, 1), __shfl_up_sync(FULL, f2.y, 1));
      s_top = __fmul2_rn(s_top, g2);  // (lane 0: its own)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        rw.W[r] = __fmul2_rn(rw.W[r], f2);
        rw.s[r] = __fmul2_rn(rw.s[r], f2);
      }
      u_bot = __fmul2_rn(u_bot, f2);
    }
    // s_top came from the lane above (lane 0: from the ring, in its own scale)
    s_top = __fmul2_rn(s_top, make_float2(__shfl_up_sync(FULL, f.x, 1), __shfl_up_sync(FULL, f.y, 1)));
#pragma unroll
    for (int r = 0; r < R; ++r) {
      rw.W[r] = __fmul2_rn(rw.W[r], f);
      rw.s[r] = __fmul2_rn(rw.s[r], f);
    }
    u_bot = __fmul2_rn(u_bot, f);
    // the window's inputs in lane 0's scale
    const int e0x = __shfl_sync(FULL, nx, 0), e0y = __shfl_sync(FULL, ny, 0);
    __syncwarp();
    if (stage || __shfl_sync(FULL, ex, 0) != e0x || __shfl_sync(FULL, ey, 0) != e0y) {
      const int sx = nexp.x - e0x, sy = nexp.y - e0y;
      ring[lane] = make_float4(scale2(nxt.x, sx), scale2(nxt.y, sx), scale2(nxt.z, sy), scale2(nxt.w, sy));
    }
    ex = nx;
    ey = ny;
    // inputs come in the scale of the lane above: fold the difference into row 0
    const int upx = __shfl_up_sync(FULL, ex, 1) - ex, upy = __shfl_up_sync(FULL, ey, 1) - ey;  // (lane 0: 0)
    const float2 in = make_float2(pow2T(max(-127, min(126, upx)), 0.f), pow2T(max(-127, min(126, upy)), 0.f));
    rw.hit0 = GEN ? make_float2(rw.hit[0] * in.x, rw.hit[0] * in.y) : in;
    rw.miss0 = make_float2(rw.miss[0] * in.x, rw.miss[0] * in.y);
    rw.K[0] = make_float2(K0 * in.x, K0 * in.y);
    rw.X[0] = make_float2(X0 * in.x, X0 * in.y);
    if (lane == kWarp - 1) {
      const int q = (t >> 3) & 3;
      oexp[q] = make_int2(ex, ey);
      if (SPAN == 16) oexp[q + 1] = make_int2(ex, ey);
    }
    __syncwarp();
  };

  const float2 k2 = make_float2(sc.k2, sc.k2), x = make_float2(sc.x, sc.x);
  // one step; STEADY: every lane at a column in 1 .. min(m1, m2), its bases given
  auto step = [&](auto steady_tag, const int t, uint32_t hbx, uint32_t hby) {
    constexpr bool STEADY = decltype(steady_tag)::value;
    const int p = t - lane;  // this lane's column
    const float4 rec = ring[t & (kWarp - 1)];
    if (!STEADY) {
      // before column 1 the base does not matter (the state and the diagonal
      // are zero); past a haplotype's end its columns are not used
      hbx = __ldg(hp1 + max(1, min(p, m1)));
      hby = __ldg(hp2 + max(1, min(p, m2)));
    }
    float2 u_in = shfl_up2(u_bot);
    float2 s_in = shfl_up2(rw.s[R - 1]);
    u_in = lane0 ? make_float2(rec.y, rec.w) : u_in;
    s_in = lane0 ? make_float2(rec.x, rec.z) : s_in;
    column_long(rw, hbx, hby, s_top, u_in, k2, x, u_bot);
    s_top = s_in;
    if (STEADY) {
      acc32 = __fadd2_rn(acc32, u_bot);
    } else if (p >= 0) {
      if (p <= m1) acc32.x += u_bot.x;
      if (p <= m2) acc32.y += u_bot.y;
    }
    if (lane == kWarp - 1) oring[t & (kWarp - 1)] = make_float4(rw.s[R - 1].x, u_bot.x, rw.s[R - 1].y, u_bot.y);
  };
  // the FP32 row sums move into FP64 every 8 steps
  auto flush_acc = [&]() {
    if (last) {
      accx += (double)acc32.x;
      accy += (double)acc32.y;
    }
    acc32 = make_float2(0.f, 0.f);
  };
  // the 8 bases a lane passes in a group, as three aligned words (their first
  // and last bytes may belong to a neighbour in the batch's haplotype buffer),
  // loaded a group ahead
  uint32_t px0 = 0, px1 = 0, px2 = 0, py0 = 0, py1 = 0, py2 = 0;
  int fetched = -1;
  auto fetch = [&](const int t) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(hp1 + (t - lane)), b = reinterpret_cast<uintptr_t>(hp2 + (t - lane));
    const uint32_t* qa = reinterpret_cast<const uint32_t*>(a & ~(uintptr_t)3);
    const uint32_t* qb = reinterpret_cast<const uint32_t*>(b & ~(uintptr_t)3);
    px0 = __ldg(qa);
    px1 = __ldg(qa + 1);
    px2 = __ldg(qa + 2);
    py0 = __ldg(qb);
    py1 = __ldg(qb + 1);
    py2 = __ldg(qb + 2);
    fetched = t;
  };
  auto group = [&](auto steady_tag, const int wn, const int q) {
    const int t = wn * kWarp + q * 8;
    // (the last choice of exponents in the window was the last use of its records)
    constexpr int kLoadAt = (kWarp - SPAN) / 8;
    if constexpr (decltype(steady_tag)::value) {
      if (fetched != t) fetch(t);
      if (((q * 8) & (SPAN - 1)) == 0) rescale(steady_tag, t, q == 0);
      if (q == kLoadAt && !first && wn + 1 < nwin) load_window(wn + 1);
      const int sx = ((int)reinterpret_cast<uintptr_t>(hp1) + t - lane) & 3, sy = ((int)reinterpret_cast<uintptr_t>(hp2) + t - lane) & 3;
      const uint32_t xa = __funnelshift_r(px0, px1, sx * 8), xb = __funnelshift_r(px1, px2, sx * 8);
      const uint32_t ya = __funnelshift_r(py0, py1, sy * 8), yb = __funnelshift_r(py1, py2, sy * 8);
      // (the next group's columns lie inside both haplotypes, or are not used)
      if (t + 15 <= min(m1, m2)) fetch(t + 8);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        step(steady_tag, t + u, __byte_perm(u < 4 ? xa : xb, 0, 0x4440 + (u & 3)),
             __byte_perm(u < 4 ? ya : yb, 0, 0x4440 + (u & 3)));
    } else {
      if (((q * 8) & (SPAN - 1)) == 0) rescale(steady_tag, t, q == 0);
      if (q == kLoadAt && !first && wn + 1 < nwin) load_window(wn + 1);
#pragma unroll 1
      for (int u = 0; u < 8; ++u) step(steady_tag, t + u, 0u, 0u);
    }
    flush_acc();
    // the block laid down at the end of the last window: its stores have long
    // arrived, so the release costs no wait
    if (!ALONE && q == 0 && !last && lane0 && wn > 0) st_release(word, tag | (unsigned)wn);
  };
  for (int wn = 0; wn < nwin; ++wn) {
    // columns of this window: 32 wn - 31 .. 32 wn + 31
    if (wn >= 1 && wn * kWarp + kWarp - 1 <= min(m1, m2)) {
#pragma unroll 1
      for (int q = 0; q < kWarp / 8; ++q) group(std::true_type{}, wn, q);
    } else {
#pragma unroll 1
      for (int q = 0; q < kWarp / 8; ++q) group(std::false_type{}, wn, q);
    }
    if (!ok) return false;
    if (!last) {
      // block wn: columns 32 (wn - 1) + 1 .. 32 wn, 8 columns to an exponent
      __syncwarp();
      const int p = (wn - 1) * kWarp + 1 + lane;
      const int2 e = oexp[lane >> 3];
      if (p >= 0 && p <= M) {
        const float4 rec = oring[lane];
        __stcg(dst + p, rec);
        if (p <= m1) bmx = max(bmx, state_exponent(fmaxf(rec.x, rec.y)) + e.x);
        if (p <= m2) bmy = max(bmy, state_exponent(fmaxf(rec.z, rec.w)) + e.y);
      }
      if ((lane & 7) == 0) __stcg(dst_exp + wn * (kWarp / 8) + (lane >> 3), e);
      __syncwarp();
    }
  }
  if (last) {
    add_total(accx, ex, totx, Ex);
    add_total(accy, ey, toty, Ey);
  }

  // the halves that left what this tier keeps: their decay so far is over the rate
  unsigned lost = ALONE ? failed : 0u;
  if (!ALONE && !first) {
    const unsigned long long v = wait_task(above, nwin, err, ok);
    if (!ok) return false;
    lost = task_fail(v);
  }
  const int cap = ALONE && nstrips == 1 ? INT_MAX : long_max_bits(min(n, i0 + SR));
  if (!last) {
    bmx = __reduce_max_sync(FULL, bmx);
    bmy = __reduce_max_sync(FULL, bmy);
    if (bmx < -cap) lost |= 1u;
    if (bmy < -cap) lost |= 2u;
    if (ALONE) failed = lost;
    __syncwarp();
    if (!ALONE && lane0) {
      __threadfence();
      st_release(word, tag | ((unsigned long long)lost << 30) | (unsigned)nwin);
    }
  } else {
    double lnN = 0.0;
    for (int i = lane; i < n; i += kWarp) lnN += tb->lnN[rqual[i]];
#pragma unroll
    for (int o = 16; o; o >>= 1) lnN += __shfl_xor_sync(FULL, lnN, o);
    if (lane == kWarp - 1) {
      // ln of the final sum z = f 2^e (f in [1/2, 1)) and the exponent
      auto write = [&](double z, int E, bool bad, int m, int64_t h, int64_t o) {
        int e = 0;
        const double f = frexp(z, &e);
        if (!bad && z > 0.0 && z < HUGE_VAL && e - 1 + E >= -cap) {
          bv.out[o] = log(f) - (sc.ln_c + log((double)(m + 1))) + lnN + (double)(e + E) * kLn2;
        } else {
          bv.out[o] = __longlong_as_double(0x7ff8000000000000LL);
          spill_pair<float>(qv, w.read, h, o);
        }
      };
      write(totx, Ex, (lost & 1u) != 0, m1, h1, w.out_begin + g);
      if (two) write(toty, Ey, (lost & 2u) != 0, m2, h2, w.out_begin + g + 1);
    }
    if (!ALONE && lane0) st_release(word, (unsigned)nwin);
  }
  if (!ALONE && qv.strip_runs != nullptr && lane0) {
    atomicAdd(qv.strip_runs, 1ull);
    atomicAdd(qv.strip_runs + 1, 1ull);
  }
  return true;
}

// Persistent kernel of the long-read items (FP32 semiglobal primary tier): the
// warps pull tasks (strips of pairs) in order from qv.head, in both schedules.
// qv.long_off[i] is the number of item i's first task.  Each warp owns two
// boundary buffers and alternates; a buffer is written again once the task
// that reads it is done.
template <int LO, int HI, int kBlocks, int SPAN>
__global__ void __launch_bounds__(kWarpsPerBlock * kWarp, kBlocks)
pairhmm_long_kernel(const __grid_constant__ BatchView bv, const __grid_constant__ QueueView qv,
                    const Tables<float>* __restrict__ gtab, const __grid_constant__ Scalars<float> sc) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ Tables<float> tab;
  __shared__ float4 rings[kWarpsPerBlock][2][kWarp];
  __shared__ int2 exps[kWarpsPerBlock][4];
  {
    const int words = (int)(sizeof(Tables<float>) / sizeof(int));
    const int* src = reinterpret_cast<const int*>(gtab);
    int* dst = reinterpret_cast<int*>(&tab);
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const int lane = threadIdx.x & (kWarp - 1), wid = threadIdx.x >> 5;
  const int gw = (int)(blockIdx.x * kWarpsPerBlock) + wid;
  float4* const bufs = reinterpret_cast<float4*>(qv.scratch);
  const long long half = qv.scratch_stride / 2;
  long long reader[2] = {-1, -1};  // per buffer: the task that reads what this warp last wrote there
  int reader_blocks[2] = {0, 0};   // and its blocks
  for (int turn = 0;; turn ^= 1) {
    unsigned long long k = 0;
    if (lane == 0) k = atomicAdd(qv.head, 1ull);
    k = __shfl_sync(FULL, k, 0);
    if ((long long)k >= qv.long_tasks) break;
    // the item: the last one whose first task is not past k (32-way search)
    long long lo = 0, hi = qv.n_items;
    while (hi - lo > 1) {
      const long long st = (hi - lo + kWarp - 1) / kWarp;
      const long long at = lo + lane * st;
      const unsigned b = __ballot_sync(FULL, at < hi && qv.long_off[at] <= (long long)k);
      const int c = __popc(b) - 1;
      lo += c * st;
      hi = min(hi, lo + st);
    }
    const WorkItem w = qv.items[lo];
    const int R = code_R(w.code);
    const int n = (int)(bv.read_off[w.read + 1] - bv.read_off[w.read]);
    const int nstrips = (n + kWarp * R - 1) / (kWarp * R);
    const int j = (int)((long long)k - qv.long_off[lo]);
    const int g = 2 * (j / nstrips), strip = j % nstrips;
    bool ok = true;
    unsigned failed = 0;
    if (strip < nstrips - 1) {
      if (reader[turn] >= 0) wait_task(qv.long_words + reader[turn], reader_blocks[turn], qv.error_flag, ok);
      const int64_t h = w.hap_begin + g;
      const int ma = (int)(bv.hap_off[h + 1] - bv.hap_off[h]);
      const int mb = g + 1 < w.nhap ? (int)(bv.hap_off[h + 2] - bv.hap_off[h + 1]) : ma;
      reader[turn] = (long long)k + 1;
      reader_blocks[turn] = (max(ma, mb) + kWarp - 1) / kWarp + 1;
    }
    if (ok) {
      switch (R) {
#define VD_LCASE(r)                                                                                              \
  case r:                                                                                                        \
    if constexpr (r >= LO && r <= HI)                                                                            \
      ok = long_task<r, SPAN>(bv, qv, w, g, strip, nstrips, (long long)k, &tab, sc, lane, bufs, half, 2 * gw + turn,  \
                        rings[wid][0], rings[wid][1], exps[wid], failed);                                                \
    break;
        VD_LCASE(4) VD_LCASE(5) VD_LCASE(6) VD_LCASE(7) VD_LCASE(8)
#undef VD_LCASE
        default: break;
      }
    }
    if (!__all_sync(FULL, ok)) break;  // a wait gave up: the error flag is set
  }
}

}  // namespace vd
