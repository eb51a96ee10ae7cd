// Reverse-wavefront gradient of the PairHMM log-likelihood on sm_100a.
//
// For every read x haplotype pair the kernel returns ln L and the six partial
// derivatives d ln L / d theta, theta = (gap-open Phred Qg, gap-continuation
// Phred Qx, Phred offsets o0..o3 of the four quality bins), g = 10^(-Qg/10),
// x = 10^(-Qx/10), e = 10^(-max(0, min(q,60) + o_bin(q))/10).  The reference
// has no differentiable PairHMM: this is reverse-mode differentiation of the
// scaled forward recurrence of pairhmm_core.cuh, i.e. (semiglobal mode) of
//   mu_i(j) = s_{i-1}(j-1) h_ij                 h = hit or miss of row i
//   om_i(j) = mu_i(j-1) + x om_i(j-1)
//   u_i(j)  = mu_i(j) + X_i u_{i-1}(j)          (X_n = A_n on the last row)
//   s_i(j)  = mu_i(j) + K_i u_{i-1}(j) + k2 om_i(j)
//   Zs = sum_j u_n(j),  ln L = ln Zs - ln c - ln(m+1) + sum_i ln N_i.
// Its adjoint (~ marks dZs/d(variable), scaled by a power of two rho):
//   s~_i(j)  = h_{i+1,j+1} mu~_{i+1}(j+1)
//   u~_i(j)  = X_{i+1} u~_{i+1}(j) + K_{i+1} s~_{i+1}(j)      (u~_n = rho)
//   om~_i(j) = k2 s~_i(j) + x om~_i(j+1)
//   mu~_i(j) = u~_i(j) + s~_i(j) + om~_i(j+1)
// and every folded constant collects (adjoint of its product) x (its operand):
//   per row  pu = sum_j u~ nu,  ps = sum_j s~ nu,  bM = sum_{mismatch} mu~ mu,
//            bH = sum_{match} mu~ mu (two-sided rows only)
//   global   Bk2 = sum s~ om,  Ax = sum om~_i(j+1) om_i(j)
// so that with the log-derivative tables of the constants (GradTables)
//   d ln L = [sum_rows (X pu dlnX + K ps dlnK + bM dlnmiss + bH dlnhit)
//             + k2 Bk2 dlnk2 + Ax dx] / (rho Zs) + sum_rows dlnN.
// Anchored mode differentiates Zs = (mu + A nu + g om)_n(m), the end cell, with
// the virtual row-0 emulator of the forward kernel; the end cell seeds the
// adjoint (mu~ = rho, om~ = rho g, and rho A into u~ of the row above) and A
// and g collect rho A nu and rho g om there.
//
// Layout: one warp per pair, lane L owns R consecutive rows (reads of at
// most 256 bases, one strip), the anti-diagonal sweep of the forward kernel.
// The reverse sweep runs the steps backwards: lane L takes the adjoint of the
// row below from lane L+1 by __shfl_down_sync (u~ at the same column, s~ one
// column to the right, held for a step), the mirror image of the forward.
//
// Memory: the forward values a backward step needs (mu and omega of the
// lane's rows and the u handed in from the row above: 2R+1 values per lane
// and step) are produced by recomputation.  A first forward pass stores the
// warp state every C steps (C = ceil(sqrt(T)) for T = m + 33 steps, "sqrt-L
// anti-diagonal checkpointing"); the reverse sweep replays each segment of C
// steps from its checkpoint once to lay down a state every kSub = 6 steps,
// then replays each 6-step sub-segment into a shared-memory buffer and walks
// it back from there, so the per-step values never leave the SM.  With
// store_all the first pass keeps every step in global memory (one segment of
// T steps).  Both give bit-identical results.
#pragma once
#include "pairhmm_kernel.cuh"

namespace vd {

// Derivatives of the per-quality constants with respect to the offset of the
// quality's bin, in Phred units (0 where the Phred floor at 0 binds).
struct GradTables {
  double dlnN[256];     // d ln N_q / d o
  double dlnmiss[256];  // d ln miss_q / d o
  double dlnhit[256];   // d ln hit_q / d o (two-sided rows)
  int bin[256];         // quality bin of the Phred byte
};

// Derivatives with respect to Qg and Qx, identical for every row.
struct GradScalars {
  double dlnN_g, dlnK_g, dlnX_g, dlnA_g, dlnk2_g, dlng_g;
  double dlnK_x, dlnX_x, dlnk2_x, dx_x;
};

struct GradView {
  const RescueEntry* items;          // (read, hap, out) per pair
  const unsigned long long* count;   // nullable: items to take from a device counter
  long long n_items;
  unsigned long long* head;
  double* out_ln;                    // per output slot
  double* out_jac;                   // per output slot, 6 doubles
  char* scratch;                     // per warp slot: checkpoints and the segment buffer
  long long slot_bytes;
  int store_all;
  int anchored;                      // 0: semiglobal, 1: anchored (global) model
  RescueEntry* spill;                // FP32 pass: pairs left to the FP64 pass
  unsigned long long* spill_count;
  long long spill_cap;
  int* error_flag;                   // bit 0: spill overflow, bit 1: an FP64 pair underflowed
};

// Steps of one pair's wavefront and its checkpoint interval; shared with the
// host, which sizes the scratch from it.
__host__ __device__ inline int grad_steps(int m) { return m + kWarp + 1; }
__host__ __device__ inline int grad_interval(int steps, bool store_all) {
  if (store_all) return steps;
  int c = (int)ceil(sqrt((double)steps));
  return c < 4 ? 4 : c;
}
// Steps of the shared-memory sub-segment buffer (sqrt-L mode): each sqrt(T)
// segment is replayed once to lay down a warp state every kSub steps, then
// sub-segment by sub-segment into shared memory and walked back from there.
constexpr int kSub = 6;
// Shared memory of one warp's sub-segment buffer, sized for R = 8.
template <typename T>
__host__ __device__ constexpr int grad_smem_per_warp() { return kSub * (2 * kMaxR + 1) * kWarp * (int)sizeof(T); }
// Elements of type T one warp slot needs in global memory for a pair with R
// rows per lane: the sqrt(T) checkpoints and the sub-segment states, or every
// step's buffer row when store_all.
__host__ __device__ inline long long grad_slot_elems(int R, int m, bool store_all) {
  const int steps = grad_steps(m);
  const int C = grad_interval(steps, store_all);
  const int nseg = (steps + C - 1) / C;
  if (store_all) return (long long)C * (2 * R + 1) * kWarp;
  return ((long long)nseg + (C + kSub - 1) / kSub) * (3 * R + 2) * kWarp;
}

// The adjoint starts at rho = 2^k on the last row, with rho Zs near 2^kTarget
// (k at most kMax): on the most likely path the forward values fall from c at
// the top row towards Zs and the adjoint falls from rho at the bottom towards
// rho Zs / c, so the products stay near rho Zs and the adjoint keeps the
// exponent range below it for paths away from the most likely one.
template <typename T> struct GradConsts { static constexpr int kTarget = 100, kMax = 120; };
template <> struct GradConsts<double> { static constexpr int kTarget = 600, kMax = 900; };

// Inlined so that x, k2 and the views are constant operands (40 regions: 18.4 ->
// 17.6 ms a call).
template <typename T, int R, bool GEN, bool ANCH>
__device__ __forceinline__ void grad_pair(const BatchView& bv, const GradView& gv, const RescueEntry item,
                                       const Tables<T>* __restrict__ tb, const Scalars<T>& sc,
                                       const GradTables* __restrict__ gt, const GradScalars& gs, const int lane,
                                       T* __restrict__ slot, T* __restrict__ sbuf) {
  constexpr unsigned FULL = 0xffffffffu;
  const int64_t roff = bv.read_off[item.read];
  const int n = (int)(bv.read_off[item.read + 1] - roff);
  const uint8_t* __restrict__ rbase = bv.read_bases + roff;
  const uint8_t* __restrict__ rqual = bv.read_quals + roff;
  const int64_t hoff = bv.hap_off[item.hap];
  const int m = (int)(bv.hap_off[item.hap + 1] - hoff);
  const uint8_t* __restrict__ hap = bv.hap_bases + hoff;
  const int64_t o = item.out;

  const bool store_all = gv.store_all != 0;
  const int steps = grad_steps(m);
  const int C = grad_interval(steps, store_all);
  const int nseg = (steps + C - 1) / C;
  constexpr int CKW = 3 * R + 2;  // checkpoint words per lane
  constexpr int BFW = 2 * R + 1;  // segment-buffer words per lane and step
  T* __restrict__ ck = slot;                                   // sqrt(T) checkpoints
  T* __restrict__ sub = slot + (long long)nseg * CKW * kWarp;   // states every kSub steps of a segment
  T* __restrict__ buf = slot;                                  // store_all: every step

  const T k2 = sc.k2, x = sc.x, c0 = sc.c, gfin = sc.gfin;
  const T A = tb->A[rqual[n - 1]];

  // rows of this lane: the layout of process_item for one strip.  Semiglobal:
  // row i = 32 lane ... with padding rows below the read passing u down.
  // Anchored: the read is bottom-aligned below v = 32 R - n virtual rows, the
  // lowest of them (i = -1) the emulator of row 0, fed s(-1) = c at column 0.
  const int v = ANCH ? kWarp * R - n : 0;
  int emu = -1;
  LaneRows<T, R, GEN> rw;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = lane * R + r - v;
    if (i >= 0 && i < n) {
      const unsigned q = rqual[i];
      rw.rb[r] = rbase[i];
      rw.miss[r] = tb->miss[q];
      if (GEN) rw.hit[r] = tb->hit[q];
      rw.K[r] = tb->K[q];
      rw.X[r] = (!ANCH && i == n - 1) ? A : tb->X[q];
    } else {
      const bool emulator = ANCH && i == -1;
      if (emulator) emu = r;
      rw.rb[r] = kNeverBase;
      rw.miss[r] = emulator ? T(1) : T(0);
      if (GEN) rw.hit[r] = rw.miss[r];
      rw.K[r] = T(0);
      rw.X[r] = (!ANCH && i >= n) ? T(1) : T(0);
    }
    rw.mu[r] = T(0);
    rw.om[r] = T(0);
    rw.s[r] = T(0);
  }
  T s_top = T(0), u_bot = T(0);
  double acc = 0.0;
  // anchored end cell: (M + I + D)[n][m] = mu + A nu + g om of the last row at
  // column m, the running maximum of that sum over the row (the 1e-300 floor of
  // anchored.cpp:24), and its nu and om (the operands of A and g in it)
  T cap = T(0), rmax = T(0), end_nu = T(0), end_om = T(0);

  // one forward step; with rec the lane's column values go to row t - t0 of
  // dst (the global buffer, or this warp's shared sub-segment buffer)
  auto fstep = [&](const int t, const int t0, const bool rec, T* __restrict__ dst) {
    const int j = t - lane;
    T u_in = __shfl_up_sync(FULL, u_bot, 1);
    T s_in = __shfl_up_sync(FULL, rw.s[R - 1], 1);
    if (lane == 0) { u_in = ANCH ? T(0) : c0; s_in = u_in; }
    if (j == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) { rw.mu[r] = T(0); rw.om[r] = T(0); rw.s[r] = T(0); }
      s_top = T(0);
      if (ANCH) {
        if (emu == 0) s_top = c0;
#pragma unroll
        for (int r = 1; r < R; ++r)
          if (emu == r) rw.s[r - 1] = c0;
      }
    }
    const bool act = (unsigned)j <= (unsigned)m;
    const uint32_t hb = (act && j > 0) ? (uint32_t)hap[j - 1] : 0u;
    T tmu = T(0), tnu = T(0), tom = T(0);
    column<T, R, GEN, ANCH>(rw, hb, s_top, u_in, k2, x, u_bot, tmu, tnu, tom);
    s_top = s_in;
    if (rec && act) {
      T* e = dst + (long long)(t - t0) * BFW * kWarp + lane;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        e[r * kWarp] = rw.mu[r];
        e[(R + r) * kWarp] = rw.om[r];
      }
      e[2 * R * kWarp] = u_in;
    }
    if (lane == kWarp - 1 && act) {
      if (ANCH) {
        cap = fmaT(gfin, tom, fmaT(A, tnu, tmu));
        rmax = maxT(rmax, cap);
        if (j == m) { end_nu = tnu; end_om = tom; }
      } else {
        acc += (double)u_bot;
      }
    }
  };
  auto save_state = [&](T* __restrict__ area, const int k) {
    T* e = area + (long long)k * CKW * kWarp + lane;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      e[r * kWarp] = rw.mu[r];
      e[(R + r) * kWarp] = rw.om[r];
      e[(2 * R + r) * kWarp] = rw.s[r];
    }
    e[3 * R * kWarp] = s_top;
    e[(3 * R + 1) * kWarp] = u_bot;
  };
  auto load_state = [&](const T* __restrict__ area, const int k) {
    const T* e = area + (long long)k * CKW * kWarp + lane;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      rw.mu[r] = e[r * kWarp];
      rw.om[r] = e[(R + r) * kWarp];
      rw.s[r] = e[(2 * R + r) * kWarp];
    }
    s_top = e[3 * R * kWarp];
    u_bot = e[(3 * R + 1) * kWarp];
  };

  // ---- first forward pass: Zs, and the checkpoints (or every step) ----
  for (int t = 0; t < steps; ++t) {
    if (!store_all && t % C == 0) save_state(ck, t / C);
    fstep(t, 0, store_all, buf);
  }
  const double Zs = __shfl_sync(FULL, ANCH ? (double)cap : acc, kWarp - 1);
  const double Zmax = __shfl_sync(FULL, (double)rmax, kWarp - 1);
  double lnN = 0.0;
  for (int i = lane; i < n; i += kWarp) lnN += tb->lnN[rqual[i]];
#pragma unroll
  for (int s = 16; s; s >>= 1) lnN += __shfl_xor_sync(FULL, lnN, s);
  const bool ok = Zs >= (double)sc.final_floor && Zs < HUGE_VAL;
  if (!ok) {
    // the FP32 pass hands the pair to the FP64 pass; an FP64 failure is flagged
    if (lane == 0) {
      const double nan = __longlong_as_double(0x7ff8000000000000LL);
      gv.out_ln[o] = nan;
      for (int k = 0; k < 6; ++k) gv.out_jac[o * 6 + k] = nan;
      if (gv.spill != nullptr) {
        const unsigned long long s = atomicAdd(gv.spill_count, 1ull);
        if ((long long)s < gv.spill_cap) gv.spill[s] = item;
        else atomicOr(gv.error_flag, 1);
      } else {
        atomicOr(gv.error_flag, 2);
      }
    }
    __syncwarp();
    return;
  }

  // ---- reverse sweep ----
  const int rho_log2 = min(GradConsts<T>::kMax, GradConsts<T>::kTarget - ilogb(Zs));
  const T rho = pow2T(rho_log2, T(0));
  T ome[R], ups[R], pu[R], ps[R], bM[R], bH[GEN ? R : 1];
#pragma unroll
  for (int r = 0; r < R; ++r) { ome[r] = T(0); ups[r] = T(0); pu[r] = T(0); ps[r] = T(0); bM[r] = T(0); }
#pragma unroll
  for (int r = 0; r < (GEN ? R : 1); ++r) bH[r] = T(0);
  T Bk2 = T(0), Ax = T(0);
  T top_u = T(0), top_s = T(0), pend_s = T(0);

  auto bstep = [&](const int t, const int t0, const T* __restrict__ src) {
    const int j = t - lane;
    const bool act = (unsigned)j <= (unsigned)m;
    T in_u = __shfl_down_sync(FULL, top_u, 1);
    T in_s_next = __shfl_down_sync(FULL, top_s, 1);
    // semiglobal: every (M + I)[n][j] is summed, so u of the bottom row has
    // adjoint rho; anchored: only the end cell counts (seeded below)
    if (lane == kWarp - 1) { in_u = (act && !ANCH) ? rho : T(0); in_s_next = T(0); }
    // anchored end cell at column m: d/dmu = rho, d/dom = rho g, d/dnu = rho A
    const bool seed = ANCH && lane == kWarp - 1 && j == m;
    const T in_s = pend_s;
    pend_s = in_s_next;
    if (!act) {
      top_u = T(0);
      top_s = T(0);
      return;
    }
    const T* e = src + (long long)(t - t0) * BFW * kWarp + lane;
    T muf[R], omf[R], nu[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      muf[r] = e[r * kWarp];
      omf[r] = e[(R + r) * kWarp];
    }
    nu[0] = e[2 * R * kWarp];
#pragma unroll
    for (int r = 1; r < R; ++r) nu[r] = fmaT(rw.X[r - 1], nu[r - 1], muf[r - 1]);
    const uint32_t hb = j > 0 ? (uint32_t)hap[j - 1] : 0u;
    T cu = in_u, cs = in_s;
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
      const T sb = cs, ub = cu;
      const bool sd = seed && r == R - 1;
      const T omb = fmaT(x, ome[r], k2 * sb) + (sd ? rho * gfin : T(0));
      const T mub = ub + sb + ome[r] + (sd ? rho : T(0));
      pu[r] = fmaT(ub, nu[r], pu[r]);
      ps[r] = fmaT(sb, nu[r], ps[r]);
      const bool match = rw.rb[r] == hb;
      T up_s;
      if (GEN) {
        if (match) bH[r] = fmaT(mub, muf[r], bH[r]);
        else bM[r] = fmaT(mub, muf[r], bM[r]);
        up_s = mub * (match ? rw.hit[r] : rw.miss[r]);
      } else {
        bM[r] = fmaT(match ? T(0) : mub, muf[r], bM[r]);
        up_s = match ? mub : mub * rw.miss[r];
      }
      Bk2 = fmaT(sb, omf[r], Bk2);
      Ax = fmaT(ome[r], omf[r], Ax);
      ome[r] = omb;
      cu = fmaT(rw.X[r], ub, rw.K[r] * sb) + (sd ? rho * A : T(0));
      cs = ups[r];
      ups[r] = up_s;
    }
    top_u = cu;
    top_s = ups[0];
  };

  if (store_all) {
    __syncwarp();
    for (int t = steps - 1; t >= 0; --t) bstep(t, 0, buf);
    __syncwarp();
  } else {
    for (int k = nseg - 1; k >= 0; --k) {
      const int t0 = k * C;
      const int t1 = min(steps, t0 + C);
      // lay down a state every kSub steps of the segment, then walk the
      // sub-segments back through shared memory
      load_state(ck, k);
      for (int t = t0; t < t1; ++t) {
        if ((t - t0) % kSub == 0) save_state(sub, (t - t0) / kSub);
        fstep(t, t0, false, buf);
      }
      __syncwarp();
      for (int q = (t1 - t0 - 1) / kSub; q >= 0; --q) {
        const int ta = t0 + q * kSub;
        const int tb = min(t1, ta + kSub);
        load_state(sub, q);
        for (int t = ta; t < tb; ++t) fstep(t, ta, true, sbuf);
        __syncwarp();
        for (int t = tb - 1; t >= ta; --t) bstep(t, ta, sbuf);
        __syncwarp();
      }
    }
  }

  // ---- chain rule to theta (FP64) ----
  const double inv = 1.0 / (ldexp(1.0, rho_log2) * Zs);
  double jg = 0.0, jx = 0.0, jo0 = 0.0, jo1 = 0.0, jo2 = 0.0, jo3 = 0.0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = lane * R + r - v;
    if (i >= 0 && i < n) {
      const unsigned q = rqual[i];
      const bool last = !ANCH && i == n - 1;
      const double bX = (double)rw.X[r] * (double)pu[r];
      const double bK = (double)rw.K[r] * (double)ps[r];
      jg += (bX * (last ? gs.dlnA_g : gs.dlnX_g) + bK * gs.dlnK_g) * inv + gs.dlnN_g;
      jx += (bX * (last ? 0.0 : gs.dlnX_x) + bK * gs.dlnK_x) * inv;
      const double bh = GEN ? (double)bH[r] : 0.0;
      const double d = ((double)bM[r] * gt->dlnmiss[q] + bh * gt->dlnhit[q] - (bX + bK) * gt->dlnN[q]) * inv +
                       gt->dlnN[q];
      const int b = gt->bin[q];
      jo0 += b == 0 ? d : 0.0;
      jo1 += b == 1 ? d : 0.0;
      jo2 += b == 2 ? d : 0.0;
      jo3 += b == 3 ? d : 0.0;
    }
  }
  jg += (double)k2 * (double)Bk2 * gs.dlnk2_g * inv;
  jx += ((double)k2 * (double)Bk2 * gs.dlnk2_x + (double)Ax * gs.dx_x) * inv;
  if (ANCH && lane == kWarp - 1) {
    // the end cell's own constants: A = (g/4) f_n and g (d ln g / dQg = -ln(10)/10)
    const double rho_d = ldexp(1.0, rho_log2);
    const double bA = rho_d * (double)A * (double)end_nu, bg = rho_d * (double)gfin * (double)end_om;
    const unsigned q = rqual[n - 1];
    jg += (bA * gs.dlnA_g + bg * gs.dlng_g) * inv;
    const double d = -bA * gt->dlnN[q] * inv;
    const int b = gt->bin[q];
    jo0 += b == 0 ? d : 0.0;
    jo1 += b == 1 ? d : 0.0;
    jo2 += b == 2 ? d : 0.0;
    jo3 += b == 3 ? d : 0.0;
  }
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    jg += __shfl_xor_sync(FULL, jg, s);
    jx += __shfl_xor_sync(FULL, jx, s);
    jo0 += __shfl_xor_sync(FULL, jo0, s);
    jo1 += __shfl_xor_sync(FULL, jo1, s);
    jo2 += __shfl_xor_sync(FULL, jo2, s);
    jo3 += __shfl_xor_sync(FULL, jo3, s);
  }
  if (lane == 0) {
    const double lnC0 = (double)sc.ln_c + (ANCH ? 0.0 : log((double)(m + 1)));
    // anchored.cpp:24 floors the end cell at 1e-300 of the last row's maximum;
    // the gradient is that of the unfloored value
    const double Zc = ANCH ? fmax(Zs, 1e-300 * Zmax) : Zs;
    gv.out_ln[o] = log(Zc) - lnC0 + lnN;
    double* J = gv.out_jac + o * 6;
    J[0] = jg;
    J[1] = jx;
    J[2] = jo0;
    J[3] = jo1;
    J[4] = jo2;
    J[5] = jo3;
  }
  __syncwarp();
}

// Persistent gradient kernel: warps pull pairs from gv.head.  The FP32 pass
// reads the host-built list; the FP64 pass reads what the FP32 pass spilled.
// Blocks per SM: the FP32 pass fits three (168 registers, 3 x 67 KB of shared
// memory with 6-step buffers), 18% faster than two at 178 registers; the FP64
// pass keeps its registers.
template <typename T> struct GradMinBlocks { static constexpr int value = 3; };
template <> struct GradMinBlocks<double> { static constexpr int value = 1; };

template <typename T, bool ANCH>
__global__ void __launch_bounds__(kWarpsPerBlock * kWarp, GradMinBlocks<T>::value)
pairhmm_grad_kernel(const __grid_constant__ BatchView bv, const __grid_constant__ GradView gv,
                    const Tables<T>* __restrict__ gtab, const __grid_constant__ Scalars<T> sc,
                    const GradTables* __restrict__ gtt, const __grid_constant__ GradScalars gs) {
  __shared__ Tables<T> tab;
  __shared__ GradTables gt;
  {
    const int words = (int)(sizeof(Tables<T>) / sizeof(int));
    const int* src = reinterpret_cast<const int*>(gtab);
    int* dst = reinterpret_cast<int*>(&tab);
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
    const int gwords = (int)(sizeof(GradTables) / sizeof(int));
    const int* gsrc = reinterpret_cast<const int*>(gtt);
    int* gdst = reinterpret_cast<int*>(&gt);
    for (int i = threadIdx.x; i < gwords; i += blockDim.x) gdst[i] = gsrc[i];
  }
  __syncthreads();
  extern __shared__ __align__(16) unsigned char grad_dyn[];
  const int lane = threadIdx.x & (kWarp - 1);
  const long long gw = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  T* slot = reinterpret_cast<T*>(gv.scratch + gw * gv.slot_bytes);
  T* sbuf = reinterpret_cast<T*>(grad_dyn + (threadIdx.x >> 5) * grad_smem_per_warp<T>());
  long long total = gv.n_items;
  if (gv.count != nullptr) {
    const long long c = (long long)*gv.count;
    total = c < total ? c : total;
  }
  for (;;) {
    unsigned long long i = 0;
    if (lane == 0) i = atomicAdd(gv.head, 1ull);
    i = __shfl_sync(0xffffffffu, i, 0);
    if ((long long)i >= total) break;
    const RescueEntry item = gv.items[i];
    const int code = bv.read_code[item.read];
    const bool gen = code_general(code);
#define VD_GCASE(r)                                                                          \
  case r:                                                                                    \
    if (gen) grad_pair<T, r, true, ANCH>(bv, gv, item, &tab, sc, &gt, gs, lane, slot, sbuf); \
    else grad_pair<T, r, false, ANCH>(bv, gv, item, &tab, sc, &gt, gs, lane, slot, sbuf);    \
    break;
    switch (code_R(code)) {
      VD_GCASE(1) VD_GCASE(2) VD_GCASE(3) VD_GCASE(4) VD_GCASE(5) VD_GCASE(6) VD_GCASE(7) VD_GCASE(8)
      default: break;
    }
#undef VD_GCASE
  }
}


// ---- two pairs per warp (FP32, semiglobal, one-sided emission, sqrt-L) ----------
// Two pairs with the same rows per lane go through grad_pair's passes together,
// packed as float2 (x: first pair, y: second): one issue slot serves both in the
// FMAs, and the shuffles, the buffer accesses and the step's bookkeeping are
// shared.  Every element goes through grad_pair's operations in grad_pair's
// order, so a pair's result is the same bits on either kernel (and under
// VD_CHECKPOINT_ALL, which runs there).  The rows keep W = om of the next column
// in place of mu and om, as the forward's two-read kernels do.  A half whose
// haplotype is the shorter one sees only zeros from below past its end, which add
// nothing to its sums.  What bounds it: FMA issue and the vertical chains at 8 to
// 12 warps per SM (24 registers a row).  40 regions, 3.9e9 cells: 14.7 -> 9.4 ms;
// 4,000 pairs of 100 / 150 / 250 bases x 400: 1.08 / 1.20 / 1.42 -> 0.62 / 0.69 / 1.10 ms.
template <int R, int SUB>
__device__ __forceinline__ void grad_pair2(const BatchView& bv, const GradView& gv, const RescueEntry ia,
                                           const RescueEntry ib, const Tables<float>* __restrict__ tb,
                                           const Scalars<float>& sc, const GradTables* __restrict__ gt,
                                           const GradScalars& gs, const int lane, float* __restrict__ slot,
                                           float2* __restrict__ sbuf) {
  constexpr unsigned FULL = 0xffffffffu;
  const int64_t roa = bv.read_off[ia.read], rob = bv.read_off[ib.read];
  const int na = (int)(bv.read_off[ia.read + 1] - roa), nb = (int)(bv.read_off[ib.read + 1] - rob);
  const uint8_t* __restrict__ qa = bv.read_quals + roa;
  const uint8_t* __restrict__ qb = bv.read_quals + rob;
  const int64_t hoa = bv.hap_off[ia.hap], hob = bv.hap_off[ib.hap];
  const int ma = (int)(bv.hap_off[ia.hap + 1] - hoa), mb = (int)(bv.hap_off[ib.hap + 1] - hob);
  const uint8_t* __restrict__ ha = bv.hap_bases + hoa - 1;  // ha[j] = base of column j >= 1
  const uint8_t* __restrict__ hb = bv.hap_bases + hob - 1;
  const int M = max(ma, mb);
  const int steps = grad_steps(M);
  const int C = grad_interval(steps, false);
  const int nseg = (steps + C - 1) / C;
  // a sub-segment's steps are unrolled for the fewest rows only (at 8 rows that
  // spills 2.8 KB: 4,000 pairs of 250 bases 1.10 -> 1.78 ms; at 1 row 0.33 -> 0.29)
  constexpr int kUnrollSub = R <= 2 ? SUB : 1, kUnrollRun = 4;
  constexpr int CKW = 2 * R + 2;  // checkpoint words (float2) per lane
  constexpr int BFW = 2 * R + 1;  // buffer words (float2) per lane and step
  float2* __restrict__ ck = reinterpret_cast<float2*>(slot);
  float2* __restrict__ sub = ck + (long long)nseg * CKW * kWarp;

  const float2 k2 = make_float2(sc.k2, sc.k2), x = make_float2(sc.x, sc.x), c2 = make_float2(sc.c, sc.c);
  const bool lane0 = lane == 0, lane31 = lane == kWarp - 1;
  PairRows<R> rw;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = lane * R + r;
    const unsigned q0 = i < na ? qa[i] : 0u, q1 = i < nb ? qb[i] : 0u;
    rw.ra[r] = i < na ? (uint32_t)bv.read_bases[roa + i] : kNeverBase;
    rw.rb[r] = i < nb ? (uint32_t)bv.read_bases[rob + i] : kNeverBase;
    rw.miss[r] = make_float2(i < na ? tb->miss[q0] : 0.f, i < nb ? tb->miss[q1] : 0.f);
    rw.K[r] = make_float2(i < na ? tb->K[q0] : 0.f, i < nb ? tb->K[q1] : 0.f);
    rw.X[r] = make_float2(i < na ? (i == na - 1 ? tb->A[q0] : tb->X[q0]) : 1.f,
                          i < nb ? (i == nb - 1 ? tb->A[q1] : tb->X[q1]) : 1.f);
    rw.W[r] = make_float2(0.f, 0.f);
    rw.s[r] = make_float2(0.f, 0.f);
  }
  float2 s_top = make_float2(0.f, 0.f), u_bot = make_float2(0.f, 0.f);
  double acc_a = 0.0, acc_b = 0.0;

  // one forward step; INNER: every lane at a column in 1 .. min(ma, mb); REC: the
  // lane's column values go to e (mu, om per row, u handed in); SUM: lane 31 sums its
  // bottom row
  auto fstep = [&](auto inner_tag, auto rec_tag, auto sum_tag, const int t, float2* __restrict__ e) {
    constexpr bool INNER = decltype(inner_tag)::value, REC = decltype(rec_tag)::value;
    const int j = t - lane;
    uint32_t b0, b1;
    if (INNER) {
      b0 = __ldg(ha + j);
      b1 = __ldg(hb + j);
    } else {
      b0 = j > 0 && j <= ma ? (uint32_t)__ldg(ha + j) : 0u;
      b1 = j > 0 && j <= mb ? (uint32_t)__ldg(hb + j) : 0u;
    }
    float2 u_in = shfl_up2(u_bot);
    float2 s_in = shfl_up2(rw.s[R - 1]);
    u_in = lane0 ? c2 : u_in;
    s_in = lane0 ? c2 : s_in;
    if (!INNER && j == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        rw.W[r] = make_float2(0.f, 0.f);
        rw.s[r] = make_float2(0.f, 0.f);
      }
      s_top = make_float2(0.f, 0.f);
    }
    const bool rec = REC && (INNER || (unsigned)j <= (unsigned)M);
    float2 s_above = s_top, nu = u_in;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float2 mu = s_above;
      mul_if_ne(mu.x, rw.ra[r], b0, rw.miss[r].x);
      mul_if_ne(mu.y, rw.rb[r], b1, rw.miss[r].y);
      const float2 om = rw.W[r];
      if (rec) {
        e[r * kWarp] = mu;
        e[(R + r) * kWarp] = om;
      }
      const float2 un = __ffma2_rn(rw.X[r], nu, mu);
      const float2 sn = __ffma2_rn(k2, om, __ffma2_rn(rw.K[r], nu, mu));
      s_above = rw.s[r];
      rw.W[r] = __ffma2_rn(x, om, mu);
      rw.s[r] = sn;
      nu = un;
    }
    if (rec) e[2 * R * kWarp] = u_in;
    u_bot = nu;
    s_top = s_in;
    if (decltype(sum_tag)::value && (INNER || (lane31 && j >= 0))) {
      if (INNER || j <= ma) acc_a += (double)u_bot.x;
      if (INNER || j <= mb) acc_b += (double)u_bot.y;
    }
  };
  // forward steps [ta, tz) without a record
  auto run = [&](auto sum_tag, const int ta, const int tz) {
    int t = ta;
    for (; t < tz && t < kWarp; ++t) fstep(std::false_type{}, std::false_type{}, sum_tag, t, nullptr);
    const int ti = min(tz, min(ma, mb) + 1);
#pragma unroll kUnrollRun
    for (; t < ti; ++t) fstep(std::true_type{}, std::false_type{}, sum_tag, t, nullptr);
    for (; t < tz; ++t) fstep(std::false_type{}, std::false_type{}, sum_tag, t, nullptr);
  };
  auto save_state = [&](float2* __restrict__ area, const int k) {
    float2* e = area + (long long)k * CKW * kWarp + lane;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      e[r * kWarp] = rw.W[r];
      e[(R + r) * kWarp] = rw.s[r];
    }
    e[2 * R * kWarp] = s_top;
    e[(2 * R + 1) * kWarp] = u_bot;
  };
  auto load_state = [&](const float2* __restrict__ area, const int k) {
    const float2* e = area + (long long)k * CKW * kWarp + lane;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      rw.W[r] = e[r * kWarp];
      rw.s[r] = e[(R + r) * kWarp];
    }
    s_top = e[2 * R * kWarp];
    u_bot = e[(2 * R + 1) * kWarp];
  };

  // ---- first forward pass ----
  for (int k = 0; k < nseg; ++k) {
    save_state(ck, k);
    const int t1 = min(steps, (k + 1) * C);
    run(std::true_type{}, k * C, t1);
  }
  const double Za = __shfl_sync(FULL, acc_a, kWarp - 1), Zb = __shfl_sync(FULL, acc_b, kWarp - 1);
  double lna = 0.0, lnb = 0.0;
  for (int i = lane; i < na; i += kWarp) lna += tb->lnN[qa[i]];
  for (int i = lane; i < nb; i += kWarp) lnb += tb->lnN[qb[i]];
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    lna += __shfl_xor_sync(FULL, lna, s);
    lnb += __shfl_xor_sync(FULL, lnb, s);
  }
  const bool oka = Za >= (double)sc.final_floor && Za < HUGE_VAL, okb = Zb >= (double)sc.final_floor && Zb < HUGE_VAL;
  // a half that left the FP32 range goes to the FP64 pass
  auto hand_on = [&](const RescueEntry& item) {
    if (lane == 0) {
      const double nan = __longlong_as_double(0x7ff8000000000000LL);
      gv.out_ln[item.out] = nan;
      for (int k = 0; k < 6; ++k) gv.out_jac[item.out * 6 + k] = nan;
      const unsigned long long s = atomicAdd(gv.spill_count, 1ull);
      if ((long long)s < gv.spill_cap) gv.spill[s] = item;
      else atomicOr(gv.error_flag, 1);
    }
  };
  if (!oka) hand_on(ia);
  if (!okb && ib.out >= 0) hand_on(ib);
  __syncwarp();
  if (!oka && !okb) return;

  // ---- reverse sweep ----
  auto rho_exp = [&](double Z, bool ok) {
    return ok ? min(GradConsts<float>::kMax, GradConsts<float>::kTarget - ilogb(Z)) : -126;
  };
  const int ra2 = rho_exp(Za, oka), rb2 = rho_exp(Zb, okb);
  // (a half handed on runs along from 0: nothing of it is used)
  const float2 rho = make_float2(oka ? pow2T(ra2, 0.f) : 0.f, okb ? pow2T(rb2, 0.f) : 0.f);
  float2 ome[R], ups[R], pu[R], ps[R], bM[R];
  const float2 zero = make_float2(0.f, 0.f);
#pragma unroll
  for (int r = 0; r < R; ++r) ome[r] = ups[r] = pu[r] = ps[r] = bM[r] = zero;
  float2 Bk2 = zero, Ax = zero, top_u = zero, top_s = zero, pend_s = zero;

  auto bstep = [&](auto inner_tag, const int t, const float2* __restrict__ e) {
    constexpr bool INNER = decltype(inner_tag)::value;
    const int j = t - lane;
    float2 in_u = make_float2(__shfl_down_sync(FULL, top_u.x, 1), __shfl_down_sync(FULL, top_u.y, 1));
    float2 in_s_next = make_float2(__shfl_down_sync(FULL, top_s.x, 1), __shfl_down_sync(FULL, top_s.y, 1));
    if (lane31) {
      in_u = make_float2(INNER || (unsigned)j <= (unsigned)ma ? rho.x : 0.f,
                         INNER || (unsigned)j <= (unsigned)mb ? rho.y : 0.f);
      in_s_next = zero;
    }
    const float2 in_s = pend_s;
    pend_s = in_s_next;
    uint32_t b0, b1;
    if (INNER) {
      b0 = __ldg(ha + j);
      b1 = __ldg(hb + j);
    } else {
      if ((unsigned)j > (unsigned)M) {
        top_u = zero;
        top_s = zero;
        return;
      }
      b0 = j > 0 && j <= ma ? (uint32_t)__ldg(ha + j) : 0u;
      b1 = j > 0 && j <= mb ? (uint32_t)__ldg(hb + j) : 0u;
    }
    float2 muf[R], nu[R];
#pragma unroll
    for (int r = 0; r < R; ++r) muf[r] = e[r * kWarp];
    nu[0] = e[2 * R * kWarp];
#pragma unroll
    for (int r = 1; r < R; ++r) nu[r] = __ffma2_rn(rw.X[r - 1], nu[r - 1], muf[r - 1]);
    float2 cu = in_u, cs = in_s;
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
      const float2 sb = cs, ub = cu;
      const float2 omf = e[(R + r) * kWarp];
      const float2 omb = __ffma2_rn(x, ome[r], __fmul2_rn(k2, sb));
      const float2 mub = __fadd2_rn(__fadd2_rn(ub, sb), ome[r]);
      pu[r] = __ffma2_rn(ub, nu[r], pu[r]);
      ps[r] = __ffma2_rn(sb, nu[r], ps[r]);
      // (a matching cell adds nothing to bM and keeps mub)
      float2 up = mub;
      if (rw.ra[r] != b0) { bM[r].x = __fmaf_rn(mub.x, muf[r].x, bM[r].x); up.x = mub.x * rw.miss[r].x; }
      if (rw.rb[r] != b1) { bM[r].y = __fmaf_rn(mub.y, muf[r].y, bM[r].y); up.y = mub.y * rw.miss[r].y; }
      Bk2 = __ffma2_rn(sb, omf, Bk2);
      Ax = __ffma2_rn(ome[r], omf, Ax);
      ome[r] = omb;
      cu = __ffma2_rn(rw.X[r], ub, __fmul2_rn(rw.K[r], sb));
      cs = ups[r];
      ups[r] = up;
    }
    top_u = cu;
    top_s = ups[0];
  };

  for (int k = nseg - 1; k >= 0; --k) {
    const int t0 = k * C;
    const int t1 = min(steps, t0 + C);
    load_state(ck, k);
    const int nsub = (t1 - t0 + SUB - 1) / SUB;
    for (int q = 0; q + 1 < nsub; ++q) {
      save_state(sub, q);
      run(std::false_type{}, t0 + q * SUB, t0 + (q + 1) * SUB);
    }
    for (int q = nsub - 1; q >= 0; --q) {
      const int ta = t0 + q * SUB;
      const int tz = min(t1, ta + SUB);
      if (q + 1 != nsub) load_state(sub, q);  // (the last one's state is at hand)
      // each lane reads back what it wrote itself
      if (tz - ta == SUB && ta >= kWarp && tz - 1 <= min(ma, mb)) {
#pragma unroll kUnrollSub
        for (int u = 0; u < SUB; ++u)
          fstep(std::true_type{}, std::true_type{}, std::false_type{}, ta + u, sbuf + u * BFW * kWarp + lane);
#pragma unroll kUnrollSub
        for (int u = SUB - 1; u >= 0; --u) bstep(std::true_type{}, ta + u, sbuf + u * BFW * kWarp + lane);
      } else {
        for (int t = ta; t < tz; ++t)
          fstep(std::false_type{}, std::true_type{}, std::false_type{}, t, sbuf + (t - ta) * BFW * kWarp + lane);
        for (int t = tz - 1; t >= ta; --t) bstep(std::false_type{}, t, sbuf + (t - ta) * BFW * kWarp + lane);
      }
    }
  }

  // ---- chain rule to theta (FP64), as in grad_pair ----
  auto finish = [&](const RescueEntry& item, int n, int m, const uint8_t* rq, double Z, int rho_log2, double lnN,
                    auto half) {
    const double inv = 1.0 / (ldexp(1.0, rho_log2) * Z);
    double jg = 0.0, jx = 0.0, jo0 = 0.0, jo1 = 0.0, jo2 = 0.0, jo3 = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = lane * R + r;
      if (i < n) {
        const unsigned q = rq[i];
        const bool last = i == n - 1;
        const double bX = (double)half(rw.X[r]) * (double)half(pu[r]);
        const double bK = (double)half(rw.K[r]) * (double)half(ps[r]);
        jg += (bX * (last ? gs.dlnA_g : gs.dlnX_g) + bK * gs.dlnK_g) * inv + gs.dlnN_g;
        jx += (bX * (last ? 0.0 : gs.dlnX_x) + bK * gs.dlnK_x) * inv;
        const double d = ((double)half(bM[r]) * gt->dlnmiss[q] + 0.0 * gt->dlnhit[q] - (bX + bK) * gt->dlnN[q]) * inv +
                         gt->dlnN[q];
        const int b = gt->bin[q];
        jo0 += b == 0 ? d : 0.0;
        jo1 += b == 1 ? d : 0.0;
        jo2 += b == 2 ? d : 0.0;
        jo3 += b == 3 ? d : 0.0;
      }
    }
    jg += (double)half(k2) * (double)half(Bk2) * gs.dlnk2_g * inv;
    jx += ((double)half(k2) * (double)half(Bk2) * gs.dlnk2_x + (double)half(Ax) * gs.dx_x) * inv;
#pragma unroll
    for (int s = 16; s; s >>= 1) {
      jg += __shfl_xor_sync(FULL, jg, s);
      jx += __shfl_xor_sync(FULL, jx, s);
      jo0 += __shfl_xor_sync(FULL, jo0, s);
      jo1 += __shfl_xor_sync(FULL, jo1, s);
      jo2 += __shfl_xor_sync(FULL, jo2, s);
      jo3 += __shfl_xor_sync(FULL, jo3, s);
    }
    if (lane == 0) {
      gv.out_ln[item.out] = log(Z) - ((double)sc.ln_c + log((double)(m + 1))) + lnN;
      double* J = gv.out_jac + item.out * 6;
      J[0] = jg;
      J[1] = jx;
      J[2] = jo0;
      J[3] = jo1;
      J[4] = jo2;
      J[5] = jo3;
    }
  };
  if (oka) finish(ia, na, ma, qa, Za, ra2, lna, [](const float2 v) { return v.x; });
  if (okb && ib.out >= 0) finish(ib, nb, mb, qb, Zb, rb2, lnb, [](const float2 v) { return v.y; });
  __syncwarp();
}

// Shared memory of one warp's sub-segment buffer.
constexpr int grad_pair_smem_per_warp(int max_R, int sub) { return sub * (2 * max_R + 1) * kWarp * (int)sizeof(float2); }

// Persistent kernel of the two-pair items: entries 2i and 2i + 1 of the list are
// one item (the second may be a filler, out = -1).  Rows take 24 registers each:
// 5-8 of them run 2 blocks per SM, up to 4 run 3.
template <int kLoR, int kHiR, int kSteps, int kBlocks>
__global__ void __launch_bounds__(kWarpsPerBlock * kWarp, kBlocks)
pairhmm_grad_pair_kernel(const __grid_constant__ BatchView bv, const __grid_constant__ GradView gv,
                         const Tables<float>* __restrict__ gtab, const __grid_constant__ Scalars<float> sc,
                         const GradTables* __restrict__ gtt, const __grid_constant__ GradScalars gs) {
  __shared__ Tables<float> tab;
  __shared__ GradTables gt;
  {
    const int words = (int)(sizeof(Tables<float>) / sizeof(int));
    const int* src = reinterpret_cast<const int*>(gtab);
    int* dst = reinterpret_cast<int*>(&tab);
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
    const int gwords = (int)(sizeof(GradTables) / sizeof(int));
    const int* gsrc = reinterpret_cast<const int*>(gtt);
    int* gdst = reinterpret_cast<int*>(&gt);
    for (int i = threadIdx.x; i < gwords; i += blockDim.x) gdst[i] = gsrc[i];
  }
  __syncthreads();
  extern __shared__ __align__(16) unsigned char grad_pair_dyn[];
  const int lane = threadIdx.x & (kWarp - 1);
  const long long gw = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  float* slot = reinterpret_cast<float*>(gv.scratch + gw * gv.slot_bytes);
  float2* sbuf = reinterpret_cast<float2*>(grad_pair_dyn + (threadIdx.x >> 5) * grad_pair_smem_per_warp(kHiR, kSteps));
  for (;;) {
    unsigned long long i = 0;
    if (lane == 0) i = atomicAdd(gv.head, 1ull);
    i = __shfl_sync(0xffffffffu, i, 0);
    if ((long long)i >= gv.n_items) break;
    const RescueEntry ia = gv.items[2 * i], ib = gv.items[2 * i + 1];
    switch (code_R(bv.read_code[ia.read])) {
#define VD_GPCASE(r)                                                                                           \
  case r:                                                                                                      \
    if constexpr (r >= kLoR && r <= kHiR) grad_pair2<r, kSteps>(bv, gv, ia, ib, &tab, sc, &gt, gs, lane, slot, sbuf); \
    break;
      VD_GPCASE(1) VD_GPCASE(2) VD_GPCASE(3) VD_GPCASE(4) VD_GPCASE(5) VD_GPCASE(6) VD_GPCASE(7) VD_GPCASE(8)
#undef VD_GPCASE
      default: break;
    }
  }
}

}  // namespace vd
