// kernels_sweep.cu -- the constant-pH Monte Carlo sweep on the device.
//
// Reference: soup/src/electrostatics.ts:435-496 protonationSweep (CPU, sequential, FP64 JavaScript
// numbers), electrostatics.ts:277-281 esPairEnergy, soup/src/acid-soap.ts:147-198 (acidSoapWell,
// acidSoapSiteWork), electrostatics.ts:308-315 pcgNext.
//
// The attempt chain is sequential: attempt a+1's site draw depends on whether attempt a took an
// acceptance draw, which depends on its free energy.  The energy itself is not sequential: the
// reference recomputes, per attempt, E_s = kT ln10 (pKa - pH) + the screened Coulomb work + the
// acid-soap pair work over the site's neighbours, and E_s depends on the neighbours' charges only.
// Positions are fixed during a sweep, so the change of E_t when neighbour s flips is a fixed number
// per pair.  So:
//   k_sweep_init  (all SMs, a warp per head) evaluates E_h in FP64 from the head list, and for every
//                 list entry t of h the change D_ht of E_t when h deprotonates (-D_ht when it
//                 protonates).
//   k_sweep_draws, k_sweep_pairs (all SMs) precompute every draw's site and, for the pairs of draws of one
//                 block whose sites are near one another, the change of the later draw's site energy when
//                 the earlier flips.
//   k_sweep_walk  (a group of CTAs per replica) resolves the chain a block of 512 or 256 draws at a time, a
//                 thread per draw on the group's first CTA: every draw decides from its site energy, a scan
//                 over the draws finds which of them are attempts (an attempt that needs an acceptance draw
//                 uses up the next one), the flips found change the later draws' energies, and the draws
//                 decide again until the flips stand.  The decisions up to any draw depend on the earlier
//                 ones alone, so what stands is the sequential chain's result, and draw d stands after at
//                 most d rounds (3 rounds a block at 18,659 heads, 4 to 5 where the cutoff spans the box).
//                 Then the other CTAs add the block's flips to E from the D rows.
//   What bounds the walk: latency.  One warp that resolved windows of 32 draws took 4.1 ms a sweep at 18,659
//   heads (1,075 windows of handoffs and dependent loads); blocks of 512 take 0.76 ms, some 22k cycles for each of
//   66.  By clock stamps (which add a tenth): 3 rounds of 3.5k to decide and scan, 2 pulls of 1.5k, 1.7k to commit, and
//   7.5k until the other CTAs have added the flips: 3k for the adds, 4k to 5k for the handoff there and back.
// E and D are fixed point (2^-40 kT, int64): integer adds commute, so E does not depend on the
// order the updates land in and every run is reproducible.  E_h is the FP64 sum rounded once, each
// D_ht is rounded once, so the energies agree with the reference's FP64 sums to about 1e-11 kT (the
// decisions agree unless a draw lands that close to its threshold).
// The energies are FP64 with JavaScript rounding of the minimum image, as the reference's.
#include "soup_internal.h"


namespace soup {

namespace {

__device__ __forceinline__ double es_energy(const SysParams& P, double r, double qq) {
  if (P.d_A == 0.0 || qq == 0.0 || r >= P.d_rc || r <= 0.0) return 0.0;
  const double u1 = (P.d_A * exp(-P.d_kappa * r)) / r;
  return qq * (u1 - P.d_shiftU + P.d_shiftF * (r - P.d_rc));
}
__device__ __forceinline__ double acid_well(const SysParams& P, double r) {
  if (P.d_acid <= 0.0) return 0.0;
  if (r < P.d_rcattr) return -P.d_acid * P.d_eps;
  if (r > P.d_rcattr + P.d_wc) return 0.0;
  const double c = cos((3.141592653589793 * (r - P.d_rcattr)) / (2.0 * P.d_wc));
  return -P.d_acid * P.d_eps * c * c;
}
// squared minimum-image distance, FP64.  The reference's image index is Math.round(d / L).  While the cutoffs end short
// of half the box, FP32 finds it: it can differ only near a half-box offset, where every pair is beyond them either
// way.  A live box that has shrunk further (SysParams.image64; I64: some replica's has) takes the index from
// d * (1 / L) in FP64, within an ulp of d / L.  With FP64 for all, a sweep at 18,659 heads takes 4% longer; with the
// question asked in every kernel, 1%.
template <bool I64>
__device__ __forceinline__ double image(float a, float b, bool in64, float inv, double inv64, double L) {
  const double d = (double)a - (double)b;
  if (!I64 || !in64) {
    const float n = rintf((a - b) * inv);
    return n == 0.f ? d : d - (double)n * L;
  }
  const double x = d * inv64, r = floor(x);
  return d - (x - r >= 0.5 ? r + 1.0 : r) * L;
}
template <bool I64>
__device__ __forceinline__ double dist2(const SysParams& P, const float4& a, const float4& b) {
  const bool in64 = I64 && P.image64 != 0;
  const double dx = image<I64>(a.x, b.x, in64, P.inv_box[0], P.d_inv_box[0], P.d_box[0]),
               dy = image<I64>(a.y, b.y, in64, P.inv_box[1], P.d_inv_box[1], P.d_box[1]),
               dz = image<I64>(a.z, b.z, in64, P.inv_box[2], P.d_inv_box[2], P.d_box[2]);
  return dx * dx + dy * dy + dz * dz;
}
// the energy a neighbour of charge qj at squared distance r2 contributes to a site's E
__device__ __forceinline__ double site_term(const SysParams& P, double r2, float qj, double cut2, double reach2) {
  double e = 0.0;
  if (qj != 0.f && r2 < cut2) e += es_energy(P, sqrt(r2), P.d_q * (double)qj);
  if (P.d_acid > 0.0 && r2 < reach2 && r2 > 0.0) {
    const double v = acid_well(P, sqrt(r2));
    e += (qj == 0.f) ? v : -v;
  }
  return e;
}

constexpr double kFix = 1099511627776.0;            // 2^40 fixed-point units per kT
constexpr double kUnfix = 1.0 / 1099511627776.0;
__device__ __forceinline__ long long to_fix(double x) { return __double2ll_rn(x * kFix); }
// change of a neighbour's E when a site at squared distance r2 goes from charge qo to qn
// (round-to-nearest-even is odd-symmetric, so the reverse flip gives exactly the negative)
__device__ __forceinline__ long long flip_delta(const SysParams& P, double r2, float qo, float qn, double cut2,
                                                double reach2) {
  return to_fix(site_term(P, r2, qn, cut2, reach2) - site_term(P, r2, qo, cut2, reach2));
}
// flip_delta(r2, 0, qd) with one square root (the same operations in the same order, so the same
// bits); the value of every D entry and of every in-window correction
__device__ __forceinline__ long long std_delta(const SysParams& P, double r2, float qd, double cut2, double reach2) {
  double t1 = 0.0, t0 = 0.0;
  const bool es_in = qd != 0.f && r2 < cut2;
  const bool ac_in = P.d_acid > 0.0 && r2 < reach2 && r2 > 0.0;
  if (es_in || ac_in) {
    const double rr = sqrt(r2);
    if (es_in) t1 += es_energy(P, rr, P.d_q * (double)qd);
    if (ac_in) {
      const double v = acid_well(P, rr);
      t1 += -v;
      t0 += v;
    }
  }
  return to_fix(t1 - t0);
}

// FP32 screen of pairs beyond both cutoffs, which change nothing: the squared range with a wide margin
__device__ __forceinline__ float near2(const SysParams& P) {
  const float nr = (float)(fmax(P.d_rc, P.d_rcattr + P.d_wc) * 1.001 + 1e-3);
  return nr * nr;
}
__device__ __forceinline__ float fast_r2(const SysParams& P, const float4& a, const float4& b) {
  float dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
  dx -= rintf(dx * P.inv_box[0]) * P.box[0];
  dy -= rintf(dy * P.inv_box[1]) * P.box[1];
  dz -= rintf(dz * P.inv_box[2]) * P.box[2];
  return dx * dx + dy * dy + dz * dz;
}

// E_h = kT ln10 (pKa - pH) + uEs(h) and the row D_h, a warp per head over the heads' gathered records.  The
// screened energy per unit charge product and the well are evaluated once per pair, for E and for D (the
// same operations in the same order as es_energy / std_delta, so the same bits).  Entries beyond both
// cutoffs (the list's skin) are told by an FP32 distance with a wide margin.  Bound: FP64 issue.
template <bool I64>
__global__ void __launch_bounds__(256) k_sweep_init(const SysParams* __restrict__ sp, const uint32_t* __restrict__ head_sys,
                                                    uint32_t H, const float4* __restrict__ xq,
                                                    const uint32_t* __restrict__ es_nl, const uint32_t* __restrict__ es_cnt,
                                                    uint32_t cap, long long* __restrict__ E, long long* __restrict__ D,
                                                    uint32_t only) {
  const uint32_t h = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (h >= H) return;
  const uint32_t r = head_sys[h];
  if (only != SOUP_NONE_U32 && r != only) return;
  const SysParams& P = sp[r];
  if (!P.es_on) return;
  const double cut2 = P.d_rc * P.d_rc, reach = P.d_rcattr + P.d_wc, reach2 = reach * reach;
  const float screen2 = near2(P);
  const float qd = (float)P.d_q;
  const double qqd = P.d_q * (double)qd;
  const float4 xi = xq[h];
  double es = 0.0, w = 0.0;
  const uint32_t cnt = es_cnt[h];
  const uint32_t* row = es_nl + (size_t)h * cap;
  long long* drow = D + (size_t)h * cap;
  for (uint32_t s = lane; s < cnt; s += 32) {
    const float4 xj = xq[row[s]];
    long long d = 0;
    if (fast_r2(P, xi, xj) < screen2) {
      const float qj = xj.w;
      const double r2 = dist2<I64>(P, xi, xj);
      const bool es_in = r2 < cut2, ac_in = P.d_acid > 0.0 && r2 < reach2 && r2 > 0.0;
      double t1 = 0.0, t0 = 0.0;
      if (es_in || ac_in) {
        const double rr = sqrt(r2);
        if (es_in && P.d_A != 0.0 && rr < P.d_rc && rr > 0.0) {
          const double u1 = (P.d_A * exp(-P.d_kappa * rr)) / rr;
          const double u = u1 - P.d_shiftU + P.d_shiftF * (rr - P.d_rc);
          const double qq = P.d_q * (double)qj;
          if (qq != 0.0) es += qq * u;
          if (qqd != 0.0) t1 += qqd * u;
        }
        if (ac_in) {
          const double v = acid_well(P, rr);
          w += (qj == 0.f) ? v : -v;
          t1 += -v;
          t0 += v;
        }
      }
      d = to_fix(t1 - t0);
    }
    drow[s] = d;
  }
  for (int o = 16; o > 0; o >>= 1) {
    es += __shfl_xor_sync(0xffffffffu, es, o);
    w += __shfl_xor_sync(0xffffffffu, w, o);
  }
  if (lane == 0) E[h] = to_fix(P.d_kT * 2.302585092994046 * (P.d_pka - P.d_ph) + (es + w));
}

// u < exp(-dG/kT) for dG > 0, with dG = g 2^-40 (g the fixed-point energy, g > 0) and u = v 2^-32 (v the
// draw's 32 output bits).  The walk's chain takes this decision once per attempt and again whenever
// an earlier flip of its window changes the site's energy, so the common case runs in FP32 and
// integers: for -dG/kT > -20 an FP32 estimate decides when u is more than 2e-5 (relative) away from
// it.  The estimate's error is below 6.8e-6: the exponent -g * (2^-40 / kT) carries three FP32
// roundings (1.8e-7 relative, 3.6e-6 absolute at |x| < 20), __expf adds at most 2 + 1.173 |x| ulp
// (3.0e-6), the draw's and the margin's roundings 2e-7.  Below -20 only u < 1e-8 can pass (v < 43).
// Otherwise, and near the threshold, FP64 decides: exp(-dG / kT) with dG and u exactly as the
// reference forms them.
__device__ __forceinline__ bool metropolis(long long g, uint32_t v, float x_scale, double kT) {
  const float xf = -(float)g * x_scale;
  if (xf > -20.f) {
    const float est = __expf(xf);
    const float u = (float)v * 2.3283064365386963e-10f;
    if (u < est * (1.f - 2e-5f)) return true;
    if (u > est * (1.f + 2e-5f)) return false;
  } else if (v >= 43u) {
    return false;                 // u >= 1.0012e-8 > exp(-20 + 4e-6)
  }
  return (double)v * 2.3283064365386963e-10 < exp(-((double)g * kUnfix) / kT);
}

// the pcgNext LCG (state' = a state + c mod 2^32) advanced n steps at once
struct Lcg { uint32_t a, c; };
__device__ __forceinline__ Lcg lcg_pow(uint32_t n) {
  Lcg acc{1u, 0u}, b{747796405u, 2891336453u};
  while (n) {
    if (n & 1u) acc = Lcg{acc.a * b.a, acc.c * b.a + b.c};
    b = Lcg{b.a * b.a, b.c * b.a + b.c};
    n >>= 1;
  }
  return acc;
}
// pcgNext's output bits; the draw is u = bits / 2^32
__device__ __forceinline__ uint32_t pcg_bits(uint32_t v) {
  v = ((v >> ((v >> 28u) + 4u)) ^ v) * 277803737u;
  return (v >> 22u) ^ v;
}

constexpr int kWalkThreads = 512;
constexpr uint32_t kDraws = kWalkThreads;       // draws of a block, at most (SysParams.sweep_draws: 512 or 256)
constexpr uint32_t kWalkWarps = kWalkThreads / 32;
constexpr uint32_t kEndOfSweep = 0xFFFFFFFFu;   // s_cflag once the sweep is over
constexpr uint32_t kSpinLimit = 1u << 25;       // default polls of a handoff flag before the walk gives up
constexpr uint32_t kMaxHeads = 196592;          // heads of one replica: their charge states fill CTA 0's shared memory

// device-scope release / acquire on 32-bit words: the handoffs between the CTAs of a walk
__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(uint32_t* p, uint32_t v) {
  asm volatile("st.release.gpu.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_add_release_gpu(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// whole blocks for the 2 H draws a sweep consumes at most (an attempt takes a site draw and at most one acceptance draw)
__host__ __device__ __forceinline__ uint32_t blocks_of(uint32_t heads, uint32_t W) { return (2 * heads + W - 1) / W; }
__device__ __forceinline__ uint32_t draw_blocks(const SysParams& P) { return blocks_of(P.nheads, P.sweep_draws); }
// the reference's min(H - 1, floor(u H)) for u = bits / 2^32: u H = bits H / 2^32 is exact in FP64
// (bits H < 2^52), so its floor is the high word of the 64-bit product, always below H
__device__ __forceinline__ uint32_t site_of(uint32_t bits, uint32_t H) {
  return (uint32_t)(((uint64_t)bits * H) >> 32);
}

// the site every draw of the sweep's stream selects when it is a site draw (all SMs)
__global__ void k_sweep_draws(const SysParams* __restrict__ sp, const uint32_t* __restrict__ rng_io, uint32_t only,
                              uint32_t* __restrict__ draw_site) {
  const uint32_t r = only == SOUP_NONE_U32 ? blockIdx.y : only;
  const SysParams& P = sp[r];
  const uint32_t H = P.nheads;
  if (H == 0 || !P.es_on) return;
  const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= draw_blocks(P) * P.sweep_draws) return;
  const Lcg j = lcg_pow(d + 1u);
  draw_site[P.draw_off + d] = site_of(pcg_bits(j.a * rng_io[r] + j.c), H);
}

// The pairs of draws within a block whose sites are near one another.  For place i of a block: entry e names
// an earlier place j (ascending) and the change of i's site energy when j's site deprotonates (std_delta, the
// value the D rows hold).  A place's word in pcnt packs the entry count and, from bit 10 on, 1 + the last
// earlier place of the same site (0: none; a flip changes its own site's state and not its energy).  The
// walk's threads read their entries a place each, eight entries (a group g = e / 8) to a word of pidx, in 256 columns:
// pidx [block][group][column][e % 8], pdel [block][group][e % 8][column].  A place has no more entries than there are
// places before it, so of a block of 512 places 256 + c and 255 - c share column c, the one's groups from the top down,
// the other's from the bottom up, 65 in all; a block of 256 has a column a place (folded, its sweep took 1% longer).
// 10 bytes an entry, 5.3 KB a head.
// A block of threads stages the sites' records and takes kPairDraws draws, a warp per draw at a time: it
// screens 32 earlier draws at a time and evaluates the near ones packed.
constexpr uint32_t kPairDraws = 16;
constexpr uint32_t kPairCols = 256;
__host__ __device__ __forceinline__ uint32_t pair_block(uint32_t W) { return kPairCols * (W == 512u ? 8u * 65u : W); }   // entries
// place i's column and first group, and the way to its next
__device__ __forceinline__ bool pair_up(uint32_t i, uint32_t W) { return W == 512u && i < kPairCols; }
__device__ __forceinline__ uint32_t pair_column(uint32_t i, uint32_t W) { return pair_up(i, W) ? 255u - i : i % kPairCols; }
__device__ __forceinline__ uint32_t pair_first(uint32_t i, uint32_t W) { return pair_up(i, W) ? 64u : 0u; }
__device__ __forceinline__ int pair_step(uint32_t i, uint32_t W) { return pair_up(i, W) ? -1 : 1; }
__device__ __forceinline__ uint32_t pair_group(uint32_t e, uint32_t i, uint32_t W) {
  return pair_first(i, W) + (e >> 3) * (uint32_t)pair_step(i, W);
}
__device__ __forceinline__ uint32_t pidx_at(uint32_t e, uint32_t i, uint32_t W) {
  return (pair_group(e, i, W) * kPairCols + pair_column(i, W)) * 8u + (e & 7u);
}
__device__ __forceinline__ uint32_t pdel_at(uint32_t e, uint32_t i, uint32_t W) {
  return (pair_group(e, i, W) * 8u + (e & 7u)) * kPairCols + pair_column(i, W);
}
__device__ __forceinline__ uint32_t pair_count(uint32_t w) { return w & 1023u; }
__device__ __forceinline__ int pair_same(uint32_t w) { return (int)(w >> 10) - 1; }
template <bool I64>
__global__ void __launch_bounds__(256) k_sweep_pairs(const SysParams* __restrict__ sp, const float4* __restrict__ xq,
                                                     const uint32_t* __restrict__ draw_site, uint32_t only,
                                                     uint32_t* __restrict__ pcnt, uint16_t* __restrict__ pidx,
                                                     long long* __restrict__ pdel) {
  __shared__ float4 rec[kDraws];       // w: the site
  __shared__ uint16_t buf[8][kDraws];
  const uint32_t r = only == SOUP_NONE_U32 ? blockIdx.y : only;
  const SysParams& P = sp[r];
  const uint32_t H = P.nheads;
  if (H == 0 || !P.es_on) return;
  const uint32_t W = P.sweep_draws, first = blockIdx.x * kPairDraws;   // W is a multiple of kPairDraws
  if (first >= draw_blocks(P) * W) return;
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  const size_t block0 = P.draw_off + (first / W) * W, pair0 = P.pair_off + (size_t)(first / W) * pair_block(W);
  const uint32_t i0 = first % W;
  const uint32_t* ds = draw_site + block0;
  const float4* hx = xq + P.head_off;
  for (uint32_t j = threadIdx.x; j < i0 + kPairDraws; j += 256u) {
    const uint32_t s = ds[j];
    const float4 p = hx[s];
    rec[j] = make_float4(p.x, p.y, p.z, __uint_as_float(s));
  }
  __syncthreads();
  uint16_t* near = buf[wid];
  const float screen2 = near2(P);
  const double cut2 = P.d_rc * P.d_rc, reach = P.d_rcattr + P.d_wc, reach2 = reach * reach;
  for (uint32_t i = i0 + wid; i < i0 + kPairDraws; i += 8u) {
    const float4 xi = rec[i];
    const uint32_t site = __float_as_uint(xi.w);
    uint32_t n = 0, same = 0;                          // same: 1 + the last earlier place of this site
    for (uint32_t c = 0; c < i; c += 32u) {
      const uint32_t j = c + lane;
      const float4 xj = rec[min(j, i)];
      const bool own = __float_as_uint(xj.w) == site;
      const uint32_t m = __ballot_sync(0xffffffffu, j < i && !own && fast_r2(P, xj, xi) < screen2);
      const uint32_t mo = __ballot_sync(0xffffffffu, j < i && own);
      if ((m >> lane) & 1u) near[n + __popc(m & ((1u << lane) - 1u))] = (uint16_t)j;
      n += __popc(m);
      if (mo) same = c + 32u - (uint32_t)__clz(mo);
    }
    __syncwarp();
    for (uint32_t e = lane; e < n; e += 32u) {
      const uint32_t j = near[e];
      pidx[pair0 + pidx_at(e, i, W)] = (uint16_t)j;
      pdel[pair0 + pdel_at(e, i, W)] = std_delta(P, dist2<I64>(P, rec[j], xi), (float)P.d_q, cut2, reach2);
    }
    // the last word's places beyond n name place W, which never flips
    for (uint32_t e = n + lane; e < ((n + 7u) & ~7u); e += 32u) pidx[pair0 + pidx_at(e, i, W)] = (uint16_t)W;
    if (lane == 0) pcnt[block0 + i] = n | (same << 10);
    __syncwarp();
  }
}

// The attempts among 32 draws from draw p on: an attempt whose need bit is set takes the next
// draw as its acceptance draw, and the lane after that is an attempt again.  Every run of set need
// bits (restricted to lanes >= p) therefore starts at an attempt, its attempts are the run's even
// offsets, and each of them skips the following lane.  Even offsets are read off the prefix parity
// of the need bits against the parity just before the run (spread over the run by a carry).
__device__ __forceinline__ uint32_t attempt_mask(uint32_t need_m, uint32_t p) {
  const uint32_t range = 0xffffffffu << p;
  const uint32_t x = need_m & range;
  uint32_t px = x;                      // px bit i: parity of x's bits 0..i
  px ^= px << 1;
  px ^= px << 2;
  px ^= px << 4;
  px ^= px << 8;
  px ^= px << 16;
  const uint32_t starts = ((px & ~x) << 1) & x & ~(x << 1);   // runs whose preceding parity is 1
  const uint32_t fill = (x ^ (x + starts)) & x;                 // that parity spread over the run
  const uint32_t even = x & (px ^ fill);                        // the run's even offsets
  return range & ~(even << 1);
}

// one attempt's decision from its site energy: bit 1 accepted, bit 2 took an acceptance draw
// (dG = E_s for a neutral site, -E_s for a charged one; its sign is the fixed-point value's)
__device__ __forceinline__ int decide(long long e, uint32_t f, uint32_t v_acc, float x_scale, double kT) {
  const long long g = f != 0 ? -e : e;
  if (g <= 0) return 1;
  return (metropolis(g, v_acc, x_scale, kT) ? 1 : 0) | 2;
}

// what the walk of one replica shares between its CTAs (global memory): the block's flips in draw order (site,
// its charge state before the flip from bit 28 on; the length of the site's list) and the handoffs
struct alignas(16) WalkShared {
  uint32_t flag;       // (blocks whose flips are written << 10) | flips of the last; kEndOfSweep: over
  uint32_t done;       // CTAs that have added a block's flips, summed over the blocks
  uint32_t timeout;    // a handoff gave up
  uint32_t pad;
  uint2 rec[kDraws];
};

// Add n flips to the energies of their neighbours (global int64, reductions in L2): warp `w` of `nw` takes
// whole flips, or parts of flips when there are more warps than flips.  Every load of a pass is in flight
// before the first add.  (One SM adds about a lane per cycle, so the share of an SM sets the time.)
template <bool I64>
__device__ __forceinline__ void scatter_flips(const uint2* rec, uint32_t n, const SysParams& P, uint32_t cap,
                                              const uint32_t* __restrict__ es_nl, const long long* __restrict__ D,
                                              const float4* __restrict__ xq, long long* __restrict__ E, uint32_t w,
                                              uint32_t nw) {
  constexpr int kUpd = 4;
  const uint32_t lane = threadIdx.x & 31u, off = P.head_off;
  if (n == 0) return;
  const uint32_t parts = max(1u, nw / n);
  for (uint32_t t = w; t < n * parts; t += nw) {
    const uint2 v = rec[t / parts];
    const uint32_t f = v.x >> 28, h = off + (v.x & 0x0FFFFFFFu);
    const uint32_t cnt = v.y, len = (cnt + parts - 1) / parts;
    const uint32_t s0 = (t % parts) * len, s1 = min(s0 + len, cnt);
    const size_t row = (size_t)h * cap;
    for (uint32_t b = s0; b < s1; b += 32u * kUpd) {
      uint32_t tv[kUpd];
      long long dv[kUpd];
#pragma unroll
      for (int u = 0; u < kUpd; ++u) {
        const uint32_t s = b + 32u * u + lane;
        tv[u] = s < s1 ? es_nl[row + s] : 0u;
        dv[u] = s < s1 ? D[row + s] : 0;
      }
#pragma unroll
      for (int u = 0; u < kUpd; ++u) {
        if (b + 32u * u + lane >= s1) continue;
        long long d = f == 0 ? dv[u] : -dv[u];
        if (f == 2) {   // a charge other than the standard one goes to 0
          const double cut2 = P.d_rc * P.d_rc, reach = P.d_rcattr + P.d_wc;
          d = flip_delta(P, dist2<I64>(P, xq[h], xq[tv[u]]), xq[h].w, 0.f, cut2, reach * reach);
        }
        if (d != 0) atomicAdd(reinterpret_cast<unsigned long long*>(E + (tv[u] - off)), (unsigned long long)d);
      }
    }
  }
}

// The D and head-list rows of a block's W draws into L2 (a fifth of them is scattered when the block is done):
// `t` of `nt` threads (at least W).  Every prefetched address lies inside its row.
__device__ __forceinline__ void prefetch_rows(const SysParams& P, uint32_t cap, const uint32_t* __restrict__ ds,
                                              const uint32_t* __restrict__ es_nl, const uint32_t* __restrict__ es_cnt,
                                              const long long* __restrict__ D, uint32_t W, uint32_t t, uint32_t nt) {
  const uint32_t step = nt / W, l0 = t / W;
  if (l0 >= step) return;
  const uint32_t h = P.head_off + ds[t % W], cnt = es_cnt[h];
  if (cnt == 0) return;
  const char* drow = reinterpret_cast<const char*>(D + (size_t)h * cap);
  const char* nrow = reinterpret_cast<const char*>(es_nl + (size_t)h * cap);
  const uint32_t db = cnt * 8u, nb = cnt * 4u, ld = (db + 127u) / 128u + 1u, ln = (nb + 127u) / 128u + 1u;
  for (uint32_t l = l0; l < ld + ln; l += step) {
    const char* a = l < ld ? drow + min(l * 128u, db - 1u) : nrow + min((l - ld) * 128u, nb - 1u);
    asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
  }
}

// A group of CTAs per replica (a cooperative launch: they are resident together).  Per block of draws:
//   the group's first CTA reads E and the charge states of the block's sites (E holds every flip of the
//   earlier blocks), finds the block's flips (a thread per draw) and publishes them; the others add them to E
//   (alone, it adds them itself) and it waits until all have.
// A round of a block: all draws decide; a scan finds the attempts among them and so the flips; every draw pulls
// the flips of its earlier near draws into its energy.  With W < 512 draws a block the threads hold 512 / W
// parts of every draw's entries, and the first part's threads decide; W is a replica's P.sweep_draws, and a
// launch walks the replicas of one W.  (Pushing only the flips that changed to their later
// neighbours, by shared-memory atomics, was slower: a read behind them waits about 10 cycles for each.)
// The handoffs are the block number, released at device scope once the flips are written (the E reads are
// behind it, so no add can reach E before them), and a counter of the CTAs that are done, each release
// ordering that CTA's reductions before it.  Every poll is bounded; one that gives up ends the walk and the
// host reports it.
template <uint32_t W, bool I64>
__global__ void __launch_bounds__(kWalkThreads) k_sweep_walk(
    const SysParams* __restrict__ sp, const uint32_t* __restrict__ head_slot, const float4* __restrict__ xq,
    float* __restrict__ charge, const uint32_t* __restrict__ es_nl, const uint32_t* __restrict__ es_cnt,
    const long long* __restrict__ D, uint32_t cap, long long* __restrict__ Eg, const uint32_t* __restrict__ draw_site,
    const uint32_t* __restrict__ pcnt, const uint16_t* __restrict__ pidx, const long long* __restrict__ pdel,
    WalkShared* __restrict__ shared, uint32_t* __restrict__ rng_io, double* __restrict__ out, uint32_t only,
    uint32_t group, uint32_t spin_limit) {
  extern __shared__ __align__(16) unsigned char flag[];   // the first CTA: a head's charge state
  __shared__ uint2 s_rec[kDraws];
  __shared__ long long s_part[kWalkThreads];
  __shared__ int16_t s_same[kDraws];
  __shared__ int8_t s_code[W + 1];     // 0 no flip, 1 of a neutral site, -1 of a charged one, 2 of another charge
  __shared__ uint32_t s_next[kWalkWarps];                 // per warp: is its last draw's successor used up, by carry in
  __shared__ uint32_t s_att[kWalkWarps], s_nfl[kWalkWarps], s_kill[kWalkWarps];
  __shared__ uint32_t s_dep, s_used, s_acc, s_dn, s_timeout, s_hv;
  __shared__ double s_dsum[kWalkWarps];
  const uint32_t r = (only == SOUP_NONE_U32) ? blockIdx.x / group : only, rank = blockIdx.x % group;
  const SysParams& P = sp[r];
  const uint32_t H = P.nheads;
  if (H == 0 || !P.es_on || P.sweep_draws != W) return;   // the whole group leaves
  WalkShared& G = shared[r];
  const uint32_t off = P.head_off, tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
  long long* E = Eg + off;
  const size_t d0 = P.draw_off;
  const uint32_t blocks = draw_blocks(P);

  if (rank != 0) {
    const uint32_t nt = (group - 1u) * kWalkThreads, t = (rank - 1u) * kWalkThreads + tid;
    prefetch_rows(P, cap, draw_site + d0, es_nl, es_cnt, D, W, t, nt);
    for (uint32_t blk = 0;; ++blk) {
      if (tid == 0) {
        uint32_t v, spins = 0;
        for (;;) {
          v = ld_acquire_gpu(&G.flag);
          if (v == kEndOfSweep || (v >> 10) >= blk + 1u) break;
          if (++spins > spin_limit) { v = kEndOfSweep; atomicExch(&G.timeout, 1u); break; }
        }
        s_hv = v;
      }
      __syncthreads();
      if (s_hv == kEndOfSweep) return;
      const uint32_t n = s_hv & 1023u;
      if (tid < n) s_rec[tid] = __ldcg(&G.rec[tid]);
      __syncthreads();
      scatter_flips<I64>(s_rec, n, P, cap, es_nl, D, xq, E, t >> 5, nt >> 5);
      __syncthreads();
      if (tid == 0) red_add_release_gpu(&G.done, 1u);
      if (blk + 1u < blocks) prefetch_rows(P, cap, draw_site + d0 + (size_t)(blk + 1u) * W, es_nl, es_cnt, D, W, t, nt);
    }
  }

  // 0 neutral, 1 charged with the deprotonated charge, 2 charged with another value
  const float qd = (float)P.d_q;
  int others = 0;
  for (uint32_t h = tid; h < H; h += kWalkThreads) {
    const float q = xq[off + h].w;
    flag[h] = q == 0.f ? 0 : (q == qd ? 1 : 2);
    others |= flag[h] == 2;
  }
  const bool odd = __syncthreads_or(others) != 0;   // some head holds another charge
  if (tid == 0) { s_dep = 0; s_used = 0; s_acc = 0; s_dn = 0; s_timeout = 0; s_code[W] = 0; }
  const double kT = P.d_kT;
  const float x_scale = (float)(kUnfix / P.d_kT);   // -dG/kT per fixed-point unit of dG
  const double dGintr = kT * 2.302585092994046 * (P.d_pka - P.d_ph);
  const uint32_t s0 = rng_io[r];
  const Lcg jb = lcg_pow(W);
  constexpr uint32_t parts = kWalkThreads / W, warps = W / 32u;
  const uint32_t place = tid % W, part = tid / W;
  const bool first = part == 0;        // these threads decide (whole warps)
  const uint32_t column = pair_column(place, W);
  const int step = pair_step(place, W);
  uint32_t st;                         // the stream's state behind this thread's draw
  {
    const Lcg j = lcg_pow(place + 1u);
    st = j.a * s0 + j.c;
  }
  uint32_t attempts = 0, carry = 0, accepted = 0, dcount = 0;   // carry: the block's first draw is used up
  double dsum = 0.0;
  bool over = false;
  uint32_t site = draw_site[d0 + place], word = pcnt[d0 + place], len = es_cnt[off + site];
  __syncthreads();
  for (uint32_t blk = 0; !over; ++blk) {
    const size_t b0 = d0 + (size_t)blk * W;
    // this draw's near draws: places eight to a word, changes one by one
    const size_t p0 = P.pair_off + (size_t)blk * pair_block(W);
    const uint16_t* px = pidx + p0;
    const long long* pd = pdel + p0;
    const uint32_t np = pair_count(word);
    const uint4* pi = reinterpret_cast<const uint4*>(px) + (pair_first(place, W) + part * (uint32_t)step) * kPairCols + column;
    const uint4 idx0 = 8u * part < np ? __ldg(pi) : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t v_acc = pcg_bits(st * 747796405u + 2891336453u);   // the next draw of the stream
    const long long e_base = (long long)__ldcg(reinterpret_cast<const unsigned long long*>(E + site));
    const uint32_t f_base = flag[site];
    const bool more = blk + 1u < blocks;
    const uint32_t site_next = more ? draw_site[b0 + W + place] : 0u, word_next = more ? pcnt[b0 + W + place] : 0u;
    if (first) s_same[place] = (int16_t)pair_same(word);
    if (lane == 0) s_kill[wid] = 0;
    long long e = e_base;
    uint32_t f = f_base, am = 0, need_m = 0, carry_out = 0, flips = 0;
    int code = 0, pred = -1;                     // the last earlier flip of this block on the same site
    const bool last = H - attempts <= W;   // the attempt limit can fall into this block
    for (uint32_t round = 0;; ++round) {
      const int res = first ? decide(e, f, v_acc, x_scale, kT) : 0;
      const uint32_t acc_m = __ballot_sync(0xffffffffu, res & 1);
      need_m = __ballot_sync(0xffffffffu, res & 2);
      const uint32_t am0 = attempt_mask(need_m, 0), am1 = attempt_mask(need_m, 1);
      if (lane == 0) s_next[wid] = ((am0 & need_m) >> 31) | (((am1 & need_m) >> 31) << 1);
      __syncthreads();
      // the carry into every warp: the warps' maps of carry in to carry out, composed
      uint32_t fn = lane < warps ? s_next[lane] : 2u;        // 2: the identity
#pragma unroll
      for (int o = 1; o < (int)kWalkWarps; o <<= 1) {
        const uint32_t g = __shfl_up_sync(0xffffffffu, fn, o);
        if (lane >= (uint32_t)o) fn = ((fn >> (g & 1u)) & 1u) | (((fn >> (g >> 1)) & 1u) << 1);
      }
      const uint32_t before = __shfl_sync(0xffffffffu, fn, (wid + 31u) & 31u);
      const uint32_t cin = wid == 0 || !first ? carry : (before >> carry) & 1u;
      carry_out = (__shfl_sync(0xffffffffu, fn, kWalkWarps - 1) >> carry) & 1u;
      am = first ? (cin ? am1 : am0) : 0u;
      if (last) {                      // no more than H attempts
        if (lane == 0) s_att[wid] = __popc(am);
        __syncthreads();
        const uint32_t ahead = __reduce_add_sync(0xffffffffu, lane < wid ? s_att[lane] : 0u), left = H - attempts;
        const uint32_t room = left - min(left, ahead);
        am &= __ballot_sync(0xffffffffu, __popc(am & ((1u << lane) - 1u)) < (int)room);
        __syncthreads();               // s_att is written again below
      }
      flips = am & acc_m;
      const int now = ((flips >> lane) & 1u) ? (f == 0u ? 1 : (f == 1u ? -1 : 2)) : 0, was = code;
      if (first) s_code[place] = (int8_t)now;
      code = now;
      if (lane == 0) { s_nfl[wid] = __popc(flips); s_att[wid] = __popc(am); }
      if (!__syncthreads_or(now != was)) break;
      if (round > kDraws) {            // cannot be: draw d stands after d rounds
        s_timeout = 1u;
        break;
      }
      long long sum = 0;
      uint4 nxt = idx0;
      const uint4* pw = pi;
      const long long* pv = pd + (pair_first(place, W) + part * (uint32_t)step) * (8u * kPairCols) + column;
      for (uint32_t q = 8u * part; q < np; q += 8u * parts, pv += step * (int)(8u * kPairCols * parts)) {
        const uint32_t jw[4] = {nxt.x, nxt.y, nxt.z, nxt.w};
        // the next word: stepped to with 256 draws a block (counted from the first, a sweep of 4,665 heads took 441 us and
        // not 424), counted from the first with 512 (18,659 heads, 995 and not 1013)
        if (W == 512u) pw = pi + step * (int)((q / 8u - part + parts) * kPairCols);
        else pw += kPairCols * parts;
        if (q + 8u * parts < np) nxt = __ldg(pw);
        int c[8];
        long long v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          c[u] = s_code[u & 1 ? jw[u >> 1] >> 16 : jw[u >> 1] & 0xFFFFu];
          v[u] = c[u] != 0 ? __ldg(pv + u * kPairCols) : 0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {  // c v for c = 0, 1, -1
          const long long m = c[u] >> 31;
          sum += (v[u] ^ m) - m;
        }
      }
      if (parts > 1u) {
        s_part[tid] = sum;
        __syncthreads();
        if (first)
          for (uint32_t u = 1; u < parts; ++u) sum += s_part[u * W + place];
      }
      e = e_base + sum;
      if (odd) {                       // flips from a charge other than the standard one: not D's change
        const double cut2 = P.d_rc * P.d_rc, reach = P.d_rcattr + P.d_wc, reach2 = reach * reach;
        for (uint32_t q = 0; q < np; ++q) {
          const uint32_t j = px[pidx_at(q, place, W)];
          if (s_code[j] != 2) continue;
          const uint32_t sj = off + draw_site[b0 + j];
          e += flip_delta(P, dist2<I64>(P, xq[sj], xq[off + site]), xq[sj].w, 0.f, cut2, reach2) - pd[pdel_at(q, place, W)];
        }
      }
      // the charge state behind the last earlier flip of this site
      pred = first ? s_same[place] : -1;
      while (pred >= 0 && s_code[pred] == 0) pred = s_same[pred];
      f = pred < 0 ? f_base : (s_code[pred] == 1 ? 1u : 0u);
    }
    // the flips stand: the charge states (a site flipped twice takes what its last flip left) and records
    const bool mine = code != 0;
    const uint32_t nfl = lane < warps ? s_nfl[lane] : 0u;
    const uint32_t at = __reduce_add_sync(0xffffffffu, lane < wid ? nfl : 0u), nf = __reduce_add_sync(0xffffffffu, nfl);
    const uint32_t na = __reduce_add_sync(0xffffffffu, lane < warps ? s_att[lane] : 0u);
    attempts += na;
    over = attempts == H || s_timeout != 0;
    if (mine) {
      const uint32_t p = at + __popc(flips & ((1u << lane) - 1u));
      const uint2 v = make_uint2(site | (f << 28), len);
      if (group > 1u) __stcg(&G.rec[p], v);
      else s_rec[p] = v;
      if (pred >= 0) atomicOr(&s_kill[pred >> 5], 1u << (pred & 31));
      ++accepted;
      if (f == 0) { dsum += (double)e * kUnfix - dGintr; ++dcount; }
    }
    carry = carry_out;
    if (attempts == H && am) {         // the draws the sweep used: up to its last attempt, and its acceptance draw
      const uint32_t b = 31u - (uint32_t)__clz(am);
      if (lane == 0) atomicMax(&s_used, blk * W + wid * 32u + b + 1u + ((need_m >> b) & 1u));
    }
    __syncthreads();
    if (group > 1u && !over && tid == 0) st_release_gpu(&G.flag, ((blk + 1u) << 10) | nf);
    if (mine && !((s_kill[wid] >> lane) & 1u)) flag[site] = f != 0 ? 0 : 1;
    if (over) break;                   // nothing reads E any more
    site = site_next;
    word = word_next;
    len = es_cnt[off + site];
    st = jb.a * st + jb.c;
    if (group == 1u) {
      scatter_flips<I64>(s_rec, nf, P, cap, es_nl, D, xq, E, wid, kWalkWarps);
    } else if (tid == 0) {
      const uint32_t want = (group - 1u) * (blk + 1u);
      uint32_t spins = 0;
      while (ld_acquire_gpu(&G.done) < want) {
        if (++spins > spin_limit) { s_timeout = 1u; break; }
      }
    }
    __syncthreads();
    over = s_timeout != 0;
  }
  __syncthreads();
  if (group > 1u && tid == 0) {
    if (__ldcg(&G.timeout)) s_timeout = 1u;
    st_release_gpu(&G.flag, kEndOfSweep);
  }
  // the charges from the final states (a head still in state 2 keeps its own value)
  uint32_t dep = 0;
  for (uint32_t h = tid; h < H; h += kWalkThreads) {
    const uint8_t fl = flag[h];
    if (fl != 2) charge[head_slot[off + h]] = fl == 0 ? 0.f : qd;
    dep += fl != 0;
  }
  for (int o = 16; o > 0; o >>= 1) {
    dep += __shfl_xor_sync(0xffffffffu, dep, o);
    accepted += __shfl_xor_sync(0xffffffffu, accepted, o);
    dcount += __shfl_xor_sync(0xffffffffu, dcount, o);
    dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
  }
  if (lane == 0) {
    atomicAdd(&s_dep, dep);
    atomicAdd(&s_acc, accepted);
    atomicAdd(&s_dn, dcount);
    s_dsum[wid] = dsum;
  }
  __syncthreads();
  if (tid == 0) {
    double ds = 0.0;
    for (uint32_t u = 0; u < kWalkWarps; ++u) ds += s_dsum[u];
    const Lcg j = lcg_pow(s_used);
    rng_io[r] = j.a * s0 + j.c;
    out[4 * r + 0] = s_timeout ? -1.0 : (double)H;   // -1: a handoff gave up (the host reports it)
    out[4 * r + 1] = (double)s_acc;
    out[4 * r + 2] = s_dn > 0 ? ds / kT / s_dn : 0.0;
    out[4 * r + 3] = (double)s_dep;
  }
}

// head positions and charges by head index, as they are when the sweep begins
__global__ void k_gather_heads(const uint32_t* __restrict__ head_slot, uint32_t H, const float4* __restrict__ pos,
                               const float* __restrict__ charge, float4* __restrict__ xq) {
  const uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= H) return;
  const uint32_t k = head_slot[h];
  const float4 p = pos[k];
  xq[h] = make_float4(p.x, p.y, p.z, charge[k]);
}

}  // namespace

// the mean length of the head lists of a replica (the longest of the batch's), from its head density
double sweep_list_entries(const Batch& b, uint32_t replica) {
  double most = 0.0;
  for (uint32_t r = 0; r < b.R; ++r) {
    if (replica != SOUP_NONE_U32 && r != replica) continue;
    const SoupConfig& c = b.cfg[r];
    if (!c.es_enabled || !b.hsp[r].nheads) continue;
    const double vol = c.wall_radius > 0 ? c.wall_radius * c.wall_radius * c.wall_radius * 4.18879 : c.box[0] * c.box[1] * c.box[2];
    const double range = c.es_list_range;
    most = std::max(most, b.hsp[r].nheads * std::min(1.0, range * range * range * 4.18879 / vol));
  }
  return most;
}

template <uint32_t W, bool I64>
void launch_walk(Batch& b, uint32_t replica, unsigned ry, unsigned group, size_t smem) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(ry * group);
  lc.blockDim = dim3(kWalkThreads);
  lc.dynamicSmemBytes = smem;
  lc.stream = b.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  lc.attrs = attr;
  lc.numAttrs = group > 1u ? 1 : 0;
  SOUP_CUDA_TRY(cudaLaunchKernelEx(&lc, k_sweep_walk<W, I64>, (const SysParams*)b.sp, (const uint32_t*)b.head_slot,
                                   (const float4*)b.head_pos, b.charge, (const uint32_t*)b.es_nl,
                                   (const uint32_t*)b.es_cnt, (const long long*)b.head_d, b.es_cap, b.head_e,
                                   (const uint32_t*)b.draw_site, (const uint32_t*)b.pair_cnt,
                                   (const uint16_t*)b.pair_idx, (const long long*)b.pair_del,
                                   reinterpret_cast<WalkShared*>(b.walk_shared), b.prot_rng_dev, b.sweep_out, replica,
                                   group, b.wait_limit ? b.wait_limit : kSpinLimit));
}

// replica == SOUP_NONE_U32: every replica
void launch_sweep(Batch& b, uint32_t replica) {
  if (b.H == 0) return;
  uint32_t hmax = 0, wmax = 0;
  bool far = false;
  for (uint32_t r = 0; r < b.R; ++r)
    if (replica == SOUP_NONE_U32 || r == replica) {
      far = far || b.hsp[r].image64 != 0;
      hmax = std::max(hmax, b.hsp[r].nheads);
      wmax = std::max(wmax, b.hsp[r].sweep_draws);
    }
  if (hmax == 0) return;
  b.launches += 4;
  prof_begin(b, SOUP_K_SWEEP);
  const unsigned ry = replica == SOUP_NONE_U32 ? b.R : 1;
  const uint32_t draws = (2 * hmax + kDraws - 1) / kDraws * kDraws;   // at least every replica's whole blocks
  k_gather_heads<<<(b.H + 255) / 256, 256, 0, b.stream>>>(b.head_slot, b.H, b.pos, b.charge, b.head_pos);
  (far ? k_sweep_init<true> : k_sweep_init<false>)<<<(unsigned)(((uint64_t)b.H * 32 + 255) / 256), 256, 0, b.stream>>>(
      b.sp, b.head_sys, b.H, b.head_pos, b.es_nl, b.es_cnt, b.es_cap, b.head_e, b.head_d, replica);
  k_sweep_draws<<<dim3((draws + 255) / 256, ry), 256, 0, b.stream>>>(b.sp, b.prot_rng_dev, replica, b.draw_site);
  (far ? k_sweep_pairs<true> : k_sweep_pairs<false>)<<<dim3(draws / kPairDraws, ry), 256, 0, b.stream>>>(
      b.sp, b.head_pos, b.draw_site, replica, b.pair_cnt, b.pair_idx, b.pair_del);
  // a group of CTAs per replica, all SMs together (a cooperative launch).  A handoff there and back costs 4k to 5k cycles
  // a block, in which one SM adds about 4k list entries: a replica whose blocks flip fewer than that walks alone
  // (a fifth of the draws flips; a list holds the heads within the range, at most all of them).
  const unsigned each = std::max(1u, (unsigned)b.sms / ry);
  const double entries = 0.2 * std::min(2u * hmax, wmax) * std::min<double>(hmax, sweep_list_entries(b, replica));
  const unsigned group = entries < 4000.0 ? 1u : each;
  SOUP_CUDA_TRY(cudaMemsetAsync(b.walk_shared, 0, sizeof(WalkShared) * b.R, b.stream));
  const size_t smem = ((size_t)hmax + 15) & ~(size_t)15;
  for (uint32_t w : {512u, 256u}) {   // the block sizes in use
    bool any = false;
    for (uint32_t r = 0; r < b.R; ++r)
      any = any || ((replica == SOUP_NONE_U32 || r == replica) && b.hsp[r].nheads && b.hsp[r].sweep_draws == w);
    if (!any) continue;
    b.launches += 1;
    const auto walk = w == 512u ? (far ? launch_walk<512, true> : launch_walk<512, false>)
                                : (far ? launch_walk<256, true> : launch_walk<256, false>);
    walk(b, replica, ry, group, smem);
  }
  prof_end(b);
}

uint32_t sweep_max_heads() { return kMaxHeads; }
void sweep_layout(Batch& b, size_t& draws, size_t& pairs) {
  draws = pairs = 0;
  for (SysParams& p : b.hsp) {
    const uint32_t W = p.sweep_most = p.sweep_draws, blocks = blocks_of(p.nheads, W);
    p.draw_off = (uint32_t)draws;
    p.pair_off = pairs;
    draws += (size_t)blocks * W;
    pairs += (size_t)blocks * pair_block(W);
  }
}

size_t sweep_shared_bytes(const Batch& b) { return sizeof(WalkShared) * b.R; }

void sweep_prepare(Batch& b) {
  const int most = (int)((kMaxHeads + 15) & ~15u);
  for (const void* walk : {(const void*)k_sweep_walk<512, false>, (const void*)k_sweep_walk<512, true>,
                           (const void*)k_sweep_walk<256, false>, (const void*)k_sweep_walk<256, true>})
    SOUP_CUDA_TRY(cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  SOUP_CUDA_TRY(cudaDeviceGetAttribute(&b.sms, cudaDevAttrMultiProcessorCount, b.device));
}

}  // namespace soup
