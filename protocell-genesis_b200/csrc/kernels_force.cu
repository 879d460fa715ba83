// kernels_force.cu -- the force: list pair force + bonded terms + wall, the far Debye-Hueckel half,
// and the O(N^2) brute-force twin.
//
// Reference: soup/wgsl/verlet.wgsl:132-149 soup_force_list_main (bondedForce + sum over the list of
// nonbondedSoup), soup/wgsl/step.wgsl:152-193 bondedForce, soup/wgsl/electrostatics-long.wgsl:63-103
// (far half, accumulated), soup/wgsl/wall.wgsl:42-56 (wall, accumulated), step.wgsl:277-292 brute.
//
// TPP threads (4, 8 or 16) cooperate on one particle.  A particle's force is summed in sixteen partial sums:
// list entry e and bonded term t go to sums e mod 16 and t, each in ascending order, and the sums are added
// in a fixed tree, so the result is the same bits for every TPP and run to run.  No atomics: every
// particle's force is produced by exactly one group (full list, no Newton-3).
#include "soup_internal.h"

namespace soup {

namespace {

constexpr int kBlock = 256;
inline unsigned nblocks(uint64_t n, int b = kBlock) { return (unsigned)((n + b - 1) / b); }

// One bonded term of particle (slot k, original id gi), term index t in [0, 13):
//   t < 3         FENE to slot partner t
//   3 <= t < 12   bend to partner-of-partner ((t-3)/3, (t-3)%3), skipping i itself
//   t == 12       FENE tether to the adsorbing catalyst (centerLink)
__device__ __forceinline__ void bonded_term(const Shared& S, const SysParams& P, int t, uint32_t gi, const float4& xi,
                                            const uint32_t* __restrict__ sl, uint32_t owner,
                                            const uint32_t* __restrict__ slots, const uint32_t* __restrict__ slot_of,
                                            const float4* __restrict__ pos, float& fx, float& fy, float& fz) {
  uint32_t other;
  bool fene;
  if (t < 3) { other = sl[t]; fene = true; }
  else if (t < 12) {
    uint32_t m = sl[(t - 3) / 3];
    if (m == SOUP_NONE_U32) return;
    other = slots[3 * slot_of[m] + (t - 3) % 3];
    if (other == gi) return;
    fene = false;
  } else { other = owner; fene = true; }
  if (other == SOUP_NONE_U32) return;
  float4 xo = pos[slot_of[other]];
  float dx = fast_mi(xi.x - xo.x, P.box[0], P.inv_box[0]);
  float dy = fast_mi(xi.y - xo.y, P.box[1], P.inv_box[1]);
  float dz = fast_mi(xi.z - xo.z, P.box[2], P.inv_box[2]);
  float s = bonded_scalar(S, dx * dx + dy * dy + dz * dz, fene);
  fx += s * dx; fy += s * dy; fz += s * dz;
}

// One group's pass over its particle's row up to `end`: four entries a lane and iteration, the next
// iteration's indices loaded before this one's pairs.  Rows are padded to 16 entries with the particle
// itself, and what a chunk holds beyond `end` is beyond the reach: neither adds anything.
// INSIDE: the warp's particles lie at least the reach inside every face, so their in-range neighbours are at
// their stored (wrapped) coordinates and the minimum image is the plain difference (fast_mi returns it
// unchanged; an entry beyond the reach by the plain difference is beyond it by the minimum image too).
// CHARGED: some particle of the warp is charged or of the polar class.
__device__ __forceinline__ uint4 ld_stream(const uint4* p) {   // read once: keeps the L1 for the neighbours
  uint4 v;
  asm("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
template <int TPP, bool INSIDE, bool CHARGED>
__device__ __forceinline__ void list_sum(uint32_t k, int lane, uint32_t end, const uint32_t* __restrict__ row,
                                         const float4* __restrict__ pos, const float* __restrict__ charge,
                                         const float4& xi, float qi, bool needq, uint32_t polar,
                                         const PairW* __restrict__ prow, const PairLean& L, const SysParams& P,
                                         float (&f)[16 / TPP][3]) {
  constexpr int E = 16 / TPP, C = 4 / E;          // a lane's entries of a chunk of 16, chunks an iteration
  const float bx = P.box[0], by = P.box[1], bz = P.box[2];
  const float ix = P.inv_box[0], iy = P.inv_box[1], iz = P.inv_box[2];
  const bool qi_nz = qi != 0.f;
  uint32_t nj[4];
  auto fetch = [&](uint32_t base) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const uint32_t at = base + 16u * c;
      const uint32_t* p = row + at + E * lane;
      const bool in = C == 1 || at < end;
      if (E == 4) {
        const uint4 v = in ? ld_stream(reinterpret_cast<const uint4*>(p)) : make_uint4(k, k, k, k);
        nj[0] = v.x; nj[1] = v.y; nj[2] = v.z; nj[3] = v.w;
      } else if (E == 2) {
        const uint2 v = in ? __ldg(reinterpret_cast<const uint2*>(p)) : make_uint2(k, k);
        nj[2 * c] = v.x; nj[2 * c + 1] = v.y;
      } else {
        nj[c] = in ? __ldg(p) : k;
      }
    }
  };
  if (end > 0) fetch(0);
  for (uint32_t base = 0; base < end; base += 16u * C) {
    uint32_t j[4];
    float4 xj[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) { j[u] = nj[u]; xj[u] = __ldg(pos + j[u]); }
    if (base + 16u * C < end) fetch(base + 16u * C);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float dx = xi.x - xj[u].x, dy = xi.y - xj[u].y, dz = xi.z - xj[u].z;
      if (!INSIDE) {
        dx = fast_mi(dx, bx, ix);
        dy = fast_mi(dy, by, iy);
        dz = fast_mi(dz, bz, iz);
      }
      const float r2 = dx * dx + dy * dy + dz * dz;
      // the kind, a small whole number held as a float, from the low bits of its sum with 2^23
      const uint32_t kj = __float_as_uint(xj[u].w + 8388608.0f) & (SOUP_KMAX - 1u);
      const float qj = CHARGED && needq ? __ldg(charge + j[u]) : 0.f;
      const float s = pair_lean<CHARGED>(prow[kj], L, r2, CHARGED && ((polar >> kj) & 1u), qi_nz, qi, qj);
      float (&a)[3] = f[u % E];
      a[0] += s * dx; a[1] += s * dy; a[2] += s * dz;
    }
  }
}

// eight 128-thread blocks per SM (64 registers): small blocks even out rows of unequal length (256 threads: 192
// against 183 us at 483k beads).  At 64 the four-lane forms spill 36 bytes a thread and the heads' eight-lane one 24;
// fewer registers spill more, fewer blocks hide less of the gathers' latency
constexpr int kForceBlock = 128;

// SEL: the particles are the nsel slots sel[] (the heads, after a charge sweep) instead of all N
//
// Bound: the L1's wavefronts for the neighbour gathers (two thirds of its rate) and the issue of the pair maths
// (half).  Straight-line pairs over sixteen fixed partial sums, rows read to each bead's own reach and chunks stored for the
// lanes' order took it from 250 to 168 us right after a rebuild at 483k beads, 309 to 187 over a rebuild's steps.
// Slower: gathers pipelined an iteration ahead (242), three or five blocks of 256 an SM (214, 244).
template <int TPP, bool SEL>
__global__ void __launch_bounds__(kForceBlock, 8) k_force(
    const Shared* __restrict__ Sg, const SysParams* __restrict__ sp, const uint8_t* __restrict__ sysid, uint32_t N,
    const float4* __restrict__ pos, const float* __restrict__ charge, const uint32_t* __restrict__ slots,
    const uint32_t* __restrict__ center, const uint32_t* __restrict__ id, const uint32_t* __restrict__ slot_of,
    const uint32_t* __restrict__ nl, const uint32_t* __restrict__ nl_cnt, const uint32_t* __restrict__ nl_shell,
    const uint32_t* __restrict__ drift_bits, uint32_t stride, float4* __restrict__ force,
    const uint32_t* __restrict__ sel, uint32_t nsel, const uint32_t* __restrict__ head_of, float4* __restrict__ head_xq) {
  __shared__ PairW pw[SOUP_KMAX * SOUP_KMAX];
  for (int w = threadIdx.x; w < (int)(sizeof(pw) / 4); w += kForceBlock)
    reinterpret_cast<uint32_t*>(pw)[w] = reinterpret_cast<const uint32_t*>(Sg->pw)[w];
  __syncthreads();
  constexpr int E = 16 / TPP;
  const Shared& S = *Sg;
  const uint32_t gtid = blockIdx.x * (uint32_t)kForceBlock + threadIdx.x;
  const uint32_t g = gtid / TPP;
  const int lane = (int)(gtid % TPP);
  const bool active = SEL ? g < nsel : g < N;
  const uint32_t k = SEL ? (active ? sel[g] : 0u) : (active ? g : 0u);
  const uint32_t rs = sysid[k];
  const SysParams& P = sp[rs];
  const float4 xi = pos[k];
  const int ki = (int)xi.w & (SOUP_KMAX - 1);
  const float qi = charge[k];
  const bool needq = qi != 0.f || (S.cls[ki] == 1u && P.acid > 0.f);
  const PairLean L = PairLean::of(S, P);
  const uint32_t end = active ? list_force_end(k, nl_cnt, nl_shell, __uint_as_float(drift_bits[rs]), P, list_wide(S, P, ki, qi))
                              : 0u;
  const float reach = P.reach[1] + 1e-3f;
  const bool in = xi.x >= reach && xi.x <= P.box[0] - reach && xi.y >= reach && xi.y <= P.box[1] - reach &&
                  xi.z >= reach && xi.z <= P.box[2] - reach;
  const bool inside = __all_sync(0xffffffffu, in || !active), charged = __any_sync(0xffffffffu, needq && active);
  const uint32_t polar = (S.polar >> ki) & 1u ? S.polar : 0u;   // the kinds of the polar class, for an owner of it
  const uint32_t* row = nl + (size_t)k * stride;
  const PairW* prow = pw + ki * SOUP_KMAX;
  float f[E][3] = {};
  if (inside) {
    if (charged) list_sum<TPP, true, true>(k, lane, end, row, pos, charge, xi, qi, needq, polar, prow, L, P, f);
    else list_sum<TPP, true, false>(k, lane, end, row, pos, charge, xi, qi, needq, polar, prow, L, P, f);
  } else {
    if (charged) list_sum<TPP, false, true>(k, lane, end, row, pos, charge, xi, qi, needq, polar, prow, L, P, f);
    else list_sum<TPP, false, false>(k, lane, end, row, pos, charge, xi, qi, needq, polar, prow, L, P, f);
  }
  if (active) {   // bonded terms (bondedForce), spread over the sums
    uint32_t sl[3] = {slots[3 * k], slots[3 * k + 1], slots[3 * k + 2]};
    const uint32_t owner = center[k];
    if ((sl[0] & sl[1] & sl[2] & owner) != SOUP_NONE_U32) {
      const uint32_t gi = id[k];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int t = E * lane + e;
        if (t < 13) bonded_term(S, P, t, gi, xi, sl, owner, slots, slot_of, pos, f[e][0], f[e][1], f[e][2]);
      }
    }
  }
  // the tree over the sums: neighbours first, inside the lane and then across the group
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int o = 1; o < E; o <<= 1)
#pragma unroll
      for (int e = 0; e < E; e += 2 * o) f[e][a] += f[e + o][a];
#pragma unroll
    for (int o = 1; o < TPP; o <<= 1) f[0][a] += __shfl_xor_sync(0xffffffffu, f[0][a], o);
  }
  if (active && lane == 0) {
    float fx = f[0][0], fy = f[0][1], fz = f[0][2];
    if (P.wall_r > 0.f) {   // wall.wgsl:42-56
      float d0 = xi.x - P.box[0] * 0.5f, d1 = xi.y - P.box[1] * 0.5f, d2 = xi.z - P.box[2] * 0.5f;
      float r = sqrtf(d0 * d0 + d1 * d1 + d2 * d2);
      if (r > P.wall_r) {
        float w = -P.wall_k * (r - P.wall_r) / fmaxf(r, 1e-6f);
        fx += w * d0; fy += w * d1; fz += w * d2;
      }
    }
    force[k] = make_float4(fx, fy, fz, 0.f);
    // a head's record (x, y, z, q) by head index: the far half reads one 16-byte record per list entry instead
    // of a slot lookup and two gathers
    const uint32_t h = SEL ? g : (head_of ? head_of[k] : SOUP_NONE_U32);
    if (SEL || h != SOUP_NONE_U32) head_xq[h] = make_float4(xi.x, xi.y, xi.z, qi);
  }
}

// soup/wgsl/electrostatics-long.wgsl:63-82 soup_es_force_far_main, a warp per head, on the records that the list
// force wrote.  Bound: the latency of the gathers.  A lane has four in flight and the next four entries loaded (one at
// a time: 48.9 against 39.1 us at 483k beads, 12.5 against 8.7 at 24k).
__global__ void __launch_bounds__(256) k_es_far(const SysParams* __restrict__ sp, const uint32_t* __restrict__ head_slot,
                                                const uint32_t* __restrict__ head_sys, uint32_t H,
                                                const float4* __restrict__ xq, const uint32_t* __restrict__ es_nl,
                                                const uint32_t* __restrict__ es_cnt, uint32_t cap,
                                                float4* __restrict__ force) {
  const uint32_t h = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (h >= H) return;   // warp-uniform
  const SysParams& P = sp[head_sys[h]];
  const float4 xi = xq[h];
  const float qi = xi.w;
  if (qi == 0.f || P.es_A == 0.f) return;
  const float bx = P.box[0], by = P.box[1], bz = P.box[2], ibx = P.inv_box[0], iby = P.inv_box[1], ibz = P.inv_box[2];
  const float A = P.es_A, kappa = P.es_kappa, fc = P.es_fc, r0 = P.es_split, r1 = P.es_rc;
  float fx = 0.f, fy = 0.f, fz = 0.f;
  const uint32_t cnt = es_cnt[h];
  const uint32_t* row = es_nl + (size_t)h * cap;
  uint32_t j[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) j[u] = lane + 32u * u < cnt ? __ldg(row + lane + 32u * u) : h;
  for (uint32_t s = (uint32_t)lane; s - lane < cnt; s += 128u) {
    float4 xj[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) xj[u] = __ldg(xq + j[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t n = s + 128u + 32u * u;
      j[u] = n < cnt ? __ldg(row + n) : h;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float dx = fast_mi(xi.x - xj[u].x, bx, ibx);
      const float dy = fast_mi(xi.y - xj[u].y, by, iby);
      const float dz = fast_mi(xi.z - xj[u].z, bz, ibz);
      const float r2 = dx * dx + dy * dy + dz * dz;
      const float rinv = rsqrt_ftz(r2);
      const float r = r2 * rinv;
      const float w = A * __expf(-kappa * r) * rinv;
      const float sc = qi * xj[u].w * (w * (rinv + kappa) - fc) * rinv;
      if (s + 32u * u < cnt && xj[u].w != 0.f && r >= r0 && r < r1) {   // esForceFar (electrostatics.wgsl:87-90)
        fx += sc * dx; fy += sc * dy; fz += sc * dz;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    fx += __shfl_xor_sync(0xffffffffu, fx, o);
    fy += __shfl_xor_sync(0xffffffffu, fy, o);
    fz += __shfl_xor_sync(0xffffffffu, fz, o);
  }
  if (lane == 0) {
    const uint32_t ks = head_slot[h];
    float4 f = force[ks];
    force[ks] = make_float4(f.x + fx, f.y + fy, f.z + fz, 0.f);
  }
}

// soup/wgsl/step.wgsl:277-292 + electrostatics-long.wgsl:88-103 + wall: every pair of the replica.
__global__ void __launch_bounds__(128) k_force_brute(
    const Shared* __restrict__ Sg, const SysParams* __restrict__ sp, const uint8_t* __restrict__ sysid, uint32_t N,
    const float4* __restrict__ pos, const float* __restrict__ charge, const uint32_t* __restrict__ slots,
    const uint32_t* __restrict__ center, const uint32_t* __restrict__ id, const uint32_t* __restrict__ slot_of,
    float4* __restrict__ force) {
  __shared__ Shared S;
  for (int w = threadIdx.x; w < (int)(sizeof(Shared) / 4); w += blockDim.x)
    reinterpret_cast<uint32_t*>(&S)[w] = reinterpret_cast<const uint32_t*>(Sg)[w];
  __syncthreads();
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= N) return;
  const SysParams& P = sp[sysid[k]];
  const PairLean L = PairLean::of(S, P);
  const float4 xi = pos[k];
  const int ki = (int)xi.w;
  const float qi = charge[k];
  float fx = 0.f, fy = 0.f, fz = 0.f;
  for (uint32_t j = P.slot_off; j < P.slot_off + P.n; ++j) {
    if (j == k) continue;
    const float4 xj = pos[j];
    const float dx = fast_mi(xi.x - xj.x, P.box[0], P.inv_box[0]);
    const float dy = fast_mi(xi.y - xj.y, P.box[1], P.inv_box[1]);
    const float dz = fast_mi(xi.z - xj.z, P.box[2], P.inv_box[2]);
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (r2 < 1e-12f) continue;
    const int kj = (int)xj.w;
    const float qj = charge[j];
    if (r2 < S.rmax2) {
      const float sc = pair_lean<true>(S.pw[ki * SOUP_KMAX + kj], L, r2, (S.polar >> ki) & (S.polar >> kj) & 1u, qi != 0.f,
                                       qi, qj);
      fx += sc * dx; fy += sc * dy; fz += sc * dz;
    }
    const float qq = qi * qj;
    if (qq != 0.f && P.es_A != 0.f) {
      const float r = sqrtf(r2);
      if (r >= P.es_split && r < P.es_rc) {
        const float u = P.es_A * __expf(-P.es_kappa * r) / r;
        const float s = qq * (u * (1.0f / r + P.es_kappa) - P.es_fc) / r;
        fx += s * dx; fy += s * dy; fz += s * dz;
      }
    }
  }
  uint32_t sl[3] = {slots[3 * k], slots[3 * k + 1], slots[3 * k + 2]};
  uint32_t owner = center[k];
  const uint32_t gi = id[k];
  for (int t = 0; t < 13; ++t) bonded_term(S, P, t, gi, xi, sl, owner, slots, slot_of, pos, fx, fy, fz);
  if (P.wall_r > 0.f) {
    float d0 = xi.x - P.box[0] * 0.5f, d1 = xi.y - P.box[1] * 0.5f, d2 = xi.z - P.box[2] * 0.5f;
    float r = sqrtf(d0 * d0 + d1 * d1 + d2 * d2);
    if (r > P.wall_r) {
      float w = -P.wall_k * (r - P.wall_r) / fmaxf(r, 1e-6f);
      fx += w * d0; fy += w * d1; fz += w * d2;
    }
  }
  force[k] = make_float4(fx, fy, fz, 0.f);
}

template <int TPP>
void launch_force_tpp(Batch& b, bool heads) {
  const uint32_t n = heads ? b.H : b.N;
  const unsigned blocks = nblocks((uint64_t)n * TPP, kForceBlock);
  const uint32_t* shells = b.prune ? b.nl_shell : nullptr;
  if (heads)
    k_force<TPP, true><<<blocks, kForceBlock, 0, b.stream>>>(b.shared, b.sp, b.sysid, b.N, b.pos, b.charge, b.slots, b.center, b.id,
                                                     b.slot_of, b.nl, b.nl_cnt, shells, b.drift_bits, b.list_stride,
                                                     b.force, b.head_slot, b.H, nullptr, b.head_xq);
  else
    k_force<TPP, false><<<blocks, kForceBlock, 0, b.stream>>>(b.shared, b.sp, b.sysid, b.N, b.pos, b.charge, b.slots, b.center, b.id,
                                                      b.slot_of, b.nl, b.nl_cnt, shells, b.drift_bits, b.list_stride,
                                                      b.force, nullptr, 0u, b.H ? b.head_of : nullptr, b.head_xq);
}

}  // namespace

void launch_force(Batch& b) {
  prof_begin(b, SOUP_K_FORCE);
  launch_force_list(b);
  prof_end(b);
  if (b.H > 0) {
    prof_begin(b, SOUP_K_ES_FAR);
    launch_es_far(b);
    prof_end(b);
  }
}

// Lanes per particle: the result is the same bits, so the launch's size decides.  Few particles need the lanes
// to cover the gathers' latency; many need the fewest instructions, and rows of a chunk or two leave most lanes idle.
// Measured with 4 / 8 / 16 lanes, us: 6k beads 16.1 / 14.0 / 12.3, 10k 16.8 / 15.5 / 16.3, 24k 22.0 / 21.7 / 22.5, 30k
// 23.9 / 23.9 / 26.2, 40k 30.1 / 28.1 / 31.0, 60k 36.8 / 35.4 / 41.6, 80k 43.3 / 41.9 / 52.7, 100k 52.8 / 53.8 / 65.7,
// 121k 57.7 / 64.0 / 81.8 (another mix of kinds: 80k 40.5 / 41.4 / 46.4); rows of 24 entries: 20k 11.3 / 12.3 / 12.9,
// of 5: 60k 12.5 / 15.4 / 24.4, 3k 9.5 / 9.3 / 9.9; the 700 heads of a small system 31.6 / 22 / 13.5.
int force_lanes(const Batch& b, bool heads) {
  const int set = heads ? b.tpp_heads : b.tpp;
  const uint32_t n = heads ? b.H : b.N;
  if (set) return set <= 4 ? 4 : (set <= 8 ? 8 : 16);
  if (n >= 8192u && b.mean_row < 32.0) return 4;
  return n >= 80000u ? 4 : (n >= 28000u ? 8 : 16);
}

void launch_force_list(Batch& b, bool heads) {
  const uint32_t n = heads ? b.H : b.N;
  if (n == 0) return;
  b.launches += 1;
  switch (force_lanes(b, heads)) {
    case 4: launch_force_tpp<4>(b, heads); break;
    case 8: launch_force_tpp<8>(b, heads); break;
    default: launch_force_tpp<16>(b, heads); break;
  }
}

// after a charge sweep: only the heads' forces depend on charges (when only heads are charged and
// the polar class is the heads' kind alone), so they alone are recomputed, with the same arithmetic;
// timed with the sweep it completes (the force group keeps whole passes only)
void launch_force_heads(Batch& b) {
  prof_begin(b, SOUP_K_SWEEP);
  launch_force_list(b, true);
  if (b.H > 0) launch_es_far(b);
  prof_end(b);
}

void launch_es_far(Batch& b) {
  if (b.H == 0) return;
  b.launches += 1;
  k_es_far<<<nblocks((uint64_t)b.H * 32, 256), 256, 0, b.stream>>>(b.sp, b.head_slot, b.head_sys, b.H, b.head_xq,
                                                                   b.es_nl, b.es_cnt, b.es_cap, b.force);
}

void launch_force_brute(Batch& b) {
  b.launches += 1;
  k_force_brute<<<nblocks(b.N, 128), 128, 0, b.stream>>>(b.shared, b.sp, b.sysid, b.N, b.pos, b.charge, b.slots,
                                                         b.center, b.id, b.slot_of, b.force);
}

}  // namespace soup
