// kernels_bonds.cu -- dynamic-bond Monte Carlo, deterministic.
//
// Reference: soup/wgsl/bond-verlet.wgsl:12-54 (candidate walk over the Verlet list),
// soup/wgsl/bond-dispatch.wgsl:89-142 bondFormDecide and :170-200 bond_break_main,
// soup/wgsl/bond-valence.wgsl:40-116 (tryClaimSlot / releaseSlot / releasePartnerSlot),
// soup/wgsl/bond-adsorption.wgsl:62-316 (catalyst centre bookkeeping and the two desorption valves),
// soup/wgsl/bond-common.wgsl:111-168 (matchRule, roleOf, hasBondTo, bondPcg).
//
// The reference resolves slot and centre claims by CAS races between threads, so its outcome varies
// with scheduling.  The canonical semantics here (and in the CPU oracle) are the serial execution of
// the formation pass in ascending particle order.  It is computed in parallel, exactly:
//   Phase A (a warp per particle that can react): the candidate walk and both Metropolis draws.  Neither
//     depends on claim outcomes (a pair i<j is only ever formed by i; draws consume the particle's
//     own stream), so accept decisions and the final RNG state are computed here, in parallel.
//   Phase B (all SMs): every particle with an accepted proposal, every catalyst, every particle
//     holding a centre link, and every proposal partner becomes an "item".  Items whose particle
//     sets (self, partners, the catalyst found, and their current centre links) intersect are
//     joined by union-find; different components touch disjoint state, so they commute.  Inside a
//     component the items run in ascending index order: a thread runs a whole component, and the last block
//     to finish the large ones, an item of each per round.
//   Breaking is race-free in the reference (only the lower index of a bond draws for it) and runs
//     one thread per particle.
#include "soup_internal.h"

namespace soup {

namespace {

constexpr int kBlock = 256;
inline unsigned nblocks(uint64_t n, int b = kBlock) { return (unsigned)((n + b - 1) / b); }
constexpr uint32_t NONE = SOUP_NONE_U32;
constexpr int REC = 10;   // u32 per item record: i, catId, meta(nprop | rule<<(8+2c)), j[6], root

__device__ __forceinline__ int match_rule(const Shared& S, float ti, float tj) {
  for (int r = 0; r < 2; ++r) {   // BOND_RULES = 2 (bond-common.wgsl:41)
    const float a = S.kindA[r], b = S.kindB[r];
    if ((ti == a && tj == b) || (ti == b && tj == a)) return r;
  }
  return -1;
}

// the claims' state: per bead by original id, `next` per item; items of one component are a list from its root's
// head, `count` long
struct Claims { uint32_t *parent, *head, *count, *has_item, *next; };

// Phase A
// A bead whose kind is in no rule has no candidate, draws nothing and, unless it is a catalyst or
// tethered to one, leaves no item: its walk would change nothing (water, most of a campaign's beads).
__device__ __forceinline__ bool bond_active(const Shared& S, float ti, uint32_t centre) {
  bool in_rule = false;
  for (int r = 0; r < 2; ++r) in_rule = in_rule || ti == S.kindA[r] || ti == S.kindB[r];
  return in_rule || ti == S.cat_kind || centre != NONE;
}

// the active beads' slots, compacted (a warp's in one atomic); sel[0..*nsel) in no particular order.  It also
// clears what the claims keep per bead (by original id).
__global__ void __launch_bounds__(256) k_bond_select(const Shared* __restrict__ Sg, uint32_t N,
                                                     const float4* __restrict__ pos,
                                                     const uint32_t* __restrict__ center, uint32_t* __restrict__ sel,
                                                     uint32_t* __restrict__ nsel, Claims C) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < N) {
    C.parent[k] = k;
    C.head[k] = NONE;
    C.count[k] = 0;
    C.has_item[k] = 0;
  }
  const bool act = k < N && bond_active(*Sg, pos[k].w, center[k]);
  const uint32_t m = __ballot_sync(0xffffffffu, act);
  if (!m) return;
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t base = 0;
  if (lane == (uint32_t)(__ffs(m) - 1)) base = atomicAdd(nsel, (uint32_t)__popc(m));
  base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
  if (act) sel[base + __popc(m & ((1u << lane) - 1u))] = k;
}

// A warp per active bead (k_bond_select): the lanes test 32 row entries at a time, up to where the row can hold a
// pair in contact (list_force_end: contacts lie within the force's reach).  The few that qualify are kept by
// all lanes alike, the SOUP_CAND_CAP smallest ids in order.  (A thread per bead walked its row entry by
// entry, 200 us at 3k beads and 350 us at 483k, waiting on one gather after another.)
__global__ void __launch_bounds__(128) k_bond_walk(
    const Shared* __restrict__ Sg, const SysParams* __restrict__ sp, const uint8_t* __restrict__ sysid,
    const uint32_t* __restrict__ sel, const uint32_t* __restrict__ nsel,
    const float4* __restrict__ pos, const float* __restrict__ charge, const uint32_t* __restrict__ id,
    const uint32_t* __restrict__ slots, const uint32_t* __restrict__ center, const uint32_t* __restrict__ nl,
    const uint32_t* __restrict__ nl_cnt, const uint32_t* __restrict__ nl_shell, const uint32_t* __restrict__ drift_bits,
    uint32_t stride, uint32_t* __restrict__ brng, uint32_t* __restrict__ items, uint32_t* __restrict__ nitems,
    uint32_t* __restrict__ has_item) {
  const uint32_t ns = *nsel;
  if (blockIdx.x * 4u >= ns) return;   // the whole block: past the active beads
  __shared__ Shared S;
  for (int w = threadIdx.x; w < (int)(sizeof(Shared) / 4); w += blockDim.x)
    reinterpret_cast<uint32_t*>(&S)[w] = reinterpret_cast<const uint32_t*>(Sg)[w];
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t t = blockIdx.x * 4u + (threadIdx.x >> 5); t < ns; t += gridDim.x * 4u) {
    const uint32_t k = sel[t];
    const float4 xi = pos[k];
    const float ti = xi.w;
    const uint32_t rs = sysid[k];
    const SysParams& P = sp[rs];
    const float box[3] = {P.box[0], P.box[1], P.box[2]};
    const uint32_t gi = id[k];
    const uint32_t s0 = slots[3 * k], s1 = slots[3 * k + 1], s2 = slots[3 * k + 2];
    const float cat_reach = ex_wcut(S, ex_pairB(S, ti, S.cat_kind));
    uint32_t catId = NONE;
    uint32_t cj[SOUP_CAND_CAP], cr[SOUP_CAND_CAP];
#pragma unroll
    for (int c = 0; c < SOUP_CAND_CAP; ++c) { cj[c] = NONE; cr[c] = 0; }
    const uint32_t end = list_force_end(k, nl_cnt, nl_shell, __uint_as_float(drift_bits[rs]), P,
                                        list_wide(S, P, (int)ti & (SOUP_KMAX - 1), charge[k]));
    // the force reads whole chunks: entries of the next shells lie among those up to its end
    const uint32_t last = min((end + 15u) & ~15u, nl_cnt[k]);
    const uint32_t* row = nl + (size_t)k * stride;
    for (uint32_t b = 0; b < last; b += 32u) {
      const uint32_t s = b + lane;
      const uint32_t js = s < last ? row[s] : k;
      const float4 xj = pos[js];
      const float tj = xj.w;
      const bool isCat = js != k && tj == S.cat_kind;
      const int rk = js != k ? match_rule(S, ti, tj) : -1;
      uint32_t hit_j = NONE;
      if (isCat || rk >= 0) {
        const uint32_t j = id[js];
        const float d = ex_dist(xi, xj, box);
        if (isCat && d < cat_reach) catId = min(catId, j);                  // smallest catalyst in reach
        if (rk >= 0 && j > gi && s0 != j && s1 != j && s2 != j && d < ex_wcut(S, ex_pairB(S, ti, tj))) hit_j = j;
      }
      for (uint32_t m = __ballot_sync(0xffffffffu, hit_j != NONE); m; m &= m - 1u) {
        uint32_t j = __shfl_sync(0xffffffffu, hit_j, __ffs(m) - 1);
        uint32_t r = (uint32_t)__shfl_sync(0xffffffffu, rk, __ffs(m) - 1);
#pragma unroll
        for (int c = 0; c < SOUP_CAND_CAP; ++c)      // insert, ascending; the largest drops out
          if (j < cj[c]) {
            const uint32_t oj = cj[c], orr = cr[c];
            cj[c] = j; cr[c] = r;
            j = oj; r = orr;
          }
      }
    }
    catId = __reduce_min_sync(0xffffffffu, catId);
    // draws (bondFormDecide's candidate loop up to the claims), on every lane alike
    uint32_t rng = brng[k];
    uint32_t pj[SOUP_CAND_CAP];
    uint32_t meta = 0;
    int np = 0;
#pragma unroll
    for (int c = 0; c < SOUP_CAND_CAP; ++c) {
      pj[c] = NONE;
      if (cj[c] == NONE) continue;
      const uint32_t r = cr[c];
      if (S.req_cat[r] > 0.5f && catId == NONE) continue;
      rng = pcg_hash(rng);
      if (u01(rng) >= S.att_form[r]) continue;
      rng = pcg_hash(rng);
      if (u01(rng) >= S.acc_form[r]) continue;
      pj[c] = cj[c];
      meta |= r << (8 + 2 * np);
      ++np;
    }
    if (lane == 0) {
      brng[k] = rng;
      if (np > 0 || ti == S.cat_kind || center[k] != NONE) {
        const uint32_t at = atomicAdd(nitems, 1u);
        uint32_t* rec = items + (size_t)at * REC;
        rec[0] = gi; rec[1] = catId; rec[2] = meta | (uint32_t)np;
        int n = 0;
#pragma unroll
        for (int c = 0; c < SOUP_CAND_CAP; ++c)
          if (pj[c] != NONE) rec[3 + n++] = pj[c];
        for (; n < SOUP_CAND_CAP; ++n) rec[3 + n] = NONE;
        has_item[gi] = 1;
      }
    }
  }
}

// ---- Phase B helpers: the serial body of bondFormDecide on global state ----
struct St {
  const Shared& S;
  const SysParams* sp;
  const uint8_t* sysid;
  const float4* pos;
  uint32_t* slots;
  uint32_t* center;
  uint32_t* held;
  const uint32_t* slot_of;
  uint32_t* events;
  uint32_t* desorb;

  __device__ uint32_t sl(uint32_t g) const { return slot_of[g]; }
  __device__ float kind(uint32_t g) const { return pos[sl(g)].w; }
  __device__ float dist(uint32_t a, uint32_t b) const {
    const SysParams& P = sp[sysid[sl(a)]];
    return ex_dist(pos[sl(a)], pos[sl(b)], P.box);
  }
  __device__ bool cas(uint32_t p, uint32_t e, uint32_t v) {
    uint32_t* c = &center[sl(p)];
    if (*c != e) return false;
    *c = v;
    return true;
  }
  __device__ float cat_contact(uint32_t a) const { return ex_wcut(S, ex_pairB(S, kind(a), S.cat_kind)); }
  // bond-valence.wgsl:40-98
  __device__ int claim(uint32_t p, uint32_t role, uint32_t partner) {
    uint32_t* s = &slots[3 * sl(p)];
    const bool term = S.head_terminal > 0.5f;
    if (role == 0) {
      if (s[0] == NONE) { s[0] = partner; if (term && s[2] != NONE) { s[0] = NONE; return -1; } return 0; }
      if (s[1] == NONE) { s[1] = partner; if (term && s[2] != NONE) { s[1] = NONE; return -1; } return 1; }
      return -1;
    } else if (role == 1) {
      if (s[2] == NONE) { s[2] = partner; if (term && s[0] != NONE && s[1] != NONE) { s[2] = NONE; return -1; } return 2; }
      return -1;
    }
    const uint32_t capc = (uint32_t)S.head_cap;
    for (uint32_t c = 0; c < capc; ++c) if (s[c] == NONE) { s[c] = partner; return (int)c; }
    return -1;
  }
  __device__ void release(uint32_t p, int slot) { if (slot >= 0) slots[3 * sl(p) + slot] = NONE; }
  __device__ bool within_reach(uint32_t a, uint32_t b) const { return dist(a, b) < __fadd_rn(cat_contact(a), S.wc); }
  // bond-adsorption.wgsl:87-248
  __device__ bool propagate(uint32_t i, uint32_t j, int sI, int sJ, uint32_t cat) {
    if (sI == 0 && sJ == 0) {
      if (cat == NONE) return false;
      if (dist(i, cat) >= cat_contact(i)) return false;
      if (!cas(cat, NONE, i)) return false;
      if (!cas(i, NONE, cat)) { cas(cat, i, NONE); return false; }
      held[sl(cat)] = 0;
      return true;
    }
    uint32_t tipOld, tipNew;
    if (sI == 1 && sJ == 0) { tipOld = i; tipNew = j; }
    else if (sI == 0 && sJ == 1) { tipOld = j; tipNew = i; }
    else return false;
    uint32_t owner = center[sl(tipOld)];
    bool reclaim = false;
    if (owner == NONE) { if (cat == NONE) return false; owner = cat; reclaim = true; }
    if (reclaim) { if (dist(tipOld, cat) >= cat_contact(tipOld)) return false; }
    else if (!within_reach(tipOld, owner)) return false;
    if (dist(tipNew, owner) >= cat_contact(tipNew)) return false;
    if (reclaim) {
      if (!cas(owner, NONE, tipOld)) return false;
      if (!cas(tipOld, NONE, owner)) { cas(owner, tipOld, NONE); return false; }
    }
    if (!cas(owner, tipOld, tipNew)) { if (reclaim) cas(tipOld, owner, NONE); return false; }
    if (!cas(tipNew, NONE, owner)) {
      cas(owner, tipNew, tipOld);
      if (reclaim) { cas(owner, tipOld, NONE); cas(tipOld, owner, NONE); }
      return false;
    }
    cas(tipOld, owner, NONE);
    held[sl(owner)] = 0;
    return true;
  }
  // bond-adsorption.wgsl:256-268
  __device__ bool terminate(uint32_t carbon) {
    const uint32_t owner = center[sl(carbon)];
    if (owner == NONE) return false;
    if (!within_reach(carbon, owner)) return false;
    if (!cas(carbon, owner, NONE)) return false;
    cas(owner, carbon, NONE);
    held[sl(owner)] = 0;
    return true;
  }
  // the whole item: desorption valve, then the accepted proposals in order
  __device__ void run(const uint32_t* rec) {
    const uint32_t i = rec[0], cat = rec[1], meta = rec[2];
    const int np = (int)(meta & 0xFFu);
    const uint32_t ks = sl(i);
    const uint32_t rs = sysid[ks];
    const float ti = pos[ks].w;
    if (ti == S.cat_kind) {                               // desorbTimeout (bond-adsorption.wgsl:304-316)
      const uint32_t tip = center[ks];
      if (tip != NONE) {
        const uint32_t inc = (uint32_t)S.interval;
        const uint32_t prev = held[ks];
        held[ks] = prev + inc;
        if (prev + inc > (uint32_t)S.max_hold) {
          if (cas(i, tip, NONE)) { cas(tip, i, NONE); held[ks] = 0; atomicAdd(&desorb[2 * rs + 1], 1u); }
        }
      }
    } else {
      const uint32_t owner = center[ks];                  // desorbStretch (bond-adsorption.wgsl:283-292)
      if (owner != NONE && dist(i, owner) >= S.r_inf) {
        if (cas(i, owner, NONE)) { cas(owner, i, NONE); held[sl(owner)] = 0; atomicAdd(&desorb[2 * rs + 0], 1u); }
      }
    }
    for (int c = 0; c < np; ++c) {
      const uint32_t j = rec[3 + c];
      const uint32_t r = (meta >> (8 + 2 * c)) & 3u;
      const float tj = kind(j);
      const uint32_t roleI = (ti == S.kindA[r]) ? (uint32_t)S.roleA[r] : (uint32_t)S.roleB[r];
      const uint32_t roleJ = (tj == S.kindA[r]) ? (uint32_t)S.roleA[r] : (uint32_t)S.roleB[r];
      const int sI = claim(i, roleI, j);
      if (sI < 0) continue;
      const int sJ = claim(j, roleJ, i);
      if (sJ < 0) { release(i, sI); continue; }
      bool ok;
      if (roleI == 0 && roleJ == 0) ok = propagate(i, j, sI, sJ, cat);
      else if (roleI == 1) ok = terminate(i);
      else ok = terminate(j);
      if (!ok) { release(i, sI); release(j, sJ); continue; }
      atomicAdd(&events[2 * SOUP_MAX_RULES * rs + 2 * r], 1u);   // components run concurrently
    }
  }
};

__device__ __forceinline__ uint32_t uf_find(uint32_t* parent, uint32_t x) {
  volatile uint32_t* vp = parent;
  uint32_t p = vp[x];
  while (p != x) { x = p; p = vp[x]; }
  return x;
}
__device__ __forceinline__ void uf_union(uint32_t* parent, uint32_t a, uint32_t b) {
  for (;;) {
    a = uf_find(parent, a);
    b = uf_find(parent, b);
    if (a == b) return;
    if (a > b) { uint32_t t = a; a = b; b = t; }
    if (atomicCAS(&parent[b], b, a) == b) return;   // hook the larger root under the smaller
  }
}

// the particles an item may touch, as far as the pass-start state can tell (closure under centre links)
__device__ __forceinline__ int item_set(const uint32_t* rec, const uint32_t* center, const uint32_t* slot_of,
                                        uint32_t* out) {
  int n = 0;
  auto add = [&](uint32_t g) {
    if (g == NONE) return;
    out[n++] = g;
    const uint32_t c = center[slot_of[g]];
    if (c != NONE) out[n++] = c;
  };
  add(rec[0]);
  add(rec[1]);
  const int np = (int)(rec[2] & 0xFFu);
  for (int c = 0; c < np; ++c) add(rec[3 + c]);
  return n;
}

// Phase B.  Every particle an item may touch runs its own desorption check in its turn, so it needs
// an item too (proposal partners are the only ones the walk does not already cover): added here, by
// the whole grid, before the claims.
// nitems[1] holds the walk's item count: only the walk's items add partners (nitems[0] grows meanwhile).  Items whose
// particle sets meet are joined on the way (union-find over the sets closed under centre links).
__global__ void k_bond_partners(const uint32_t* __restrict__ center, const uint32_t* __restrict__ slot_of,
                                uint32_t* __restrict__ items, uint32_t* __restrict__ nitems, uint32_t item_cap, Claims C,
                                uint32_t* __restrict__ flags) {
  const uint32_t M0 = min(nitems[1], item_cap);
  uint32_t setbuf[2 * (2 + SOUP_CAND_CAP)];
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < M0; t += gridDim.x * blockDim.x) {
    const int n = item_set(items + (size_t)t * REC, center, slot_of, setbuf);
    for (int q = 0; q < n; ++q) {
      const uint32_t x = setbuf[q];
      if (q) uf_union(C.parent, setbuf[0], x);
      if (atomicCAS(&C.has_item[x], 0u, 1u) == 0u) {
        const uint32_t at = atomicAdd(nitems, 1u);
        if (at < item_cap) {
          uint32_t* nr = items + (size_t)at * REC;
          nr[0] = x; nr[1] = NONE; nr[2] = 0;
          for (int c = 0; c < SOUP_CAND_CAP; ++c) nr[3 + c] = NONE;
          const uint32_t cx = center[slot_of[x]];
          if (cx != NONE) uf_union(C.parent, x, cx);
        } else {
          flags[6] = 1u;
        }
      }
    }
  }
}

// the components' lists of items, in no particular order
__global__ void k_bond_lists(uint32_t* __restrict__ items, const uint32_t* __restrict__ nitems, uint32_t item_cap, Claims C) {
  const uint32_t M = min(*nitems, item_cap);
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < M; t += gridDim.x * blockDim.x) {
    const uint32_t root = uf_find(C.parent, items[(size_t)t * REC]);
    items[(size_t)t * REC + 9] = root;
    C.next[t] = atomicExch(&C.head[root], t);
    atomicAdd(&C.count[root], 1u);
  }
}

// Phase B, the claims: the items of a component in ascending order of their ids, which is all that the serial order
// decides (components touch disjoint particles).  A thread runs a component of up to kClaimSerial items, its
// list sorted first; eight threads of a warp work, so that components of unequal length hold up few others.  The
// items of larger components are left to the last block to finish, which runs them in rounds: of every
// component the pending item with the smallest id.
// Bound: the chain of gathers of an item.  (One CTA a replica ran all of them: 549 us at 483k beads, 31 now and 6 for
// the lists.)
constexpr uint32_t kClaimSerial = 24;
__global__ void __launch_bounds__(256) k_bond_claims(
    const Shared* __restrict__ Sg, const SysParams* __restrict__ sp, const uint8_t* __restrict__ sysid,
    const float4* __restrict__ pos, uint32_t* __restrict__ slots, uint32_t* __restrict__ center,
    uint32_t* __restrict__ held, const uint32_t* __restrict__ slot_of, const uint32_t* __restrict__ items,
    uint32_t* __restrict__ nitems, uint32_t item_cap, Claims C, uint32_t* __restrict__ large,
    uint32_t* __restrict__ events, uint32_t* __restrict__ desorb) {
  __shared__ bool last;
  const uint32_t M = min(*nitems, item_cap);
  St st{*Sg, sp, sysid, pos, slots, center, held, slot_of, events, desorb};
  if ((threadIdx.x & 3u) == 0) {
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; t < M; t += (gridDim.x * blockDim.x) >> 2) {
      const uint32_t* rec = items + (size_t)t * REC;
      const uint32_t root = rec[9], n = C.count[root];
      if (n > kClaimSerial) {
        large[atomicAdd(&nitems[3], 1u)] = t;
      } else if (n == 1) {
        st.run(rec);
      } else if (C.head[root] == t) {
        uint32_t at[kClaimSerial], key[kClaimSerial];
        uint32_t m = 0;
        for (uint32_t u = t; u != NONE; u = C.next[u], ++m) {
          const uint32_t id = items[(size_t)u * REC];
          uint32_t p = m;
          for (; p > 0 && key[p - 1] > id; --p) { key[p] = key[p - 1]; at[p] = at[p - 1]; }
          key[p] = id;
          at[p] = u;
        }
        for (uint32_t p = 0; p < m; ++p) st.run(items + (size_t)at[p] * REC);
      }
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&nitems[4], 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const uint32_t L = *(volatile uint32_t*)&nitems[3];
  volatile uint32_t* big = large;
  volatile uint32_t* low = C.head;                       // by root: the smallest pending id
  for (uint32_t u = threadIdx.x; u < L; u += blockDim.x) low[items[(size_t)big[u] * REC + 9]] = NONE;
  for (;;) {
    int pending = 0;
    __syncthreads();
    for (uint32_t u = threadIdx.x; u < L; u += blockDim.x) {
      const uint32_t t = big[u];
      if (t == NONE) continue;
      pending = 1;
      atomicMin(&C.head[items[(size_t)t * REC + 9]], items[(size_t)t * REC]);
    }
    if (!__syncthreads_or(pending)) break;
    for (uint32_t u = threadIdx.x; u < L; u += blockDim.x) {
      const uint32_t t = big[u];
      if (t == NONE) continue;
      const uint32_t* rec = items + (size_t)t * REC;
      if (low[rec[9]] == rec[0]) { st.run(rec); big[u] = NONE; }
    }
    __syncthreads();
    for (uint32_t u = threadIdx.x; u < L; u += blockDim.x) {
      const uint32_t t = big[u];
      if (t != NONE) low[items[(size_t)t * REC + 9]] = NONE;
    }
  }
}

// bond-dispatch.wgsl:170-200 bond_break_main
__global__ void k_bond_break(const Shared* __restrict__ Sg, const uint8_t* __restrict__ sysid, uint32_t N,
                             const float4* __restrict__ pos, const uint32_t* __restrict__ id,
                             const uint32_t* __restrict__ slot_of, uint32_t* __restrict__ slots,
                             uint32_t* __restrict__ brng, uint32_t* __restrict__ events) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= N) return;
  const Shared& S = *Sg;
  const uint32_t gi = id[k];
  const float ti = pos[k].w;
  uint32_t rng = brng[k];
  bool touched = false;
  for (int s = 0; s < 3; ++s) {
    const uint32_t partner = slots[3 * k + s];
    if (partner == NONE || partner < gi) continue;
    const uint32_t ps = slot_of[partner];
    const int r = match_rule(S, ti, pos[ps].w);
    if (r < 0) continue;
    touched = true;
    rng = pcg_hash(rng);
    if (u01(rng) >= S.att_break[r]) continue;
    rng = pcg_hash(rng);
    if (u01(rng) >= S.acc_break[r]) continue;
    slots[3 * k + s] = NONE;
    for (int t = 0; t < 3; ++t) {
      if (atomicCAS(&slots[3 * ps + t], gi, NONE) == gi) break;
    }
    atomicAdd(&events[2 * SOUP_MAX_RULES * sysid[k] + 2 * r + 1], 1u);
  }
  if (touched) brng[k] = rng;
}

}  // namespace

void launch_bonds(Batch& b) {
  b.launches += 6;
  prof_begin(b, SOUP_K_BONDS);
  const Claims C{b.uf_parent, b.comp_head, b.comp_count, b.has_item, b.item_next};
  cudaMemsetAsync(b.bond_nitems, 0, 5 * sizeof(uint32_t), b.stream);
  k_bond_select<<<nblocks(b.N, 256), 256, 0, b.stream>>>(b.shared, b.N, b.pos, b.center, b.bond_sel,
                                                         b.bond_nitems + 2, C);
  k_bond_walk<<<std::min(nblocks(b.N, 4), 148u * 16u), 128, 0, b.stream>>>(
      b.shared, b.sp, b.sysid, b.bond_sel, b.bond_nitems + 2, b.pos, b.charge, b.id, b.slots, b.center, b.nl, b.nl_cnt,
      b.prune ? b.nl_shell : nullptr, b.drift_bits, b.list_stride, b.brng, b.bond_items, b.bond_nitems, b.has_item);
  cudaMemcpyAsync(b.bond_nitems + 1, b.bond_nitems, sizeof(uint32_t), cudaMemcpyDeviceToDevice, b.stream);
  const unsigned over_items = std::max(1u, std::min(nblocks(b.N, 256) / 8u, 592u));
  k_bond_partners<<<over_items, 256, 0, b.stream>>>(b.center, b.slot_of, b.bond_items, b.bond_nitems, b.N, C, b.flags);
  k_bond_lists<<<over_items, 256, 0, b.stream>>>(b.bond_items, b.bond_nitems, b.N, C);
  // (the walk is over: its selection's buffer takes the large components' items)
  k_bond_claims<<<std::min(nblocks(b.N, 256), 592u), 256, 0, b.stream>>>(
      b.shared, b.sp, b.sysid, b.pos, b.slots, b.center, b.held, b.slot_of, b.bond_items, b.bond_nitems, b.N, C, b.bond_sel,
      b.events, b.desorb);
  k_bond_break<<<nblocks(b.N), kBlock, 0, b.stream>>>(b.shared, b.sysid, b.N, b.pos, b.id, b.slot_of, b.slots,
                                                      b.brng, b.events);
  prof_end(b);
}

}  // namespace soup
