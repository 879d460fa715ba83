// kernels_grid.cu -- cell binning, the deterministic re-sort, and the Verlet / head list builds.
//
// Reference: engine/wgsl/neighbor.wgsl:19-64 (clear/count/prefix/fill: an atomic counting sort with a
// one-thread prefix sum and an atomic, run-to-run varying fill order), soup/wgsl/verlet.wgsl:53-92
// (per-particle walk of (2R+1)^3 cells, keep |mi3(xi-xj)| < listRange), soup/wgsl/
// electrostatics-long.wgsl:15-56 (serial head compaction, O(N_h^2) head list).
//
// Here: a parallel counting sort whose order inside a cell is fixed (ascending original index), so
// every array is physically reordered into cell order at each rebuild (coalesced neighbour reads);
// list membership uses the exact f32 test of the reference, so the lists equal the oracle's sets.
// Walks are over x-rows of cells (contiguous slot ranges), a row at a time.
#include <type_traits>

#include "soup_internal.h"

namespace soup {

namespace {

constexpr int kBlock = 256;
inline unsigned nblocks(uint64_t n, int b = kBlock) { return (unsigned)((n + b - 1) / b); }

__global__ void k_cell_index(const float4* __restrict__ pos, const uint8_t* __restrict__ sysid,
                             const SysParams* __restrict__ sp, uint32_t N, uint32_t* __restrict__ cell_of,
                             uint32_t* __restrict__ count) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= N) return;
  const SysParams& P = sp[sysid[k]];
  float4 p = pos[k];
  int cx = ex_cell_axis(p.x, P.box[0], P.dims[0]);
  int cy = ex_cell_axis(p.y, P.box[1], P.dims[1]);
  int cz = ex_cell_axis(p.z, P.box[2], P.dims[2]);
  uint32_t c = P.cell_off + (uint32_t)(cx + P.dims[0] * (cy + P.dims[1] * cz));
  cell_of[k] = c;
  atomicAdd(&count[c], 1u);
}

// Exclusive scan, 4 elements per thread, 1024 threads per block: block-local scan + block totals.
__global__ void k_scan_block(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t n,
                             uint32_t* __restrict__ block_sums) {
  __shared__ uint32_t warp_tot[32];
  const uint32_t base = blockIdx.x * 4096u + threadIdx.x * 4u;
  uint32_t v[4];
  uint32_t t = 0;
  for (int e = 0; e < 4; ++e) { v[e] = (base + e < n) ? in[base + e] : 0u; t += v[e]; }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t incl = t;
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  if (w == 0) {
    uint32_t x = warp_tot[lane];
    uint32_t xi = x;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, xi, o);
      if (lane >= o) xi += y;
    }
    warp_tot[lane] = xi - x;  // exclusive
    if (lane == 31 && block_sums) block_sums[blockIdx.x] = xi;
  }
  __syncthreads();
  uint32_t run = warp_tot[w] + incl - t;
  for (int e = 0; e < 4; ++e) {
    if (base + e < n) out[base + e] = run;
    run += v[e];
  }
}
// The blocks' offsets added, a block of threads per scanned block, and the total behind the last.  RAW: `sums` are
// the blocks' own totals (at most 1024), and each block of threads adds up those before it; otherwise their scan.
template <bool RAW>
__global__ void __launch_bounds__(1024) k_scan_add(uint32_t* __restrict__ out, uint32_t n, const uint32_t* __restrict__ sums) {
  __shared__ uint32_t before;
  if (threadIdx.x == 0) before = RAW ? 0u : sums[blockIdx.x];
  __syncthreads();
  if (RAW) {
    const uint32_t v = __reduce_add_sync(0xffffffffu, threadIdx.x < blockIdx.x ? sums[threadIdx.x] : 0u);
    if ((threadIdx.x & 31u) == 0 && v) atomicAdd(&before, v);
    __syncthreads();
  }
  const uint32_t off = before;
#pragma unroll
  for (uint32_t e = 0; e < 4u; ++e) {
    const uint32_t i = blockIdx.x * 4096u + e * 1024u + threadIdx.x;
    if (i < n) out[i] += off;
  }
  if (threadIdx.x == 0 && blockIdx.x + 1u == gridDim.x) out[n] = RAW ? off + sums[blockIdx.x] : sums[gridDim.x];
}

}  // namespace

// exclusive scan of in[0..n) into out[0..n), out[n] = total; tmp must hold >= 2*ceil(n/4096)+2 words.
// One launch to 4096 words, two to 4M (a rebuild of a small system is a chain of launches of 2 us each), and
// beyond that, where a block's offset would be a sum of more than 1024 totals, the totals are scanned first.
// With two, five and more launches, and memsets of their own for the cursors and the head cells, a force
// evaluation of 1,220 beads took 112 us (99 now) and ten steps of 3,277 beads 412 (398).
// Returns the kernels it launched (no shared counter: calls from several host threads do not race).
uint64_t exclusive_scan(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* tmp, cudaStream_t st) {
  if (n == 0) return 0;
  const uint32_t nb = (n + 4095) / 4096;
  if (nb == 1) {
    k_scan_block<<<1, 1024, 0, st>>>(in, out, n, out + n);
    return 1;
  }
  uint32_t* sums = tmp;
  k_scan_block<<<nb, 1024, 0, st>>>(in, out, n, sums);
  if (nb <= 1024) {
    k_scan_add<true><<<nb, 1024, 0, st>>>(out, n, sums);
    return 2;
  }
  uint32_t* offs = tmp + nb + 1;
  const uint64_t launches = exclusive_scan(sums, offs, nb, offs + nb + 1, st);
  k_scan_add<false><<<nb, 1024, 0, st>>>(out, n, offs);
  return launches + 2;
}

namespace {

__global__ void k_scatter(const uint32_t* __restrict__ cell_of, const uint32_t* __restrict__ start, uint32_t N,
                          uint32_t* __restrict__ count, uint32_t* __restrict__ perm) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= N) return;
  uint32_t c = cell_of[k];
  perm[start[c] + atomicSub(&count[c], 1u) - 1u] = k;   // the counts count the places down
}

// Inside each cell, order by original index: the atomic scatter order above varies run to run, this
// makes the slot order (and therefore every summation order) deterministic.
__global__ void k_sort_cells(const uint32_t* __restrict__ start, uint32_t ncells, const uint32_t* __restrict__ id,
                             uint32_t* __restrict__ perm) {
  uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  uint32_t a = start[c], e = start[c + 1];
  for (uint32_t x = a + 1; x < e; ++x) {
    uint32_t v = perm[x];
    uint32_t key = id[v];
    uint32_t y = x;
    while (y > a && id[perm[y - 1]] > key) { perm[y] = perm[y - 1]; --y; }
    perm[y] = v;
  }
}

__global__ void k_gather(uint32_t N, const uint32_t* __restrict__ perm,
                         const float4* __restrict__ pos, const float4* __restrict__ vel, const float4* __restrict__ force,
                         const float* __restrict__ charge, const uint32_t* __restrict__ slots,
                         const uint32_t* __restrict__ center, const uint32_t* __restrict__ held,
                         const uint32_t* __restrict__ brng, const uint32_t* __restrict__ trng,
                         const uint8_t* __restrict__ frozen, const uint32_t* __restrict__ id,
                         float4* __restrict__ pos2, float4* __restrict__ vel2, float4* __restrict__ force2,
                         float* __restrict__ charge2, uint32_t* __restrict__ slots2, uint32_t* __restrict__ center2,
                         uint32_t* __restrict__ held2, uint32_t* __restrict__ brng2, uint32_t* __restrict__ trng2,
                         uint8_t* __restrict__ frozen2, uint32_t* __restrict__ id2, uint32_t* __restrict__ slot_of,
                         float4* __restrict__ pos_ref) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= N) return;
  uint32_t o = perm[k];
  float4 p = pos[o];
  pos2[k] = p;
  pos_ref[k] = p;
  vel2[k] = vel[o];
  force2[k] = force[o];
  charge2[k] = charge[o];
  slots2[3 * k + 0] = slots[3 * o + 0];
  slots2[3 * k + 1] = slots[3 * o + 1];
  slots2[3 * k + 2] = slots[3 * o + 2];
  center2[k] = center[o];
  held2[k] = held[o];
  brng2[k] = brng[o];
  trng2[k] = trng[o];
  frozen2[k] = frozen[o];
  uint32_t g = id[o];
  id2[k] = g;
  slot_of[g] = k;
}

// the gathered arrays back into the primary buffers, so every array keeps its address across rebuilds
// (a captured step graph holds them as kernel arguments).  The replicas' drifts are zeroed here (a memset of its own
// is a launch)
__global__ void k_copy_back(uint32_t N, const float4* __restrict__ pos2, const float4* __restrict__ vel2,
                            const float4* __restrict__ force2, const float* __restrict__ charge2,
                            const uint32_t* __restrict__ slots2, const uint32_t* __restrict__ center2,
                            const uint32_t* __restrict__ held2, const uint32_t* __restrict__ brng2,
                            const uint32_t* __restrict__ trng2, const uint8_t* __restrict__ frozen2,
                            const uint32_t* __restrict__ id2, float4* __restrict__ pos, float4* __restrict__ vel,
                            float4* __restrict__ force, float* __restrict__ charge, uint32_t* __restrict__ slots,
                            uint32_t* __restrict__ center, uint32_t* __restrict__ held, uint32_t* __restrict__ brng,
                            uint32_t* __restrict__ trng, uint8_t* __restrict__ frozen, uint32_t* __restrict__ id,
                            uint32_t* __restrict__ head_of, uint32_t R, uint32_t* __restrict__ drift_bits) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= N) return;
  if (k < R) drift_bits[k] = 0u;   // a replica has a bead at least
  head_of[k] = SOUP_NONE_U32;   // k_head_index names the heads
  pos[k] = pos2[k]; vel[k] = vel2[k]; force[k] = force2[k]; charge[k] = charge2[k];
  slots[3 * k] = slots2[3 * k]; slots[3 * k + 1] = slots2[3 * k + 1]; slots[3 * k + 2] = slots2[3 * k + 2];
  center[k] = center2[k]; held[k] = held2[k]; brng[k] = brng2[k]; trng[k] = trng2[k]; frozen[k] = frozen2[k];
  id[k] = id2[k];
}

// At most two [lo,hi] intervals of cells along one axis.
struct AxisRange { int lo[2], hi[2], n; };

// The cells lo..hi (unwrapped, hi - lo + 1 <= dim) as at most two wrapped [lo,hi] intervals.
__device__ __forceinline__ AxisRange span_ranges(int lo, int hi, int dim) {
  AxisRange a;
  if (lo < 0) { a.n = 2; a.lo[0] = lo + dim; a.hi[0] = dim - 1; a.lo[1] = 0; a.hi[1] = hi; }
  else if (hi >= dim) { a.n = 2; a.lo[0] = lo; a.hi[0] = dim - 1; a.lo[1] = 0; a.hi[1] = hi - dim; }
  else { a.n = 1; a.lo[0] = lo; a.hi[0] = hi; }
  if (a.n == 2 && a.lo[1] > a.hi[1]) a.n = 1;
  if (a.n == 2 && a.lo[0] > a.hi[0]) { a.n = 1; a.lo[0] = a.lo[1]; a.hi[0] = a.hi[1]; }
  return a;
}
// distance from p to the cell interval [c cs, (c + 1) cs) along one axis (unwrapped c), less a
// margin for the rounding of the cell assignment
__device__ __forceinline__ float gap_to_cell(float p, int c, float cs) {
  const float lo = (float)c * cs - p, hi = (float)(c + 1) * cs - p;
  return fmaxf(0.f, fmaxf(lo, -hi) - 1e-4f);
}

// The build-distance shell of a list entry, carried in its top three bits until its row is grouped: 0
// inside the force's reach, 1..7 the rest of the list range (list_shell_width2).  A force pass needs shell
// s > 0 only once the largest displacement since the build can have closed the distance from the reach to
// that shell's inner edge (list_force_end).
struct Shells {
  float mul, add;                                        // r2 mul + add = (shell + fraction) / kShells
  __device__ __forceinline__ static Shells of(float reach2, float list_range) {
    const float scale = 1.0f / fmaxf(list_shell_width2(reach2, list_range), 1e-12f);
    return Shells{scale * (1.0f / kShells), (1.0f - reach2 * scale) * (1.0f / kShells)};
  }
  // (a shell edge may fall to either side by rounding: list_force_end's margin is far wider)
  __device__ __forceinline__ uint32_t tag(float r2) const {
    const float x = __saturatef(fmaf(r2, mul, add));
    return __float_as_uint(__fmaf_rz(x, (float)kShells * 0.999999f, 8388608.0f)) << 29;   // floor in the low bits
  }
};

// ---- the neighbour walk of one particle by a warp -------------------------------------------------
// The cells within the walk radius of a particle's cell form rows along x, and the beads of a row (they are
// in cell order) one or two contiguous runs.  The lanes take a row each: the runs trimmed to the x cells that
// can reach the list sphere, rows wholly beyond it dropped, and an axis on which the walk would wrap onto
// itself visited once, whole.  The runs then make one flat sequence of candidates, and the warp takes 32 of
// them at a time whatever run they lie in, so every lane has work but in the last 32.  (A run holds about 20
// candidates: run by run, half the lanes would idle; a thread per particle diverges at every accepted
// candidate and leaves a small system's chain of dependent loads uncovered.)
constexpr uint32_t kWalkRuns = 128;                    // runs: two per row, (2 * 3 + 1)^2 rows at walk 3
constexpr uint32_t kWalkSpan = 2048;                   // candidates whose run starts are marked at a time
constexpr uint32_t kWalkWords = 2 * kWalkRuns + 2 * kWalkSpan / 32;   // shared words a warp's walk needs

struct WalkGrid { int dims[3]; int walk, walk_x; uint32_t cell_off; float range; float cell[3]; float inv_cell_x; };

__device__ __forceinline__ float sqrt_approx(float x) {   // under the walk's margins
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// take(j0, j1): warp-wide, 2 x 32 candidates (indices into the cell-ordered array; self: the walk's own bead there)
template <class Take>
__device__ __forceinline__ void warp_walk(const float4& xi, uint32_t self, const float* box, const WalkGrid& G,
                                          const uint32_t* __restrict__ start, uint32_t* __restrict__ sm, Take&& take) {
  uint32_t* shift = sm;                                // candidate q of run s is bead q + shift[s]
  uint32_t* first = sm + kWalkRuns;                    // its first candidate
  uint2* mark = reinterpret_cast<uint2*>(sm + 2 * kWalkRuns);   // per 32 candidates: a bit where a run starts; the
                                                       // runs that start before them, less one
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u, le = lt | (1u << lane);
  const int R = G.walk, D = 2 * R + 1, Rx = G.walk_x;
  const int dx = G.dims[0], dy = G.dims[1], dz = G.dims[2];
  const int qx = ex_cell_axis(xi.x, box[0], dx), qy = ex_cell_axis(xi.y, box[1], dy), qz = ex_cell_axis(xi.z, box[2], dz);
  const bool fx = dx < 2 * Rx + 1, fy = dy < D, fz = dz < D;    // this axis is visited whole
  const int ny = fy ? dy : D, nz = fz ? dz : D;
  const float csy = G.cell[1], csz = G.cell[2], icx = G.inv_cell_x;
  const float lrm = G.range * (1.0f + 1e-5f) + 1e-3f, lrm2 = lrm * lrm;
  uint32_t runs = 0, total = 0;
  for (int r0 = 0; r0 < ny * nz; r0 += 32) {
    const int rr = r0 + (int)lane;
    uint32_t a0 = 0, l0 = 0, a1 = 0, l1 = 0;
    if (rr < ny * nz) {
      const int iz = ny == 5 ? (rr * 205) >> 10 : rr / ny, iy = rr - iz * ny;   // rr < 51 where ny is 5
      const int y = fy ? iy : qy - R + iy, z = fz ? iz : qz - R + iz;
      const float gy = fy ? 0.f : gap_to_cell(xi.y, y, csy), gz = fz ? 0.f : gap_to_cell(xi.z, z, csz);
      const float g2 = gy * gy + gz * gz;
      if (g2 < lrm2) {
        const int wy = y < 0 ? y + dy : (y >= dy ? y - dy : y), wz = z < 0 ? z + dz : (z >= dz ? z - dz : z);
        const uint32_t row = G.cell_off + (uint32_t)(dx * (wy + dy * wz));
        if (fx) {
          a0 = start[row];
          l0 = start[row + (uint32_t)dx] - a0;
        } else {
          const float ext = sqrt_approx(lrm2 - g2) + 1e-3f;
          const int xlo = max(qx - Rx, (int)floorf((xi.x - ext) * icx)), xhi = min(qx + Rx, (int)floorf((xi.x + ext) * icx));
          if (xlo <= xhi) {
            const AxisRange xr = span_ranges(xlo, xhi, dx);
            a0 = start[row + (uint32_t)xr.lo[0]];
            l0 = start[row + (uint32_t)xr.hi[0] + 1] - a0;
            if (xr.n == 2) {
              a1 = start[row + (uint32_t)xr.lo[1]];
              l1 = start[row + (uint32_t)xr.hi[1] + 1] - a1;
            }
          }
        }
      }
    }
    uint32_t incl = l0 + l1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (uint32_t)o) incl += v;
    }
    const uint32_t at = total + incl - (l0 + l1);
    const uint32_t b0 = __ballot_sync(0xffffffffu, l0 != 0), b1 = __ballot_sync(0xffffffffu, l1 != 0);
    uint32_t s = runs + __popc(b0 & lt) + __popc(b1 & lt);
    if (l0) { shift[s] = a0 - at; first[s] = at; ++s; }
    if (l1) { shift[s] = a1 - (at + l0); first[s] = at + l0; }
    runs += __popc(b0) + __popc(b1);
    total += __shfl_sync(0xffffffffu, incl, 31);
  }
  __syncwarp();
  uint32_t before = 0xFFFFFFFFu;                       // the runs that start before the span, less one
  for (uint32_t w0 = 0; w0 < total; w0 += kWalkSpan) {
    const uint32_t n = min(total - w0, kWalkSpan), words = (n + 63u) / 64u * 2u;
    for (uint32_t i = lane; i < words; i += 32u) mark[i].x = 0;
    __syncwarp();
    for (uint32_t s = lane; s < runs; s += 32u) {
      const uint32_t p = first[s] - w0;                // the spans ahead wrap round
      if (p < n) atomicOr(&mark[p >> 5].x, 1u << (p & 31u));
    }
    __syncwarp();
    for (uint32_t i0 = 0; i0 < words; i0 += 32u) {
      const uint32_t own = i0 + lane < words ? __popc(mark[i0 + lane].x) : 0u;
      uint32_t incl = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
      }
      if (i0 + lane < words) mark[i0 + lane].y = before + incl - own;
      before += __shfl_sync(0xffffffffu, incl, 31);
    }
    __syncwarp();
#pragma unroll 1
    for (uint32_t c = 0; c < n; c += 64u) {            // a place past the end stands for the walk's own bead
      const uint4 m = *reinterpret_cast<const uint4*>(&mark[c >> 5]);
      const uint32_t q0 = w0 + c + lane, q1 = q0 + 32u;
      const uint32_t j0 = shift[m.y + __popc(m.x & le)] + q0, j1 = shift[m.w + __popc(m.z & le)] + q1;
      take(q0 < total ? j0 : self, q1 < total ? j1 : self);
    }
    __syncwarp();
  }
}

// words behind a row: one entry too many, and the 64 candidates behind that
constexpr uint32_t kRowSlack = 80;

// A row with more candidates than its shared words hold, or than the capacity (a clump, an overflow to report, or
// candidates on the edge of the range that the exact distance leaves out).  The exact distance decides before an
// entry counts, as the reference does, and no entry is kept in between: the row is walked twice, to count the
// shells and to place the entries, in k_build_list's order.  Apart, so that k_build_list keeps its registers.
__device__ __noinline__ void build_long_row(const Shared& S, const SysParams& P, const float4* __restrict__ pos, float q,
                                            const uint32_t* __restrict__ start, uint32_t k, uint32_t cap,
                                            uint32_t* __restrict__ sm, uint32_t* __restrict__ out,
                                            uint32_t* __restrict__ nl_cnt, uint32_t* __restrict__ shell_end,
                                            uint32_t* __restrict__ flags) {
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  const float4 xi = pos[k];
  const float box[3] = {P.box[0], P.box[1], P.box[2]};
  const float inv[3] = {P.inv_box[0], P.inv_box[1], P.inv_box[2]};
  const float lr = P.list_range, lr2_lo = lr * lr * (1.0f - 1e-5f), lr2_hi = lr * lr * (1.0f + 1e-5f);
  const Shells sh = Shells::of(list_wide(S, P, (int)xi.w & (SOUP_KMAX - 1), q) ? S.rmax2 : S.rplain2, lr);
  const WalkGrid G{{P.dims[0], P.dims[1], P.dims[2]}, P.walk, P.walk * P.fine, P.cell_off, lr, {P.cell[0], P.cell[1], P.cell[2]}, P.inv_cell[0]};
  const uint32_t y0 = (lane & 1u) - 1u, y1 = ((lane >> 1) & 1u) - 1u, y2 = ((lane >> 2) & 1u) - 1u;
  uint32_t next = 0, cnt = 0, found = 0;               // lane l: the entries, then the next place, of shell l mod 8
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    const uint32_t whole = cnt & ~15u;
    found = 0;
    auto put = [&](uint32_t j) {
      const float4 xj = pos[j];
      const float dx = fast_mi(xi.x - xj.x, box[0], inv[0]);
      const float dy = fast_mi(xi.y - xj.y, box[1], inv[1]);
      const float dz = fast_mi(xi.z - xj.z, box[2], inv[2]);
      const float r2 = dx * dx + dy * dy + dz * dz;
      bool in = j != k && r2 <= lr2_hi;
      if (in && r2 >= lr2_lo) in = ex_dist(xi, xj, box) < lr;
      const uint32_t hits = __ballot_sync(0xffffffffu, in);
      in = in && found + __popc(hits & lt) < cap;      // what is behind the capacity is dropped, and reported
      found += __popc(hits);
      const uint32_t t = in ? sh.tag(r2) >> 29 : 0u, m = __ballot_sync(0xffffffffu, in);
      const uint32_t b0 = __ballot_sync(0xffffffffu, t & 1u), b1 = __ballot_sync(0xffffffffu, t & 2u),
                     b2 = __ballot_sync(0xffffffffu, t & 4u);
      if (pass == 1) {
        const uint32_t x0 = (t & 1u) - 1u, x1 = ((t >> 1) & 1u) - 1u, x2 = ((t >> 2) & 1u) - 1u;
        const uint32_t at = __shfl_sync(0xffffffffu, next, (int)t) + __popc(m & (b0 ^ x0) & (b1 ^ x1) & (b2 ^ x2) & lt);
        if (in) out[at < whole ? (at & ~15u) + 4u * (at & 3u) + ((at >> 2) & 3u) : at] = j;
      }
      next += __popc(m & (b0 ^ y0) & (b1 ^ y1) & (b2 ^ y2));
    };
    warp_walk(xi, k, box, G, start, sm, [&](uint32_t j0, uint32_t j1) {
      put(j0);
      put(j1);
    });
    if (pass == 1) break;
    cnt = min(found, cap);
    uint32_t incl = next;                              // the shells' ends
#pragma unroll
    for (int o = 1; o < kShells; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if ((lane & 7u) >= (uint32_t)o) incl += y;
    }
    if (lane < (uint32_t)kShells) shell_end[lane] = lane + 1u < (uint32_t)kShells ? incl : cnt;
    next = incl - next;
  }
  if (cnt + lane < ((cnt + 15u) & ~15u)) out[cnt + lane] = k;   // rows are padded with the particle itself
  if (lane == 0) {
    *nl_cnt = cnt;
    if (found > cap) flags[0] = 1u;
  }
}

// soup/wgsl/verlet.wgsl:53-92, a warp per particle (warp_walk).  The fast squared distance decides unless it
// lies within 1e-5 of the range, where the reference's arithmetic decides (the minimum image cannot differ
// there: range < box/2), so the list is the reference's set.  The accepted entries are compacted into the
// warp's shared row with ballots (a row of more candidates than `most` is built by build_long_row), then the row is grouped by build-distance shell, keeping its order inside
// a shell, straight into memory.  Every whole chunk of 16 entries is stored transposed (entry 4 e + l at
// place 4 l + e), so that the force's four lanes of a particle, which read four places each, gather four
// successive entries at a time: beads of one run, which share cache lines.
//
// Bound: instruction issue (78% of the slots, with the shared rows holding 32 warps an SM): at a range of 4.45 sigma
// about 600 candidates a bead, 295 of them in range.  At 483k beads a thread per bead and a second pass that grouped
// the rows took 1533 + 411 us, this 1185; at 24k 306 and 57, at 3.3k 393 and 18.
__global__ void __launch_bounds__(128, 9) k_build_list(
    const Shared* __restrict__ Sg, const float4* __restrict__ pos, const float* __restrict__ charge,
    const uint8_t* __restrict__ sysid, const SysParams* __restrict__ sp, const uint32_t* __restrict__ start, uint32_t N,
    uint32_t cap, uint32_t most, uint32_t stride, uint32_t* __restrict__ nl, uint32_t* __restrict__ nl_cnt,
    uint32_t* __restrict__ shell_end, uint32_t* __restrict__ flags) {
  extern __shared__ __align__(16) uint32_t sm[];
  const uint32_t wib = threadIdx.x >> 5, lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  const uint32_t held = (most + 15u) & ~15u;           // most: the candidates a shared row takes, cap at most
  uint32_t* row = sm + (size_t)wib * (held + kRowSlack + kWalkWords);
  const uint32_t k = blockIdx.x * (blockDim.x >> 5) + wib;
  if (k >= N) return;   // whole warps
  const SysParams& P = sp[sysid[k]];
  const float4 xi = pos[k];
  const float box[3] = {P.box[0], P.box[1], P.box[2]};
  const float inv[3] = {P.inv_box[0], P.inv_box[1], P.inv_box[2]};
  const float lr = P.list_range;
  const Shells sh = Shells::of(list_wide(*Sg, P, (int)xi.w & (SOUP_KMAX - 1), charge[k]) ? Sg->rmax2 : Sg->rplain2, lr);
  const float lr2_lo = lr * lr * (1.0f - 1e-5f), lr2_hi = lr * lr * (1.0f + 1e-5f);
  // a particle at least the list range inside every face screens with plain differences: a candidate within
  // the range sits at its stored coordinates, and one beyond it by the plain difference is beyond it by
  // the minimum image too
  const float rm = lr * (1.0f + 1e-5f) + 1e-3f;
  const bool direct = xi.x >= rm && xi.x <= box[0] - rm && xi.y >= rm && xi.y <= box[1] - rm && xi.z >= rm &&
                      xi.z <= box[2] - rm;
  const WalkGrid G{{P.dims[0], P.dims[1], P.dims[2]}, P.walk, P.walk * P.fine, P.cell_off, lr, {P.cell[0], P.cell[1], P.cell[2]}, P.inv_cell[0]};
  uint32_t cnt = 0;
  bool edge = false;
  // 32 candidates: the accepted ones, tagged, behind the row
  auto put = [&](auto image, uint32_t j, const float4& xj) {
    float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
    if (decltype(image)::value) {
      dx = fast_mi(dx, box[0], inv[0]);
      dy = fast_mi(dy, box[1], inv[1]);
      dz = fast_mi(dz, box[2], inv[2]);
    }
    const float r2 = dx * dx + dy * dy + dz * dz;
    const bool in = j != k && r2 <= lr2_hi;
    edge |= in && r2 >= lr2_lo;
    const uint32_t m = __ballot_sync(0xffffffffu, in), at = cnt + __popc(m & lt);
    if (in) row[at] = j + sh.tag(r2);
    cnt += __popc(m);
  };
  auto walk = [&](auto image) {
    warp_walk(xi, k, box, G, start, row + held + kRowSlack, [&](uint32_t j0, uint32_t j1) {
      const float4 x0 = pos[j0], x1 = pos[j1];
      put(image, j0, x0);
      put(image, j1, x1);
      cnt = min(cnt, most + 1u);                       // a row that is too long ends in the slack
    });
  };
  if (direct) walk(std::false_type{});
  else walk(std::true_type{});
  uint32_t* out = nl + (size_t)k * stride;
  if (cnt > most) {
    build_long_row(*Sg, P, pos, charge[k], start, k, cap, row + held + kRowSlack, out, nl_cnt + k,
                   shell_end + (size_t)kShells * k, flags);
    return;
  }
  if (__any_sync(0xffffffffu, edge)) {                 // the exact distance decides within 1e-5 of the range (rare)
    uint32_t kept = 0;
#pragma unroll 1
    for (uint32_t s0 = 0; s0 < cnt; s0 += 32u) {
      __syncwarp();
      const uint32_t v = s0 + lane < cnt ? row[s0 + lane] : 0u;
      const bool in = s0 + lane < cnt && ex_dist(xi, pos[v & 0x1FFFFFFFu], box) < lr;
      const uint32_t m = __ballot_sync(0xffffffffu, in);
      if (in) row[kept + __popc(m & lt)] = v;
      kept += __popc(m);
    }
    cnt = kept;
  }
  __syncwarp();
  // group the row by shell, keeping the walk's order inside a shell: 32 entries at a time, three ballots of the
  // shell's bits give every lane the entries of its own shell (its place among them) and lane s those of shell s
  // (the shells' running ends).  The loops stay rolled: unrolled, with the row in registers, the kernel outgrew the instruction cache
  // lane l stands for shell l mod 8: a ballot of bit i xor this is ones where bit i is the shell's
  const uint32_t y0 = (lane & 1u) - 1u, y1 = ((lane >> 1) & 1u) - 1u, y2 = ((lane >> 2) & 1u) - 1u;
  uint32_t end = 0;
#pragma unroll 1
  for (uint32_t c = 0; c < cnt; c += 32u) {
    const uint32_t v = c + lane < cnt ? row[c + lane] : SOUP_NONE_U32;   // beyond the row: the last shell
    const uint32_t b0 = __ballot_sync(0xffffffffu, v & 0x20000000u), b1 = __ballot_sync(0xffffffffu, v & 0x40000000u),
                   b2 = __ballot_sync(0xffffffffu, v & 0x80000000u);
    end += __popc((b0 ^ y0) & (b1 ^ y1) & (b2 ^ y2));
  }
  uint32_t incl = end;                                 // the shells' ends
#pragma unroll
  for (int o = 1; o < kShells; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if ((lane & 7u) >= (uint32_t)o) incl += y;
  }
  uint32_t next = incl - end;                          // the shells' next places
  const uint32_t whole = cnt & ~15u;
#pragma unroll 1
  for (uint32_t c = 0; c < cnt; c += 32u) {
    const uint32_t v = c + lane < cnt ? row[c + lane] : SOUP_NONE_U32;
    const uint32_t b0 = __ballot_sync(0xffffffffu, v & 0x20000000u), b1 = __ballot_sync(0xffffffffu, v & 0x40000000u),
                   b2 = __ballot_sync(0xffffffffu, v & 0x80000000u);
    const uint32_t x0 = ~(uint32_t)((int)(v << 2) >> 31), x1 = ~(uint32_t)((int)(v << 1) >> 31),
                   x2 = ~(uint32_t)((int)v >> 31);
    const uint32_t at = __shfl_sync(0xffffffffu, next, (int)(v >> 29)) + __popc((b0 ^ x0) & (b1 ^ x1) & (b2 ^ x2) & lt);
    const uint32_t to = at < whole ? (at & ~15u) + 4u * (at & 3u) + ((at >> 2) & 3u) : at;
    if (c + lane < cnt) out[to] = v & 0x1FFFFFFFu;
    next += __popc((b0 ^ y0) & (b1 ^ y1) & (b2 ^ y2));
  }
  if (cnt + lane < ((cnt + 15u) & ~15u)) out[cnt + lane] = k;   // rows are padded with the particle itself
  if (lane < (uint32_t)kShells) shell_end[(size_t)kShells * k + lane] = lane + 1u < (uint32_t)kShells ? incl : cnt;
  if (lane == 0) nl_cnt[k] = cnt;
}

// heads: bin into the coarse head grid (replica-local cells), deterministic order inside a cell.  The cells' counts
// are zero before and after: k_head_scatter counts them down
__global__ void k_head_index(const uint32_t* __restrict__ heads, const uint32_t* __restrict__ head_sys, uint32_t H,
                             const uint32_t* __restrict__ slot_of, const float4* __restrict__ pos,
                             const SysParams* __restrict__ sp, uint32_t* __restrict__ hcell_of,
                             uint32_t* __restrict__ hcount, uint32_t* __restrict__ head_slot,
                             uint32_t* __restrict__ head_of) {
  uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= H) return;
  const SysParams& P = sp[head_sys[h]];
  const uint32_t ks = slot_of[heads[h]];
  head_slot[h] = ks;
  head_of[ks] = h;
  float4 p = pos[ks];
  int cx = ex_cell_axis(p.x, P.box[0], P.hdims[0]);
  int cy = ex_cell_axis(p.y, P.box[1], P.hdims[1]);
  int cz = ex_cell_axis(p.z, P.box[2], P.hdims[2]);
  uint32_t c = P.hcell_off + (uint32_t)(cx + P.hdims[0] * (cy + P.hdims[1] * cz));
  hcell_of[h] = c;
  atomicAdd(&hcount[c], 1u);
}
__global__ void k_head_scatter(const uint32_t* __restrict__ hcell_of, const uint32_t* __restrict__ hstart, uint32_t H,
                               uint32_t* __restrict__ hcount, uint32_t* __restrict__ hsorted) {
  uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= H) return;
  uint32_t c = hcell_of[h];
  hsorted[hstart[c] + atomicSub(&hcount[c], 1u) - 1u] = h;
}
__global__ void k_head_sort_cells(const uint32_t* __restrict__ hstart, uint32_t ncells, uint32_t* __restrict__ hsorted) {
  uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  uint32_t a = hstart[c], e = hstart[c + 1];
  for (uint32_t x = a + 1; x < e; ++x) {
    uint32_t v = hsorted[x];
    uint32_t y = x;
    while (y > a && hsorted[y - 1] > v) { hsorted[y] = hsorted[y - 1]; --y; }
    hsorted[y] = v;
  }
}

// the heads in head-cell order with their positions: the list build reads one 16-byte record per
// candidate instead of the index, the head's slot and its position one after another
__global__ void k_head_gather_sorted(const uint32_t* __restrict__ hsorted, uint32_t H,
                                     const uint32_t* __restrict__ head_slot, const float4* __restrict__ pos,
                                     float4* __restrict__ xg) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= H) return;
  const uint32_t g = hsorted[t];
  const float4 p = pos[head_slot[g]];
  xg[t] = make_float4(p.x, p.y, p.z, __uint_as_float(g));
}

// soup/wgsl/electrostatics-long.wgsl:31-56 head list at rc_es + skin, via the head grid, a warp per head
// (warp_walk over the heads in head-cell order); hits are compacted with a ballot.  Entries are the
// neighbours' HEAD indices (head_slot maps them to slots); membership uses the exact test near the
// range, so the set equals the reference's.
__global__ void __launch_bounds__(128) k_build_es_list(const uint32_t* __restrict__ head_sys, uint32_t H,
                                                       const SysParams* __restrict__ sp, const uint32_t* __restrict__ hstart,
                                                       const float4* __restrict__ hxg, uint32_t cap,
                                                       uint32_t* __restrict__ es_nl, uint32_t* __restrict__ es_cnt,
                                                       uint32_t* __restrict__ flags) {
  __shared__ __align__(16) uint32_t sm[4][kWalkWords];
  const uint32_t wib = threadIdx.x >> 5, lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  const uint32_t place = blockIdx.x * 4u + wib;        // in head-cell order: the warps of a block share candidates
  if (place >= H) return;   // whole warps
  const float4 xi = hxg[place];
  const uint32_t h = __float_as_uint(xi.w);
  const SysParams& P = sp[head_sys[h]];
  const float box[3] = {P.box[0], P.box[1], P.box[2]};
  const float inv[3] = {P.inv_box[0], P.inv_box[1], P.inv_box[2]};
  const float lr = P.es_list_range;
  const float lo = lr * lr * (1.0f - 1e-5f), hi = lr * lr * (1.0f + 1e-5f);
  const WalkGrid G{{P.hdims[0], P.hdims[1], P.hdims[2]}, P.hwalk, P.hwalk * P.hfine, P.hcell_off, lr, {P.hcell[0], P.hcell[1], P.hcell[2]},
                   P.inv_hcell[0]};
  uint32_t cnt = 0;
  uint32_t* row = es_nl + (size_t)h * cap;
  auto put = [&](const float4& xj) {
    const uint32_t g = __float_as_uint(xj.w);
    const float dx = fast_mi(xi.x - xj.x, box[0], inv[0]);
    const float dy = fast_mi(xi.y - xj.y, box[1], inv[1]);
    const float dz = fast_mi(xi.z - xj.z, box[2], inv[2]);
    const float r2 = dx * dx + dy * dy + dz * dz;
    bool hit = g != h && r2 <= hi;
    if (hit && r2 >= lo) hit = ex_dist(xi, xj, box) < lr;
    const uint32_t m = __ballot_sync(0xffffffffu, hit);
    const uint32_t at = cnt + __popc(m & lt);
    if (hit && at < cap) row[at] = g;
    cnt += __popc(m);
  };
  warp_walk(xi, place, box, G, hstart, sm[wib], [&](uint32_t j0, uint32_t j1) {
    const float4 x0 = hxg[j0], x1 = hxg[j1];
    put(x0);
    put(x1);
  });
  if (lane == 0) {
    if (cnt > cap) { flags[1] = 1u; cnt = cap; }
    es_cnt[h] = cnt;
  }
}

}  // namespace

void launch_cell_index(Batch& b) {
  b.launches += 1;
  prof_begin(b, SOUP_K_SORT);
  cudaMemsetAsync(b.cell_count, 0, sizeof(uint32_t) * (b.ncells + 1), b.stream);
  k_cell_index<<<nblocks(b.N), kBlock, 0, b.stream>>>(b.pos, b.sysid, b.sp, b.N, b.cell_of_slot, b.cell_count);
  prof_end(b);
}

void launch_sort_and_gather(Batch& b) {
  prof_begin(b, SOUP_K_SORT);
  const uint64_t scans = exclusive_scan(b.cell_count, b.cell_start, b.ncells, b.scan_tmp, b.stream);
  k_scatter<<<nblocks(b.N), kBlock, 0, b.stream>>>(b.cell_of_slot, b.cell_start, b.N, b.cell_count, b.perm);
  k_sort_cells<<<nblocks(b.ncells), kBlock, 0, b.stream>>>(b.cell_start, b.ncells, b.id, b.perm);
  k_gather<<<nblocks(b.N), kBlock, 0, b.stream>>>(b.N, b.perm, b.pos, b.vel, b.force, b.charge, b.slots, b.center,
                                                   b.held, b.brng, b.trng, b.frozen, b.id, b.pos2, b.vel2, b.force2,
                                                   b.charge2, b.slots2, b.center2, b.held2, b.brng2, b.trng2,
                                                   b.frozen2, b.id2, b.slot_of, b.pos_ref);
  k_copy_back<<<nblocks(b.N), kBlock, 0, b.stream>>>(b.N, b.pos2, b.vel2, b.force2, b.charge2, b.slots2, b.center2,
                                                      b.held2, b.brng2, b.trng2, b.frozen2, b.id2, b.pos, b.vel, b.force,
                                                      b.charge, b.slots, b.center, b.held, b.brng, b.trng, b.frozen,
                                                      b.id, b.head_of, b.R, b.drift_bits);
  b.launches += 4 + scans;
  prof_end(b);
}

void launch_build_lists(Batch& b) {
  b.launches += 1;
  prof_begin(b, SOUP_K_LIST);
  // A shared row takes 1280 candidates, with which eight blocks fit an SM, or as many as twice the row a bead has in
  // liquid (1.1 beads a sigma^3, or the replica's own density), up to 4096: two blocks an SM, behind which walking a row
  // twice more costs less than a third block gives.  The capacity alone is no measure: sized by it, a
  // capacity of 8192 took 1563 us at 121k beads and 6143 at 483k (382 and 1299 at 1126; lists and head lists)
  double want = 1280.0;
  uint32_t n = 0;
  for (uint32_t r = 0; r < b.R; ++r) {
    const SoupConfig& c = b.cfg[r];
    n = std::max(n, c.n);
    const double vol = c.wall_radius > 0 ? 4.18879 * c.wall_radius * c.wall_radius * c.wall_radius : c.box[0] * c.box[1] * c.box[2];
    const double density = std::max(c.n / vol, 1.1 / (c.sigma * c.sigma * c.sigma));
    want = std::max(want, 2.0 * density * 4.18879 * c.list_range * c.list_range * c.list_range);
  }
  const uint32_t most = std::min({b.list_cap, n, (uint32_t)std::min(want, 4096.0)}), held = (most + 15u) & ~15u;
  constexpr uint32_t wpb = 4;
  const size_t smem = wpb * sizeof(uint32_t) * ((size_t)held + kRowSlack + kWalkWords);
  if (smem > 48u * 1024u && !b.list_smem_open) {       // to all an SM has: the setting is the device's, not this batch's
    SOUP_CUDA_TRY(cudaFuncSetAttribute(k_build_list, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    b.list_smem_open = true;
  }
  k_build_list<<<nblocks(b.N, wpb), 32 * wpb, smem, b.stream>>>(
      b.shared, b.pos, b.charge, b.sysid, b.sp, b.cell_start, b.N, b.list_cap, most, b.list_stride, b.nl, b.nl_cnt, b.nl_shell,
      b.flags);
  prof_end(b);
}

void launch_build_es_lists(Batch& b) {
  if (b.H == 0) return;
  prof_begin(b, SOUP_K_LIST);
  k_head_index<<<nblocks(b.H), kBlock, 0, b.stream>>>(b.heads, b.head_sys, b.H, b.slot_of, b.pos, b.sp, b.hcell_of,
                                                       b.hcell_count, b.head_slot, b.head_of);
  const uint64_t scans = exclusive_scan(b.hcell_count, b.hcell_start, b.nhcells, b.scan_tmp, b.stream);
  k_head_scatter<<<nblocks(b.H), kBlock, 0, b.stream>>>(b.hcell_of, b.hcell_start, b.H, b.hcell_count, b.hsorted);
  k_head_sort_cells<<<nblocks(b.nhcells), kBlock, 0, b.stream>>>(b.hcell_start, b.nhcells, b.hsorted);
  k_head_gather_sorted<<<nblocks(b.H), kBlock, 0, b.stream>>>(b.hsorted, b.H, b.head_slot, b.pos, b.hsorted_xg);
  k_build_es_list<<<nblocks(b.H, 4), 128, 0, b.stream>>>(b.head_sys, b.H, b.sp, b.hcell_start, b.hsorted_xg, b.es_cap, b.es_nl, b.es_cnt, b.flags);
  b.launches += 6 + scans;
  prof_end(b);
}

}  // namespace soup
