// io_kernels.cuh -- layout conversion between the reference's [x][y][z]
// arrays and the internal structure-of-arrays lattice, and the device
// reductions behind the phase statistics.
#pragma once

#include "lattice.cuh"

namespace mlbm {

// Reference layout index: ((x * ly + y) * lz + z), z fastest
// (include/lbm_model.cuh:18-22).
__device__ __forceinline__ long long ref_index(const Geom& g, int x, int y,
                                               int z) {
  return ((long long)x * g.ly + y) * g.lz + z;
}

// Internal-layout kernels use blockDim (32, 4) over (x, y) and grid.z = z.
#define MLBM_NODE_COORDS                              \
  const int x = blockIdx.x * 32 + threadIdx.x;        \
  const int y = blockIdx.y * blockDim.y + threadIdx.y; \
  const int z = blockIdx.z;

// Both layouts are dense with opposite fastest axes, so a copy is a transpose
// of the (x, z) planes: a block moves a 32 x 32 tile of one y through shared
// memory, reading and writing runs of 32 values (one value per thread straight
// across touched a sector per 4 bytes on one side: 56 us for the 64 MB of a
// 200^3 FP32 field).  blockDim (32, kTileRows), grid (x tiles of every y, z
// tiles): y has no place among the grid's short dimensions (up to 2^24 rows).
// The density coming in moves 32 x kSpanZ tiles, runs of 512 bytes read (384^3:
// 250 -> 177 us a call); on the way out the wider tile gains at 200^3 (23 -> 21
// us) and loses at 384^3 (181 -> 189) and 64^3.
constexpr int kTileRows = 8;
constexpr int kSpanZ = 128;
#define MLBM_SPAN_COORDS                                             \
  const int xt = (int)(blockIdx.x % (unsigned)g.wpr), x0 = xt * 32;  \
  const int y = (int)(blockIdx.x / (unsigned)g.wpr);                 \
  const int z0 = blockIdx.y * kSpanZ, lane = threadIdx.x;
inline dim3 span_grid(const Geom& g) {
  return dim3((unsigned)g.wpr * (unsigned)g.ly, (g.lz + kSpanZ - 1) / kSpanZ, 1);
}
#define MLBM_TILE_COORDS                                             \
  const int xt = (int)(blockIdx.x % (unsigned)g.wpr), x0 = xt * 32;  \
  const int y = (int)(blockIdx.x / (unsigned)g.wpr);                 \
  const int z0 = blockIdx.y * 32, lane = threadIdx.x;

inline dim3 tile_block() { return dim3(32, kTileRows, 1); }
inline dim3 tile_grid(const Geom& g) {
  return dim3((unsigned)g.wpr * (unsigned)g.ly, (g.lz + 31) / 32, 1);
}

// Pack a uint8 [x][y][z] fluid array into the bit mask.
__global__ void k_pack_mask(const uint8_t* __restrict__ fluid_ref,
                            uint32_t* __restrict__ mask, Geom g) {
  __shared__ uint8_t t[32][33];
  MLBM_TILE_COORDS
  for (int r = threadIdx.y; r < 32; r += kTileRows) {
    const int x = x0 + r, z = z0 + lane;
    t[r][lane] = x < g.lx && z < g.lz && fluid_ref[ref_index(g, x, y, z)] != 0;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32 && z0 + r < g.lz; r += kTileRows) {
    const uint32_t w = __ballot_sync(0xffffffffu, t[lane][r] != 0);
    if (lane == 0) mask[((long long)(z0 + r) * g.ly + y) * g.wpr + xt] = w;
  }
}

__global__ void k_rho_from_ref(const float* __restrict__ rho_ref,
                               float* __restrict__ rho_int, Geom g) {
  __shared__ float t[32][kSpanZ + 1];
  MLBM_SPAN_COORDS
#pragma unroll
  for (int r = threadIdx.y; r < 32; r += kTileRows) {
#pragma unroll
    for (int c = 0; c < kSpanZ; c += 32) {
      const int x = x0 + r, z = z0 + c + lane;
      if (x < g.lx && z < g.lz) t[r][c + lane] = rho_ref[ref_index(g, x, y, z)];
    }
  }
  __syncthreads();
  if (x0 + lane >= g.lx) return;
  for (int r = threadIdx.y; r < kSpanZ && z0 + r < g.lz; r += kTileRows)
    rho_int[node_index(g, x0 + lane, y, z0 + r)] = t[lane][r];
}

// field: 0 rho, 1 pressure, 2 psi -> reference layout.
template <typename R, typename O>
__global__ void k_scalar_to_ref(const R* __restrict__ rho, O* __restrict__ out,
                                Geom g, Phys p, int field) {
  __shared__ O t[32][33];
  MLBM_TILE_COORDS
  for (int r = threadIdx.y; r < 32; r += kTileRows) {
    const int x = x0 + lane, z = z0 + r;
    if (x >= g.lx || z >= g.lz) continue;
    const R v = rho[node_index(g, x, y, z)];
    t[lane][r] = (O)(field == 0 ? v : field == 1 ? pressure_of<R>(p, v) : psi_of<R>(p, v));
  }
  __syncthreads();
  if (z0 + lane >= g.lz) return;
  for (int r = threadIdx.y; r < 32 && x0 + r < g.lx; r += kTileRows)
    out[ref_index(g, x0 + r, y, z0 + lane)] = t[r][lane];
}

__global__ void k_fluid_to_ref(const uint32_t* __restrict__ mask,
                               uint8_t* __restrict__ out, Geom g) {
  MLBM_TILE_COORDS
  if (z0 + lane >= g.lz) return;
  // a warp writes 32 z of one x; its 32 mask words serve the tile's 32 x
  const uint32_t w = mask[((long long)(z0 + lane) * g.ly + y) * g.wpr + xt];
  for (int r = threadIdx.y; r < 32 && x0 + r < g.lx; r += kTileRows)
    out[ref_index(g, x0 + r, y, z0 + lane)] = (w >> r) & 1u;
}

// The three components of a node stay together: runs of 96 values.
template <typename O>
__global__ void k_vel_to_ref(const float* __restrict__ vel,
                             O* __restrict__ out, Geom g) {
  __shared__ float t[32][97];  // [z][3 x + c]
  MLBM_TILE_COORDS
  const int nx = min(32, g.lx - x0), nz = min(32, g.lz - z0);
  for (int r = threadIdx.y; r < nz; r += kTileRows) {
    const float* src = vel + 3 * node_index(g, x0, y, z0 + r);
    for (int c = lane; c < 3 * nx; c += 32) t[r][c] = src[c];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < nx; r += kTileRows) {
    O* dst = out + 3 * ref_index(g, x0 + r, y, z0);
    for (int c = lane; c < 3 * nz; c += 32) dst[c] = (O)t[c / 3][3 * r + c % 3];
  }
}

// Post-collision populations f*_i in the reference layout [x][y][z][19].
// Phase 0: f*_i(x) = pop[opp(i)][x].  Phase 1 (fluid nodes): pop[i][x+e_i]
// when x+e_i is fluid, else pop[opp(i)][x].  Solid nodes keep their
// initial values, stored at pop[opp(i)][x] in either phase.
template <typename T, typename O>
__global__ void k_pop_to_ref(const T* __restrict__ pop,
                             const uint32_t* __restrict__ mask,
                             O* __restrict__ out, Geom g, Phys p, int phase) {
  using R = typename Pop<T>::Real;
  MLBM_NODE_COORDS
  if (x >= g.lx || y >= g.ly) return;
  const long long n = node_index(g, x, y, z), r = ref_index(g, x, y, z);
  const bool fl = fluid_at(mask, g, x, y, z);
  const R shift = R(p.rho_shift);
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const R s = shift * weight<R>(i);
    long long src = opp(i) * g.plane + n;
    if (phase == 1 && fl && i != 0) {
      const int xd = wrapc(x + ex(i), g.lx), yd = wrapc(y + ey(i), g.ly),
                zd = wrapc(z + ez(i), g.lz);
      if (fluid_at(mask, g, xd, yd, zd))
        src = i * g.plane + node_index(g, xd, yd, zd);
    }
    out[(long long)Q * r + i] = (O)Pop<T>::ld(pop + src, s);
  }
}

// ---- phase statistics ----------------------------------------------------------
// Per node of the fluid: counts (fluid, liquid, vapour, liquid-solid and
// liquid-vapour boundary nodes), FP64 sums (mass, liquid/vapour pressure and
// density) and min/max of rho and p.  calc_cluster, src/multiphase_lbm.cu:
// 240-316; write_stats, :1061-1072.
enum { ST_NF, ST_NL, ST_NV, ST_NLS, ST_NLV, ST_MASS, ST_PL, ST_PV, ST_RL,
       ST_RV, ST_MINR, ST_MAXR, ST_MINP, ST_MAXP, ST_COUNT };

constexpr int kStatThreads = 256;

__device__ __forceinline__ double stat_op(int k, double v, double o) {
  return (k == ST_MINR || k == ST_MINP) ? fmin(v, o)
         : (k == ST_MAXR || k == ST_MAXP) ? fmax(v, o)
                                           : v + o;
}
__device__ __forceinline__ double stat_identity(int k) {
  return (k == ST_MINR || k == ST_MINP) ? 1e9
         : (k == ST_MAXR || k == ST_MAXP) ? -1e-9
                                           : 0.0;
}

// The columns that the bulk statistics compute; the others are written as 0.
__host__ __device__ constexpr bool stat_bulk_column(int k) {
  return k == ST_NF || k == ST_NL || k == ST_NV || k == ST_MASS ||
         k == ST_RL || k == ST_RV || k == ST_MINR || k == ST_MAXR;
}

// Warp then block reduction of acc in a fixed order (deterministic); thread 0
// .. ST_COUNT - 1 of the block write the block's record.  256 threads.
__device__ __forceinline__ void stat_block_reduce(double (&acc)[ST_COUNT],
                                                  int tid, double* record) {
#pragma unroll
  for (int k = 0; k < ST_COUNT; ++k) {
    double v = acc[k];
    for (int off = 16; off > 0; off >>= 1)
      v = stat_op(k, v, __shfl_down_sync(0xffffffffu, v, off));
    acc[k] = v;
  }
  __shared__ double sh[kStatThreads / 32][ST_COUNT];
  const int warp = tid >> 5, lane = tid & 31;
  if (lane == 0)
    for (int k = 0; k < ST_COUNT; ++k) sh[warp][k] = acc[k];
  __syncthreads();
  if (tid < ST_COUNT) {
    const int k = tid;
    double v = sh[0][k];
    for (int w = 1; w < kStatThreads / 32; ++w) v = stat_op(k, v, sh[w][k]);
    record[k] = v;
  }
}

// Scratch of one statistics reduction (8-byte slots): the arrival counter and
// the two boundary counts (zero between calls), then the block records
// (ST_COUNT each), then the ST_COUNT results and the device error flag.
struct StatScratch {
  unsigned* counter;
  unsigned long long* boundary;  // liquid-solid, liquid-vapour
  double* records;
  double* out;
};
constexpr int kStatCounters = 3;

// Called by every thread of a block once the block's part is in the scratch.
// The last of `arrivals` blocks to arrive folds the `nrecords` records (of this
// launch or of the one before) -- in a fixed order, so the result does not
// depend on which block is last: thread t folds records t, t + 256, ...
// ascending, then the warps' shuffle trees, then the warps in order -- writes
// the results and the device error flag and re-arms the counters.  Records are
// read through L2 (ld.global.cg): other SMs wrote them.  256 threads.
__device__ __forceinline__ void stat_last_block(StatScratch s, unsigned arrivals,
                                                unsigned nrecords,
                                                const int* __restrict__ err,
                                                int tid, bool full) {
  __shared__ bool last;
  __shared__ double sh[kStatThreads / 32][ST_COUNT];
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(s.counter, 1u) == arrivals - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  double v[ST_COUNT];
#pragma unroll
  for (int k = 0; k < ST_COUNT; ++k) v[k] = stat_identity(k);
  for (unsigned b = tid; b < nrecords; b += kStatThreads) {
    const double* rec = s.records + (size_t)b * ST_COUNT;
    double r[ST_COUNT];
#pragma unroll
    for (int k = 0; k < ST_COUNT; ++k) r[k] = __ldcg(rec + k);
#pragma unroll
    for (int k = 0; k < ST_COUNT; ++k) v[k] = stat_op(k, v[k], r[k]);
  }
#pragma unroll
  for (int k = 0; k < ST_COUNT; ++k)
    for (int off = 16; off > 0; off >>= 1)
      v[k] = stat_op(k, v[k], __shfl_down_sync(0xffffffffu, v[k], off));
  const int warp = tid >> 5, lane = tid & 31;
  if (lane == 0)
    for (int k = 0; k < ST_COUNT; ++k) sh[warp][k] = v[k];
  __syncthreads();
  if (tid < ST_COUNT) {
    double r = sh[0][tid];
    for (int w = 1; w < kStatThreads / 32; ++w) r = stat_op(tid, r, sh[w][tid]);
    if (full && (tid == ST_NLS || tid == ST_NLV))
      r = (double)atomicExch(s.boundary + (tid - ST_NLS), 0ull);
    s.out[tid] = full || stat_bulk_column(tid) ? r : 0.0;  // not computed: 0
  }
  if (tid == 0) {
    s.out[ST_COUNT] = err ? (double)*err : 0.0;
    *s.counter = 0u;
  }
}

// Sums, counts and extrema of the fluid nodes.  A warp takes kStatWords x 32
// nodes at a time -- the padded rows make the nodes of consecutive mask words
// consecutive densities -- with all their loads in flight: no node needs a
// table entry first (walking the fluid nodes' table, two dependent loads a
// node, took 35 us at 200^3, the 18 neighbours' densities of the boundary test
// another 32; 31 and 23 us for both parts now).  What bounds it: instruction
// issue, 71 per 32 nodes.
// Counts are integers and extrema are in the densities' type; sums are FP64,
// each lane over its nodes in order, then the fixed trees of
// stat_block_reduce.  FULL: the pressures too, and for the boundary test the
// words of the liquid nodes and of the fluid nodes below rhol; the fold is then
// k_stats_boundary's.
constexpr int kStatWords = 16;
template <typename R, bool FULL>
__global__ void __launch_bounds__(kStatThreads, sizeof(R) == 8 ? 2 : 4)
    k_stats_nodes(const R* __restrict__ rho, const uint32_t* __restrict__ mask,
                  int nwords, Phys p, StatScratch sc, uint32_t* __restrict__ liquid,
                  uint32_t* __restrict__ low, const int* __restrict__ err) {
  const int lane = threadIdx.x & 31;
  const int warp = blockIdx.x * (kStatThreads / 32) + threadIdx.x / 32;
  const int warps = gridDim.x * (kStatThreads / 32);
  const R rhol = R(p.rhol_spinodal), rhog = R(p.rhog_spinodal);
  unsigned nf = 0, nl = 0, nv = 0;
  double mass = 0, pl = 0, pv = 0, rl = 0, rv = 0;
  R minr = R(INFINITY), maxr = R(-INFINITY), minp = minr, maxp = maxr;
#pragma unroll 1
  for (int c = warp; c <= (nwords - 1) / kStatWords; c += warps) {
    const int w = c * kStatWords + lane;
    const uint32_t m = lane < kStatWords && w < nwords ? __ldg(mask + w) : 0u;
    const R* r0 = rho + (size_t)c * (kStatWords * 32) + lane;
    R r[kStatWords];
    uint32_t fl = 0;  // bit j: this lane's node of word j is fluid
#pragma unroll
    for (int j = 0; j < kStatWords; ++j) {
      const uint32_t mj = __shfl_sync(~0u, m, j);
      const uint32_t b = (mj >> lane) & 1u;
      fl |= b << j;
      r[j] = R(0);
      if (b) r[j] = __ldg(r0 + j * 32);
    }
    uint32_t wl = 0, wb = 0;
#pragma unroll
    for (int j = 0; j < kStatWords; ++j) {
      const R v = r[j];
      const bool fluid = (fl >> j) & 1u, liq = fluid && v > rhol;
      if (fluid) {
        const R pr = FULL ? pressure_of<R>(p, v) : R(0);
        mass += (double)v;
        if (liq) {
          ++nl;
          rl += (double)v;
          if (FULL) pl += (double)pr;
        } else if (v < rhog) {
          ++nv;
          rv += (double)v;
          if (FULL) pv += (double)pr;
        }
        minr = fmin(minr, v);
        maxr = fmax(maxr, v);
        if (FULL) {
          minp = fmin(minp, pr);
          maxp = fmax(maxp, pr);
        }
      }
      if (FULL) {
        const uint32_t l = __ballot_sync(~0u, liq);
        const uint32_t b = __ballot_sync(~0u, fluid && v < rhol);
        if (lane == j) {
          wl = l;
          wb = b;
        }
      }
    }
    nf += __popc(fl);
    if (FULL && lane < kStatWords && w < nwords) {
      liquid[w] = wl;
      low[w] = wb;
    }
  }
  double acc[ST_COUNT];
#pragma unroll
  for (int k = 0; k < ST_COUNT; ++k) acc[k] = stat_identity(k);
  acc[ST_NF] = nf;
  acc[ST_NL] = nl;
  acc[ST_NV] = nv;
  acc[ST_MASS] = mass;
  acc[ST_PL] = pl;
  acc[ST_PV] = pv;
  acc[ST_RL] = rl;
  acc[ST_RV] = rv;
  acc[ST_MINR] = fmin(acc[ST_MINR], (double)minr);
  acc[ST_MAXR] = fmax(acc[ST_MAXR], (double)maxr);
  if (FULL) {
    acc[ST_MINP] = fmin(acc[ST_MINP], (double)minp);
    acc[ST_MAXP] = fmax(acc[ST_MAXP], (double)maxp);
  }
  stat_block_reduce(acc, threadIdx.x, sc.records + (long long)blockIdx.x * ST_COUNT);
  if (!FULL) stat_last_block(sc, gridDim.x, gridDim.x, err, threadIdx.x, false);
}

// 32 neighbours at x + dx of the nodes of word w of a row of bits (periodic).
__device__ __forceinline__ uint32_t row_shift(const uint32_t* __restrict__ row, int w,
                                              int dx, const Geom& g) {
  const uint32_t v = row[w];
  const int end = (g.lx - 1) & 31, last = g.wpr - 1;
  if (dx < 0)
    return (v << 1) | (w > 0 ? row[w - 1] >> 31 : (row[last] >> end) & 1u);
  if (dx > 0)
    return w < last ? (v >> 1) | (row[w + 1] << 31)
                    : (v >> 1) | ((row[0] & 1u) << end);
  return v;
}

// Liquid-solid and liquid-vapour boundary nodes, 32 at a time in bits: for a
// liquid node the first neighbour x - e_i (i = 1..18) that is solid or below
// rhol decides, as calc_cluster does.  After k_stats_nodes<R, true>, whose
// records the last block folds.
static __global__ void __launch_bounds__(kStatThreads)
    k_stats_boundary(const uint32_t* __restrict__ mask,
                     const uint32_t* __restrict__ liquid,
                     const uint32_t* __restrict__ low, int nwords, Geom g,
                     unsigned nrecords, StatScratch sc,
                     const int* __restrict__ err) {
  unsigned ls = 0, lv = 0;
  for (int i = blockIdx.x * kStatThreads + threadIdx.x; i < nwords;
       i += gridDim.x * kStatThreads) {
    uint32_t open = liquid[i];  // liquid nodes no neighbour has decided yet
    if (!open) continue;
    const int w = i % g.wpr, r = i / g.wpr;
    const int y = r % g.ly, z = r / g.ly;
#pragma unroll
    for (int k = 1; k < Q; ++k) {
      const int q = (wrapc(z - ez(k), g.lz) * g.ly + wrapc(y - ey(k), g.ly)) * g.wpr;
      const uint32_t solid = ~row_shift(mask + q, w, -ex(k), g);
      const uint32_t below = row_shift(low + q, w, -ex(k), g);
      ls += __popc(open & solid);
      lv += __popc(open & ~solid & below);
      open &= ~(solid | below);
    }
  }
  ls = __reduce_add_sync(~0u, ls);
  lv = __reduce_add_sync(~0u, lv);
  __shared__ unsigned sum[2];
  if (threadIdx.x < 2) sum[threadIdx.x] = 0u;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    if (ls) atomicAdd(sum, ls);
    if (lv) atomicAdd(sum + 1, lv);
  }
  __syncthreads();
  if (threadIdx.x < 2 && sum[threadIdx.x])
    atomicAdd(sc.boundary + threadIdx.x, (unsigned long long)sum[threadIdx.x]);
  stat_last_block(sc, gridDim.x, nrecords, err, threadIdx.x, true);
}

// Per-x-plane fluid / liquid node counts (integers: deterministic).  A thread
// counts a column of kProfileRows rows (y, z) at its x, a block adds its
// columns up and adds one number per plane (two atomics per fluid node on lx
// counters took 210 us at 200^3).  blockDim (32, 8), grid x tiles of
// every row group.
constexpr int kProfileRows = 16;
template <typename R>
__global__ void k_plane_profile(const R* __restrict__ rho,
                                const uint32_t* __restrict__ mask, Geom g,
                                Phys p, unsigned long long* __restrict__ nf,
                                unsigned long long* __restrict__ nl) {
  __shared__ unsigned sf[8][32], sl[8][32];
  const int lane = threadIdx.x, w = (int)(blockIdx.x % (unsigned)g.wpr);
  const int x = w * 32 + lane;
  const long long rows = (long long)g.ly * g.lz;
  const long long r0 =
      ((long long)(blockIdx.x / (unsigned)g.wpr) * 8 + threadIdx.y) * kProfileRows;
  unsigned f = 0, l = 0;
#pragma unroll 4
  for (long long r = r0; r < min(r0 + kProfileRows, rows); ++r) {
    const bool fl = (mask[r * g.wpr + w] >> lane) & 1u;
    f += fl;
    // padding columns are never fluid, and lie inside the array
    l += fl && rho[r * g.px + x] > R(p.rhol_spinodal);
  }
  sf[threadIdx.y][lane] = f;
  sl[threadIdx.y][lane] = l;
  __syncthreads();
  if (threadIdx.y) return;
  for (int j = 1; j < 8; ++j) {
    f += sf[j][lane];
    l += sl[j][lane];
  }
  if (x >= g.lx) return;
  if (f) atomicAdd(nf + x, (unsigned long long)f);
  if (l) atomicAdd(nl + x, (unsigned long long)l);
}
inline dim3 profile_grid(const Geom& g) {
  const long long rows = (long long)g.ly * g.lz;
  return dim3((unsigned)(g.wpr * ((rows + 8 * kProfileRows - 1) / (8 * kProfileRows))));
}

}  // namespace mlbm
