// moments.cu -- host side of the moment step (moments.cuh): lists, buffers, launches, and the way back to populations.
#include <cuda_runtime.h>

#include <cub/cub.cuh>

#include "capi_internal.h"
#include "launch.cuh"
#include "moments.cuh"

namespace mlbm {

namespace {

size_t up256(size_t n) { return (n + 255) / 256 * 256; }

// Sizes of the parts of the buffer for a list of `pairs`.
struct Parts {
  size_t m, psi, n, words, xyz;
  Parts(const Geom& g, int storage, size_t pairs) {
    const size_t real = real_bytes(storage);
    m = up256((size_t)node_elems(g) * 4 * real);
    psi = up256((size_t)node_elems(g) * real);
    n = up256(pairs * 8 * real);
    words = up256(pairs * sizeof(uint2));
    xyz = up256(pairs * sizeof(uint32_t));
  }
  size_t total() const { return m + psi + n + words + xyz; }
};

// Pair list of the current mask and slabs, and the
// buffers (one allocation).  Waits for the counts.
mlbm_status build_list(mlbm_lattice* lat) {
  MomentState& s = lat->mom;
  const Geom& g = lat->g;
  const long long grid = TileGrid(g).count();
  size_t temp_bytes = 0;
  uint32_t* counts = nullptr;
  cudaError_t e = cub::DeviceScan::ExclusiveSum(
      nullptr, temp_bytes, counts, counts, grid + 1, lat->stream);
  if (e != cudaSuccess) return cuda_fail(e, "moment lists");
  // scratch of the scan: the transfer buffer an upload has left (same
  // stream), else an allocation of its own
  const size_t counts_bytes = up256((size_t)(grid + 1) * sizeof(uint32_t));
  char* own = nullptr;
  char* buf = static_cast<char*>(lat->staging);
  if (lat->staging_bytes < counts_bytes + temp_bytes) {
    e = lattice_try_malloc(lat, (void**)&own, counts_bytes + temp_bytes);
    if (e != cudaSuccess) return cuda_fail(e, "moment lists");
    buf = own;
  }
  counts = reinterpret_cast<uint32_t*>(buf);
  const unsigned threads = 32 * kPairRows;
  k_mom_tiles<true><<<(unsigned)grid, threads, 0, lat->stream>>>(
      lat->nbw, counts, nullptr, nullptr, nullptr, g);
  e = cub::DeviceScan::ExclusiveSum(buf + counts_bytes, temp_bytes, counts, counts,
                                    grid + 1, lat->stream);
  uint32_t total = 0;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&total, counts + grid, sizeof total,
                        cudaMemcpyDeviceToHost, lat->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(lat->stream);
  const Parts part(g, lat->storage, total);
  const size_t need = part.total();
  if (e == cudaSuccess && need > s.buffer_bytes) {
    cudaFree(s.buffer);
    s.buffer = nullptr;
    s.buffer_bytes = 0;
    e = lattice_try_malloc(lat, &s.buffer, need);
    if (e == cudaSuccess) s.buffer_bytes = need;
  }
  if (e == cudaSuccess) {
    char* at = static_cast<char*>(s.buffer);
    s.m = at;
    s.psi = at += part.m;
    s.n = at += part.psi;
    s.words = reinterpret_cast<uint2*>(at += part.n);
    s.xyz = reinterpret_cast<uint32_t*>(at += part.words);
    s.npairs = (int)total;
    if (total)
      k_mom_tiles<false><<<(unsigned)grid, threads, 0, lat->stream>>>(
          lat->nbw, nullptr, counts, s.words, s.xyz, g);
    e = cudaGetLastError();
  }
  cudaFree(own);
  if (e != cudaSuccess) return cuda_fail(e, "moment lists");
  s.list_built = true;
  ++lat->changes;
  return MLBM_OK;
}

PairList pair_list(const MomentState& s) { return PairList{s.words, s.xyz, s.npairs}; }

unsigned pair_blocks(const MomentState& s) {
  return (unsigned)((s.npairs + kMomThreads - 1) / kMomThreads);
}

template <typename T, bool WR>
void launch_gather(mlbm_lattice* lat, const StepArgs& a, bool inj, bool overlap) {
  using R = typename Pop<T>::Real;
  MomentState& s = lat->mom;
  R* rho = static_cast<R*>(lat->rho);
  R* psi = static_cast<R*>(s.psi);
  MomPair<R>* n = static_cast<MomPair<R>*>(s.n);
  const unsigned grid = pair_blocks(s);
  if (s.active) {
    launch_overlapped(overlap, k_mom_gather<T, WR>, grid, kMomThreads, 0, lat->stream,
                      (const Mom<R>*)s.m, pair_list(s), n, rho, psi, lat->g,
                      lat->phys, a, inj, s.shift);
    return;
  }
  const Geom& g = lat->g;
  k_mom_psi<R><<<dim3((g.lx + 31) / 32, (g.ly + 7) / 8, g.lz + 2), dim3(32, 8), 0,
                 lat->stream>>>(static_cast<const R*>(lat->psi), psi, g);
  const T* pop = static_cast<const T*>(lat->pop);
  if (lat->phase == 0)
    k_mom_gather_pop<T, 0, WR><<<grid, kMomThreads, 0, lat->stream>>>(
        pop, pair_list(s), n, rho, psi, g, lat->phys, a, inj);
  else
    k_mom_gather_pop<T, 1, WR><<<grid, kMomThreads, 0, lat->stream>>>(
        pop, pair_list(s), n, rho, psi, g, lat->phys, a, inj);
}

template <typename T>
mlbm_status to_populations(mlbm_lattice* lat) {
  using R = typename Pop<T>::Real;
  const MomentState& s = lat->mom;
  if (s.npairs == 0) return MLBM_OK;
  const Mom<R>* m = static_cast<const Mom<R>*>(s.m);
  T* pop = static_cast<T*>(lat->pop);
  if (lat->phase == 0)
    k_mom_populations<T, 0><<<pair_blocks(s), kMomThreads, 0, lat->stream>>>(
        m, pair_list(s), pop, lat->g, s.shift);
  else
    k_mom_populations<T, 1><<<pair_blocks(s), kMomThreads, 0, lat->stream>>>(
        m, pair_list(s), pop, lat->g, s.shift);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "populations of the moments");
  return MLBM_OK;
}

}  // namespace

// Packed coordinates and 32-bit node indexes bound the lattice.
bool moments_supported(const Geom& g) {
  return g.lx <= kC2MaxX && g.ly <= kC2MaxY && g.lz <= kC2MaxZ &&
         node_elems(g) < (1LL << 31);
}

size_t moments_max_bytes(const Geom& g, int storage) {
  if (!moments_supported(g)) return 0;
  return Parts(g, storage, (size_t)g.lx * g.ly * ((g.lz + 1) / 2)).total();
}

bool moments_apply(const mlbm_lattice* lat) {
  return lat->phys.omega == 1.f && !lat->slab && !lat->mom.no_room &&
         moments_supported(lat->g);
}

mlbm_status moments_prepare(mlbm_lattice* lat) {
  MomentState& s = lat->mom;
  if (s.list_built) return MLBM_OK;
  const mlbm_status st = build_list(lat);
  if (st == MLBM_ERR_NOMEM) {
    s.no_room = true;
    cudaGetLastError();  // not an error of the step: it runs on populations
  }
  return st;
}

template <typename T>
mlbm_status launch_moment_step(mlbm_lattice* lat, const StepArgs& a, bool write_u,
                               bool write_rho) {
  using R = typename Pop<T>::Real;
  MomentState& s = lat->mom;
  const Phys& p = lat->phys;
  const bool inj = p.rho_inject_period != 0ull &&
                   (unsigned long long)a.step % p.rho_inject_period == 0ull;
  if (s.npairs > 0) {
    const bool overlap = !stream_capturing(lat->stream);
    if (write_rho) launch_gather<T, true>(lat, a, inj, overlap);
    else launch_gather<T, false>(lat, a, inj, overlap);
    auto collide = write_u ? k_mom_collide<R, true> : k_mom_collide<R, false>;
    launch_overlapped(overlap, collide, pair_blocks(s), kMomThreads, 0, lat->stream,
                      (const MomPair<R>*)s.n, pair_list(s), (const R*)s.psi, (Mom<R>*)s.m,
                      lat->vel, lat->g, lat->phys);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "moment step launch");
  }
  s.active = true;
  s.shift = p.rho_shift;
  return MLBM_OK;
}
template mlbm_status launch_moment_step<float>(mlbm_lattice*, const StepArgs&, bool, bool);
template mlbm_status launch_moment_step<__half>(mlbm_lattice*, const StepArgs&, bool, bool);
template mlbm_status launch_moment_step<double>(mlbm_lattice*, const StepArgs&, bool, bool);

mlbm_status moments_sync_dense(mlbm_lattice* lat) {
  if (!lat->mom.active) return MLBM_OK;
  switch (lat->storage) {
    case MLBM_STORE_F32: return to_populations<float>(lat);
    case MLBM_STORE_F16: return to_populations<__half>(lat);
    default: return to_populations<double>(lat);
  }
}

mlbm_status moments_leave(mlbm_lattice* lat) {
  if (!lat->mom.active) return MLBM_OK;
  if (mlbm_status st = moments_sync_dense(lat)) return st;
  lat->mom.active = false;
  if (lat->mom.npairs == 0) return MLBM_OK;
  const Geom& g = lat->g;
  const dim3 grid((g.lx + 31) / 32, (g.ly + 7) / 8, g.lz), block(32, 8);
  if (lat->storage == MLBM_STORE_F64)
    k_mom_psi_back<double><<<grid, block, 0, lat->stream>>>(
        static_cast<const double*>(lat->mom.psi), static_cast<double*>(lat->psi), g);
  else
    k_mom_psi_back<float><<<grid, block, 0, lat->stream>>>(
        static_cast<const float*>(lat->mom.psi), static_cast<float*>(lat->psi), g);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "psi of the moments");
  return MLBM_OK;
}

mlbm_status moments_release(mlbm_lattice* lat) {
  MomentState& s = lat->mom;
  if (!s.buffer) return MLBM_OK;
  if (mlbm_status st = moments_leave(lat)) return st;
  const cudaError_t e = cudaStreamSynchronize(lat->stream);
  if (e != cudaSuccess) return cuda_fail(e, "moment buffers");
  moments_free(lat);
  return MLBM_OK;
}

// The lists stay where mask and slabs do: a step after a new initial state then
// allocates nothing and waits for nothing, so it can be captured into a graph.
void moments_reset(mlbm_lattice* lat) {
  MomentState& s = lat->mom;
  if (s.inlet != lat->phys.inlet_width || s.outlet != lat->phys.outlet_width)
    s.list_built = false;
  s.inlet = lat->phys.inlet_width;
  s.outlet = lat->phys.outlet_width;
  s.no_room = false;
  s.active = false;
}

void moments_free(mlbm_lattice* lat) {
  cudaFree(lat->mom.buffer);
  lat->mom = MomentState{};
}

}  // namespace mlbm
