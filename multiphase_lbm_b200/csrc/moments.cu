// moments.cu -- host side of the moment step (moments.cuh): node list, buffers,
// launches, and the way back to populations.
#include <cuda_runtime.h>

#include <cub/cub.cuh>

#include "capi_internal.h"
#include "launch.cuh"
#include "moments.cuh"

namespace mlbm {

namespace {

unsigned blocks_of(long long n, int threads) {
  return (unsigned)((n + threads - 1) / threads);
}

size_t up256(size_t n) { return (n + 255) / 256 * 256; }

// The node list of the current mask, and the buffers (one allocation: m, n,
// list).  Waits for the node count.
mlbm_status build_list(mlbm_lattice* lat) {
  MomentState& s = lat->mom;
  const Geom& g = lat->g;
  const long long nwords = mom_tile_words(g);
  uint32_t* start = nullptr;
  size_t temp_bytes = 0;
  uint32_t count = 0;
  cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, temp_bytes, start, start,
                                                nwords + 1, lat->stream);
  if (e != cudaSuccess) return cuda_fail(e, "moment list");
  // scratch of the scan: the transfer buffer an upload has left (same
  // stream), else an allocation of its own
  const size_t words_bytes = up256((size_t)(nwords + 1) * sizeof(uint32_t));
  char* own = nullptr;
  char* buf = static_cast<char*>(lat->staging);
  if (lat->staging_bytes < words_bytes + temp_bytes) {
    e = cudaMalloc((void**)&own, words_bytes + temp_bytes);
    if (e != cudaSuccess) return cuda_fail(e, "moment list");
    buf = own;
  }
  start = reinterpret_cast<uint32_t*>(buf);
  k_mom_counts<<<blocks_of(nwords + 1, 256), 256, 0, lat->stream>>>(
      lat->mask, start, nwords, g);
  e = cub::DeviceScan::ExclusiveSum(buf + words_bytes, temp_bytes, start, start,
                                    nwords + 1, lat->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&count, start + nwords, sizeof count,
                        cudaMemcpyDeviceToHost, lat->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(lat->stream);
  if (e == cudaSuccess && (!s.buffer || count > s.list_cap)) {
    cudaFree(s.buffer);
    s.buffer = nullptr;
    s.list_cap = 0;
    const size_t node = 4 * real_bytes(lat->storage);
    const size_t m_bytes = up256((size_t)psi_elems(g) * node);
    const size_t n_bytes = up256((size_t)count * node);
    e = cudaMalloc(&s.buffer, m_bytes + n_bytes + (size_t)count * sizeof(uint2));
    if (e == cudaSuccess) {
      s.m = s.buffer;
      s.n = static_cast<char*>(s.buffer) + m_bytes;
      s.list = reinterpret_cast<uint2*>(static_cast<char*>(s.n) + n_bytes);
      s.list_cap = count;
    } else {
      s.buffer = nullptr;
    }
  }
  if (e == cudaSuccess && count) {
    k_mom_list<<<blocks_of(nwords * 32, 256), 256, 0, lat->stream>>>(
        lat->mask, lat->nbw, start, s.list, nwords, g);
    e = cudaGetLastError();
  }
  cudaFree(own);
  if (e != cudaSuccess) return cuda_fail(e, "moment list");
  s.count = (int)count;
  s.list_built = s.words_current = true;
  return MLBM_OK;
}

template <typename T, bool WR>
void launch_gather(mlbm_lattice* lat, const StepArgs& a, bool inj, bool overlap) {
  using R = typename Pop<T>::Real;
  MomentState& s = lat->mom;
  R* rho = static_cast<R*>(lat->rho);
  R* psi = static_cast<R*>(lat->psi);
  Mom<R>* n = static_cast<Mom<R>*>(s.n);
  const unsigned grid = blocks_of(s.count, kMomThreads);
  if (s.active) {
    launch_overlapped(overlap, k_mom_gather<T, WR>, grid, kMomThreads, lat->stream,
                      (const Mom<R>*)s.m, (const uint2*)s.list, s.count, n, rho,
                      psi, lat->g, lat->phys, a, inj, s.shift);
  } else {
    const T* pop = static_cast<const T*>(lat->pop);
    if (lat->phase == 0)
      k_mom_gather_pop<T, 0, WR><<<grid, kMomThreads, 0, lat->stream>>>(
          pop, s.list, s.count, n, rho, psi, lat->g, lat->phys, a, inj);
    else
      k_mom_gather_pop<T, 1, WR><<<grid, kMomThreads, 0, lat->stream>>>(
          pop, s.list, s.count, n, rho, psi, lat->g, lat->phys, a, inj);
  }
}

template <typename T>
mlbm_status to_populations(mlbm_lattice* lat) {
  using R = typename Pop<T>::Real;
  const MomentState& s = lat->mom;
  if (s.count == 0) return MLBM_OK;
  const unsigned grid = blocks_of(s.count, kMomThreads);
  const Mom<R>* m = static_cast<const Mom<R>*>(s.m);
  T* pop = static_cast<T*>(lat->pop);
  if (lat->phase == 0)
    k_mom_populations<T, 0><<<grid, kMomThreads, 0, lat->stream>>>(
        m, s.list, s.count, pop, lat->g, s.shift);
  else
    k_mom_populations<T, 1><<<grid, kMomThreads, 0, lat->stream>>>(
        m, s.list, s.count, pop, lat->g, s.shift);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "populations of the moments");
  return MLBM_OK;
}

}  // namespace

// Packed coordinates and 32-bit offsets bound the lattice.
bool moments_supported(const Geom& g) {
  return g.lx <= kC2MaxX && g.ly <= kC2MaxY && g.lz <= kC2MaxZ &&
         psi_elems(g) < (1LL << 31);
}

bool moments_apply(const mlbm_lattice* lat) {
  return lat->phys.omega == 1.f && !lat->slab && !lat->mom.no_room &&
         moments_supported(lat->g);
}

mlbm_status moments_prepare(mlbm_lattice* lat) {
  MomentState& s = lat->mom;
  mlbm_status st = MLBM_OK;
  if (!s.list_built) {
    st = build_list(lat);
  } else if (!s.words_current) {
    if (s.count)
      k_mom_words<<<blocks_of(s.count, 256), 256, 0, lat->stream>>>(
          lat->nbw, s.list, s.count, lat->g);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "moment list");
    s.words_current = true;
  }
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
  if (s.count > 0) {
    const bool overlap = !stream_capturing(lat->stream);
    if (write_rho) launch_gather<T, true>(lat, a, inj, overlap);
    else launch_gather<T, false>(lat, a, inj, overlap);
    auto collide = write_u ? k_mom_collide<R, true> : k_mom_collide<R, false>;
    launch_overlapped(overlap, collide, blocks_of(s.count, kMomThreads),
                      kMomThreads, lat->stream, (const Mom<R>*)s.n,
                      (const uint2*)s.list, s.count, (const R*)lat->psi,
                      (Mom<R>*)s.m, lat->vel, lat->g, lat->phys);
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
  if (mlbm_status st = moments_sync_dense(lat)) return st;
  lat->mom.active = false;
  return MLBM_OK;
}

void moments_invalidate(mlbm_lattice* lat) {
  lat->mom.list_built = false;
  moments_reset(lat);
}

void moments_reset(mlbm_lattice* lat) {
  lat->mom.words_current = false;
  lat->mom.no_room = false;
  lat->mom.active = false;
}

void moments_free(mlbm_lattice* lat) {
  MomentState& s = lat->mom;
  cudaFree(s.buffer);
  s = MomentState{};
}

}  // namespace mlbm
