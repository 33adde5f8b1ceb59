// batch_compact.cuh -- the batched time step over the compact (fluid-only)
// layout: the density pass and the update pass of every domain of a batch,
// one launch each, with the per-node work of the single-lattice compact
// kernels (pair.cuh), so a domain advanced in a batch is bit-identical to the
// same domain advanced alone.
//
// Each domain owns a contiguous range of blocks.  The AA phase of a domain
// at batch step s is phase_base ^ (s & 1).  Both passes run one node per
// thread in the gather step and one pair per thread in the local step, so a
// domain's block count depends on the parity of s: two block-prefix tables,
// one per parity, and the launch grid covers the larger total.  The batch step
// s is read from the device counter (graph replays advance it), so a captured
// graph stays valid for every start parity.
#pragma once

#include "batch.cuh"
#include "compact2.cuh"
#include "lattice.cuh"

#include <type_traits>

namespace mlbm {

constexpr int kBCThreads = kC2Threads;

struct CDomain {
  Geom g;
  Phys p;
  void* cpop;                 // [Q][cs] populations (T)
  const uint2* cinfo;         // [cs]
  const uint2* wtab;          // mask word table
  float* psi;
  float* rho;
  uint32_t cs;
  int nfluid;                 // compact slots (even)
  int phase_base;
  long long step_origin;
};

// Domain and local block of this block at batch step s, in reverse order (as
// k_cupdate's) or not; false if the block has no work at this parity.
template <bool REVERSE>
__device__ __forceinline__ bool bc_locate(const long long* __restrict__ pre,
                                          int n, long long s, int& d,
                                          long long& local) {
  const int par = (int)(s & 1);
  const long long* pp = pre + (size_t)par * (n + 1);
  const long long b = REVERSE ? pp[n] - 1 - blockIdx.x : blockIdx.x;
  if (REVERSE ? b < 0 : b >= pp[n]) return false;
  d = find_domain(pp, n, b);
  local = b - pp[d];
  return true;
}

// Blocks per SM, (density, update): 24 domains of edges 32-128 at tau 0.9, us per
// step FP32 / FP16: (10, 8) 302 / 270; (8, 7) 312 / 284, (10, 7) 309 / 274, (6, 8)
// 304 / 276, (12, 8) 311 / 279, (10, 10) 332 / 294; updates by pairs in both
// phases, blocks of 256, 321 / 291.
template <typename T, bool WRITE_RHO>
__global__ void __launch_bounds__(kBCThreads, 10)
    k_batch_cdensity(const CDomain* __restrict__ doms,
                     const long long* __restrict__ pre, int n,
                     const long long* __restrict__ step, int delta, int reverse,
                     unsigned inject_type) {
  const long long s = *step + delta;
  int d;
  long long local;
  if (!bc_locate<false>(pre, n, s, d, local)) return;
  const CDomain& D = doms[d];
  const int ph = D.phase_base ^ (int)(s & 1);
  StepArgs a{s - D.step_origin, reverse, inject_type};
  const bool inj = batch_inject(D.p, a.step);
  const long long t = local * kBCThreads + threadIdx.x;
  if (ph == 0) {
    if (t >= D.nfluid) return;
    node_density0<T, WRITE_RHO>(static_cast<const T*>(D.cpop), D.cs, D.cinfo,
                                D.wtab, (int)t, D.rho, D.psi, D.g, D.p, a, inj);
  } else {
    if (2 * t >= D.nfluid) return;
    pair_density<T, WRITE_RHO>(static_cast<const T*>(D.cpop), D.cs, D.cinfo,
                               (int)(2 * t), D.nfluid, D.rho, D.psi, D.g, D.p, a,
                               inj);
  }
}

template <typename T>
__global__ void __launch_bounds__(kBCThreads, 8)
    k_batch_cupdate(const CDomain* __restrict__ doms,
                    const long long* __restrict__ pre, int n,
                    const long long* __restrict__ step, int delta, int reverse,
                    unsigned inject_type) {
  const long long s = *step + delta;
  int d;
  long long local;
  if (!bc_locate<true>(pre, n, s, d, local)) return;
  const CDomain& D = doms[d];
  const int ph = D.phase_base ^ (int)(s & 1);
  StepArgs a{s - D.step_origin, reverse, inject_type};
  const bool inj = batch_inject(D.p, a.step);
  const long long t = local * kBCThreads + threadIdx.x;
  if ((ph == 0 ? t : 2 * t) >= D.nfluid) return;
  auto update = [&](auto eq) {
    if (ph == 0)
      node_update0<T, false, decltype(eq)::value>(
          static_cast<T*>(D.cpop), D.cs, D.cinfo, D.wtab, (int)t, D.psi, nullptr,
          D.g, D.p, a, inj);
    else
      pair_update<T, false, decltype(eq)::value>(
          static_cast<T*>(D.cpop), D.cs, D.cinfo, (int)(2 * t), D.nfluid, D.psi,
          nullptr, D.g, D.p, a, inj);
  };
  if (D.p.omega == 1.f) update(std::true_type());  // a batch with other taus beside
  else update(std::false_type());
}

}  // namespace mlbm
