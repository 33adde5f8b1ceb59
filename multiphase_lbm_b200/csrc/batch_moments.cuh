// batch_moments.cuh -- the batched time step of domains with tau = 1, held as
// moments (moments.cuh): the gather pass and the collide pass of every domain
// of a batch, one launch each, with the per-pair work of the single-lattice
// kernels, so a domain advanced in a batch is bit-identical to the same domain
// advanced alone.
//
// Each domain owns a contiguous range of blocks.  The domains' descriptions and
// first blocks are a kernel parameter: what a block needs before its first load
// (the search for its domain, pointers, sizes) comes from the constant cache, and
// the sizes and parameters stay out of L1 and, mostly, of registers.  In device
// memory, with a table of every block's domain, they cost a chain of two loads at
// the head of each block and some 40 uniform loads a warp, and the gather spilled.
// 8 domains of 128^3 / 48 of edges 32-128 / 100 of 32^3, us per step: FP32 293 /
// 394 / 60 -> 265 / 360 / 56, FP16 281 / 378 / 57 -> 268 / 361 / 56, FP64 637 / 847 /
// 134 -> 485 / 649 / 106 (the injection test in 32 bits a good part of FP64's).
// A parameter holds 128 domains (23 KB of 32), more take more launches; up to 16
// the launch carries less: 1 / 8 / 16 domains of 32^3 6.7 / 10.8 / 15.9 us per
// step, with the parameter of 128 7.3 / 11.4 / 16.9; of 64^3 11.0 / 45.0 / 95.9
// against 11.6 / 47.3 / 98.7.  The batch step is read from the device counter,
// which graph replays advance.
#pragma once

#include "batch.cuh"
#include "moments.cuh"

namespace mlbm {

struct MomDomain {
  Geom g;
  Phys p;
  void* m;      // Mom<R>, dense (node_element)
  void* n;      // MomPair<R>, pair list
  void* psi;    // R, dense (node_element)
  void* rho;    // R, dense
  PairList list;
  long long step_origin;
};

struct MomBlock {
  int domain, first;  // first pair
};

// The domains of a launch and the first block of each (the entries past the last
// domain: INT_MAX).
template <int N>
struct MomDomains {
  MomDomain d[N];
  int block[N];

  __device__ __forceinline__ MomBlock find(int b) const {
    int lo = 0;
#pragma unroll
    for (int h = N / 2; h; h /= 2)
      if (block[lo + h] <= b) lo += h;
    return MomBlock{lo, (b - block[lo]) * kMomThreads};
  }
};

template <typename T, bool WRITE_RHO, int N>
__global__ void __launch_bounds__(kMomThreads, mom_gather_blocks<T>())
    k_batch_mom_gather(const __grid_constant__ MomDomains<N> doms,
                       const long long* __restrict__ step, int delta, int reverse,
                       unsigned inject_type) {
  using R = typename Pop<T>::Real;
  const MomBlock b = doms.find((int)blockIdx.x);
  const MomDomain& D = doms.d[b.domain];
  const StepArgs a{*step + delta - D.step_origin, reverse, inject_type};
  const bool inj = batch_inject(D.p, a.step);
  const int k = b.first + (int)threadIdx.x;
  if (k >= D.list.count) return;
  const PairAt q = pair_at(D.g, D.list, k);
  Gather<T> c{static_cast<const Mom<R>*>(D.m) + q.at, Columns(D.g, q.x, q.y),
              q.na, q.nb, D.p.rho_shift, D.p.rho_shift};
  c.run();
  mom_put<R, WRITE_RHO>(q, c.sum.pair(), static_cast<MomPair<R>*>(D.n), k,
                        static_cast<R*>(D.rho), static_cast<R*>(D.psi), D.g, D.p, a,
                        inj);
}

template <typename R, int N>
__global__ void __launch_bounds__(kMomThreads, sizeof(R) == 8 ? 7 : 8)
    k_batch_mom_collide(const __grid_constant__ MomDomains<N> doms) {
  const MomBlock b = doms.find((int)(gridDim.x - 1 - blockIdx.x));
  const MomDomain& D = doms.d[b.domain];
  const int k = b.first + (int)threadIdx.x;
  if (k < D.list.count)
    mom_collide<R, false, false>(static_cast<const MomPair<R>*>(D.n), D.list, k,
                                 static_cast<const R*>(D.psi),
                                 static_cast<Mom<R>*>(D.m), nullptr, D.g, D.p);
}

}  // namespace mlbm
