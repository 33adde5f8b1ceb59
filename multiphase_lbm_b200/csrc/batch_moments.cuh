// batch_moments.cuh -- the batched time step of domains with tau = 1, held as
// moments (moments.cuh): the gather pass and the collide pass of every domain
// of a batch, one launch each, with the per-pair work of the single-lattice
// kernels, so a domain advanced in a batch is bit-identical to the same domain
// advanced alone.
//
// Each domain owns a contiguous range of blocks; a table gives every block its
// domain and its place in the domain's pair list (one load; a search over the
// domains' block prefixes would be a chain of dependent ones).  The batch step
// is read from the device counter, which graph replays advance.
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

template <typename T, bool WRITE_RHO>
__global__ void __launch_bounds__(kMomThreads, mom_gather_blocks<T>())
    k_batch_mom_gather(const MomDomain* __restrict__ doms,
                       const MomBlock* __restrict__ blocks,
                       const long long* __restrict__ step, int delta, int reverse,
                       unsigned inject_type) {
  using R = typename Pop<T>::Real;
  const MomBlock b = blocks[blockIdx.x];
  const MomDomain& D = doms[b.domain];
  const StepArgs a{*step + delta - D.step_origin, reverse, inject_type};
  const bool inj = D.p.rho_inject_period != 0ull &&
                   (unsigned long long)a.step % D.p.rho_inject_period == 0ull;
  const int k = b.first + (int)threadIdx.x;
  mom_gather<T, WRITE_RHO, false>(
      static_cast<const Mom<R>*>(D.m), D.list, k,
      static_cast<MomPair<R>*>(D.n), static_cast<R*>(D.rho),
      static_cast<R*>(D.psi), D.g, D.p, a, inj, D.p.rho_shift);
}

template <typename R>
__global__ void __launch_bounds__(kMomThreads, sizeof(R) == 8 ? 6 : 8)
    k_batch_mom_collide(const MomDomain* __restrict__ doms,
                        const MomBlock* __restrict__ blocks) {
  const MomBlock b = blocks[gridDim.x - 1 - blockIdx.x];
  const MomDomain& D = doms[b.domain];
  const int k = b.first + (int)threadIdx.x;
  if (k < D.list.count)
    mom_collide<R, false, false>(static_cast<const MomPair<R>*>(D.n), D.list, k,
                                 static_cast<const R*>(D.psi),
                                 static_cast<Mom<R>*>(D.m), nullptr, D.g, D.p);
}

}  // namespace mlbm
