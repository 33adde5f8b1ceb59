// moments.cuh -- the two-pass time step of a lattice with tau = 1, held as
// the four moments (rho, u) of every fluid node instead of 19 populations.
//
// BGK with omega = 1/tau = 1 leaves f*_i = f_i + (feq_i - f_i) = feq_i(rho, u):
// the post-collision populations of a node are functions of its density and
// (force-shifted) velocity alone, so the state of a step is 4 numbers a node.
// Every kernel of this library computes f*_i = feq_i in that case (collide,
// collide2), and this step forms the same feq_i, with the same operations in
// the same order, where a node reads it; so it gives the bits of the
// population kernels, at 16 bytes read and 16 written per node and pass in
// place of 76.
//
// State between steps: m, one Mom per node in a dense array with a ghost
// layer on every side (psi_index), so that the 18 neighbours of any node sit
// at fixed offsets, periodic boundaries included.  Solid nodes' entries are
// never read.  A step is
//   gather   per fluid node: pulls f_i(x) = f*_i(x - e_i) of its neighbours
//            (its own f*_opp(i) where x - e_i is solid: halfway
//            bounce-back), sums rho and the momentum j, writes psi(rho) and
//            n[k] = (rho, j);
//   collide  per fluid node: Shan-Chen force from the neighbours' psi,
//            u = (j + tau F)/rho, writes m = (rho, u) and its ghost copies.
// n is indexed by the node's place k in the node list (k_mom_list): fluid
// nodes only, ordered by tiles of 32 x kTileY x kTileZ nodes, so the nodes of
// one block are neighbours in all three directions and share their loads in
// L1 (list entry: neighbour word with NB_EDGE, packed coordinates).
//
// FP16 storage keeps its meaning: a population read by the gather is rounded
// to half(f* - t_i rho_shift) exactly as the population kernels store it.
#pragma once

#include "compact.cuh"
#include "compact2.cuh"
#include "kernels.cuh"
#include "lattice.cuh"

namespace mlbm {

constexpr int kMomThreads = 256;
constexpr int kTileY = 4, kTileZ = 4;  // node list tiles: 32 x kTileY x kTileZ
// Bit of a node list entry's neighbour word: the node lies on a face of the
// box, so its psi and moments have ghost copies.
constexpr uint32_t NB_EDGE = 1u << 21;

template <typename R>
struct alignas(4 * sizeof(R)) Mom {
  R d, x, y, z;  // density; velocity (m) or momentum (n)
};

// Call st(index) for a node and each of its periodic ghost copies.
template <typename St>
__device__ __forceinline__ void for_ghosts(const Geom& g, int x, int y, int z,
                                           St st) {
  const int xs[3] = {x, x == 0 ? g.lx : INT_MIN, x == g.lx - 1 ? -1 : INT_MIN};
  const int ys[3] = {y, y == 0 ? g.ly : INT_MIN, y == g.ly - 1 ? -1 : INT_MIN};
  const int zs[3] = {z, z == 0 ? g.lz : INT_MIN, z == g.lz - 1 ? -1 : INT_MIN};
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    if (zs[c] == INT_MIN) continue;
#pragma unroll 1
    for (int b = 0; b < 3; ++b) {
      if (ys[b] == INT_MIN) continue;
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (xs[a] != INT_MIN) st((uint32_t)psi_index(g, xs[a], ys[b], zs[c]));
    }
  }
}

struct MomNode {
  uint32_t nb;
  int x, y, z;
  uint32_t i;  // psi_index
};

__device__ __forceinline__ MomNode mom_node(const Geom& g, uint2 e) {
  MomNode n;
  n.nb = e.x;
  n.x = (int)(e.y & 2047u);
  n.y = (int)((e.y >> 11) & 2047u);
  n.z = (int)(e.y >> 22);
  n.i = (uint32_t)((n.z + 1) * (g.ly + 2) + n.y + 1) * (uint32_t)g.pxg +
        (uint32_t)n.x + 4u;
  return n;
}

// f*_i = feq_i of a node with moments m, for a node reached against (flip)
// or along direction i: collide()'s equilibrium, operation for operation.
template <typename R>
__device__ __forceinline__ R eq_population(int i, const Mom<R>& m, bool flip) {
  const R usq15 = rmul(R(1.5), rfma(m.z, m.z, rfma(m.y, m.y, rmul(m.x, m.x))));
  const R base = rsub(R(1), usq15);
  if (i == 0) return rmul(rmul(weight<R>(0), m.d), base);
  R eu = R(0);
  if (ex(i)) eu = ex(i) > 0 ? m.x : -m.x;
  if (ey(i)) eu = ex(i) ? (ey(i) > 0 ? radd(eu, m.y) : rsub(eu, m.y))
                        : (ey(i) > 0 ? m.y : -m.y);
  if (ez(i)) eu = ex(i) || ey(i) ? (ez(i) > 0 ? radd(eu, m.z) : rsub(eu, m.z))
                                 : (ez(i) > 0 ? m.z : -m.z);
  eu = flip ? -eu : eu;
  const R sym = rfma(rmul(R(4.5), eu), eu, base);
  const R anti = rmul(R(3), eu);
  const R wd = rmul(weight<R>(i), m.d);
  return rmul(wd, radd(sym, anti));
}

// A population as the storage format T holds it: stored with shift s_st,
// read back with shift s_ld (both t_i times a rho_shift).
template <typename T>
__device__ __forceinline__ typename Pop<T>::Real stored(
    typename Pop<T>::Real f, typename Pop<T>::Real s_st,
    typename Pop<T>::Real s_ld) {
  T v;
  Pop<T>::st(&v, f, s_st);
  return Pop<T>::ld(&v, s_ld);
}

// Density injection with its step test hoisted out (inject_on for any R).
template <typename R>
__device__ __forceinline__ R mom_inject(const Phys& p, const Geom& g,
                                        const StepArgs& s, bool on, int y, R d) {
  if (!on || !((float)y < p.inject_position * (float)g.ly)) return d;
  const R inc = rmul(R(p.rho_increment), R(s.reverse));
  switch (s.inject_type) {
    case 0: return radd(d, inc);
    case 1: return d < R(p.rhol_spinodal) ? radd(d, inc) : d;
    case 2: return d > R(p.rhol_spinodal) ? radd(d, inc) : d;
    default: return d;
  }
}

// rho and j of the populations f, in the order of sum_density() / collide();
// injection and the slab density applied to rho.
template <typename R>
__device__ __forceinline__ Mom<R> mom_sums(const Phys& p, const Geom& g,
                                           const StepArgs& a, bool inj, int y,
                                           const R (&f)[Q]) {
  Mom<R> n{R(0), R(0), R(0), R(0)};
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    n.d = radd(n.d, f[i]);
    if (ex(i)) n.x = ex(i) > 0 ? radd(n.x, f[i]) : rsub(n.x, f[i]);
    if (ey(i)) n.y = ey(i) > 0 ? radd(n.y, f[i]) : rsub(n.y, f[i]);
    if (ez(i)) n.z = ez(i) > 0 ? radd(n.z, f[i]) : rsub(n.z, f[i]);
  }
  n.d = mom_inject<R>(p, g, a, inj, y, n.d);
  return n;
}

// What a gather leaves of one node.
template <typename R, bool WRITE_RHO>
__device__ __forceinline__ void mom_put(const MomNode& q, const Mom<R>& s,
                                        Mom<R>* n, int k, R* rho, R* psi,
                                        const Geom& g, const Phys& p) {
  n[k] = s;
  if (WRITE_RHO) rho[node_index(g, q.x, q.y, q.z)] = s.d;
  const R v = psi_of<R>(p, s.d);
  if (q.nb & NB_EDGE)
    for_ghosts(g, q.x, q.y, q.z, [&](uint32_t i) { psi[i] = v; });
  else
    psi[q.i] = v;
}

// Gather pass from moments.  m is read with plain loads only after the gate:
// the launch before wrote it.
template <typename T, bool WRITE_RHO>
__device__ __forceinline__ void mom_gather(const Mom<typename Pop<T>::Real>* m,
                                           uint2 e, int k,
                                           Mom<typename Pop<T>::Real>* n,
                                           typename Pop<T>::Real* rho,
                                           typename Pop<T>::Real* psi,
                                           const Geom& g, const Phys& p,
                                           const StepArgs& a, bool inj,
                                           float shift_st) {
  using R = typename Pop<T>::Real;
  const MomNode q = mom_node(g, e);
  Mom<R> s;
  if (nb_kind(q.nb)) {
    s = Mom<R>{R(slab_density(p, nb_kind(q.nb))), R(0), R(0), R(0)};
  } else {
    const int sy = g.pxg, sz = (g.ly + 2) * g.pxg;
    const R st = R(shift_st), ld = R(p.rho_shift);
    R f[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const bool own = i == 0 || !((q.nb >> i) & 1u);
      const int o = ex(i) + ey(i) * sy + ez(i) * sz;
      const Mom<R> v = m[own ? q.i : q.i - o];
      f[i] = stored<T>(eq_population<R>(i, v, i != 0 && own), st * weight<R>(i),
                       ld * weight<R>(i));
    }
    s = mom_sums<R>(p, g, a, inj, q.y, f);
  }
  mom_put<R, WRITE_RHO>(q, s, n, k, rho, psi, g, p);
}

// Collide pass.
template <typename R, bool WRITE_U>
__device__ __forceinline__ void mom_collide(const Mom<R>* n, uint2 e, int k,
                                            const R* psi, Mom<R>* m, float* vel,
                                            const Geom& g, const Phys& p) {
  const MomNode q = mom_node(g, e);
  Mom<R> s = n[k];
  if (nb_kind(q.nb)) {
    s.x = s.y = s.z = R(0);
  } else {
    const int py = g.pxg, pz = (g.ly + 2) * g.pxg;
    R sx = R(0), sy = R(0), sz = R(0);
#pragma unroll
    for (int i = 1; i < Q; ++i) {
      const R wp = rmul(weight<R>(i), psi[q.i + (ex(i) + ey(i) * py + ez(i) * pz)]);
      if (ex(i)) sx = ex(i) > 0 ? radd(sx, wp) : rsub(sx, wp);
      if (ey(i)) sy = ey(i) > 0 ? radd(sy, wp) : rsub(sy, wp);
      if (ez(i)) sz = ez(i) > 0 ? radd(sz, wp) : rsub(sz, wp);
    }
    const R gp = rmul(-R(p.G), psi[q.i]);
    const R tau = R(p.tau);
    const R inv_rho = rrcp(s.d);
    s.x = rmul(rfma(tau, rmul(gp, sx), s.x), inv_rho);
    s.y = rmul(rfma(tau, rmul(gp, sy), s.y), inv_rho);
    s.z = rmul(rfma(tau, rmul(gp, sz), s.z), inv_rho);
  }
  if (WRITE_U) {
    float* v = vel + 3 * node_index(g, q.x, q.y, q.z);
    v[0] = (float)s.x;
    v[1] = (float)s.y;
    v[2] = (float)s.z;
  }
  if (q.nb & NB_EDGE)
    for_ghosts(g, q.x, q.y, q.z, [&](uint32_t i) { m[i] = s; });
  else
    m[q.i] = s;
}

// ---- kernels ----------------------------------------------------------------

template <typename T, bool WRITE_RHO>
__global__ void __launch_bounds__(kMomThreads, 3)
    k_mom_gather(const Mom<typename Pop<T>::Real>* m,
                 const uint2* __restrict__ list, int count,
                 Mom<typename Pop<T>::Real>* n, typename Pop<T>::Real* rho,
                 typename Pop<T>::Real* psi, Geom g, Phys p, StepArgs a,
                 bool inj, float shift_st) {
  const int k = blockIdx.x * kMomThreads + threadIdx.x;
  if (k >= count) return;
  const uint2 e = __ldg(list + k);
  pdl_gate<true>();
  mom_gather<T, WRITE_RHO>(m, e, k, n, rho, psi, g, p, a, inj, shift_st);
}

// The gather of a step that starts from populations (the dense layout in AA
// phase PHASE): initial states, restored checkpoints, another tau before.
template <typename T, int PHASE, bool WRITE_RHO>
__global__ void __launch_bounds__(kMomThreads)
    k_mom_gather_pop(const T* __restrict__ pop, const uint2* __restrict__ list,
                     int count, Mom<typename Pop<T>::Real>* n,
                     typename Pop<T>::Real* rho, typename Pop<T>::Real* psi,
                     Geom g, Phys p, StepArgs a, bool inj) {
  using R = typename Pop<T>::Real;
  const int k = blockIdx.x * kMomThreads + threadIdx.x;
  if (k >= count) return;
  const MomNode q = mom_node(g, __ldg(list + k));
  Mom<R> s;
  if (nb_kind(q.nb)) {
    s = Mom<R>{R(slab_density(p, nb_kind(q.nb))), R(0), R(0), R(0)};
  } else {
    Nbr w;
    w.init(g, q.x, q.y, q.z);
    R f[Q];
    gather<T, PHASE>(pop, g.plane, w, q.nb, w.n, R(p.rho_shift), f);
    s = mom_sums<R>(p, g, a, inj, q.y, f);
  }
  mom_put<R, WRITE_RHO>(q, s, n, k, rho, psi, g, p);
}

// Blocks run in reverse list order: what the gather wrote last is still in L2
// when the collide starts with it, and the next gather starts where the
// collide ended.
template <typename R, bool WRITE_U>
__global__ void __launch_bounds__(kMomThreads, 4)
    k_mom_collide(const Mom<R>* n, const uint2* __restrict__ list, int count,
                  const R* psi, Mom<R>* m, float* vel, Geom g, Phys p) {
  const int k = (int)(gridDim.x - 1 - blockIdx.x) * kMomThreads + threadIdx.x;
  if (k >= count) return;
  const uint2 e = __ldg(list + k);
  pdl_gate<true>();
  mom_collide<R, WRITE_U>(n, e, k, psi, m, vel, g, p);
}

// The populations of the fluid nodes, in the dense layout in AA phase PHASE
// (a step "from" the other phase leaves it): what the population kernels hold
// after the same steps, bit for bit.
template <typename T, int PHASE>
__global__ void __launch_bounds__(kMomThreads)
    k_mom_populations(const Mom<typename Pop<T>::Real>* __restrict__ m,
                      const uint2* __restrict__ list, int count,
                      T* __restrict__ pop, Geom g, float shift_st) {
  using R = typename Pop<T>::Real;
  const int k = blockIdx.x * kMomThreads + threadIdx.x;
  if (k >= count) return;
  const MomNode q = mom_node(g, __ldg(list + k));
  const Mom<R> v = m[q.i];
  R f[Q];
#pragma unroll
  for (int i = 0; i < Q; ++i) f[i] = eq_population<R>(i, v, false);
  Nbr w;
  w.init(g, q.x, q.y, q.z);
  scatter<T, PHASE ^ 1>(pop, g.plane, w, q.nb, w.n, R(shift_st), f);
}

// ---- node list ----------------------------------------------------------------
// Mask words in tile order: word t of the list's order -> (x / 32, y, z).
__device__ __forceinline__ bool mom_tile_word(const Geom& g, long long t, int& w,
                                              int& y, int& z) {
  const int nty = (g.ly + kTileY - 1) / kTileY;
  const int in = (int)(t % (kTileY * kTileZ));
  long long tile = t / (kTileY * kTileZ);
  w = (int)(tile % g.wpr);
  tile /= g.wpr;
  y = (int)(tile % nty) * kTileY + in % kTileY;
  z = (int)(tile / nty) * kTileZ + in / kTileY;
  return y < g.ly && z < g.lz;
}
__host__ __device__ __forceinline__ long long mom_tile_words(const Geom& g) {
  return (long long)((g.ly + kTileY - 1) / kTileY) * ((g.lz + kTileZ - 1) / kTileZ) *
         g.wpr * kTileY * kTileZ;
}

static __global__ void k_mom_counts(const uint32_t* __restrict__ mask,
                                    uint32_t* __restrict__ counts,
                                    long long nwords, Geom g) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t > nwords) return;
  int w, y, z;
  uint32_t c = 0;
  if (t < nwords && mom_tile_word(g, t, w, y, z))
    c = __popc(mask[((long long)z * g.ly + y) * g.wpr + w]);
  counts[t] = c;
}

__device__ __forceinline__ uint32_t mom_word(const uint32_t* __restrict__ nbw,
                                             const Geom& g, int x, int y, int z) {
  const bool edge = x == 0 || y == 0 || z == 0 || x == g.lx - 1 ||
                    y == g.ly - 1 || z == g.lz - 1;
  return nbw[node_index(g, x, y, z)] | (edge ? NB_EDGE : 0u);
}

// The list's neighbour words again (a new initial state may move the slabs).
static __global__ void k_mom_words(const uint32_t* __restrict__ nbw,
                                   uint2* __restrict__ list, int count, Geom g) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const uint32_t c = list[k].y;
  list[k].x = mom_word(nbw, g, (int)(c & 2047u), (int)((c >> 11) & 2047u),
                       (int)(c >> 22));
}

// One warp per mask word; start[t] = list place of the word's first node.
static __global__ void k_mom_list(const uint32_t* __restrict__ mask,
                                  const uint32_t* __restrict__ nbw,
                                  const uint32_t* __restrict__ start,
                                  uint2* __restrict__ list, long long nwords,
                                  Geom g) {
  const long long t =
      ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  if (t >= nwords) return;
  const int lane = threadIdx.x & 31;
  int w, y, z;
  if (!mom_tile_word(g, t, w, y, z)) return;
  const uint32_t bits = mask[((long long)z * g.ly + y) * g.wpr + w];
  if (!((bits >> lane) & 1u)) return;
  const int x = 32 * w + lane;
  list[start[t] + __popc(bits & low_bits(lane))] =
      make_uint2(mom_word(nbw, g, x, y, z), pack_xyz(x, y, z));
}

}  // namespace mlbm
