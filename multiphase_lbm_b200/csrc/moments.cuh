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
// A step is
//   gather   per fluid node: pulls f_i(x) = f*_i(x - e_i) of its neighbours
//            (its own f*_opp(i) where x - e_i is solid: halfway
//            bounce-back), sums rho and the momentum j, writes psi(rho) and
//            n = (rho, j);
//   collide  per fluid node: Shan-Chen force from the neighbours' psi,
//            u = (j + tau F)/rho, writes m = (rho, u).
//
// Layout.  m and psi are dense, node (x, y, z) at ((z + 1) ly + y) px + x;
// planes z = -1 and z = lz hold the periodic images of the last and the first
// (x and y wrap by the offsets of a node's columns: with ghost copies in all
// axes the stores of the images took longer than the rest of the collide).
// A thread owns the nodes z and z + 1 (z even): the 36 populations of the pair
// come from 28 nodes in 9 columns, and what depends on the source node alone
// (1 - 1.5 u^2, the weights times rho) is formed once for the up to three
// populations that the pair takes from it.  Solid nodes' moments are never
// used.  Threads run over a list of the pairs that hold fluid (a pair with one
// solid node, 4-8 % of the nodes in the benchmarks' packings, idles half),
// ordered by tiles of 32 x kTileY x kTileZ nodes and by rows within, so that a
// block's loads share lines in all three directions.
//
// What bounds it: the gather (two thirds of a step) instruction issue and L1
// together -- about 750 instructions per warp of pairs, and the cache lines its
// loads touch: a warp of the list spans 2-3 runs of fluid along x, so a 16-byte
// load of its lanes touches 6 lines where a full row would touch 4 --, the
// collide the latency of its loads.  At 200^3, tau = 1, the population kernels
// (compact2.cuh) take 183 us a step in FP32 and 152 in FP16 storage, this step
// 109 and 112.  Tried there (FP32): one node per thread 155; the two
// nodes of a pair side by side with 32-byte loads 117 (19 requests in place of
// 28, but 9.7 lines each); pairs whose neighbours are all fluid listed first in
// each tile, to skip their bounce-back selects, 119 (the runs break up: 7.9
// lines); tiles staged in shared memory with packed FP32 arithmetic 190 (bank
// conflicts take the place of the lines); packed sums or own populations in
// registers 112-127; gather and collide blocks side by side in one launch
// 140-154; other tile shapes and block-to-SM orders, no gain.
//
// FP16 storage keeps its meaning: a population read by the gather is rounded
// to half(f* - t_i rho_shift) exactly as the population kernels store it.
#pragma once

#include "compact.cuh"
#include "compact2.cuh"
#include "kernels.cuh"
#include "lattice.cuh"

#include <type_traits>

namespace mlbm {

constexpr int kTileX = 32, kTileY = 8, kTileZ = 4;  // order of the pair list
constexpr int kMomThreads = 128;

// Neighbour words of the lists (k_build_nbr's, bits 0-20) also hold:
constexpr uint32_t NB_EDGE = 1u << 21;   // z = 0 or lz - 1: has an image

template <typename R>
struct alignas(4 * sizeof(R)) Mom {
  R d, x, y, z;  // density; velocity (m) or momentum (n)
};
template <typename R>
struct alignas(8 * sizeof(R)) MomPair {
  Mom<R> a, b;  // z, z + 1
};
template <typename R>
struct Two {
  R a, b;
};

// Node (x, y, z), 0 <= x < lx, 0 <= y < ly, -1 <= z <= lz, of m and psi.
__host__ __device__ __forceinline__ uint32_t node_element(const Geom& g, int x, int y,
                                                          int z) {
  return (uint32_t)((z + 1) * g.ly + y) * (uint32_t)g.px + (uint32_t)x;
}
// (one plane more, read for the node beside the box's last one when lz is odd)
__host__ __device__ __forceinline__ long long node_elems(const Geom& g) {
  return (long long)(g.lz + 3) * g.ly * g.px;
}

// Offsets of the columns around a node's (periodic in x and y) and of the
// plane above it.
struct Columns {
  int xm, xp, ym, yp, plane;
  __device__ __forceinline__ Columns(const Geom& g, int x, int y) {
    const int row = g.px;
    xm = x == 0 ? g.lx - 1 : -1;
    xp = x == g.lx - 1 ? 1 - g.lx : 1;
    ym = y == 0 ? (g.ly - 1) * row : -row;
    yp = y == g.ly - 1 ? (1 - g.ly) * row : row;
    plane = g.ly * row;
  }
  __device__ __forceinline__ int at(int dx, int dy) const {
    return (dx < 0 ? xm : dx > 0 ? xp : 0) + (dy < 0 ? ym : dy > 0 ? yp : 0);
  }
};

// Whole pairs move with one access (FP32: 32 bytes).
__device__ __forceinline__ MomPair<float> ld_pair(const MomPair<float>* p) {
  MomPair<float> v;
  asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v.a.d), "=f"(v.a.x), "=f"(v.a.y), "=f"(v.a.z), "=f"(v.b.d),
                 "=f"(v.b.x), "=f"(v.b.y), "=f"(v.b.z)
               : "l"(p));
  return v;
}
__device__ __forceinline__ void st_pair(MomPair<float>* p, const MomPair<float>& v) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p),
               "f"(v.a.d), "f"(v.a.x), "f"(v.a.y), "f"(v.a.z), "f"(v.b.d),
               "f"(v.b.x), "f"(v.b.y), "f"(v.b.z)
               : "memory");
}
__device__ __forceinline__ MomPair<double> ld_pair(const MomPair<double>* p) {
  return *p;
}
__device__ __forceinline__ void st_pair(MomPair<double>* p, const MomPair<double>& v) {
  *p = v;
}

// Call st(element) for the image of a node with z = 0 or z = lz - 1 (both in a
// box of one plane).
template <typename St>
__device__ __forceinline__ void for_images(const Geom& g, int x, int y, int z, St st) {
  if (z == 0) st(node_element(g, x, y, g.lz));
  if (z == g.lz - 1) st(node_element(g, x, y, -1));
}

// ---- the pair list --------------------------------------------------------------
struct PairList {
  const uint2* words;   // neighbour words of z and z + 1 (0: solid, outside)
  const uint32_t* xyz;  // pack_xyz of the first node (z even)
  int count;
};
struct PairAt {
  uint32_t na, nb;
  int x, y, z;
  uint32_t at;  // node_element of the first node
};
__device__ __forceinline__ PairAt pair_at(const Geom& g, const PairList& l, int k) {
  const uint2 w = __ldg(l.words + k);
  const uint32_t c = __ldg(l.xyz + k);
  PairAt q;
  q.na = w.x;
  q.nb = w.y;
  q.x = (int)(c & 2047u);
  q.y = (int)((c >> 11) & 2047u);
  q.z = (int)(c >> 22);
  q.at = node_element(g, q.x, q.y, q.z);
  return q;
}

__host__ __device__ constexpr int direction(int dx, int dy, int dz) {
  for (int i = 0; i < Q; ++i)
    if (ex(i) == dx && ey(i) == dy && ez(i) == dz) return i;
  return -1;
}

// ---- equilibrium ----------------------------------------------------------------
// A node's moments with what every population of it shares.
template <typename T>
struct Source {
  using R = typename Pop<T>::Real;
  Mom<R> m;
  R base, wd1, wd2;  // of Equilibrium; axis and diagonal weight times rho
  __device__ __forceinline__ explicit Source(const Mom<R>& v) : m(v) {
    base = Equilibrium<T>::base(rfma(v.z, v.z, rfma(v.y, v.y, rmul(v.x, v.x))));
    wd1 = rmul(weight<R>(1), v.d);
    wd2 = rmul(weight<R>(4), v.d);
  }
};

// e_i . u, added as collide() adds it (the opposite direction's is its negative).
template <typename R>
__device__ __forceinline__ R e_dot_u(int i, const Mom<R>& m) {
  R eu = R(0);
  if (ex(i)) eu = ex(i) > 0 ? m.x : -m.x;
  if (ey(i)) eu = ex(i) ? (ey(i) > 0 ? radd(eu, m.y) : rsub(eu, m.y))
                        : (ey(i) > 0 ? m.y : -m.y);
  if (ez(i)) eu = ex(i) || ey(i) ? (ez(i) > 0 ? radd(eu, m.z) : rsub(eu, m.z))
                                 : (ez(i) > 0 ? m.z : -m.z);
  return eu;
}
__host__ __device__ constexpr bool is_axis(int i) {
  return ex(i) * ex(i) + ey(i) * ey(i) + ez(i) * ez(i) == 1;
}

// feq_i of collide(), operation for operation.
template <typename T>
__device__ __forceinline__ typename Pop<T>::Real eq_population(int i,
                                                               const Source<T>& s) {
  using R = typename Pop<T>::Real;
  if (i == 0) return rmul(rmul(weight<R>(0), s.m.d), s.base);
  return rmul(is_axis(i) ? s.wd1 : s.wd2,
              Equilibrium<T>::term(s.base, e_dot_u<R>(i, s.m)));
}

// Both nodes' population as the storage format T holds it: stored with shift
// s_st, read back with shift s_ld (both t_i times a rho_shift).
template <typename T>
struct Stored {
  using R = typename Pop<T>::Real;
  static __device__ __forceinline__ Two<R> pass(Two<R> f, float, float) { return f; }
};
template <>
struct Stored<__half> {
  static __device__ __forceinline__ Two<float> pass(Two<float> f, float s_st,
                                                    float s_ld) {
    const float2 v = __half22float2(__float22half2_rn(
        make_float2(__fsub_rn(f.a, s_st), __fsub_rn(f.b, s_st))));
    return Two<float>{__fadd_rn(v.x, s_ld), __fadd_rn(v.y, s_ld)};
  }
};

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

// One population into a node's sums, in the order of sum_density() / collide().
template <typename R>
__device__ __forceinline__ void mom_sum(int i, R f, Mom<R>& n) {
  n.d = radd(n.d, f);
  if (ex(i)) n.x = ex(i) > 0 ? radd(n.x, f) : rsub(n.x, f);
  if (ey(i)) n.y = ey(i) > 0 ? radd(n.y, f) : rsub(n.y, f);
  if (ez(i)) n.z = ez(i) > 0 ? radd(n.z, f) : rsub(n.z, f);
}

// The sums of a pair.  FP16 storage adds both nodes at once in packed
// arithmetic (200^3: 117 us a step against 119); in FP32 and FP64 the register
// pairs cost more than the instructions saved (112 against 109).
template <typename T>
struct PairSums {
  using R = typename Pop<T>::Real;
  Mom<R> a{R(0), R(0), R(0), R(0)}, b{R(0), R(0), R(0), R(0)};
  __device__ __forceinline__ void add(int i, const Two<R>& f) {
    mom_sum(i, f.a, a);
    mom_sum(i, f.b, b);
  }
  __device__ __forceinline__ MomPair<R> pair() const { return MomPair<R>{a, b}; }
};
template <>
struct PairSums<__half> {
  float2 d = make_float2(0.f, 0.f), x = d, y = d, z = d;
  __device__ __forceinline__ void add(int i, const Two<float>& t) {
    const float2 f = make_float2(t.a, t.b);
    d = p_add(d, f);
    if (ex(i)) x = ex(i) > 0 ? p_add(x, f) : p_sub(x, f);
    if (ey(i)) y = ey(i) > 0 ? p_add(y, f) : p_sub(y, f);
    if (ez(i)) z = ez(i) > 0 ? p_add(z, f) : p_sub(z, f);
  }
  __device__ __forceinline__ MomPair<float> pair() const {
    return MomPair<float>{{d.x, x.x, y.x, z.x}, {d.y, x.y, y.y, z.y}};
  }
};

// What a gather leaves of one pair: its sums, after injection and the slabs'
// densities, and psi (and rho).
template <typename R, bool WRITE_RHO>
__device__ __forceinline__ void mom_put(const PairAt& q, MomPair<R> s,
                                        MomPair<R>* n, int k, R* rho, R* psi,
                                        const Geom& g, const Phys& p,
                                        const StepArgs& a, bool inj) {
  const int kind = nb_kind(q.na | q.nb);  // the same x: the same slab
  if (kind) {
    const R d = R(slab_density(p, kind));
    s.a = s.b = Mom<R>{d, R(0), R(0), R(0)};
  } else {
    s.a.d = mom_inject<R>(p, g, a, inj, q.y, s.a.d);
    s.b.d = mom_inject<R>(p, g, a, inj, q.y, s.b.d);
  }
  st_pair(n + k, s);
  const R va = psi_of<R>(p, s.a.d), vb = psi_of<R>(p, s.b.d);
  if (WRITE_RHO) {
    const int at = (int)node_index(g, q.x, q.y, q.z);
    if (q.na) rho[at] = s.a.d;
    if (q.nb) rho[at + g.ly * g.px] = s.b.d;
  }
  if (q.na) psi[q.at] = va;
  if (q.nb) psi[q.at + g.ly * g.px] = vb;
  if ((q.na | q.nb) & NB_EDGE) {
    if (q.na) for_images(g, q.x, q.y, q.z, [&](uint32_t i) { psi[i] = va; });
    if (q.nb) for_images(g, q.x, q.y, q.z + 1, [&](uint32_t i) { psi[i] = vb; });
  }
}

// ---- kernels ----------------------------------------------------------------------

// The populations of one pair, in the order the sums take them.
template <typename T>
struct Gather {
  using R = typename Pop<T>::Real;
  const Mom<R>* at;  // the first node's own moments
  Columns col;
  uint32_t na, nb;
  float st, ld;
  MomPair<R> own;
  PairSums<T> sum;

  // f_i of one node from source s, or from itself (o, the opposite direction)
  // where that is solid.  FP32 and FP64 form both and take one; FP16, whose
  // equilibrium is two operations longer, takes one of the operands first
  // (200^3: 113 us a step against 117; FP32 116 against 109).
  static __device__ __forceinline__ R one(int i, bool fluid, const Source<T>& s,
                                          const Source<T>& o) {
    if constexpr (std::is_same<T, __half>::value) {
      const R es = e_dot_u<R>(i, s.m), eo = e_dot_u<R>(i, o.m);
      const R ws = is_axis(i) ? s.wd1 : s.wd2, wo = is_axis(i) ? o.wd1 : o.wd2;
      return rmul(fluid ? ws : wo,
                  Equilibrium<T>::term(fluid ? s.base : o.base, fluid ? es : -eo));
    } else {
      const R fs = eq_population<T>(i, s), fo = eq_population<T>(opp(i), o);
      return fluid ? fs : fo;
    }
  }
  // f_i of both nodes from the sources sa, sb
  __device__ __forceinline__ Two<R> population(int i, const Source<T>& sa,
                                               const Source<T>& sb) {
    Two<R> f;
    if (i == 0)
      f = Two<R>{eq_population<T>(i, sa), eq_population<T>(i, sb)};
    else
      f = Two<R>{one(i, (na >> i) & 1u, sa, Source<T>(own.a)),
                 one(i, (nb >> i) & 1u, sb, Source<T>(own.b))};
    return Stored<T>::pass(f, st * weight<float>(i), ld * weight<float>(i));
  }
  // the three populations from the column (dx, dy): levels z - 1 .. z + 2
  __device__ __forceinline__ void column(int dx, int dy, Two<R>& f0, Two<R>& up,
                                         Two<R>& down) {
    const Mom<R>* c = at + col.at(dx, dy);
    const Source<T> lo(c[-col.plane]), a(dx || dy ? c[0] : own.a),
        b(dx || dy ? c[col.plane] : own.b), hi(c[2 * col.plane]);
    f0 = population(direction(-dx, -dy, 0), a, b);
    up = population(direction(-dx, -dy, 1), lo, a);
    down = population(direction(-dx, -dy, -1), b, hi);
  }
  __device__ __forceinline__ Two<R> diagonal(int dx, int dy) {
    const Mom<R>* c = at + col.at(dx, dy);
    return population(direction(-dx, -dy, 0), Source<T>(c[0]), Source<T>(c[col.plane]));
  }
  __device__ __forceinline__ void add(int i, const Two<R>& f) { sum.add(i, f); }
  __device__ __forceinline__ void run() {
    own.a = at[0];
    own.b = at[col.plane];
    Two<R> f0, f3, f12, f1, f6, f7, f2, f8, f9;
    column(0, 0, f0, f12, f3);
    add(0, f0);
    column(1, 0, f1, f7, f6);
    add(1, f1);
    column(0, 1, f2, f9, f8);
    add(2, f2);
    add(3, f3);
    add(4, diagonal(1, 1));
    add(5, diagonal(1, -1));
    add(6, f6);
    add(7, f7);
    add(8, f8);
    add(9, f9);
    Two<R> f10, f15, f16, f11, f17, f18;
    column(-1, 0, f10, f15, f16);
    add(10, f10);
    column(0, -1, f11, f17, f18);
    add(11, f11);
    add(12, f12);
    add(13, diagonal(-1, -1));
    add(14, diagonal(-1, 1));
    add(15, f15);
    add(16, f16);
    add(17, f17);
    add(18, f18);
  }
};

// Resident blocks the registers are held to.  FP32: 72 registers ran a 200^3
// step in 109 us and a 96^3 one in 14.9, 64 registers (8 blocks) in 112 and
// 15.4, 80 (6) in 111 and 15.2, 51 (10) in 121 and 17.9.  FP16: 64 registers 113
// at 200^3, 72 115.
template <typename T>
constexpr int mom_gather_blocks() { return sizeof(typename Pop<T>::Real) == 8 ? 4 : sizeof(T) == 2 ? 8 : 7; }

// Gather pass of pair k of a list.  A thread past its end passes the gate with
// the others (a branch around the gate cost 4 % of the step).
template <typename T, bool WRITE_RHO, bool PDL>
__device__ __forceinline__ void mom_gather(
    const Mom<typename Pop<T>::Real>* m, const PairList& list, int k,
    MomPair<typename Pop<T>::Real>* n, typename Pop<T>::Real* rho,
    typename Pop<T>::Real* psi, const Geom& g, const Phys& p, const StepArgs& a,
    bool inj, float shift_st) {
  using R = typename Pop<T>::Real;
  const bool some = k < list.count;
  const PairAt q = pair_at(g, list, some ? k : list.count - 1);
  pdl_gate<PDL>();
  if (!some) return;
  Gather<T> c{m + q.at, Columns(g, q.x, q.y), q.na, q.nb, shift_st, p.rho_shift};
  c.run();
  mom_put<R, WRITE_RHO>(q, c.sum.pair(), n, k, rho, psi, g, p, a, inj);
}

template <typename T, bool WRITE_RHO>
__global__ void __launch_bounds__(kMomThreads, mom_gather_blocks<T>())
    k_mom_gather(const Mom<typename Pop<T>::Real>* m, PairList list,
                 MomPair<typename Pop<T>::Real>* n, typename Pop<T>::Real* rho,
                 typename Pop<T>::Real* psi, Geom g, Phys p, StepArgs a, bool inj,
                 float shift_st) {
  const int k = blockIdx.x * kMomThreads + threadIdx.x;
  mom_gather<T, WRITE_RHO, true>(m, list, k, n, rho, psi, g, p, a, inj, shift_st);
}

// The gather of a step that starts from populations (the dense layout in AA
// phase PHASE): initial states, restored checkpoints, another tau before.
template <typename T, int PHASE>
__device__ __forceinline__ Mom<typename Pop<T>::Real> gather_node(
    const T* __restrict__ pop, uint32_t nb, int x, int y, int z, const Geom& g,
    const Phys& p) {
  using R = typename Pop<T>::Real;
  Mom<R> s{R(0), R(0), R(0), R(0)};
  if (!(nb & NB_SELF) || nb_kind(nb)) return s;
  Nbr w;
  w.init(g, x, y, z);
  R f[Q];
  gather<T, PHASE>(pop, g.plane, w, nb, w.n, R(p.rho_shift), f);
#pragma unroll
  for (int i = 0; i < Q; ++i) mom_sum(i, f[i], s);
  return s;
}

template <typename T, int PHASE, bool WRITE_RHO>
__global__ void __launch_bounds__(kMomThreads)
    k_mom_gather_pop(const T* __restrict__ pop, PairList list,
                     MomPair<typename Pop<T>::Real>* n, typename Pop<T>::Real* rho,
                     typename Pop<T>::Real* psi, Geom g, Phys p, StepArgs a,
                     bool inj) {
  using R = typename Pop<T>::Real;
  const int k = blockIdx.x * kMomThreads + threadIdx.x;
  if (k >= list.count) return;
  const PairAt q = pair_at(g, list, k);
  MomPair<R> s;
  s.a = gather_node<T, PHASE>(pop, q.na, q.x, q.y, q.z, g, p);
  s.b = gather_node<T, PHASE>(pop, q.nb, q.x, q.y, q.z + 1, g, p);
  mom_put<R, WRITE_RHO>(q, s, n, k, rho, psi, g, p, a, inj);
}

// Force, velocity shift of one node: collide()'s, operation for operation.
// s holds w_i psi sums; n the density and momentum.
template <typename R>
__device__ __forceinline__ void force_add(int i, R psi, R& sx, R& sy, R& sz) {
  const R wp = rmul(weight<R>(i), psi);
  if (ex(i)) sx = ex(i) > 0 ? radd(sx, wp) : rsub(sx, wp);
  if (ey(i)) sy = ey(i) > 0 ? radd(sy, wp) : rsub(sy, wp);
  if (ez(i)) sz = ez(i) > 0 ? radd(sz, wp) : rsub(sz, wp);
}
template <typename R>
__device__ __forceinline__ Mom<R> shifted_velocity(const Phys& p, const Mom<R>& n,
                                                   R psi, R sx, R sy, R sz,
                                                   int kind) {
  if (kind) return Mom<R>{n.d, R(0), R(0), R(0)};
  const R gp = rmul(-R(p.G), psi), tau = R(p.tau), inv = rrcp(n.d);
  return Mom<R>{n.d, rmul(rfma(tau, rmul(gp, sx), n.x), inv),
                rmul(rfma(tau, rmul(gp, sy), n.y), inv),
                rmul(rfma(tau, rmul(gp, sz), n.z), inv)};
}

// Collide pass of pair k of a list (k < list.count).
template <typename R, bool WRITE_U, bool PDL>
__device__ __forceinline__ void mom_collide(const MomPair<R>* n, const PairList& list,
                                            int k, const R* psi, Mom<R>* m,
                                            float* vel, const Geom& g, const Phys& p) {
  const PairAt q = pair_at(g, list, k);
  const Columns col(g, q.x, q.y);
  pdl_gate<PDL>();
  const MomPair<R> s = ld_pair(n + k);
  const R* at = psi + q.at;
  // psi of the columns: [dy + 1][dx + 1], levels z - 1, z, z + 1, z + 2
  Two<R> mid[9];
  R lo[9], hi[9];
#pragma unroll
  for (int j = 0; j < 9; ++j) {
    const int dx = j % 3 - 1, dy = j / 3 - 1;
    const R* c = at + col.at(dx, dy);
    mid[j] = Two<R>{c[0], c[col.plane]};
    if (dx * dy == 0) {
      lo[j] = c[-col.plane];
      hi[j] = c[2 * col.plane];
    }
  }
  R ax = R(0), ay = R(0), az = R(0), bx = R(0), by = R(0), bz = R(0);
#pragma unroll
  for (int i = 1; i < Q; ++i) {
    const int j = (ey(i) + 1) * 3 + ex(i) + 1;
    force_add(i, ez(i) == 0 ? mid[j].a : ez(i) > 0 ? mid[j].b : lo[j], ax, ay, az);
    force_add(i, ez(i) == 0 ? mid[j].b : ez(i) > 0 ? hi[j] : mid[j].a, bx, by, bz);
  }
  const int kind = nb_kind(q.na | q.nb);
  MomPair<R> u;
  u.a = shifted_velocity<R>(p, s.a, mid[4].a, ax, ay, az, kind);
  u.b = shifted_velocity<R>(p, s.b, mid[4].b, bx, by, bz, kind);
  if (WRITE_U) {
    const long long at0 = node_index(g, q.x, q.y, q.z);
    float* v = vel + 3 * at0;
    if (q.na) {
      v[0] = (float)u.a.x;
      v[1] = (float)u.a.y;
      v[2] = (float)u.a.z;
    }
    v += 3ll * g.ly * g.px;
    if (q.nb) {
      v[0] = (float)u.b.x;
      v[1] = (float)u.b.y;
      v[2] = (float)u.b.z;
    }
  }
  if (q.na) m[q.at] = u.a;
  if (q.nb) m[q.at + col.plane] = u.b;
  if ((q.na | q.nb) & NB_EDGE) {
    if (q.na) for_images(g, q.x, q.y, q.z, [&](uint32_t i) { m[i] = u.a; });
    if (q.nb) for_images(g, q.x, q.y, q.z + 1, [&](uint32_t i) { m[i] = u.b; });
  }
}

// Blocks run in reverse list order: what the gather wrote last is still in L2
// when the collide starts with it, and the next gather starts where the
// collide ended.
template <typename R, bool WRITE_U>
__global__ void __launch_bounds__(kMomThreads, sizeof(R) == 8 ? 6 : 8)
    k_mom_collide(const MomPair<R>* n, PairList list, const R* psi, Mom<R>* m,
                  float* vel, Geom g, Phys p) {
  const int k = (int)(gridDim.x - 1 - blockIdx.x) * kMomThreads + threadIdx.x;
  if (k < list.count) mom_collide<R, WRITE_U, true>(n, list, k, psi, m, vel, g, p);
}

// The populations of the fluid nodes, in the dense layout in AA phase PHASE
// (a step "from" the other phase leaves it): what the population kernels hold
// after the same steps, bit for bit.
template <typename T, int PHASE>
__global__ void __launch_bounds__(kMomThreads)
    k_mom_populations(const Mom<typename Pop<T>::Real>* __restrict__ m,
                      PairList list, T* __restrict__ pop, Geom g, float shift_st) {
  using R = typename Pop<T>::Real;
  const int k = blockIdx.x * kMomThreads + threadIdx.x;
  if (k >= list.count) return;
  const PairAt q = pair_at(g, list, k);
  for (int b = 0; b < 2; ++b) {
    const uint32_t nb = b ? q.nb : q.na;
    if (!nb) continue;
    const Source<T> s(m[q.at + b * g.ly * g.px]);
    R f[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) f[i] = eq_population<T>(i, s);
    Nbr w;
    w.init(g, q.x, q.y, q.z + b);
    scatter<T, PHASE ^ 1>(pop, g.plane, w, nb, w.n, R(shift_st), f);
  }
}

// psi of every node into this step's layout, the images in z included (the
// solid nodes' psi(rhos), which only initialisation writes).
template <typename R>
__global__ void k_mom_psi(const R* __restrict__ psi, R* __restrict__ out, Geom g) {
  const int x = blockIdx.x * 32 + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int z = (int)blockIdx.z - 1;
  if (x >= g.lx || y >= g.ly) return;
  out[node_element(g, x, y, z)] = psi[psi_index(g, x, y, z)];
}

// And back, ghost copies included: what the population kernels' passes find.
template <typename R>
__global__ void k_mom_psi_back(const R* __restrict__ psi, R* __restrict__ out, Geom g) {
  const int x = blockIdx.x * 32 + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int z = (int)blockIdx.z;
  if (x >= g.lx || y >= g.ly) return;
  store_psi<R>(out, g, x, y, z, psi[node_element(g, x, y, z)]);
}

// ---- tiles and lists -----------------------------------------------------------
struct TileGrid {
  int nx, ny, nz;
  __host__ __device__ explicit TileGrid(const Geom& g)
      : nx((g.lx + kTileX - 1) / kTileX), ny((g.ly + kTileY - 1) / kTileY),
        nz((g.lz + kTileZ - 1) / kTileZ) {}
  __host__ __device__ long long count() const { return (long long)nx * ny * nz; }
};

constexpr int kPairRows = kTileY * kTileZ / 2;
__device__ __forceinline__ uint32_t tile_word(const uint32_t* __restrict__ nbw,
                                              const Geom& g, int x, int y, int z) {
  if (x >= g.lx || y >= g.ly || z >= g.lz) return 0u;
  const uint32_t nb = nbw[node_index(g, x, y, z)];
  if (!(nb & NB_SELF)) return 0u;
  return nb | (z == 0 || z == g.lz - 1 ? NB_EDGE : 0u);
}

// One block of kPairRows warps per tile (warp = row (y, z / 2), lane = x).
// COUNT: counts[tile] = its pairs, for the host's scan.  Otherwise the list, at
// the places at[tile] that the scan gave.
template <bool COUNT>
__global__ void __launch_bounds__(32 * kPairRows)
    k_mom_tiles(const uint32_t* __restrict__ nbw, uint32_t* counts,
                const uint32_t* __restrict__ at, uint2* __restrict__ words,
                uint32_t* __restrict__ xyz, Geom g) {
  __shared__ uint32_t row_pairs[kPairRows];
  const TileGrid tg(g);
  const long long tile = blockIdx.x;
  const int lane = threadIdx.x & 31, row = threadIdx.x / 32;
  const int x = (int)(tile % tg.nx) * kTileX + lane,
            y = (int)(tile / tg.nx % tg.ny) * kTileY + row % kTileY,
            z = (int)(tile / ((long long)tg.nx * tg.ny)) * kTileZ + row / kTileY * 2;
  const uint32_t na = tile_word(nbw, g, x, y, z), nb = tile_word(nbw, g, x, y, z + 1);
  const bool any = (na | nb) != 0u;
  const uint32_t bp = __ballot_sync(~0u, any);
  if (lane == 0) row_pairs[row] = __popc(bp);
  __syncthreads();
  uint32_t pairs = 0, before = 0;
  for (int r = 0; r < kPairRows; ++r) {
    if (r == row) before = pairs;
    pairs += row_pairs[r];
  }
  if (COUNT) {
    if (threadIdx.x == 0) counts[tile] = pairs;
    return;
  }
  if (!any) return;
  const uint32_t k = at[tile] + before + __popc(bp & ((1u << lane) - 1u));
  words[k] = make_uint2(na, nb);
  xyz[k] = pack_xyz(x, y, z);
}

}  // namespace mlbm
