// capi_internal.h -- the lattice handle behind the C ABI (not exported).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <vector>

#include "../../include/mlbm.h"
#include "errors.h"
#include "lattice.cuh"
#include "update_tma.cuh"

namespace mlbm {
// Fluid-only population layout (compact.cuh).  Built from the mask on first
// use; the dense buffers stay allocated, and the state moves between the two
// layouts on demand.
struct CompactState {
  bool built = false;      // tables match the current mask
  bool active = false;     // the compact buffer holds the current state
  long long nfluid = 0, cs = 0;
  void* cpop = nullptr;        // [Q][cs] populations (T)
  uint2* cinfo = nullptr;      // [cs] (neighbour word, packed x, y, z); with cpop
  uint2* wtab = nullptr;       // [rows * wpr + 1] (mask word, wbase); with wbase
  bool two_pass_ok = false;    // the compact kernels fit the lattice
  uint32_t* wbase = nullptr;   // [rows * wpr + 1]
  long long cap = 0;           // cs the buffers were allocated for
  size_t table_bytes = 0, pop_bytes = 0, alt_bytes = 0;  // of wbase, cpop, cpop_alt
  std::vector<long long> plane_start;  // [lz + 1] first compact index of each plane
  std::vector<uint32_t> row_start;     // [lz * ly + 1] first compact index of each row
  // one-pass step (band.cuh): the second population buffer and the tiling
  void* cpop_alt = nullptr;            // [Q][cs] populations (T)
  int band_rows = 4, band_planes = 24;  // requested rows per band, planes per chunk
  // stage size (compact slots) of the shape last launched, and its key
  int band_slot = 0, band_slot_rows = -1, band_slot_nb = -1, band_slot_storage = -1;
};

// The moment step (moments.cuh): lists and buffers, built on first use.
struct MomentState {
  bool list_built = false;  // the lists match the mask and the slabs
  int inlet = -1, outlet = -1;  // widths of the slabs of the initial state
  bool no_room = false;     // a buffer was refused: population kernels run
  bool active = false;      // m holds the current state
  void* buffer = nullptr;   // one allocation for all of the following
  size_t buffer_bytes = 0;
  void* m = nullptr;        // [node_elems] Mom<R>: density, velocity
  void* psi = nullptr;      // [node_elems] R
  void* n = nullptr;        // [npairs] MomPair<R>: density, momentum
  uint2* words = nullptr;   // [npairs] node pairs: neighbour words,
  uint32_t* xyz = nullptr;  //          packed x, y, z
  int npairs = 0;
  float shift = 0.f;        // rho_shift the state was produced under
};

// Bound of the step kernels' device waits, and the test switch that makes
// one wait run out.
constexpr unsigned long long kDefaultWaitNs = 1000000000ull;  // 1 s
}  // namespace mlbm

struct mlbm_lattice {
  int device = 0;
  int storage = MLBM_STORE_F32;
  mlbm::Geom g{};
  mlbm_params params{};
  mlbm::Phys phys{};
  cudaStream_t stream = nullptr;
  bool stream_owned_sync = true;

  void* buffer = nullptr;       // one allocation for pop .. nbw and err
  size_t buffer_bytes = 0;
  bool cleared = false;         // what starts as zeros is (lattice_clear)
  size_t memory_limit = 0;      // mlbm_test_memory_limit; 0: none
  void* pop = nullptr;          // 19 planes of g.plane elements (T)
  void* rho = nullptr;          // density, R per node
  void* psi = nullptr;          // pseudopotential, R per node
  float* rho_init = nullptr;    // uploaded initial density (internal layout)
  uint32_t* mask = nullptr;     // 1 bit per node, 1 = fluid
  uint32_t* nbw = nullptr;      // per-node neighbour word (kernels.cuh)
  float* vel = nullptr;         // [node][3], written on request
  void* staging = nullptr;      // reference-layout transfer buffer
  size_t staging_bytes = 0;
  uint32_t* stat_words = nullptr;  // [2][mask words] bits of the statistics pass
  double* stats_scratch = nullptr;
  size_t stats_scratch_bytes = 0;

  // update pass: z-march tiles and the TMA descriptor of the psi tensor
  mlbm::ZMarch zm{};
  alignas(64) CUtensorMap psi_map;

  int* err = nullptr;                      // device error flag (wait timeout)
  int step_kernel = 0;                     // MLBM_KERNEL_*
  mlbm::CompactState compact{};            // fluid-only layout (compact.cuh)
  mlbm::MomentState mom{};                 // moment step (moments.cuh)

  unsigned long long wait_ns = mlbm::kDefaultWaitNs;  // bounded waits
  bool stall_test = false;  // the next step launch makes a wait run out
  int phase = 0;  // 0: post-collision at opp slots of own node; 1: pushed
  // count the calls on this lattice after which tables made of it (batch.cu)
  // are out of date: of its parameters and lists, of its phase and layout
  unsigned long long changes = 0, moves = 0;
  bool slab = false;  // planes 0 and lz - 1 are halo planes (slab.cu)
  bool has_params = false, has_mask = false, has_rho = false;
  bool initialized = false;
  bool vel_valid = false;
};

namespace mlbm {
mlbm_status cuda_fail(cudaError_t e, const char* where);
// Before a lattice's first work: its psi, initial density, mask and error flag
// start as zeros (on its stream).
mlbm_status lattice_clear(mlbm_lattice* lat);
// Zero velocity everywhere (where the field is allocated): solid nodes are never
// written and read zero, so a new mask needs it too.
cudaError_t velocity_clear(mlbm_lattice* lat);
// Device bytes a lattice holds.
size_t held_bytes(const mlbm_lattice* lat);
// Device memory for a lattice.  Where it is refused while the lattice holds
// the moment step's buffers, lattice_malloc gives those back (the lattice then
// runs on populations) and asks again: they are there for speed, and what ran
// without them must run beside them.
cudaError_t lattice_try_malloc(const mlbm_lattice* lat, void** p, size_t bytes);
cudaError_t lattice_malloc(mlbm_lattice* lat, void** p, size_t bytes);
size_t pop_elem_bytes(int storage);
size_t real_bytes(int storage);
Geom make_geom(int lx, int ly, int lz);
// (Re)build the update pass's tile shape and psi tensor map.
mlbm_status setup_update(mlbm_lattice* lat, int rows, int planes);
struct StepArgs;
// The fluid-only layout (compact.cu); compact_leave and compact_sync_dense
// also take a state held as moments to dense populations.
mlbm_status compact_enter(mlbm_lattice* lat);   // dense -> compact state
mlbm_status compact_leave(mlbm_lattice* lat);   // compact -> dense state
mlbm_status compact_sync_dense(mlbm_lattice* lat);  // dense copy, stay compact
void compact_invalidate(mlbm_lattice* lat);     // the mask changed
void compact_free(mlbm_lattice* lat);
template <typename T>
mlbm_status launch_compact_two_pass(mlbm_lattice* lat, const StepArgs& a,
                                    bool write_u, bool write_rho);
template <typename T>
mlbm_status launch_compact_pass(mlbm_lattice* lat, const StepArgs& a, int pass,
                                bool write_u, bool write_rho);
bool compact_two_pass_supported(int lx, int ly, int lz, int storage);
// One-pass step over the compact layout with two buffers (compact.cu,
// band.cuh); starts and ends in AA phase 1.
template <typename T>
mlbm_status launch_compact_band(mlbm_lattice* lat, const StepArgs& a,
                                bool write_u, bool write_rho);
bool compact_band_supported(const mlbm_lattice* lat);
// Whether the lattice's bands fit shared memory (tables built); where they
// do not, BAND steps run as compact two-pass steps.
bool compact_band_fits(mlbm_lattice* lat);
// The moment step (moments.cu): tau = 1, any storage, whole lattices.
bool moments_supported(const Geom& g);
bool moments_apply(const mlbm_lattice* lat);
size_t moments_max_bytes(const Geom& g, int storage);  // every node fluid; 0: unsupported
mlbm_status moments_prepare(mlbm_lattice* lat);      // lists and buffers
// One step; starts from moments, or from populations in the dense layout.
template <typename T>
mlbm_status launch_moment_step(mlbm_lattice* lat, const StepArgs& a,
                               bool write_u, bool write_rho);
mlbm_status moments_sync_dense(mlbm_lattice* lat);   // dense copy, stay
mlbm_status moments_leave(mlbm_lattice* lat);        // moments -> dense state
mlbm_status moments_release(mlbm_lattice* lat);      // leave; buffers freed
void moments_reset(mlbm_lattice* lat);  // a new initial state
void moments_free(mlbm_lattice* lat);
mlbm_status compact_set_band_shape(mlbm_lattice* lat, int rows, int planes);
}  // namespace mlbm
