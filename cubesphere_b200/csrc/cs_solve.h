// Host-side description of one resident solve (geometry + state on one
// device, one stream).  Shared by the launch wrappers of every .cu file.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <functional>
#include <memory>
#include <string>
#include <vector>

#include "cs_dev.cuh"

namespace cs {

struct FillMap {
  // Gather-then-scatter ghost exchange, one entry per ghost destination:
  // tmp[n] = value(src[n]) (negated when meta bit 3 is set; averaged with
  // the destination's pre-exchange value when bit 4 is set), then
  // field[dst[n]] = tmp[n].  meta bits 0-2 select the destination field
  // and bits 5-7 the source field: 0 U (offsets include the component),
  // 1 ent, 2 Bxf, 3 Byf, 4 Bzf.
  int32_t* d_src = nullptr;
  int32_t* d_dst = nullptr;
  uint8_t* d_meta = nullptr;
  double* d_tmp = nullptr;
  long long n = 0;
};

// Panel-edge ownership maps on the device (see build_sync_maps).
struct PanelSync {
  int32_t *f_dst = nullptr, *f_src = nullptr;
  int8_t *f_ddir = nullptr, *f_sdir = nullptr;
  int32_t *e_dst = nullptr, *e_src = nullptr;
  int8_t *e_df = nullptr, *e_sf = nullptr, *e_sign = nullptr;
  int32_t* e_cls = nullptr;  // ncls + 1 starts: the entries of one edge (its copies but the owner's)
  long long nf = 0, ne = 0, ncls = 0;
};

// Per-kernel device timing with CUDA events recorded on the solve's
// stream between consecutive launches (enabled by cs_profile_begin).
struct Prof {
  bool on = false;
  std::vector<cudaEvent_t> ev;     // ev[0]: start; ev[i]: end of launch i
  std::vector<const char*> name;   // name[i]: launch ending at ev[i]
  int n = 0;                       // events recorded since the last harvest
  std::vector<std::string> keys;   // accumulated per kernel name
  std::vector<double> ms;
  std::vector<long long> count;
};

// What depends on the mesh parameters only: the host geometry, its device
// copy, the ghost-exchange and panel-ownership maps and the resident
// geometry-only operators.  Built once and shared read-only by every solve
// on the same mesh (cs_mesh_share, the serving mesh cache); freed with its
// last user.
struct MeshRes {
  GeomHost host;
  DGeom g{};
  FillMap fill{};       // d_tmp stays null here: the staging buffer is per solve
  PanelSync psync{};
  void* op_m9 = nullptr;   // least-squares inverses in the state's type (FP32 in the precision form)
  void* op_m10 = nullptr;
  void* lsq_map = nullptr;  // LsqPanelMap[6] when row weights are panel 1's only
  bool m9_shared = false, m10_shared = false;  // which of op_m9 / op_m10 are panel 1's only
  float* pos_ext = nullptr;  // half extents of the zones for the positivity bound, [3][6 S]
  void* op_p2v = nullptr;  // CS_FLAG_P2 one-sided stencil inverses (state's type)
  void* op_p2e = nullptr;
  bool p2_shared = false;  // op_p2v / op_p2e are panel 1's only
  void* adp_lu = nullptr;   // per-panel factors (FP64) or the panel-shared inverse (state's type)
  int8_t* adp_piv = nullptr;
  int8_t* adp_pmap = nullptr;  // inverse shared by the panels: per panel [unknown map][sign]
  std::vector<void*> allocs;
  size_t bytes = 0;     // device bytes held
  bool on_device = false;
  MeshRes() = default;
  MeshRes(const MeshRes&) = delete;
  MeshRes& operator=(const MeshRes&) = delete;
  ~MeshRes() {
    for (void* q : allocs) cudaFree(q);
  }
};

struct Solve {
  cs_params p{};
  Dims d{};
  PhysC ph{};
  DGeom g{};
  DState st{};                // state of the plain (FP64) form
  DStateT<float> stF{};       // state of the precision (FP32 bulk) form
  bool fp32 = false;          // which of the two this solve uses
  std::shared_ptr<MeshRes> mesh = std::make_shared<MeshRes>();
  std::vector<void*> allocs;  // device allocations owned by the solve
  FillMap fill;
  PanelSync psync;
  cudaStream_t stream = nullptr;
  cudaMemPool_t pool = nullptr;  // stream-ordered pool of the solve's own arrays
  unsigned char* init_buf = nullptr;  // seeded harmonic terms of cs_init_problem
  size_t init_buf_bytes = 0;
  double* diag_buf = nullptr;         // cs_diag: result and partial sums
  unsigned long long* step10_keys = nullptr;  // STEP 10 min (9) and max (9) keys, with CS_FLAG_STEP10
  int device = 0;
  int sm_count = 148;
  bool has_mesh = false, has_state = false;
  bool first_rates = false;  // the last stage's rates are in the first stage's arrays (IMEX)
  long long launches = 0;  // kernels launched by this solve
  cudaGraph_t graph = nullptr;           // one step, captured by cs_steps / cs_batch_steps
  cudaGraphExec_t graph_exec = nullptr;  // its executable form
  long long graph_kernels = 0;           // kernels in that graph
  double grid_frac = 1.0;                // share of the SMs a launch's grid is sized for (autotuned in batches)
  // Asked before the mesh (first argument, bytes) or this solve (second) takes
  // device memory that cs_estimate_device_bytes does not count; where it says no
  // they do without.  Unset: the device's own room decides.
  std::function<bool(size_t, size_t)> reserve;
  Prof prof;
  std::string err;
};

// Attaches a solve (parameters set, no mesh yet) to a resident mesh and
// allocates its own state; builds the mesh first when it is not on the
// device yet.  Defined with the C ABI.
int mesh_attach(Solve& sv, const std::shared_ptr<MeshRes>& m);
// One whole step at the device-resident time step (stages and CFL
// reduction), and its capture into sv.graph / sv.graph_exec (kept until
// drop_graph or the solve's end).  Defined with the C ABI.
int run_step(Solve& sv);
int step_graph(Solve& sv);
void drop_graph(Solve& sv);
// Device-to-host read of the next time step and of the error flags.
int read_dt(Solve& sv, double* out);
int fail(Solve& sv, int code, const std::string& msg);
int cuda_fail(Solve& sv, cudaError_t e, const char* what);
// Device allocation owned by the solve (stream-ordered, zero-filled).
void* solve_alloc(Solve& sv, size_t bytes, cudaError_t& e);
// The seeded initial state built on the device (cs_init_problem).
int init_problem_device(Solve& sv, const cs_init_desc& desc);
// Layers beyond the panel's sides and beyond its radial ends that STEP 8.d
// solves.  The stage reads E in one layer (the edge EMFs); P12's STEPS 9.b / 9.c
// run on it and read point values of E, made of the ADP modes, one layer
// further, P2's stencils, run on one layer more where there are four, two.  Past
// the sides no more is needed, since the next stage's fill sets those zones
// anew; past the radial ends the zone B that STEP 8.d sets goes into what the
// ghosts carry to the next stage, so all layers are solved that have faces.
// Both follow from the mesh parameters and flags that solves on one mesh share.
struct AdpLayers {
  int side, radial;
};
inline AdpLayers adp_layers(const cs_params& p) { return {(p.flags & CS_FLAG_P2) ? p.nghost - 1 : 2, p.nghost - 1}; }
// Identity of the mesh a parameter set needs (solves with equal keys can
// share one MeshRes).
std::string mesh_key(const cs_params& p);

// Called after every launch (kernel == false for copies): counts kernel
// launches and, when profiling, records an event on the stream.
void mark(Solve& sv, const char* name, bool kernel = true);
// Records the start event of a profiled sequence (no-op when off).
void prof_start(Solve& sv);

// SMs a launch of this solve sizes its grid for (every kernel loops over
// its range with a grid stride, so the grid size never changes results).
inline int grid_sms(const Solve& sv) {
  const int n = (int)(sv.sm_count * sv.grid_frac + 0.5);
  return n < 1 ? 1 : n;
}

inline int blocks_for(long long n, int threads, int sm_count) {
  long long b = (n + threads - 1) / threads;
  long long cap = (long long)sm_count * 64;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

// Blocks of a launch over nt tiles that share data with their neighbours: one
// a tile, so that the tiles run in order and L2 still holds what a stretch of
// the mesh shares with the one before.  Blocks that stride over the mesh run
// far apart: k_flux 21.3 ms of a 6 x 128^2 x 64 step against 20.7 (FP32 14.1 /
// 13.1), k_faceB 6.0 / 5.6 (4.2 / 3.8), k_weno_slopes 7.5 / 6.8 (5.9 / 5.4);
// kernels that read each word once gain nothing.  A solve with a share of the
// device strides with per_sm blocks an SM of its share.
inline int tile_blocks(const Solve& sv, long long nt, int per_sm) {
  return (int)(sv.grid_frac < 1.0 ? std::min<long long>(nt, (long long)grid_sms(sv) * per_sm) : std::min<long long>(nt, 1 << 30));
}

// The panel's own columns with w radial ghosts at either end: what a stage
// moves.  The fill that starts the next stage sets every ghost beside the panel
// from such a column.  The radial ghosts carry over: all of their state where it
// is the caller's, and with outflow the entropy, which the padding leaves alone
// and which gives a ghost at the pressure floor its pressure (without the ghosts
// a 6 x 32^2 x 1 step would take 0.77 ms, not 0.81, a 6 x 128^2 x 64 one 67 of 68).
inline Range3 own_columns(const Dims& d, int w) { return {1, d.N, 1, d.N, 1 - w, d.nr + w}; }

}  // namespace cs

// The opaque context of the C ABI: one resident solve.
struct cs_ctx {
  cs::Solve sv;
};
