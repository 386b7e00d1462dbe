// mhc_engine.cuh -- host-side engine shared by the C ABI translation units:
// cases, groups of cases that share kernel templates, per-phase work lists,
// and the persistent launch helper.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <map>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/mahyco_b200.h"
#include "mhc_launch.cuh"
#include "mhc_resident.h"

namespace mhc {

// records the calling thread's error message (mhc_last_error) and returns code
int set_err(int code, const std::string& msg);

#define CK(x)                                                                              \
  do {                                                                                     \
    cudaError_t e_ = (x);                                                                  \
    if (e_ != cudaSuccess) return ::mhc::set_err(MHC_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_)); \
  } while (0)

enum Stage { S_IDLE = 0, S_SAVED, S_VELOCITY, S_BC, S_POSITION, S_GEOM, S_DENSITY, S_VISCO, S_ELASTO, S_ENERGY, S_REMAP,
             S_SWEPT /* remap sweeps done, remapVariables pending */ };

inline int cdiv(long long a, int b) { return (int)((a + b - 1) / b); }

}  // namespace mhc

struct Engine;

using namespace mhc;

struct mhc_case {
  mhc_case_params P;
  Mesh M;
  int DIM = 3, NE = 1, NV = 4;
  Fields F;
  Scalars* d_scal = nullptr;
  mhc_case_params* d_params = nullptr;
  cudaStream_t stream = nullptr;   // allocation stream (and launches when standalone)
  bool own_stream = false;
  std::vector<void*> allocs;
  std::vector<size_t> alloc_bytes;  // size of each allocation (checkpoints)
  std::vector<void*> scratch;       // allocations that hold nothing between iterations (not checkpointed)
  // asynchronous status read-back: two pinned slots and their events
  Scalars* h_scal = nullptr;
  cudaEvent_t scal_ev[2] = {nullptr, nullptr};
  int scal_next = 0;
  long long it_host = 1;           // iteration the next launched cycle runs
  int stage = S_IDLE;
  bool initialised = false;
  Engine* solo = nullptr;          // private engine of a standalone case
  int slot = -1;                   // index inside its engine
};

// ---------------------------------------------------------------------------
// engine
// ---------------------------------------------------------------------------
struct DevList {
  size_t off_cases = 0;  // offsets inside the engine's int arena
  size_t off_start = 0;
  int n = 0;             // member cases
  int total = 0;         // virtual blocks of all members
  int solo = -1;         // engine slot of the only member (n = 1)
};

struct Group {
  int DIM, NE, EULER, skip;
  int EL = 0, HG = 0;          // elasto-plastic model; anti-hourglass correction
  int CBC = 0;                 // cell-variable boundary conditions (Density, Energy, Pressure)
  int LIM = 0;                 // node-sweep instance: limiter 0-2, LIM_ORDER1 or LIM_GEN
  int CLIM = 0;                // cell-sweep instance: the same, LIM_O3 (third order) or LIM_PB (pente-borne)
  int TILE = 0;                // bit D: the classical cell sweep along D goes through a shared-memory tile
  int NTILE = 0;               // bit D: the same for the node sweep
  int ADV = 0;                 // sans-lagrange: prescribed velocities, no Lagrange phase, no dual projection
  int CSTS = 0;                // schema-csts with the remap: half-step velocity updates around the step
  int CET = 0;                 // a member has conservation-energie-totale (finalize cells reads the dual variables)
  long long it0;               // iteration of the members when the lists were built
  std::vector<int> members;
  // the same launches as another group (their lists aside): kernels, members
  // and the phase of the sweep rotation
  bool same_launches(const Group& o) const {
    return DIM == o.DIM && NE == o.NE && EULER == o.EULER && skip == o.skip && EL == o.EL && HG == o.HG &&
           CBC == o.CBC && LIM == o.LIM && CLIM == o.CLIM && TILE == o.TILE && NTILE == o.NTILE &&
           ADV == o.ADV && CSTS == o.CSTS && CET == o.CET && it0 % 6 == o.it0 % 6 &&
           members == o.members;
  }
  DevList init_cells, init_nodes, lag_nodes, lag_cells, fin_cells, fin_nodes, dt;
  DevList sw_cells[3], sw_nodes[3];
  DevList cases;               // offset into the case-index arena
};

struct Engine {
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::vector<mhc_case*> cases;
  CaseDesc* d_desc = nullptr;
  int desc_cap = 0;
  std::vector<CaseDesc> h_desc;  // the same on the host: a launch over one case passes its descriptor by value
  int* d_ints = nullptr;   // case indices and block prefix sums of every list
  size_t ints_cap = 0;
  std::vector<Group> groups;
  std::vector<int> h_ints;       // the int arena as last uploaded
  bool dirty = true;
  bool graph_stale = false;      // a launch setting changed: the captured graph is not kept by a rebuild
  long long cycles_since_build = 0;
  int nsm = 0;
  // timing
  bool timing = false;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  double stage_ms[MHC_NUM_STAGES] = {0};
  long long stage_launches[MHC_NUM_STAGES] = {0};
  // graph of one rotation period
  cudaGraphExec_t graph = nullptr;
  // grid of the work-list launches: 0 = one block per work item (the block
  // scheduler balances), k > 0 = k x the blocks the device holds at once
  // (persistent blocks striding over the list)
  int grid_scale = 0;
  // per-phase override of grid_scale (-1 = use grid_scale), set by a tuner
  int stage_scale[MHC_NUM_STAGES] = {-1, -1, -1, -1, -1, -1, -1};
  int cur_stage = -1;  // phase being launched (StageTimer scope)
  // side stream of the node sweeps (NodeFork), made at the first remap
  cudaStream_t side = nullptr;
  cudaEvent_t fork_ev = nullptr;
  cudaEvent_t node_ev[3] = {nullptr, nullptr, nullptr};  // after the node sweeps of sweep k
  bool side_failed = false;
  int forked = 0;  // sweeps of this remap whose node sweeps are on the side stream, not joined yet
  // layout of the y / z sweeps of classical-limiter cases, set by a caller
  // or the tuner (mhc_*_set_sweep_layout): 1 = warp per line, 0, 2 and 3 =
  // shared-memory tile
  int cell_layout = 0, node_layout = 0;
  // kernels this engine put on the GPU (graph replays count their nodes)
  long long launches = 0;
  long long graph_launches = 0;  // kernel nodes of the captured graph
  // page-locked staging of the launch lists (case descriptors, then the
  // int arena) and the event after their last upload, so that a rebuild
  // does not wait for the work in flight
  char* h_stage = nullptr;
  size_t stage_cap = 0;
  cudaEvent_t stage_ev = nullptr;
  // status gather of every case (one kernel + one copy)
  Scalars* d_gather = nullptr;
  Scalars* h_gather = nullptr;   // pinned
  int gather_cap = 0;
};


struct StageTimer {
  Engine* e;
  int stage;
  StageTimer(Engine* e_, int s) : e(e_), stage(s) {
    e->cur_stage = s;
    if (e->timing) cudaEventRecord(e->ev[0], e->stream);
  }
  ~StageTimer() {
    e->cur_stage = -1;
    if (!e->timing) return;
    cudaEventRecord(e->ev[1], e->stream);
    cudaEventSynchronize(e->ev[1]);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e->ev[0], e->ev[1]);
    e->stage_ms[stage] += ms;
    e->stage_launches[stage] += 1;
  }
};

// The node sweep of a direction needs that direction's mass fluxes and the
// node sweep before it; the next cell sweep, and the finalize pass of the
// cells, need only the cell sweeps.  So the node sweeps run on a side stream
// beside them: forked after their cell sweep, joined before the finalize pass
// of the nodes (side_join).  The mass fluxes have two buffers, by the parity
// of the sweep: the cell sweep k waits for the node sweep k - 2, which read
// the buffer it writes (side_reuse).  Within the scope e->stream is the side
// stream.  A timed cycle keeps one stream.
struct NodeFork {
  Engine* e;
  cudaStream_t main;
  int k;
  bool on;
  NodeFork(Engine* e_, int k_) : e(e_), main(e_->stream), k(k_), on(false) {
    if (e->timing || e->side_failed) return;
    if (!e->side) {
      int prio = 0;
      bool ok = cudaStreamGetPriority(main, &prio) == cudaSuccess &&
                cudaStreamCreateWithPriority(&e->side, cudaStreamNonBlocking, prio) == cudaSuccess &&
                cudaEventCreateWithFlags(&e->fork_ev, cudaEventDisableTiming) == cudaSuccess;
      for (cudaEvent_t& ev : e->node_ev) ok = ok && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) == cudaSuccess;
      if (!ok) {
        cudaGetLastError();
        e->side_failed = true;
        return;
      }
    }
    cudaEventRecord(e->fork_ev, main);
    cudaStreamWaitEvent(e->side, e->fork_ev, 0);
    e->stream = e->side;
    on = true;
  }
  ~NodeFork() {
    if (!on) return;
    e->stream = main;
    cudaEventRecord(e->node_ev[k], e->side);
    e->forked = k + 1;
  }
};

// before the cell sweep k: the node sweep that read its mass flux buffer
inline void side_reuse(Engine* e, int k) {
  if (k >= 2 && e->forked >= k - 1) cudaStreamWaitEvent(e->stream, e->node_ev[k - 2], 0);
}

// the main stream waits for every node sweep forked (the last one follows
// the others on the side stream)
inline void side_join(Engine* e) {
  if (e->forked == 0) return;
  cudaStreamWaitEvent(e->stream, e->node_ev[e->forked - 1], 0);
  e->forked = 0;
}

// sweep instances of a case (the template argument LIM of kb_sweep_nodes /
// kb_sweep_cells)
inline int node_sweep_mode(const mhc_case_params& P) {
  if (P.ordre_projection == 1) return LIM_ORDER1;
  return P.projection_limiteur_id >= MHC_MINMOD_G ? LIM_GEN : P.projection_limiteur_id;
}
inline int cell_sweep_mode(const mhc_case_params& P) {
  if (P.projection_pente_borne) return LIM_PB;
  return P.ordre_projection == 3 ? LIM_O3 : node_sweep_mode(P);
}

// Directions whose classical cell (nodes: node) sweep goes through a
// shared-memory tile (body_sweep_cells_tile: coalesced loads and stores, the
// warp-per-line arithmetic): every y / z sweep, unless the engine's layout is
// 1 (warp per line) or MHC_SWEEP_TILE=0 is in the environment.  Layout 3, once
// one thread per line chunk, is the tile too.
inline int tile_mask(const mhc_case* h, int layout, bool nodes) {
  // the seven elasto variables ride through the warp-per-line cell sweeps only
  if (!nodes && h->P.env[0].elasto_model && h->P.with_projection) return 0;
  if ((nodes ? node_sweep_mode(h->P) : cell_sweep_mode(h->P)) > LIM_ORDER1) return 0;
  const char* s = getenv("MHC_SWEEP_TILE");
  if (layout == 1 || (layout == 0 && s && *s == '0')) return 0;
  return h->DIM == 3 ? 6 : 2;
}

inline int group_node_phase(int LIM, int NTILE, int D) {
  return ((NTILE >> D) & 1) ? PH_SWNT0 + D : node_sweep_phase(LIM, D);
}

// phase of the cell sweep of a group along D
inline int group_cell_phase(int CLIM, int TILE, int D) {
  return ((TILE >> D) & 1) ? PH_SWCT0 + D : cell_sweep_phase(CLIM, D);
}

// directions the remap does not sweep: one cell thick, or not the axis of a
// per-axis Euler scheme (RemapADIService.cc:26-32)
inline int skip_mask(const mhc_case* h) {
  int m = 0;
  if (h->M.ncx == 1) m |= 1;
  if (h->M.ncy == 1) m |= 2;
  if (h->DIM == 3 && h->M.ncz == 1) m |= 4;
  const int s = h->P.is_euler_scheme;
  if (s >= MHC_EULER_X && s <= MHC_EULER_Z) m |= 7 & ~(1 << (s - MHC_EULER_X));
  return m;
}

// persistent grid for a kernel: resident blocks on the device
template <class K>
inline int resident_blocks(Engine* e, K kernel, int threads, size_t smem) {
  static ResidentBlocks cache;
  return e->nsm * cache.get((const void*)kernel, threads, smem, [&] {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1)
      per_sm = 1;
    return per_sm;
  });
}

template <class K, class... Args>
inline void plaunch(Engine* e, K kernel, int threads, size_t smem, const DevList& L, Args... args) {
  if (L.total <= 0) return;
  const int sc = (e->cur_stage >= 0 && e->stage_scale[e->cur_stage] >= 0) ? e->stage_scale[e->cur_stage] : e->grid_scale;
  int grid = sc == 0 ? L.total : std::min(L.total, resident_blocks(e, kernel, threads, smem) * sc);
  const PhaseList pl{e->d_ints + L.off_cases, e->d_ints + L.off_start, L.n, L.total};
  kernel<<<grid, threads, smem, e->stream>>>(e->d_desc, pl, args...);
  ++e->launches;
}


// a phase kernel over a list: the instance that takes the descriptor by value
// when the list holds one case, the one that reads the table otherwise.
// `pick` (MHC_KERNEL) names both.  STRIDED: the first one strides over the case
// itself, a device full of blocks is enough.
#define MHC_KERNEL(...) [](auto solo_) { constexpr bool SOLO = decltype(solo_)::value; return __VA_ARGS__; }

// `split`: blocks per item.
template <bool STRIDED = false, class Pick, class... Args>
inline void plaunch_split(Engine* e, Pick pick, int threads, size_t smem, const DevList& L, int split, Args... args) {
  if (L.total <= 0) return;
  const int sc = (e->cur_stage >= 0 && e->stage_scale[e->cur_stage] >= 0) ? e->stage_scale[e->cur_stage] : e->grid_scale;
  const PhaseList pl{e->d_ints + L.off_cases, e->d_ints + L.off_start, L.n, L.total};
  auto launch = [&](auto kernel, const auto& table) {
    const int k = sc == 0 && STRIDED && L.solo >= 0 ? 1 : sc;
    const int items = L.total * split;
    const int grid = k == 0 ? items : std::min(items, resident_blocks(e, kernel, threads, smem) * k);
    kernel<<<grid, threads, smem, e->stream>>>(table, pl, args...);
  };
  if (L.solo >= 0) launch(pick(std::true_type{}), CaseTable<true>{e->h_desc[L.solo]});
  else launch(pick(std::false_type{}), CaseTable<false>{e->d_desc});
  ++e->launches;
}

template <bool STRIDED = false, class Pick, class... Args>
inline void plaunch_case(Engine* e, Pick pick, int threads, size_t smem, const DevList& L, Args... args) {
  plaunch_split<STRIDED>(e, pick, threads, smem, L, 1, args...);
}

// Blocks a classical cell sweep of one case spends on an item, each with a
// share of the nv variables: up to 3 while all of them fit the device at once.
// A small sweep's time is the chain of its variables, one after another (211 x
// 157 cells, two environments, van Leer: 9.8 -> 8.3 us along x, 11.2 -> 8.2
// along y); with the device full a split only repeats the faces' geometry.
// The splitting blocks are an instance of their own: the shares' bounds as
// run-time values cost the full sweeps 3 % (256x64x64).
template <class Pick>
inline int variable_split(Engine* e, Pick pick, int threads, size_t smem, const DevList& L, int nv) {
  if (L.solo < 0 || L.total <= 0) return 1;
  const int room = resident_blocks(e, pick(std::true_type{}), threads, smem) / L.total;
  return std::max(1, std::min({3, nv, room}));
}

// a classical cell sweep of nv variables; `share` names the instance whose
// blocks split them
template <class Pick, class Share>
inline void plaunch_cells(Engine* e, Pick pick, Share share, int threads, size_t smem, const DevList& L, int nv, int k) {
  const int split = variable_split(e, share, threads, smem, L, nv);
  if (split > 1) plaunch_split(e, share, threads, smem, L, split, k, split);
  else plaunch_split(e, pick, threads, smem, L, 1, k, 1);
}

#define DISPATCH_GROUP(g, CALL)                                   \
  do {                                                            \
    if ((g).DIM == 2) {                                           \
      constexpr int DIM_ = 2;                                     \
      switch ((g).NE) {                                           \
        case 1: { constexpr int NE_ = 1; CALL; } break;           \
        case 2: { constexpr int NE_ = 2; CALL; } break;           \
        case 3: { constexpr int NE_ = 3; CALL; } break;           \
        default: { constexpr int NE_ = 4; CALL; } break;          \
      }                                                           \
    } else {                                                      \
      constexpr int DIM_ = 3;                                     \
      switch ((g).NE) {                                           \
        case 1: { constexpr int NE_ = 1; CALL; } break;           \
        case 2: { constexpr int NE_ = 2; CALL; } break;           \
        case 3: { constexpr int NE_ = 3; CALL; } break;           \
        default: { constexpr int NE_ = 4; CALL; } break;          \
      }                                                           \
    }                                                             \
  } while (0)


// one performed sweep (cells, then nodes) of direction D as the k-th of the
// cycle, for the members of a group (mhc_sweeps.cu)
void sweep_step_any(Engine* e, Group& g, int D, int k);

// engine operations defined in mhc_capi.cu and shared with the other C ABI
// translation units (mhc_services.cu)
namespace mhc {
int engine_rebuild_shared(Engine* e);
int solo_engine_shared(mhc_case* h);
void launch_remap_sweeps_shared(Engine* e);
void launch_remap_variables_shared(Engine* e);
int fetch_shared(cudaStream_t s, const void* dev, void* host, size_t bytes);
}  // namespace mhc
