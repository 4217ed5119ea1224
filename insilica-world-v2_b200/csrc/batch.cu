// Batched step: every registered stack (a Layers object with its state, optionally its Transport and tracers)
// advanced by one time-split RK3 step, its receiving masses and one FCT transport step, as ONE CUDA graph per step.
//
// Each phase is one kernel over every stack at once: a table of chunks (stack, up to 256 items of its cells, edges,
// vertices or tracer rows), one chunk per block, the stack's descriptor staged in shared memory. Stacks may sit on
// different grids and have different layer counts. The barotropic fast loop of a stage and the stage's end are one
// cooperative kernel over tiles per precision form (fast_tiles.cu): k sub-steps per exchange between neighbouring tiles
// instead of two launches per sub-step; stacks whose tiles would not fit on chip take the sub-steps, the limiter and the
// stage's end as grid-wide kernels. The phase functions are the per-call path's (layers_fp64.cuh, transport_fp64.cuh), so
// every stack's result is bit-identical to stepping it alone, whatever else shares the launches.
//
// Per step: init (+ first Laplacian pass) | lap e | lap cv | lap e | per stage: A, E, S, tiles (untiled: sub-steps, CS, D) |
// vmix + FCT stage-1 edge fluxes | P1 (receiving masses, td, p1) | P2E | P2 | P3E | P3 | P4 (and M <- M1).
//
// The tile kernel's waits (and the persistent grid-wide loop's barrier) are iteration-bounded, time-bounded spins
// (globaltimer): if a wait runs out it records ISW_ETIMEOUT in the batch's status word and every block returns. The last
// stage's end checks every new thickness and records ISW_ENOTFINITE for a NaN or Inf. The kernel that records a failure also
// writes it to a mapped host word, and isw_batch_step refuses to run while that word is set (until isw_batch_status resets
// it), so a caller that never polls cannot step on a half-updated state.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <list>
#include <map>
#include <memory>
#include <vector>

#include "batch.cuh"
#include "common.cuh"
#include "handles.cuh"
#include "layers_air.cuh"
#include "layers_fp64.cuh"
#include "tiles.cuh"
#include "transport_fp64.cuh"

namespace isw {
using namespace bt;
namespace {

// The grid-wide sub-step passes over a wide chunk: PH_ETA's cells, PH_UF's edges (also forming the layer fluxes on
// the stack's last sub-step); air stacks and sub-step 0's cell pass (which also forms the slot
// coefficients) item by item.
template <int PH, int LMAXK, bool EXT>
__device__ __forceinline__ void substep_chunk(const StackDesc &d, int st, int j, const Chunk &ch) {
  if (j >= d.n[st]) return;
  const LayersDev &M = d.M;
  const double tau = d.tau[st];
  const int first = ch.begin + (int)threadIdx.x;
  if (EXT && M.air) {
    for (int i = first; i < ch.end; i += THREADS) {
      if (PH == PH_ETA) ISW_BATCH_L(d.L, LMAXK, fp64::af_muphi_cell<LL>(M, tau, i));
      else ISW_BATCH_L(d.L, LMAXK, fp64::af_u_edge<LL>(M, tau, i));
    }
  } else if (PH == PH_ETA) {
    if (j == 0)
      for (int i = first; i < ch.end; i += THREADS) fp64::bt_eta_cell_y(M, tau, 0, i);
    else
      fp64::bt_eta_cells_y<SUB_WC>(M, tau, first, ch.end);
  } else {
    fp64::bt_u_edges_y<SUB_W_FP64, EXT>(M, tau, first, ch.end);
    if (j == d.n[st] - 1) {
      const StageArgs a = stage_args(d, st);
      for (int i = first; i < ch.end; i += THREADS) fp64::flux_edge<EXT>(M, a, M.acc[i], i);
    }
  }
}

// EXT: the kernel also carries the air branch and the option branches (walls, the shelf and its bed flags, per-cell
// buoyancy, the tide, the bottom's drag), instantiated only for batches holding such stacks, so that the plain
// Boussinesq phases keep their register count.
template <int PH, int LMAXK, bool EXT, int MINB = 0>
__global__ void __launch_bounds__(THREADS, MINB) k_phase(const StackDesc *__restrict__ S, const Sched sc, int st, int j) {
  Chunk ch{0, 0, 0};
  const int kind = phase_chunk<PH>(sc, blockIdx.x, ch);
  if (kind < 0) return;
  const StackDesc &d = stage_desc(S, ch.s);
  pdl_wait();
  pdl_trigger();
  if (Dom<PH>::wide) {                       // the grid-wide sub-step passes: a wide chunk, SUB_W items a thread
    substep_chunk<PH, LMAXK, EXT>(d, st, j, ch);
    return;
  }
  const int i = ch.begin + (int)threadIdx.x;
  if (PH == PH_S && d.s_stage) {             // the block stages its rows' distinct neighbour records, then computes
    extern __shared__ __align__(16) double stg[];
    const StageArgs a = stage_args(d, st);
    ISW_BATCH_L(d.L, LMAXK, fp64::stage_pk<LL>(d.M, ch.begin / THREADS, stg));
    __syncthreads();
    if (i < ch.end) ISW_BATCH_L(d.L, LMAXK, (fp64::slow_edge<LL, EXT, true>(d.M, a.cdt, i, nullptr, stg)));
    return;
  }
  if (i >= ch.end) return;
  const LayersDev &M = d.M;
  if (PH == PH_ONBED) {                      // the shelf's bed flags of every layer, before the step's first pass reads them
    if (EXT && M.ob) ISW_BATCH_L(d.L, LMAXK, fp64::onbed_cell<LL>(M, d.h, i));
  } else if (PH == PH_INIT) {
    if (kind == 0) {
      if (EXT && M.air) ISW_BATCH_L(d.L, LMAXK, fp64::air_stiff_cell<LL>(M, d.h, d.theta, i));
      else ISW_BATCH_L(d.L, LMAXK, fp64::eta0_cell<LL>(M, d.h, i));
      if (M.nu4 != 0) ISW_BATCH_L(d.L, LMAXK, fp64::div_cell<LL>(M, d.u, i));
    } else if (kind == 1) {
      if (!(EXT && M.air)) ISW_BATCH_L(d.L, LMAXK, fp64::ubar0_edge<LL, EXT>(M, d.h, d.u, i));
    } else if (M.nu4 != 0) {
      ISW_BATCH_L(d.L, LMAXK, fp64::curl_vertex<LL>(M, d.u, i));
    }
  } else if (PH == PH_LAPE1 || PH == PH_LAPE2) {
    if (M.nu4 != 0) ISW_BATCH_L(d.L, LMAXK, fp64::lap_edge<LL>(M, PH == PH_LAPE1 ? M.L1 : M.L2, i));
  } else if (PH == PH_LAPCV) {
    if (M.nu4 != 0) {
      if (kind == 0) ISW_BATCH_L(d.L, LMAXK, fp64::div_cell<LL>(M, M.L1, i));
      else ISW_BATCH_L(d.L, LMAXK, fp64::curl_vertex<LL>(M, M.L1, i));
    }
  } else if (PH == PH_A) {
    const StageArgs a = stage_args(d, st);
    if (kind == 0) {
      if (EXT && M.air) {
        ISW_BATCH_L(d.L, LMAXK, fp64::air_bern_cell<LL>(M, a.hs, a.us, d.theta, i));
        ISW_BATCH_L(d.L, LMAXK, fp64::air_fast_init_cell<LL>(M, a.h0, i));
      } else {
        ISW_BATCH_L(d.L, LMAXK, fp64::bern_cell<LL, EXT>(M, a.hs, a.us, i));
      }
    } else {
      ISW_BATCH_L(d.L, LMAXK, fp64::pv_vertex<LL>(M, a.hs, a.us, i));
    }
  } else if (PH == PH_E) {
    const StageArgs a = stage_args(d, st);
    ISW_BATCH_L(d.L, LMAXK, fp64::edge_hq<LL, EXT>(M, a.hs, a.us, i));
    if (EXT && M.air) ISW_BATCH_L(d.L, LMAXK, fp64::air_fast_init_edge<LL>(M, a.u0, i));
  } else if (PH == PH_S) {
    const StageArgs a = stage_args(d, st);
    ISW_BATCH_L(d.L, LMAXK, fp64::slow_edge<LL, EXT>(M, a.cdt, i, EXT && M.air ? d.theta : nullptr));
  } else if (PH == PH_CS) {
    const StageArgs a = stage_args(d, st);
    if (EXT && M.air) ISW_BATCH_L(d.L, LMAXK, fp64::air_scale_cell<LL>(M, a, i));
    else ISW_BATCH_L(d.L, LMAXK, fp64::scale_sum_cell<LL>(M, a, i));
  } else if (PH == PH_D) {
    const StageArgs a = stage_args(d, st);
    if (kind == 0) {
      ISW_BATCH_L(d.L, LMAXK, fp64::h_cell<LL>(M, a, i));
      if (st == 2 && d.check) check_finite_column(d.h, M.g.N, d.L, i, sc.status);
    } else if (EXT && M.air) {
      ISW_BATCH_L(d.L, LMAXK, fp64::air_u_edge<LL>(M, a, i));
    } else {
      ISW_BATCH_L(d.L, LMAXK, fp64::u_edge<LL, EXT>(M, a, i));
    }
  } else if (PH == PH_VMIX) {
    if ((M.vmix != 0 || M.vmix_cd != 0) && d.L > 1) ISW_BATCH_L(d.L, LMAXK, fp64::vmix_edge<LL, EXT>(M, d.h, d.u, d.dt, i));
  } else if (PH == PH_VHEAT) {
    if (EXT && M.air && d.theta && (M.vmix != 0 || M.vmix_cd != 0) && d.L > 1)
      ISW_BATCH_L(d.L, LMAXK, fp64::vmix_heat_cell<LL>(M, d.h, d.theta, i));
  } else if (PH == PH_HF1) {
    const EdgeRow r = edge_row(d, i);
    ISW_BATCH_L(d.L, LMAXK, fp64::tr_hf_edge<LL>(d.T, d.tr, 1, r.j0, r.j1, r.e));
  } else if (PH == PH_POST) {
    if (kind == 1) {
      if ((M.vmix != 0 || M.vmix_cd != 0) && d.L > 1) ISW_BATCH_L(d.L, LMAXK, fp64::vmix_edge<LL, EXT>(M, d.h, d.u, d.dt, i));
    } else {
      const EdgeRow r = edge_row(d, i);
      ISW_BATCH_L(d.L, LMAXK, fp64::tr_hf_edge<LL>(d.T, d.tr, 1, r.j0, r.j1, r.e));
    }
  } else if (PH == PH_P1 || PH == PH_P1G) {
    const CellRow r = cell_row(d, i);
    ISW_BATCH_L(d.L, LMAXK, (fp64::tr_c1<LL, phase_tracers<PH>()>(d.T, d.tr, r.j0, r.n, r.c)));
  } else if (PH == PH_P2E) {
    const EdgeRow r = edge_row(d, i);
    ISW_BATCH_L(d.L, LMAXK, fp64::tr_hf_edge<LL>(d.T, d.tr, 2, r.j0, r.j1, r.e));
  } else if (PH == PH_P2 || PH == PH_P2G) {
    const CellRow r = cell_row(d, i);
    ISW_BATCH_L(d.L, LMAXK, (fp64::tr_c2<LL, phase_tracers<PH>()>(d.T, d.tr, r.j0, r.n, r.c)));
  } else if (PH == PH_P3E) {
    const EdgeRow r = edge_row(d, i);
    ISW_BATCH_L(d.L, LMAXK, fp64::tr_a_edge<LL>(d.T, d.tr, r.j0, r.j1, r.e));
  } else if (PH == PH_P3) {
    ISW_BATCH_L(d.L, LMAXK, fp64::tr_c3<LL>(d.T, d.tr, i / M.g.N, i % M.g.N));
  } else if (PH == PH_P4) {
    const int jj = i / M.g.N, c = i % M.g.N;
    ISW_BATCH_L(d.L, LMAXK, fp64::tr_p4<LL>(d.T, d.tr, jj, c));
    if (jj == 0)
      for (int l = 0; l < d.L; l++) d.Mm[(size_t)l * M.g.N + c] = d.tr.M1[(size_t)l * M.g.N + c];
  }
}

// The grid-wide fast loop of stage `st` for the untiled FP64 stacks as ONE cooperative launch of co-resident blocks: each
// sub-step every block walks its share of the cell chunks (the eta pass), all blocks meet at the bounded grid barrier,
// walk the edge chunks (the ubar pass; a stack's last sub-step also forms its layer fluxes, as PH_UF does) and meet
// again. The per-item arithmetic is PH_ETA's and PH_UF's, which otherwise take two launches
// per sub-step; the barrier's acquire makes every block's writes of one pass visible to the next pass.
template <int LMAXK, bool EXT>
__global__ void __launch_bounds__(THREADS) k_fast_grid(const StackDesc *__restrict__ S, const Sched sc, int st, int nsub,
                                                        GridBarrier *bar, BatchStatus *status, long long timeout_ns) {
  __shared__ __align__(16) unsigned char buf[sizeof(StackDesc)];
  const StackDesc &d = *reinterpret_cast<const StackDesc *>(buf);
  int cur = -1;
  auto select = [&](int s) {                 // the chunk's stack descriptor in shared memory (s is block-uniform)
    if (s == cur) return;
    __syncthreads();
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(S + s);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(buf);
    for (int w = threadIdx.x; w < (int)(sizeof(StackDesc) / 8); w += blockDim.x) dst[w] = src[w];
    __syncthreads();
    cur = s;
  };
  for (int j = 0; j < nsub; j++) {
    for (int c = blockIdx.x; c < sc.nwcell; c += gridDim.x) {
      const Chunk ch = sc.wcell[c];
      select(ch.s);
      const int i = ch.begin + (int)threadIdx.x;
      if (i < ch.end && j < d.n[st]) {
        if (EXT && d.M.air) ISW_BATCH_L(d.L, LMAXK, fp64::af_muphi_cell<LL>(d.M, d.tau[st], i));
        else fp64::bt_eta_cell_y(d.M, d.tau[st], j, i);
      }
    }
    if (!grid_sync(bar, status, timeout_ns)) return;
    for (int c = blockIdx.x; c < sc.nuedge; c += gridDim.x) {
      const Chunk ch = sc.uedge[c];
      select(ch.s);
      const int i = ch.begin + (int)threadIdx.x;
      if (i < ch.end && j < d.n[st]) {
        if (EXT && d.M.air) {
          ISW_BATCH_L(d.L, LMAXK, fp64::af_u_edge<LL>(d.M, d.tau[st], i));
        } else {
          fp64::bt_u_edge_y<EXT>(d.M, d.tau[st], i);
          if (j == d.n[st] - 1) fp64::flux_edge<EXT>(d.M, stage_args(d, st), d.M.acc[i], i);
        }
      }
    }
    if (!grid_sync(bar, status, timeout_ns)) return;
  }
}

template <bool EXT>
const void *fast_grid_kernel_t(int lmax) {
  switch (lmax) {
    case 2: return (const void *)k_fast_grid<2, EXT>;
    case 3: return (const void *)k_fast_grid<3, EXT>;
    case 5: return (const void *)k_fast_grid<5, EXT>;
    default: return (const void *)k_fast_grid<8, EXT>;
  }
}

const void *fast_grid_kernel(int lmax, bool ext) { return ext ? fast_grid_kernel_t<true>(lmax) : fast_grid_kernel_t<false>(lmax); }

}  // namespace
}  // namespace isw

using namespace isw;

struct BatchSlot {
  bool used = false;
  isw_layers *layers = nullptr;
  isw_transport *tr = nullptr;
  double *h = nullptr, *u = nullptr, *Fm = nullptr, *M = nullptr, *M1 = nullptr;
  double *theta = nullptr;                  // air layers: the layers' potential temperature (L x N), else null
  int version = 0;                          // the layers' option version the descriptors were built from
  double *tracers[TRMAX] = {};
  int ntr = 0;
  double dt = 0;
  int nfast = 0;
};

struct FastGroup {
  int begin = 0, count = 0, form = 0, cap = 0;   // its tiles [begin, begin + count), their form, the kernel's capacity
  bool walls = false;                       // a stack of it has thin walls
  int waited = -1;                          // a tile of it that another waits for (-1: every stack is one tile)
  size_t smem = 0;
};

// One tiling of a grid: the host tables (layouts are planned on them) and, once a batch steps with it, the device's.
struct TileCache {
  TileSetDev dev{};
  TileSetHost host;
  std::vector<void *> allocs;
  ~TileCache() {
    for (void *p : allocs) cudaFree(p);
  }
};

// A grid's tile sets, kept with the grid so that the batches (and Layers) on it build each tiling once: at most
// TILE_STORE_MAX of them, the oldest that no batch uses dropped first (a batch holds those it steps with).
constexpr size_t TILE_STORE_MAX = 24;
struct TileStore {
  std::map<int, std::vector<int32_t>> parts;                                   // cell owners per tile count
  std::list<std::pair<std::pair<int, int>, std::shared_ptr<TileCache>>> sets;  // (tiles, interval), newest first
};

struct isw_batch {
  int device;
  std::vector<BatchSlot> slots;
  bool dirty = true;
  StackDesc *d_desc = nullptr;
  Chunk *d_chunks = nullptr;
  TileRef *d_refs = nullptr;
  Sched scf[2] = {};                          // chunk tables of the FP64 stacks [0] and the mixed ones [1]
  int lmax = 1, nstacks = 0, ntiles = 0, nsub[3] = {0, 0, 0}, kused = 0;
  std::vector<FastGroup> groups;              // cooperative launches of the fast loop (tiles [begin, begin + count))
  int any_nu4 = 0, any_vmix = 0, any_tr = 0, any_untiled = 0, any_air = 0;
  int any_ext = 0;                            // air or option stacks: the phase kernels with those branches
  int any_ob = 0;                             // a stack with the shelf's bed flags: their pass opens the step
  size_t fast_smem = 0;
  int fast_bps = 2;                           // tile blocks per SM: 2 (384 threads each) or 1 (768 threads)
  GridBarrier *bar = nullptr;
  unsigned *flags = nullptr;                  // the tiles' exchange flags, TILE_FLAG_STRIDE apart
  BatchStatus *status = nullptr;              // device status word (code + the mirror's device address)
  int *status_host = nullptr;                 // mapped pinned host mirror of the code, written by the failing kernel
  int tile_k = 8;
  int tiles_enabled = 1;
  int tile_cells = 0;                         // packed layout's owned cells per tile (0: by blocks per SM)
  int force_bps = 0;                          // 0: choose; 1 or 2 tile blocks per SM
  int layout = 0;                             // 0: choose; 1 shared; 2 packed
  // per grid level: 0 follows the batch (default); 1 untiled; 2 packed tiles of about `cells` owned cells (0: the
  // batch's), exchange interval at most `k` (0: the batch's)
  struct LevelLayout {
    int mode = 0, cells = 0, k = 0;
  };
  std::map<int, LevelLayout> levels;
  bool check = true;                          // false: thicknesses are not looked at (a Layers' own batch with options)
  bool pdl = true;                            // programmatic dependent launch between phase kernels
  bool fast_grid = false;                     // untiled stacks' sub-steps: one cooperative launch per stage (k_fast_grid)
  int cell_tracers[2] = {1, 1};               // per form: tracers of one thread of the first two cell passes (mixed: one)
  int untiled_form[2] = {0, 0};               // per form (FP64, mixed): any untiled stack
  size_t s_smem[2] = {0, 0};                  // per form: dynamic shared memory of the slow-tendency launch (staging)
  int grid_blocks[2] = {0, 0};                // per form: co-resident blocks of the cooperative grid-wide fast loop
  // pipelined steps: step n's dynamics beside step n-1's transport (two branches of one graph), Fm double-buffered.
  // desc[q] describes a step whose dynamics write Fm_q and whose transport reads it: Fm_0 the registered Fm, Fm_1 fm_alt
  bool pipeline = false, primed = false;
  int parity = 0;
  StackDesc *d_desc1 = nullptr;
  std::vector<void *> fm_alt;
  std::vector<std::pair<double *, size_t>> fm_pairs;  // (registered Fm, bytes) per stack, for the flush's copy-back
  cudaGraphExec_t pexec[6] = {};              // dynamics D_0, D_1; both branches DT_0, DT_1; transport T_0, T_1
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  const StackDesc *cur = nullptr;             // the descriptors the launches being queued use
  std::vector<std::shared_ptr<TileCache>> tiles;   // the tile sets the descriptors point into
  cudaStream_t cap = nullptr;
  cudaGraphExec_t exec = nullptr;
  int sms = 0;
};

namespace {

template <class F>
int guarded(F f) {
  try {
    f();
    return ISW_OK;
  } catch (const Error &e) {
    set_last_error(e.msg);
    return e.status;
  } catch (const std::bad_alloc &) {
    set_last_error("host allocation failed");
    return ISW_ENOMEM;
  }
}

constexpr long long DEFAULT_TIMEOUT_NS = 2000000000LL;   // 2 s: far beyond any stage; only a broken grid reaches it
constexpr size_t SMEM_TWO = 112 * 1024;                  // per tile block when two share an SM
constexpr size_t SMEM_ONE = 224 * 1024;                  // per tile block alone on an SM
constexpr int K_PROBE = FAST_KMAX;                       // the largest exchange interval considered

template <class T>
T *dupload(std::vector<void *> &allocs, const std::vector<T> &v) {
  void *p = nullptr;
  ISW_CUDA(cudaMalloc(&p, sizeof(T) * (v.empty() ? 1 : v.size())));
  allocs.push_back(p);
  if (!v.empty()) ISW_CUDA(cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice));
  return (T *)p;
}

std::shared_ptr<TileCache> tiles_for(isw_grid *g, int P, int k);
int fitting_k(const TileSetHost &h, int L, bool mixed, int bps);

// The largest exchange interval a tiling of g into P tiles fits in the budget, or 0 when no tiling can be built (a
// region too large or too scattered for the tiles' 16-bit local ids): the planners then leave the stack untiled.
int fitting_k_or_none(isw_grid *g, int L, bool mixed, int P, int kcap, int bps) {
  try {
    return fitting_k(tiles_for(g, P, std::min(K_PROBE, kcap))->host, L, mixed, bps);
  } catch (const Error &) {
    return 0;
  }
}

std::shared_ptr<TileCache> tiles_for(isw_grid *g, int P, int k) {
  std::lock_guard<std::mutex> lock(g->tile_mu);
  if (!g->tile_store) g->tile_store = std::make_shared<TileStore>();
  TileStore &store = *std::static_pointer_cast<TileStore>(g->tile_store);
  const auto key = std::make_pair(P, k);
  for (auto it = store.sets.begin(); it != store.sets.end(); ++it)
    if (it->first == key) {
      store.sets.splice(store.sets.begin(), store.sets, it);
      return store.sets.front().second;
    }
  auto part = store.parts.find(P);
  if (part == store.parts.end()) {
    if (store.parts.size() >= TILE_STORE_MAX) store.parts.clear();
    part = store.parts.emplace(P, partition_cells(g->d.N, g->h_nbr.data(), P)).first;
  }
  auto c = std::make_shared<TileCache>();
  c->host = build_tiles(g->d.N, g->d.E, g->h_nbr.data(), g->h_cellEdge.data(), g->h_cellSign.data(), g->h_eI.data(),
                        g->h_eJ.data(), part->second, P, k);
  store.sets.emplace_front(key, c);
  for (auto it = std::prev(store.sets.end()); store.sets.size() > TILE_STORE_MAX && it != store.sets.begin();) {
    const auto cur = it--;
    if (cur->second.use_count() == 1) store.sets.erase(cur);
  }
  return c;
}

// The set's device tables, uploaded the first time a batch steps with it.
const TileSetDev &tiles_on_device(isw_grid *g, TileCache *c) {
  std::lock_guard<std::mutex> lock(g->tile_mu);
  const TileSetHost &h = c->host;
  TileSetDev &t = c->dev;
  if (t.P) return t;
  t.cell_off = dupload(c->allocs, h.cell_off);
  t.edge_off = dupload(c->allocs, h.edge_off);
  t.ncnt = dupload(c->allocs, h.ncnt);
  t.ecnt = dupload(c->allocs, h.ecnt);
  t.eown = dupload(c->allocs, h.eown);
  t.nbr_off = dupload(c->allocs, h.nbr_off);
  t.nbrs = dupload(c->allocs, h.nbrs);
  t.cedge = reinterpret_cast<const uint4 *>(dupload(c->allocs, h.cedge));
  t.casc = reinterpret_cast<const uint4 *>(dupload(c->allocs, h.casc));
  t.eix = reinterpret_cast<const int2 *>(dupload(c->allocs, h.eix));
  std::vector<double> el(2 * h.edges.size()), aarea(h.cells.size());
  std::vector<float> el32(2 * h.edges.size()), rA32(h.cells.size());
  for (size_t q = 0; q < h.edges.size(); q++) {
    const double l = g->h_le[h.edges[q]], dd = g->h_de[h.edges[q]];
    el[2 * q] = l;
    el[2 * q + 1] = dd;
    el32[2 * q] = (float)l;
    el32[2 * q + 1] = (float)(1.0 / dd);
  }
  for (size_t q = 0; q < h.cells.size(); q++) {
    aarea[q] = g->h_areaCell[h.cells[q]];
    rA32[q] = (float)(1.0 / aarea[q]);
  }
  t.el = reinterpret_cast<const double2 *>(dupload(c->allocs, el));
  t.el32 = reinterpret_cast<const float2 *>(dupload(c->allocs, el32));
  t.aarea = dupload(c->allocs, aarea);
  t.arA32 = dupload(c->allocs, rA32);
  t.k = h.k;
  t.P = h.P;
  return t;
}

// Layers the stage's end takes at once at interval k: every layer where each tile's share fits a block, else an even split
// into as few groups as fit (0: not even one layer does).
int end_group(const TileSetHost &h, int k, int L, bool mixed, int bps) {
  const size_t budget = bps == 2 ? SMEM_TWO : SMEM_ONE;
  for (int n = 1; n <= L; n++) {
    const int lg = (L + n - 1) / n;
    bool ok = true;
    for (int p = 0; p < h.P && ok; p++) {
      const int32_t *nc = &h.ncnt[(size_t)p * (h.k + 1)], *ne = &h.ecnt[(size_t)p * (h.k + 1)];
      ok = tile_smem_bytes(nc[k], ne[k], nc[1], ne[0], lg, n > 1, mixed) <= budget;
    }
    if (ok) return lg;
  }
  return 0;
}

// The smallest kernel capacity whose registers hold every tile of a tiling at interval k (-1: none).
int tiles_cap(const TileSetHost &h, int k, int bps) {
  const int nt = fast_tiles_threads(bps);
  for (int cap = 0; cap < 2; cap++) {
    bool ok = true;
    for (int p = 0; p < h.P && ok; p++) {
      const int32_t *nc = &h.ncnt[(size_t)p * (h.k + 1)], *ne = &h.ecnt[(size_t)p * (h.k + 1)];
      ok = nc[k] <= nt * TILE_CAP[cap].C && ne[k] <= nt * TILE_CAP[cap].E && ne[0] <= nt * TILE_CAP[cap].A;
    }
    if (ok) return cap;
  }
  return -1;
}

// The largest k' <= the probe's k at which every tile fits a block: its cells, edges and own cells' edges the
// threads' registers, what its threads share the block's shared memory (0 if none). An interval at which the stage's end
// takes every layer at once comes before a longer one at which it does not.
int fitting_k(const TileSetHost &h, int L, bool mixed, int bps) {
  int grouped = 0;
  for (int kk = h.k; kk >= 1; kk--) {
    if (tiles_cap(h, kk, bps) < 0) continue;
    const int lg = end_group(h, kk, L, mixed, bps);
    if (lg == L) return kk;
    if (lg > 0 && grouped == 0) grouped = kk;
  }
  return grouped;
}

// Dynamic shared memory of the largest tile of a tile set whose stage's end takes lg of L layers at once.
size_t tiles_smem(const TileSetHost &h, int lg, int L, bool mixed) {
  size_t worst = 0;
  for (int p = 0; p < h.P; p++) {
    const int32_t *nc = &h.ncnt[(size_t)p * (h.k + 1)], *ne = &h.ecnt[(size_t)p * (h.k + 1)];
    worst = std::max(worst, tile_smem_bytes(h.cell_off[p + 1] - h.cell_off[p], h.edge_off[p + 1] - h.edge_off[p], nc[1], ne[0], lg, lg < L, mixed));
  }
  return worst;
}

int kernel_lmax(int L) { return L <= 2 ? 2 : L <= 3 ? 3 : L <= 5 ? 5 : 8; }

// The fast-loop tiling of the registered stacks. Two layouts; left to choose, the one with the lower modelled time wins:
//  - shared: one cooperative group over all stacks, each stack cut into tiles in proportion to its share of the cells,
//    filling the SMs (small batches: one member, a few members);
//  - packed: each stack cut into tiles of about tile_cells owned cells (a fixed size per grid, so tile sets are reused
//    as stacks come and go), the stacks packed in order into groups of at most SMs x blocks-per-SM tiles, one
//    cooperative launch per group and stage (large ensembles, serving).
// Stacks whose tiles would not fit in shared memory at all take the grid-wide sub-step kernels.
struct Tiling {
  int k = 0, bps = 2;                          // k: the smallest exchange interval over the stacks
  bool grouped = false;                        // a stack's end takes its layers in groups
  double us = 0;                               // modelled time of the step's tile launches
  std::vector<int> P;                          // tiles per slot (0: untiled)
  std::vector<int> K;                          // exchange interval per slot
  std::vector<int> group;                      // group per slot
};

int form_of(const BatchSlot &sl) { return sl.layers->d.precision == ISW_MIXED ? 1 : 0; }

// Stacks with option branches: walls, the shelf (and its bed flags), per-cell buoyancy, the tide, the bottom's drag.
bool has_options(const isw::LayersDev &d) {
  return d.wall || d.ob || d.shelf > 0 || d.sig || d.tide || d.cbot || d.cd_bot > 0;
}

isw_batch::LevelLayout level_layout(const isw_batch *b, const BatchSlot &sl) {
  const auto it = b->levels.find(sl.layers->grid->n);
  return it == b->levels.end() ? isw_batch::LevelLayout{} : it->second;
}

bool tiles_form(const isw_batch *b, const BatchSlot &sl) {
  return sl.used && !sl.layers->d.air && level_layout(b, sl).mode != 1;
}

// Modelled time (us) of a stack's tile launches in one step at exchange interval k <= the probe's: per stage a fixed part
// (staging, the stage's end), per exchange its latency, per sub-step the edges the largest tile updates. It ranks tilings
// against one another, not against the grid-wide sub-steps (Batch.autotune times both). The constants are B200 timings of
// an earlier form of the kernel, 1,024 threads: staging and end 22 us for tiles of 553 cells (two or three layers; some 36
// at 1,107), an exchange 3.5 us, a sub-step 0.76 ns (FP64) or 0.40 ns (mixed) per edge and tile on the SM and at least 0.7.
// The present form's at 553 cells: 19 us, 2.4 to 3.0 us, 1.9 us a sub-step (FP64) or 1.1.
double tiles_us(const TileSetHost &h, int k, int L, int nfast, bool mixed, int bps) {
  const double cs[3] = {1.0 / 3.0, 1.0 / 2.0, 1.0};
  const int lg = end_group(h, k, L, mixed, bps);
  std::vector<int> edges(k + 1, 0);            // most edges of ring <= r in a tile
  for (int p = 0; p < h.P; p++)
    for (int r = 0; r <= k; r++) edges[r] = std::max(edges[r], (int)h.ecnt[(size_t)p * (h.k + 1) + r]);
  double us = 0;
  for (double c : cs) {
    const int n = std::max(1, (int)std::ceil(c * nfast));
    us += 22.0 + 3.5 * ((L + lg - 1) / lg - 1);
    for (int done = 0; done < n; done += k) {
      const int K = std::min(k, n - done);
      us += 3.5;
      for (int m = 1; m <= K; m++) us += std::max(0.7, edges[K - m] * bps * (mixed ? 0.40e-3 : 0.76e-3));
    }
  }
  return us;
}

// The exchange interval of a stack's tiling: the largest that fits when the layout was asked for, else the fastest by
// the model.
int pick_k(isw_batch *b, const BatchSlot &sl, int P, int kcap, int bps, double *us, bool *grouped) {
  const bool mixed = form_of(sl) == 1;
  int k = fitting_k_or_none(sl.layers->grid, sl.layers->d.L, mixed, P, kcap, bps);
  if (k == 0) return 0;
  const std::shared_ptr<TileCache> set = tiles_for(sl.layers->grid, P, std::min(K_PROBE, kcap));
  const TileSetHost &h = set->host;
  *us = tiles_us(h, k, sl.layers->d.L, sl.nfast, mixed, bps);
  if (b->layout == 0)
    for (int kk = k - 1; kk >= 1; kk--) {
      const double t = tiles_us(h, kk, sl.layers->d.L, sl.nfast, mixed, bps);
      if (t < *us) { *us = t; k = kk; }
    }
  if (end_group(h, k, sl.layers->d.L, mixed, bps) < sl.layers->d.L) *grouped = true;
  return k;
}

Tiling plan_shared(isw_batch *b, int bps) {
  Tiling t;
  t.bps = bps;
  t.P.assign(b->slots.size(), 0);
  t.K.assign(b->slots.size(), 0);
  t.group.assign(b->slots.size(), 0);
  double form_us[2] = {0, 0};
  const int slots = b->sms * bps;
  long long cells_total[2] = {0, 0};           // per form: a launch each
  for (auto &sl : b->slots)
    if (tiles_form(b, sl)) cells_total[form_of(sl)] += sl.layers->grid->d.N;
  int kmin = b->tile_k;
  bool any = false;
  for (size_t q = 0; q < b->slots.size(); q++) {
    const BatchSlot &sl = b->slots[q];
    if (!tiles_form(b, sl)) continue;
    const int N = sl.layers->grid->d.N;
    const int Pq = std::max(1, (int)((long long)slots * N / std::max(1LL, cells_total[form_of(sl)])));
    if (Pq * 16 > N) return Tiling{};          // tiles of at least 16 owned cells, for every stack
    double us = 0;
    const int kf = pick_k(b, sl, Pq, b->tile_k, bps, &us, &t.grouped);
    if (kf == 0) return Tiling{};
    t.P[q] = Pq;
    t.K[q] = kf;
    form_us[form_of(sl)] = std::max(form_us[form_of(sl)], us);
    t.group[q] = cells_total[0] > 0 ? form_of(sl) : 0;
    kmin = std::min(kmin, kf);
    any = true;
  }
  t.k = any ? kmin : 0;
  if (b->layout != 0) t.K.assign(b->slots.size(), t.k);
  t.us = form_us[0] + form_us[1];
  return t;
}

Tiling plan_packed(isw_batch *b, int bps) {
  Tiling t;
  t.bps = bps;
  t.P.assign(b->slots.size(), 0);
  t.K.assign(b->slots.size(), 0);
  t.group.assign(b->slots.size(), 0);
  const int cap = b->sms * bps;
  std::vector<double> slot_us(b->slots.size(), 0.0);
  const int cells_b = b->tile_cells > 0 ? b->tile_cells : (bps == 2 ? 384 : 768);
  int kmin = b->tile_k;
  bool any = false;
  for (size_t q = 0; q < b->slots.size(); q++) {
    const BatchSlot &sl = b->slots[q];
    if (!tiles_form(b, sl)) continue;
    const isw_batch::LevelLayout lv = level_layout(b, sl);       // the level's own tile size and interval, if set
    const int cells = lv.mode == 2 && lv.cells > 0 ? lv.cells : cells_b;
    const int kcap = lv.mode == 2 && lv.k > 0 ? std::min(lv.k, b->tile_k) : b->tile_k;
    const int N = sl.layers->grid->d.N;
    const int Pq = std::min(cap, std::max(1, (N + cells - 1) / cells));
    if (Pq * 16 > N) continue;
    const int kf = pick_k(b, sl, Pq, kcap, bps, &slot_us[q], &t.grouped);
    if (kf == 0) continue;
    t.P[q] = Pq;
    t.K[q] = kf;                               // each stack its own interval: a group's rounds follow its slowest
    kmin = std::min(kmin, kf);
    any = true;
  }
  if (!any) return Tiling{};
  t.k = kmin;
  int g = -1;
  for (int f = 0; f < 2; f++) {                // a group's stacks are of one form
    int fill = cap;
    for (size_t q = 0; q < b->slots.size(); q++) {
      if (t.P[q] == 0 || form_of(b->slots[q]) != f) continue;
      if (fill + t.P[q] > cap) { g++; fill = 0; }
      t.group[q] = g;
      fill += t.P[q];
    }
  }
  std::vector<double> group_us(g + 1, 0.0);
  for (size_t q = 0; q < b->slots.size(); q++)
    if (t.P[q] > 0) group_us[t.group[q]] = std::max(group_us[t.group[q]], slot_us[q]);
  for (double us : group_us) t.us += us;
  return t;
}

// Whether every tile block of each group can be resident at once, as the cooperative launch needs.
bool resident(isw_batch *b, const Tiling &t) {
  for (int f = 0; f < 2; f++) {
    std::map<int, int> count;
    size_t smax = 0;
    for (size_t q = 0; q < b->slots.size(); q++)
      if (t.P[q] > 0 && form_of(b->slots[q]) == f) {
        count[t.group[q]] += t.P[q];
        const std::shared_ptr<TileCache> set = tiles_for(b->slots[q].layers->grid, t.P[q], t.K[q]);
        const int L = b->slots[q].layers->d.L;
        smax = std::max(smax, tiles_smem(set->host, end_group(set->host, t.K[q], L, f == 1, t.bps), L, f == 1));
      }
    if (count.empty()) continue;
    for (int kind = 0; kind < (f == 1 ? 3 : 6); kind++) {      // capacities, then (FP64) with walls
      const void *fn = fast_tiles_kernel(t.bps, kind % 3, kind >= 3 ? 2 : f);
      // the kernel's limit is one setting for every batch: always the most a tile may ask for
      ISW_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(t.bps == 2 ? SMEM_TWO : SMEM_ONE)));
      int per = 0;
      ISW_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, fast_tiles_threads(t.bps), smax));
      for (const auto &kv : count)
        if ((long long)per * b->sms < kv.second) return false;
    }
  }
  return true;
}

void rebuild(isw_batch *b) {
  std::vector<StackDesc> desc;
  std::vector<Chunk> cell[2], edge[2], vert[2], rows[2], erows[2], grows[2];      // per form: [0] FP64 stacks, [1] mixed
  std::vector<Chunk> wcell[2], wedge[2], uedge[2];                      // the untiled stacks': the sub-step passes' wide chunks, plain edges
  int nsub[3] = {0, 0, 0};
  int any_nu4 = 0, any_vmix = 0, any_tr = 0, any_untiled = 0, any_air = 0, any_ext = 0, any_ob = 0, lmax = 1;
  int untiled[2] = {0, 0};
  size_t s_smem[2] = {0, 0};
  const double cs[3] = {1.0 / 3.0, 1.0 / 2.0, 1.0};
  int most_layers = 1;                                                  // over both forms: the phase kernels' L
  for (auto &sl : b->slots)
    if (sl.used) most_layers = std::max(most_layers, sl.layers->d.L);
  long long edge_items[2] = {0, 0}, cell_items[2] = {0, 0};             // per form: (tracer, edge) and (tracer, cell) pairs
  for (auto &sl : b->slots)
    if (sl.used && sl.tr) {
      edge_items[form_of(sl)] += (long long)sl.ntr * sl.layers->grid->d.E;
      cell_items[form_of(sl)] += (long long)sl.ntr * sl.layers->grid->d.N;
    }
  int used = 0;
  for (auto &sl : b->slots) used += sl.used ? 1 : 0;
  Tiling best;
  if (b->tiles_enabled && used > 0) {
    for (int bps = 2; bps >= 1; bps--) {
      if (b->force_bps && bps != b->force_bps) continue;
      for (int lay = 1; lay <= 2; lay++) {
        if (b->layout != 0 && b->layout != lay) continue;
        Tiling t = lay == 1 ? plan_shared(b, bps) : plan_packed(b, bps);
        // (layers in groups only where no layout takes them together)
        if (t.k > 0 && (best.k == 0 || t.grouped < best.grouped || (t.grouped == best.grouped && t.us < best.us))) best = t;
      }
    }
  }
  if (best.k > 0 && !resident(b, best)) best = Tiling{};
  const int kbest = best.k;
  const int ngroups = kbest > 0 ? 1 + *std::max_element(best.group.begin(), best.group.end()) : 0;
  std::vector<std::vector<TileRef>> grefs(ngroups);
  std::vector<size_t> gsmem(ngroups, 0);
  std::vector<int> gform(ngroups, 0), gcap(ngroups, 0), gwalls(ngroups, 0), gwaited(ngroups, -1);
  std::vector<std::shared_ptr<TileCache>> used_tiles;
  std::vector<std::pair<size_t, int>> gfirst;     // per tiled stack in order: its group, its first tile within the group
  for (auto &sl : b->slots) {
    if (!sl.used) continue;
    StackDesc d;
    std::memset(&d, 0, sizeof(d));
    d.M = sl.layers->d;
    d.h = sl.h; d.u = sl.u; d.Fm = sl.Fm; d.Mm = sl.M;
    d.theta = sl.theta;
    if (d.M.air) any_air = 1;
    if (d.M.air || has_options(d.M)) any_ext = 1;
    if (d.M.ob) any_ob = 1;
    d.check = b->check ? 1 : 0;
    d.dt = sl.dt;
    d.L = d.M.L;
    lmax = std::max(lmax, d.L);
    for (int st = 0; st < 3; st++) {
      const double c = cs[st];
      const double cn = std::ceil(c * sl.nfast);
      d.n[st] = cn > 1 ? (int)cn : 1;
      d.cdt[st] = c * sl.dt;
      d.tau[st] = c * sl.dt / d.n[st];
      d.inv_n[st] = 1.0 / d.n[st];
      nsub[st] = std::max(nsub[st], d.n[st]);
    }
    if (d.M.nu4 != 0) any_nu4 = 1;
    if ((d.M.vmix != 0 || d.M.vmix_cd != 0) && d.L > 1) any_vmix = 1;
    if (sl.tr) {
      d.has_tr = 1;
      any_tr = 1;
      d.T = sl.tr->d;
      d.tr.M0 = sl.M; d.tr.M1 = sl.M1; d.tr.Fm = sl.Fm; d.tr.L = d.L; d.tr.rows = sl.ntr * d.L; d.tr.beta = sl.tr->beta;
      for (int j = 0; j < sl.ntr; j++) d.tr.tr[j] = sl.tracers[j];
    }
    const int s = (int)desc.size();
    d.tiled = 0;
    const size_t q = (size_t)(&sl - &b->slots[0]);
    if (kbest > 0 && best.P[q] > 0) {
      const std::shared_ptr<TileCache> tc = tiles_for(sl.layers->grid, best.P[q], best.K[q]);
      used_tiles.push_back(tc);
      const int g = best.group[q];
      d.tiled = 1;
      d.tiles = tiles_on_device(sl.layers->grid, tc.get());
      d.lg = end_group(tc->host, best.K[q], d.L, form_of(sl) == 1, best.bps);
      gsmem[g] = std::max(gsmem[g], tiles_smem(tc->host, d.lg, d.L, form_of(sl) == 1));
      gform[g] = form_of(sl);
      if (d.M.wall) gwalls[g] = 1;
      gcap[g] = std::max(gcap[g], d.lg < d.L ? 2 : tiles_cap(tc->host, best.K[q], best.bps));
      gfirst.emplace_back((size_t)g, (int)grefs[g].size());
      if (best.P[q] > 1 && gwaited[g] < 0) gwaited[g] = (int)grefs[g].size();
      for (int p = 0; p < best.P[q]; p++) grefs[g].push_back(TileRef{s, p});
    }
    if (!d.tiled) any_untiled = 1;
    {                                            // the mixed form's slow tendency stages its neighbour records when they fit
      // (measured: S 80.0 -> 76.2 us a level-6 member step in the mixed form; 97.4 -> 113.1 in FP64, whose 80-byte
      // records are staged about twice per block against the L1 hits of direct gathers, so FP64 gathers directly)
      const size_t need = (size_t)d.M.g.sMax * (size_t)d.L * sizeof(float4);
      d.s_stage = form_of(sl) == 1 && need <= S_STAGE_MAX ? 1 : 0;
      if (d.s_stage) s_smem[form_of(sl)] = std::max(s_smem[form_of(sl)], need);
    }
    auto chunks = [&](std::vector<Chunk> &v, int n, int w = THREADS) {
      for (int i = 0; i < n; i += w) v.push_back(Chunk{s, i, std::min(n, i + w)});
    };
    const int f = form_of(sl);
    if (!d.tiled) untiled[f] = 1;
    chunks(cell[f], d.M.g.N);
    chunks(edge[f], d.M.g.E);
    chunks(vert[f], d.M.g.NV);
    if (!d.tiled) {
      chunks(wcell[f], d.M.g.N, SUB_WC * THREADS);
      chunks(wedge[f], d.M.g.E, (f == 0 ? SUB_W_FP64 : SUB_W) * THREADS);
      chunks(uedge[f], d.M.g.E);
    }
    if (d.has_tr) chunks(rows[f], sl.ntr * d.M.g.N);       // (tracer, cell) pairs
    if (d.has_tr) {                                        // (tracers of a thread, cell), (tracers of a thread, edge)
      d.cg = f == 0 ? fp64::cell_tracers(cell_items[0], most_layers) : 1;
      chunks(grows[f], (sl.ntr + d.cg - 1) / d.cg * d.M.g.N);
      d.eg = fp64::tracers_a_thread(edge_items[f], sl.ntr);
      chunks(erows[f], (sl.ntr + d.eg - 1) / d.eg * d.M.g.E);
    }
    desc.push_back(d);
  }
  b->nstacks = (int)desc.size();
  cudaFree(b->d_desc);                       // (waits for the steps in flight, which read the old tile sets too)
  b->tiles.swap(used_tiles);
  cudaFree(b->d_chunks);
  cudaFree(b->d_refs);
  cudaFree(b->flags);
  b->d_desc = nullptr;
  b->d_chunks = nullptr;
  b->d_refs = nullptr;
  b->flags = nullptr;
  b->cur = nullptr;
  b->groups.clear();
  b->ntiles = 0;
  if (b->exec) {
    cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
  }
  for (auto &x : b->pexec)
    if (x) {
      cudaGraphExecDestroy(x);
      x = nullptr;
    }
  cudaFree(b->d_desc1);
  b->d_desc1 = nullptr;
  for (void *q : b->fm_alt) cudaFree(q);
  b->fm_alt.clear();
  b->fm_pairs.clear();
  b->primed = false;
  b->parity = 0;
  b->dirty = false;
  if (desc.empty()) return;
  std::vector<Chunk> all;
  for (int f = 0; f < 2; f++) {
    all.insert(all.end(), cell[f].begin(), cell[f].end());
    all.insert(all.end(), edge[f].begin(), edge[f].end());
    all.insert(all.end(), vert[f].begin(), vert[f].end());
    all.insert(all.end(), rows[f].begin(), rows[f].end());
    all.insert(all.end(), erows[f].begin(), erows[f].end());
    all.insert(all.end(), grows[f].begin(), grows[f].end());
    all.insert(all.end(), wcell[f].begin(), wcell[f].end());
    all.insert(all.end(), wedge[f].begin(), wedge[f].end());
    all.insert(all.end(), uedge[f].begin(), uedge[f].end());
  }
  ISW_CUDA(cudaMalloc(&b->d_desc, sizeof(StackDesc) * desc.size()));
  ISW_CUDA(cudaMalloc(&b->d_chunks, sizeof(Chunk) * all.size()));
  ISW_CUDA(cudaMemcpy(b->d_chunks, all.data(), sizeof(Chunk) * all.size(), cudaMemcpyHostToDevice));
  std::vector<TileRef> refs;
  for (int g = 0; g < ngroups; g++) {
    FastGroup fg;
    fg.begin = (int)refs.size();
    fg.count = (int)grefs[g].size();
    fg.smem = gsmem[g];
    fg.form = gform[g];
    fg.cap = gcap[g];
    fg.walls = gwalls[g] != 0;
    fg.waited = gwaited[g];
    refs.insert(refs.end(), grefs[g].begin(), grefs[g].end());
    b->groups.push_back(fg);
  }
  b->fast_bps = best.bps;
  {                                          // a stack's tiles are consecutive in the list: where they (and their flags) start
    size_t at = 0;
    for (auto &d : desc)
      if (d.tiled) {
        d.tile_base = b->groups[gfirst[at].first].begin + gfirst[at].second;
        at++;
      }
  }
  ISW_CUDA(cudaMemcpy(b->d_desc, desc.data(), sizeof(StackDesc) * desc.size(), cudaMemcpyHostToDevice));
  if (b->pipeline) {                         // the other parity's descriptors: the same stacks with a second Fm
    std::vector<StackDesc> desc1 = desc;
    for (auto &d : desc1) {
      const size_t bytes = sizeof(double) * (size_t)d.L * d.M.g.E;
      void *alt = nullptr;
      ISW_CUDA(cudaMalloc(&alt, bytes));
      ISW_CUDA(cudaMemset(alt, 0, bytes));
      b->fm_alt.push_back(alt);
      b->fm_pairs.emplace_back(d.Fm, bytes);
      d.Fm = (double *)alt;
      d.tr.Fm = (double *)alt;
    }
    ISW_CUDA(cudaMalloc(&b->d_desc1, sizeof(StackDesc) * desc1.size()));
    ISW_CUDA(cudaMemcpy(b->d_desc1, desc1.data(), sizeof(StackDesc) * desc1.size(), cudaMemcpyHostToDevice));
  }
  if (!refs.empty()) {
    ISW_CUDA(cudaMalloc(&b->d_refs, sizeof(TileRef) * refs.size()));
    ISW_CUDA(cudaMemcpy(b->d_refs, refs.data(), sizeof(TileRef) * refs.size(), cudaMemcpyHostToDevice));
    const size_t fb = sizeof(unsigned) * TILE_FLAG_STRIDE * refs.size();
    ISW_CUDA(cudaMalloc(&b->flags, fb));
    ISW_CUDA(cudaMemset(b->flags, 0, fb));
  }
  const Chunk *base = b->d_chunks;
  for (int f = 0; f < 2; f++) {
    Sched &sc = b->scf[f];
    sc.status = b->status;
    sc.cell = base;
    sc.ncell = (int)cell[f].size();
    sc.edge = sc.cell + sc.ncell;
    sc.nedge = (int)edge[f].size();
    sc.vert = sc.edge + sc.nedge;
    sc.nvert = (int)vert[f].size();
    sc.rows = sc.vert + sc.nvert;
    sc.nrows = (int)rows[f].size();
    sc.erows = sc.rows + sc.nrows;
    sc.nerows = (int)erows[f].size();
    sc.grows = sc.erows + sc.nerows;
    sc.ngrows = (int)grows[f].size();
    sc.wcell = sc.grows + sc.ngrows;
    sc.nwcell = (int)wcell[f].size();
    sc.wedge = sc.wcell + sc.nwcell;
    sc.nwedge = (int)wedge[f].size();
    sc.uedge = sc.wedge + sc.nwedge;
    sc.nuedge = (int)uedge[f].size();
    base = sc.uedge + sc.nuedge;
  }
  b->ntiles = (int)refs.size();
  size_t smax = 0;
  for (auto &fg : b->groups) smax = std::max(smax, fg.smem);
  b->fast_smem = smax;
  for (int st = 0; st < 3; st++) b->nsub[st] = nsub[st];
  b->kused = b->ntiles > 0 ? kbest : 0;
  b->any_nu4 = any_nu4;
  b->any_vmix = any_vmix;
  b->any_tr = any_tr;
  b->any_untiled = any_untiled;
  b->any_air = any_air;
  b->any_ext = any_ext;
  b->any_ob = any_ob;
  b->lmax = kernel_lmax(lmax);
  b->cell_tracers[0] = fp64::cell_tracers(cell_items[0], most_layers);
  b->s_smem[0] = s_smem[0];
  b->s_smem[1] = s_smem[1];
  if (s_smem[0] > 48 * 1024)
    for (const void *fn : {(const void *)k_phase<PH_S, 2, false>, (const void *)k_phase<PH_S, 3, false>,
                           (const void *)k_phase<PH_S, 5, false>, (const void *)k_phase<PH_S, 8, false>,
                           (const void *)k_phase<PH_S, 2, true>, (const void *)k_phase<PH_S, 3, true>,
                           (const void *)k_phase<PH_S, 5, true>, (const void *)k_phase<PH_S, 8, true>})
      ISW_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s_smem[0]));
  if (s_smem[1] > 48 * 1024) slow_phase_smem_mixed(s_smem[1]);
  for (int f = 0; f < 2; f++) {
    b->untiled_form[f] = untiled[f];
    b->grid_blocks[f] = 0;
    if (!untiled[f]) continue;
    int per = 0;
    const void *fn = f == 0 ? fast_grid_kernel(b->lmax, b->any_ext) : fast_grid_kernel_mixed();
    ISW_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, THREADS, 0));
    b->grid_blocks[f] = std::max(1, per) * b->sms;
  }
}

// A phase over the stacks of form f.
template <int PH>
void launch_form(isw_batch *b, cudaStream_t st, int f, int stage, int j, bool pdl) {
  const Sched &sc = b->scf[f];
  const int nb = phase_blocks<PH>(sc);
  if (!b->cur) fail(ISW_EINVAL, "batch: no stack descriptors selected for the launch");
  if (f == 1) {
    launch_phase_mixed(PH, b->lmax, nb, st, pdl, PH == PH_S ? b->s_smem[1] : 0, b->cur, sc, stage, j);
    return;
  }
  const size_t smem = PH == PH_S ? b->s_smem[0] : 0;
  constexpr int MB = phase_blocks_an_sm(PH, 8, false);
  const bool bounded = more_blocks(nb, MB);
  if (b->any_ext) {
    switch (b->lmax) {
      case 2: launch_kernel(k_phase<PH, 2, true>, nb, st, pdl, smem, b->cur, sc, stage, j); break;
      case 3: launch_kernel(k_phase<PH, 3, true>, nb, st, pdl, smem, b->cur, sc, stage, j); break;
      case 5: launch_kernel(k_phase<PH, 5, true>, nb, st, pdl, smem, b->cur, sc, stage, j); break;
      default: launch_kernel(bounded ? k_phase<PH, 8, true, MB> : k_phase<PH, 8, true>, nb, st, pdl, smem, b->cur, sc, stage, j); break;
    }
  } else {
    switch (b->lmax) {
      case 2: launch_kernel(k_phase<PH, 2, false>, nb, st, pdl, smem, b->cur, sc, stage, j); break;
      case 3: launch_kernel(k_phase<PH, 3, false>, nb, st, pdl, smem, b->cur, sc, stage, j); break;
      case 5: launch_kernel(k_phase<PH, 5, false>, nb, st, pdl, smem, b->cur, sc, stage, j); break;
      default: launch_kernel(bounded ? k_phase<PH, 8, false, MB> : k_phase<PH, 8, false>, nb, st, pdl, smem, b->cur, sc, stage, j); break;
    }
  }
}

// A phase over every stack: one kernel per precision form present (the FP64 stacks' first); PHG in its place for a form
// whose cell passes take several tracers a thread. pdl: the first of them is launched as a programmatic dependent of the
// kernel before it in the stream (never directly after a cooperative tile launch, which keeps plain stream order); a
// second one always is.
template <int PH, int PHG = PH>
void launch_phase(isw_batch *b, cudaStream_t st, int stage, int j, bool pdl = true) {
  bool first = true;
  for (int f = 0; f < 2; f++) {
    if (phase_blocks<PH>(b->scf[f]) == 0) continue;
    const bool p = (first ? pdl : true) && b->pdl;
    first = false;
    if (PHG != PH && b->cell_tracers[f] > 1) launch_form<PHG>(b, st, f, stage, j, p);
    else launch_form<PH>(b, st, f, stage, j, p);
  }
}

void launch_fast(isw_batch *b, cudaStream_t st, int stage, long long timeout_ns, int fault_block) {
  if (!b->groups.empty() && !b->cur) fail(ISW_EINVAL, "batch: no stack descriptors selected for the launch");
  for (const FastGroup &fg : b->groups) {
    if (fg.count == 0) continue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)fg.count);
    cfg.blockDim = dim3((unsigned)fast_tiles_threads(b->fast_bps));
    cfg.dynamicSmemBytes = fg.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    launch_fast_tiles(b->fast_bps, fg.cap, fg.walls ? 2 : fg.form, cfg, b->cur, b->d_refs + fg.begin, stage, b->flags, b->status, timeout_ns, fault_block);
    if (fault_block >= 0) break;             // the failure test runs the first group only
  }
}

// The untiled stacks' sub-steps of stage `stage` as one cooperative launch per form present.
void launch_fast_grid(isw_batch *b, cudaStream_t st, int stage) {
  for (int f = 0; f < 2; f++) {
    const Sched &sc = b->scf[f];
    if (!b->untiled_form[f] || sc.nwcell == 0) continue;
    if (!b->cur) fail(ISW_EINVAL, "batch: no stack descriptors selected for the launch");
    ISW_CUDA(cudaMemsetAsync(b->bar, 0, sizeof(GridBarrier), st));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)b->grid_blocks[f]);
    cfg.blockDim = dim3(THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (f == 0) {
      const int ns = b->nsub[stage];
      long long to = DEFAULT_TIMEOUT_NS;
      void *args[] = {(void *)&b->cur, (void *)&sc, (void *)&stage, (void *)&ns, (void *)&b->bar,
                      (void *)&b->status, (void *)&to};
      ISW_CUDA(cudaLaunchKernelExC(&cfg, fast_grid_kernel(b->lmax, b->any_ext), args));
    } else
      launch_fast_grid_mixed(cfg, b->cur, sc, stage, b->nsub[stage], b->bar, b->status, DEFAULT_TIMEOUT_NS);
  }
}

// The dynamics of one step (through the last stage's end); returns whether its last launch was a tile kernel. The first kernel and the first after a tile launch (or a
// memset) take plain stream order; the others are programmatic dependents of the kernel before them.
bool enqueue_dyn(isw_batch *b, cudaStream_t st) {
  if (b->any_ob) launch_phase<PH_ONBED>(b, st, 0, 0, false);
  launch_phase<PH_INIT>(b, st, 0, 0, !b->any_ob ? false : true);
  if (b->any_nu4) {
    launch_phase<PH_LAPE1>(b, st, 0, 0);
    launch_phase<PH_LAPCV>(b, st, 0, 0);
    launch_phase<PH_LAPE2>(b, st, 0, 0);
  }
  bool after_tiles = false;
  for (int s = 0; s < 3; s++) {
    launch_phase<PH_A>(b, st, s, 0, !after_tiles);
    launch_phase<PH_E>(b, st, s, 0);
    launch_phase<PH_S>(b, st, s, 0);
    launch_fast(b, st, s, DEFAULT_TIMEOUT_NS, -1);      // the tiled stacks' fast loop and stage end
    if (b->any_untiled) {
      bool pdl = b->groups.empty();                      // not directly after a tile launch
      if (b->fast_grid) {
        launch_fast_grid(b, st, s);
        pdl = false;
      } else {
        for (int j = 0; j < b->nsub[s]; j++) {
          launch_phase<PH_ETA>(b, st, s, j, pdl);
          launch_phase<PH_UF>(b, st, s, j);
          pdl = true;
        }
      }
      launch_phase<PH_CS>(b, st, s, 0, pdl);
      launch_phase<PH_D>(b, st, s, 0);
    }
    after_tiles = !b->any_untiled;
  }
  return after_tiles;
}

// The transport passes after the stage-1 edge fluxes (P1 .. P4, M <- M1).
void enqueue_tr_tail(isw_batch *b, cudaStream_t st) {
  launch_phase<PH_P1, PH_P1G>(b, st, 0, 0);
  launch_phase<PH_P2E>(b, st, 0, 0);
  launch_phase<PH_P2, PH_P2G>(b, st, 0, 0);
  launch_phase<PH_P3E>(b, st, 0, 0);
  launch_phase<PH_P3>(b, st, 0, 0);
  launch_phase<PH_P4>(b, st, 0, 0);
}

// One step in the plain order: dynamics, then the interfacial stress with the transport's stage-1 edge fluxes, then
// the transport.
void enqueue(isw_batch *b, cudaStream_t st) {
  b->cur = b->d_desc;
  const bool pdl = !enqueue_dyn(b, st);
  if (b->any_air) {
    // air stacks: the interfacial stress's heat goes back to theta before the transport reads the tracers (theta is
    // one of them in the reference's world tick, world.py:291-301), so the stress, its heat and the stage-1 edge fluxes
    // are three passes here
    if (b->any_vmix) {
      launch_phase<PH_VMIX>(b, st, 0, 0, pdl);
      launch_phase<PH_VHEAT>(b, st, 0, 0);
    }
    if (b->any_tr) {
      launch_phase<PH_HF1>(b, st, 0, 0, pdl || b->any_vmix);
      enqueue_tr_tail(b, st);
    }
  } else {
    if (b->any_vmix || b->any_tr) launch_phase<PH_POST>(b, st, 0, 0, pdl);
    if (b->any_tr) enqueue_tr_tail(b, st);
  }
  ISW_CUDA(cudaGetLastError());
}

// Pipelined: the dynamics of the step described by `dyn` (with its interfacial stress) on `st`, and beside it on the
// side stream the transport of the step described by `tr` (the previous one); either may be null.
void enqueue_pipelined(isw_batch *b, cudaStream_t st, const StackDesc *dyn, const StackDesc *tr) {
  if (b->any_air) fail(ISW_EUNSUPPORTED, "batch: air stacks step in the plain order (the stress's heat precedes the transport)");
  const bool trans = tr && b->any_tr;
  if (trans && dyn) {
    ISW_CUDA(cudaEventRecord(b->ev_fork, st));
    ISW_CUDA(cudaStreamWaitEvent(b->side, b->ev_fork, 0));
  }
  cudaStream_t ts = trans && dyn ? b->side : st;
  if (trans) {
    b->cur = tr;
    launch_phase<PH_HF1>(b, ts, 0, 0, false);
    enqueue_tr_tail(b, ts);
  }
  if (dyn) {
    b->cur = dyn;
    const bool pdl = !enqueue_dyn(b, st);
    if (b->any_vmix) launch_phase<PH_VMIX>(b, st, 0, 0, pdl);
  }
  if (trans && dyn) {
    ISW_CUDA(cudaEventRecord(b->ev_join, b->side));
    ISW_CUDA(cudaStreamWaitEvent(st, b->ev_join, 0));
  }
  ISW_CUDA(cudaGetLastError());
}

void prepare(isw_batch *b) {
  if (b->dirty) rebuild(b);
}

// Queue `body` on st: directly when st is capturing a graph of the caller's, else as a graph of our own (captured on
// the private stream the first time, cached in *exec).
template <class F>
void run_graph(isw_batch *b, cudaStream_t st, cudaGraphExec_t *exec, F body) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  ISW_CUDA(cudaStreamIsCapturing(st, &cs));
  if (cs != cudaStreamCaptureStatusNone) {    // inside the caller's capture: queue the launches themselves
    body(st);
    return;
  }
  if (!*exec) {
    cudaGraph_t graph = nullptr;
    ISW_CUDA(cudaStreamBeginCapture(b->cap, cudaStreamCaptureModeThreadLocal));
    try {
      body(b->cap);
    } catch (...) {
      cudaStreamEndCapture(b->cap, &graph);
      if (graph) cudaGraphDestroy(graph);
      throw;
    }
    ISW_CUDA(cudaStreamEndCapture(b->cap, &graph));
    const cudaError_t ie = cudaGraphInstantiate(exec, graph, 0);
    cudaGraphDestroy(graph);
    ISW_CUDA(ie);
  }
  ISW_CUDA(cudaGraphLaunch(*exec, st));
}

const StackDesc *desc_of(isw_batch *b, int q) { return q == 0 ? b->d_desc : b->d_desc1; }

// Complete a pipelined batch: the last step's transport, and its Fm back into the registered arrays.
void flush(isw_batch *b, cudaStream_t st) {
  if (!b->pipeline || !b->primed) return;
  const int q = b->parity ^ 1;                // the last step's buffers
  if (b->any_tr) run_graph(b, st, &b->pexec[4 + q], [&](cudaStream_t s2) { enqueue_pipelined(b, s2, nullptr, desc_of(b, q)); });
  if (q == 1)
    for (size_t i = 0; i < b->fm_alt.size(); i++)
      ISW_CUDA(cudaMemcpyAsync(b->fm_pairs[i].first, b->fm_alt[i], b->fm_pairs[i].second, cudaMemcpyDeviceToDevice, st));
  b->primed = false;
}

// Flush a primed pipelined batch before its stacks or settings change (synchronising its private stream).
void settle(isw_batch *b) {
  if (b->pipeline && b->primed) {
    flush(b, b->cap);
    ISW_CUDA(cudaStreamSynchronize(b->cap));
  }
}

void step(isw_batch *b, cudaStream_t st) {
  for (auto &sl : b->slots)                  // an option set on a registered stack since: rebuild its descriptor
    if (sl.used && sl.version != sl.layers->version) {
      sl.version = sl.layers->version;
      b->dirty = true;
    }
  prepare(b);
  if (b->nstacks == 0) return;
  if (b->pipeline) {
    const int p = b->parity;
    const bool both = b->primed;
    run_graph(b, st, &b->pexec[both ? 2 + p : p],
              [&](cudaStream_t s2) { enqueue_pipelined(b, s2, desc_of(b, p), both ? desc_of(b, p ^ 1) : nullptr); });
    b->parity ^= 1;
    b->primed = true;
    return;
  }
  run_graph(b, st, &b->exec, [&](cudaStream_t s2) { enqueue(b, s2); });
}

}  // namespace

extern "C" {

int isw_batch_create(int device, isw_batch **out) {
  return guarded([&] {
    if (!out) fail(ISW_EINVAL, "batch: null output handle");
    ISW_CUDA(cudaSetDevice(device));
    isw_batch *b = new isw_batch();
    b->device = device;
    if (const char *e = std::getenv("ISW_NO_PDL")) b->pdl = e[0] != '1';   // diagnostics: plain stream order
    try {
      ISW_CUDA(cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, device));
      ISW_CUDA(cudaMalloc(&b->bar, sizeof(GridBarrier)));
      ISW_CUDA(cudaMemset(b->bar, 0, sizeof(GridBarrier)));
      ISW_CUDA(cudaMalloc(&b->status, sizeof(BatchStatus)));
      ISW_CUDA(cudaHostAlloc((void **)&b->status_host, sizeof(int), cudaHostAllocMapped));
      *b->status_host = 0;
      BatchStatus init{0, 0, nullptr};
      ISW_CUDA(cudaHostGetDevicePointer((void **)&init.mirror, b->status_host, 0));
      ISW_CUDA(cudaMemcpy(b->status, &init, sizeof(BatchStatus), cudaMemcpyHostToDevice));
      ISW_CUDA(cudaStreamCreateWithFlags(&b->cap, cudaStreamNonBlocking));
      ISW_CUDA(cudaStreamCreateWithFlags(&b->side, cudaStreamNonBlocking));
      ISW_CUDA(cudaEventCreateWithFlags(&b->ev_fork, cudaEventDisableTiming));
      ISW_CUDA(cudaEventCreateWithFlags(&b->ev_join, cudaEventDisableTiming));
    } catch (...) {
      cudaFree(b->bar);
      cudaFree(b->status);
      if (b->status_host) cudaFreeHost(b->status_host);
      delete b;
      throw;
    }
    *out = b;
  });
}

int isw_batch_destroy(isw_batch *b) {
  if (!b) return ISW_OK;
  cudaSetDevice(b->device);
  if (b->exec) cudaGraphExecDestroy(b->exec);
  for (auto x : b->pexec)
    if (x) cudaGraphExecDestroy(x);
  if (b->cap) cudaStreamDestroy(b->cap);
  if (b->side) cudaStreamDestroy(b->side);
  if (b->ev_fork) cudaEventDestroy(b->ev_fork);
  if (b->ev_join) cudaEventDestroy(b->ev_join);
  cudaFree(b->d_desc1);
  for (void *q : b->fm_alt) cudaFree(q);
  cudaFree(b->d_desc);
  cudaFree(b->d_chunks);
  cudaFree(b->d_refs);
  cudaFree(b->flags);
  cudaFree(b->bar);
  cudaFree(b->status);
  if (b->status_host) cudaFreeHost(b->status_host);
  delete b;
  (void)cudaGetLastError();         // a failure while freeing must not surface in the caller's next call
  return ISW_OK;
}

namespace {

int batch_add(isw_batch *b, isw_layers *layers, isw_transport *tr, double *h, double *u, double *Fm, double *theta, double *M,
              double *M1, double *const *tracers, int ntr, double dt, int nfast, int *slot) {
  return guarded([&] {
    if (!b || !layers || !h || !u || !Fm || !slot) fail(ISW_EINVAL, "batch.add: null argument");
    if (layers->grid->device != b->device) fail(ISW_EINVAL, "batch.add: the stack is on another device");
    if (layers->d.air && !theta) fail(ISW_EINVAL, "batch.add: air layers need their theta (isw_batch_add_air)");
    if (!layers->d.air && theta) fail(ISW_EINVAL, "batch.add: theta is for air layers");
    if (has_options(layers->d) && layers->d.precision != ISW_FP64)
      fail(ISW_EUNSUPPORTED, "batch.add: the option branches step in the FP64 form");
    if (!(dt > 0) || !std::isfinite(dt) || nfast < 1) fail(ISW_EINVAL, "batch.add: dt must be positive and nfast >= 1");
    if (tr) {
      if (!M || !M1 || !tracers) fail(ISW_EINVAL, "batch.add: transport needs M, M1 and the tracers");
      if (ntr < 1 || ntr > tr->T) fail(ISW_EINVAL, "batch.add: ntr outside 1..tracers of the transport");
      if (tr->L != layers->d.L || tr->grid != layers->grid) fail(ISW_EINVAL, "batch.add: transport and layers differ in grid or L");
      if (tr->precision != layers->d.precision) fail(ISW_EINVAL, "batch.add: transport and layers differ in precision form");
    }
    ISW_CUDA(cudaSetDevice(b->device));
    settle(b);
    BatchSlot sl;
    sl.used = true;
    sl.layers = layers;
    sl.tr = tr;
    sl.h = h; sl.u = u; sl.Fm = Fm; sl.M = M; sl.M1 = M1;
    sl.theta = theta;
    sl.version = layers->version;
    if (layers->d.air && layers->d.nu4 != 0) layers->nu4dt = layers->d.nu4 * dt;   // the step's nabla^4 loss (exchange heat)
    sl.ntr = tr ? ntr : 0;
    for (int j = 0; j < sl.ntr; j++) {
      if (!tracers[j]) fail(ISW_EINVAL, "batch.add: null tracer");
      sl.tracers[j] = tracers[j];
    }
    sl.dt = dt;
    sl.nfast = nfast;
    size_t k = 0;
    while (k < b->slots.size() && b->slots[k].used) k++;
    if (k == b->slots.size()) b->slots.push_back(sl);
    else b->slots[k] = sl;
    b->dirty = true;
    *slot = (int)k;
  });
}

}  // namespace

int isw_batch_add(isw_batch *b, isw_layers *layers, isw_transport *tr, double *h, double *u, double *Fm, double *M, double *M1,
                  double *const *tracers, int ntr, double dt, int nfast, int *slot) {
  return batch_add(b, layers, tr, h, u, Fm, nullptr, M, M1, tracers, ntr, dt, nfast, slot);
}

int isw_batch_add_air(isw_batch *b, isw_layers *layers, isw_transport *tr, double *h, double *u, double *Fm, double *theta,
                      double *M, double *M1, double *const *tracers, int ntr, double dt, int nfast, int *slot) {
  return batch_add(b, layers, tr, h, u, Fm, theta, M, M1, tracers, ntr, dt, nfast, slot);
}

// (library side: handles.cuh)
void isw_batch_set_check(isw_batch *b, int on) {
  if (b->check == (on != 0)) return;
  b->check = on != 0;
  b->dirty = true;
}

int isw_batch_pending(const isw_batch *b) { return *(volatile int *)b->status_host; }

int isw_batch_remove(isw_batch *b, int slot) {
  return guarded([&] {
    if (!b || slot < 0 || slot >= (int)b->slots.size() || !b->slots[slot].used) fail(ISW_EINVAL, "batch.remove: no such slot");
    ISW_CUDA(cudaSetDevice(b->device));
    settle(b);
    b->slots[slot] = BatchSlot();
    b->dirty = true;
  });
}

int isw_batch_config(isw_batch *b, int tiles_enabled, int tile_k, int layout, int tile_cells, int blocks_per_sm) {
  return guarded([&] {
    if (!b) fail(ISW_EINVAL, "batch.config: null handle");
    if (tile_k < 1 || tile_k > K_PROBE) fail(ISW_EINVAL, "batch.config: tile_k outside 1..8");
    if (layout < 0 || layout > 2) fail(ISW_EINVAL, "batch.config: layout must be 0 (choose), 1 (shared) or 2 (packed)");
    if (tile_cells != 0 && (tile_cells < 64 || tile_cells > 4096)) fail(ISW_EINVAL, "batch.config: tile_cells outside 64..4096");
    if (blocks_per_sm < 0 || blocks_per_sm > 2) fail(ISW_EINVAL, "batch.config: blocks_per_sm must be 0 (choose), 1 or 2");
    ISW_CUDA(cudaSetDevice(b->device));
    settle(b);
    b->tiles_enabled = tiles_enabled ? 1 : 0;
    b->tile_k = tile_k;
    b->layout = layout;
    b->tile_cells = tile_cells;
    b->force_bps = blocks_per_sm;
    b->dirty = true;
  });
}

int isw_batch_level_layout(isw_batch *b, int level, int mode, int tile_cells, int tile_k) {
  return guarded([&] {
    if (!b) fail(ISW_EINVAL, "batch.level_layout: null handle");
    if (level < 0 || level > 12) fail(ISW_EINVAL, "batch.level_layout: level outside 0..12");
    if (mode < 0 || mode > 2) fail(ISW_EINVAL, "batch.level_layout: mode must be 0 (the batch's), 1 (untiled) or 2 (packed)");
    if (tile_cells != 0 && (tile_cells < 64 || tile_cells > 4096)) fail(ISW_EINVAL, "batch.level_layout: tile_cells outside 64..4096");
    if (tile_k < 0 || tile_k > K_PROBE) fail(ISW_EINVAL, "batch.level_layout: tile_k outside 0..8");
    ISW_CUDA(cudaSetDevice(b->device));
    settle(b);
    if (mode == 0) b->levels.erase(level);
    else b->levels[level] = isw_batch::LevelLayout{mode, tile_cells, tile_k};
    b->dirty = true;
  });
}

int isw_batch_grid_loop(isw_batch *b, int mode) {
  return guarded([&] {
    if (!b) fail(ISW_EINVAL, "batch.grid_loop: null handle");
    ISW_CUDA(cudaSetDevice(b->device));
    settle(b);
    if (mode != ISW_GRID_SPLIT && mode != ISW_GRID_PERSISTENT) fail(ISW_EINVAL, "batch.grid_loop: mode must be 0 or 1");
    b->fast_grid = mode == ISW_GRID_PERSISTENT;
    b->dirty = true;
  });
}

int isw_batch_info(isw_batch *b, int *stacks, int *tiles, int *tile_k, long long *smem_bytes, int *groups, int *blocks_per_sm) {
  return guarded([&] {
    if (!b || !stacks || !tiles || !tile_k || !smem_bytes || !groups || !blocks_per_sm) fail(ISW_EINVAL, "batch.info: null argument");
    ISW_CUDA(cudaSetDevice(b->device));
    prepare(b);
    *stacks = b->nstacks;
    *tiles = b->ntiles;
    *tile_k = b->ntiles > 0 ? b->kused : 0;
    *smem_bytes = (long long)b->fast_smem;
    *groups = (int)b->groups.size();
    *blocks_per_sm = b->ntiles > 0 ? b->fast_bps : 0;
  });
}

int isw_batch_step(isw_batch *b, void *stream) {
  return guarded([&] {
    if (!b) fail(ISW_EINVAL, "batch.step: null handle");
    const int code = *(volatile int *)b->status_host;
    if (code == ISW_ETIMEOUT)
      fail(code, "batch.step: refused: an earlier step's wait on the device timed out, so the state is half-updated; restore "
                 "it and clear the status (isw_batch_status with reset) to step again");
    if (code != ISW_OK)
      fail(code, "batch.step: refused: an earlier step left a non-finite thickness; restore the state and clear the status "
                 "(isw_batch_status with reset) to step again");
    ISW_CUDA(cudaSetDevice(b->device));
    step(b, (cudaStream_t)stream);
  });
}

int isw_batch_pipeline(isw_batch *b, int on) {
  return guarded([&] {
    if (!b) fail(ISW_EINVAL, "batch.pipeline: null handle");
    ISW_CUDA(cudaSetDevice(b->device));
    settle(b);
    b->pipeline = on != 0;
    b->dirty = true;
  });
}

int isw_batch_flush(isw_batch *b, void *stream) {
  return guarded([&] {
    if (!b) fail(ISW_EINVAL, "batch.flush: null handle");
    ISW_CUDA(cudaSetDevice(b->device));
    flush(b, (cudaStream_t)stream);
  });
}

int isw_batch_status(isw_batch *b, void *stream, int reset) {
  int out = ISW_OK;
  const int rc = guarded([&] {
    if (!b) fail(ISW_EINVAL, "batch.status: null handle");
    ISW_CUDA(cudaSetDevice(b->device));
    int st = 0;
    if (reset) ISW_CUDA(cudaDeviceSynchronize());   // steps in flight on any stream: they raise flags and may yet fail
    ISW_CUDA(cudaMemcpyAsync(&st, &b->status->code, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    ISW_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    if (reset && st != ISW_OK) {             // (nothing to clear otherwise; the batch refuses to step until it is cleared)
      ISW_CUDA(cudaMemset(&b->status->code, 0, sizeof(int)));
      if (st == ISW_ETIMEOUT && b->flags)    // a launch that timed out left its tiles' flags apart
        ISW_CUDA(cudaMemset(b->flags, 0, sizeof(unsigned) * TILE_FLAG_STRIDE * (size_t)b->ntiles));
      ISW_CUDA(cudaDeviceSynchronize());
      *(volatile int *)b->status_host = 0;
    }
    out = st;
  });
  return rc != ISW_OK ? rc : out;
}

int isw_batch_fault_test(isw_batch *b, long long timeout_ns, void *stream) {
  return guarded([&] {
    if (!b) fail(ISW_EINVAL, "batch.fault_test: null handle");
    if (timeout_ns < 1000000 || timeout_ns > 2000000000LL) fail(ISW_EINVAL, "batch.fault_test: timeout outside 1 ms .. 2 s");
    ISW_CUDA(cudaSetDevice(b->device));
    prepare(b);
    if (b->ntiles == 0) fail(ISW_EUNSUPPORTED, "batch.fault_test: no tiled stack in the batch");
    if (b->groups[0].waited < 0) fail(ISW_EUNSUPPORTED, "batch.fault_test: stacks of one tile wait for no other");
    b->cur = b->d_desc;
    launch_fast(b, (cudaStream_t)stream, 0, timeout_ns, b->groups[0].waited);   // stage 0: it writes scratch only, every stage ends in an exchange
  });
}

}  // extern "C"
