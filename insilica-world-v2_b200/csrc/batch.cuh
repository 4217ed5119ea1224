// Definitions shared by the batched step's translation units (batch.cu: plain FP64 phases and the step's host side;
// batch_mixed.cu: the mixed form's phases, compiled with fused multiply-adds): the stack descriptor, chunk tables,
// tiles, the bounded grid barrier of the persistent loop, the phase list.
#pragma once
#include <cuda/atomic>

#include "common.cuh"
#include "transport_fp64.cuh"

namespace isw {
namespace bt {

constexpr int FAST_KMAX = 8;                  // the largest exchange interval of the tiled fast loop

struct TileSetDev {
  int P, k;
  const int *cell_off, *edge_off, *ncnt, *ecnt, *eown, *nbr_off, *nbrs;
  const uint4 *cedge, *casc;
  const int2 *eix;
  const double2 *el;                          // (l_e, d_e) per local edge
  const float2 *el32;                         // the mixed form's (l_e, 1 / d_e)
  const double *aarea;                        // the area per local cell
  const float *arA32;                         // and its FP32 reciprocal
};

struct StackDesc {
  LayersDev M;
  TransportDev T;
  TrArgs tr;                 // M0 = the stack's M, M1, Fm, tracers, L, rows, beta
  double *h, *u, *Fm, *Mm;
  double *theta;             // air layers: potential temperature (L x N); null for Boussinesq layers
  double dt;
  int L, has_tr, tiled;
  int eg, cg;                // tracers of one thread of the transport's edge passes, of its first two cell passes
  int check;                 // the step's end looks for non-finite thicknesses
  int s_stage;               // the slow tendency stages its blocks' neighbour records in shared memory
  int n[3];
  double cdt[3], tau[3], inv_n[3];
  TileSetDev tiles;
  int lg;                    // tiled: layers whose fluxes the stage's end holds at once
  int tile_base;             // the stack's first tile in the batch's list (and its first flag)
};

struct Chunk {
  int s, begin, end;
};

struct TileRef {
  int s, p;
};

// The batch's status word on the device, and where a kernel that sets it also writes the code for the host: a mapped
// pinned host word, so that the next isw_batch_step can refuse to run without synchronising the stream.
struct BatchStatus {
  int code;
  int pad;
  volatile int *mirror;
};

// Record the first failure of a step (later ones keep the first code) and publish it to the host.
__device__ __forceinline__ void raise_status(BatchStatus *s, int code) {
  if (atomicCAS(&s->code, 0, code) == 0 && s->mirror) {
    *s->mirror = code;
    __threadfence_system();
  }
}

struct Sched {
  const Chunk *cell, *edge, *vert, *rows, *erows;   // rows: (tracer, cell) pairs; erows: (tracers of a thread, edge)
  const Chunk *grows;                               // (tracers of a thread, cell)
  int ncell, nedge, nvert, nrows, nerows, ngrows;
  const Chunk *wcell, *wedge, *uedge;               // untiled stacks only: the sub-step passes' chunks (SUB_W... x THREADS),
  int nwcell, nwedge, nuedge;                       // and their edges in plain chunks
  BatchStatus *status;
};

// The step's result check: every layer of cell i must hold a finite thickness after the last stage, else the batch's
// status becomes ISW_ENOTFINITE (a NaN or Inf in a wind reaches the thicknesses through the layer fluxes in the same step).
__device__ __forceinline__ void check_finite_column(const double *__restrict__ h, int N, int L, int i, BatchStatus *s) {
  bool ok = true;
  for (int k = 0; k < L; k++) ok = ok && isfinite(h[(size_t)k * N + i]);
  if (!ok) raise_status(s, ISW_ENOTFINITE);
}

struct GridBarrier {
  unsigned count, gen;
};

__device__ __forceinline__ long long globaltimer() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Block-wide grid barrier with a bounded wait. Returns false once any block has recorded a failure.
__device__ inline bool grid_sync(GridBarrier *b, BatchStatus *status, long long timeout_ns) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    cuda::atomic_ref<unsigned, cuda::thread_scope_device> gen(b->gen), cnt(b->count);
    cuda::atomic_ref<int, cuda::thread_scope_device> st(status->code);
    const unsigned g0 = gen.load(cuda::memory_order_acquire);
    __threadfence();
    if (cnt.fetch_add(1u, cuda::memory_order_acq_rel) == gridDim.x - 1) {
      cnt.store(0u, cuda::memory_order_relaxed);
      gen.fetch_add(1u, cuda::memory_order_release);
    } else {
      const long long t0 = globaltimer();
      unsigned it = 0;
      while (gen.load(cuda::memory_order_acquire) == g0) {
        ++it;
        if ((it & 63) == 0) {
          if (st.load(cuda::memory_order_relaxed) != 0) { ok = 0; break; }
          if (globaltimer() - t0 > timeout_ns) {
            raise_status(status, ISW_ETIMEOUT);
            ok = 0;
            break;
          }
        }
        if (it > (1u << 30)) { ok = 0; break; }
      }
    }
    __threadfence();
    if (st.load(cuda::memory_order_relaxed) != 0) ok = 0;
  }
  __syncthreads();
  return ok != 0;
}

#define ISW_BATCH_L(LV, LMAXK, ...)                                                             \
  do {                                                                                          \
    switch (LV) {                                                                               \
      case 1: { constexpr int LL = 1; __VA_ARGS__; } break;                                     \
      case 2: if (LMAXK >= 2) { constexpr int LL = 2 <= LMAXK ? 2 : 1; __VA_ARGS__; } break;    \
      case 3: if (LMAXK >= 3) { constexpr int LL = 3 <= LMAXK ? 3 : 1; __VA_ARGS__; } break;    \
      case 4: if (LMAXK >= 4) { constexpr int LL = 4 <= LMAXK ? 4 : 1; __VA_ARGS__; } break;    \
      case 5: if (LMAXK >= 5) { constexpr int LL = 5 <= LMAXK ? 5 : 1; __VA_ARGS__; } break;    \
      case 6: if (LMAXK >= 6) { constexpr int LL = 6 <= LMAXK ? 6 : 1; __VA_ARGS__; } break;    \
      case 7: if (LMAXK >= 7) { constexpr int LL = 7 <= LMAXK ? 7 : 1; __VA_ARGS__; } break;    \
      case 8: if (LMAXK >= 8) { constexpr int LL = 8 <= LMAXK ? 8 : 1; __VA_ARGS__; } break;    \
      default: break;                                                                           \
    }                                                                                           \
  } while (0)

__device__ __forceinline__ StageArgs stage_args(const StackDesc &d, int st) {
  StageArgs a;
  a.h0 = d.h;
  a.u0 = d.u;
  a.hs = st == 0 ? d.h : st == 1 ? d.M.h1 : d.M.h2;
  a.us = st == 0 ? d.u : st == 1 ? d.M.u1 : d.M.u2;
  a.hn = st == 0 ? d.M.h1 : st == 1 ? d.M.h2 : d.h;
  a.un = st == 0 ? d.M.u1 : st == 1 ? d.M.u2 : d.u;
  a.Fm = st == 2 ? d.Fm : nullptr;
  a.cdt = d.cdt[st];
  a.dt = d.dt;
  a.tau = d.tau[st];
  a.inv_n = d.inv_n[st];
  a.n = d.n[st];
  return a;
}

// The block's stack descriptor, staged in shared memory (one chunk per block, so one stack per block).
__device__ __forceinline__ const StackDesc &stage_desc(const StackDesc *S, int s) {
  __shared__ __align__(16) unsigned char buf[sizeof(StackDesc)];
  const unsigned long long *src = reinterpret_cast<const unsigned long long *>(S + s);
  unsigned long long *dst = reinterpret_cast<unsigned long long *>(buf);
  for (int w = threadIdx.x; w < (int)(sizeof(StackDesc) / 8); w += blockDim.x) dst[w] = src[w];
  __syncthreads();
  return *reinterpret_cast<const StackDesc *>(buf);
}

// The FCT step's passes: POST (edges: interfacial stress; (tracer, edge): stage-1 fluxes), P1 (cells: M1, td, p1),
// P2E (stage-2 fluxes), P2 (cells: p2), P3E (antidiffusive fluxes), P3 (cells: ratios), P4 (cells: limited update).
// A pipelined batch splits POST into VMIX (edges, the dynamics' last pass) and HF1 ((tracer, edge), the transport's first);
// a batch with air stacks runs VMIX, VHEAT (cells: the stress's heat back to theta) and HF1 in place of POST.
// PH_ETA / PH_UF: the grid-wide cell and edge sub-steps of the untiled stacks (UF also forms the layer fluxes on a stack's
// last sub-step); PH_CS and PH_D: their limiter and their stage's end (tiled stacks end their stage in the tile kernel).
// PH_P1G / PH_P2G: PH_P1 / PH_P2 with CELL_TRACERS tracers a thread (kernels of their own: they need more registers).
enum Phase { PH_INIT, PH_LAPE1, PH_LAPCV, PH_LAPE2, PH_A, PH_E, PH_S, PH_ETA, PH_UF, PH_CS, PH_D, PH_POST, PH_P2, PH_P3, PH_P4,
             PH_P1, PH_P2E, PH_P3E, PH_VMIX, PH_HF1, PH_VHEAT, PH_ONBED, PH_P1G, PH_P2G };

// Blocks an SM that a launch bound asks of a pass (0: none), where the registers of its own accord leave one block fewer: the
// instances of six to eight layers (and the mixed P1 of three, at 66). A launch takes the bounded kernel when it has more
// blocks than fit without it. With one block fewer, cold caches, 7 layers: P1 30.4 against 21.2 us and P4 32.1 against 22.6
// (FP64, level 6), S 133.9 against 115.8 (mixed, level 7); four mixed level-6 stacks of 7 layers and a tracer 1.348 ms a step
// against 1.263. But where every block fits anyway the bound's spills cost: a mixed level-5 stack of 7 layers 0.228 ms
// against 0.217.
__host__ __device__ constexpr int phase_blocks_an_sm(int ph, int lmax, bool mixed) {
  if (lmax == 3) return ph == PH_P1 && mixed ? 4 : 0;
  if (lmax < 8) return 0;
  return ph == PH_P1 || (ph == PH_P4 && !mixed) ? 2 : ph == PH_S && mixed ? 3 : 0;
}

// Item i of the transport's edge passes: its edge, and its tracers [j0, j1).
struct EdgeRow {
  int j0, j1, e;
};
__device__ __forceinline__ EdgeRow edge_row(const StackDesc &d, int i) {
  const int g = i / d.M.g.E, ntr = d.tr.rows / d.L, j0 = g * d.eg;
  return EdgeRow{j0, min(j0 + d.eg, ntr), i - g * d.M.g.E};
}

// Item i of the first two cell passes: its cell, its first tracer and how many.
struct CellRow {
  int j0, n, c;
};
template <int PH>
__host__ __device__ constexpr int phase_tracers() { return PH == PH_P1G || PH == PH_P2G ? fp64::CELL_TRACERS : 1; }
__device__ __forceinline__ CellRow cell_row(const StackDesc &d, int i) {
  const int g = i / d.M.g.N, ntr = d.tr.rows / d.L, j0 = g * d.cg;
  return CellRow{j0, min(d.cg, ntr - j0), i - g * d.M.g.N};
}

// Domains of a phase, in block order: which chunk tables its blocks walk.
template <int PH>
struct Dom {
  static constexpr bool cell = PH == PH_INIT || PH == PH_LAPCV || PH == PH_A || PH == PH_ETA || PH == PH_D || PH == PH_CS ||
                               PH == PH_VHEAT || PH == PH_ONBED;
  static constexpr bool edge = PH == PH_INIT || PH == PH_LAPE1 || PH == PH_LAPE2 || PH == PH_E || PH == PH_S || PH == PH_D ||
                               PH == PH_POST || PH == PH_VMIX || PH == PH_UF;
  static constexpr bool vert = PH == PH_INIT || PH == PH_LAPCV || PH == PH_A;
  static constexpr bool rows = PH == PH_P3 || PH == PH_P4;
  static constexpr bool grows = PH == PH_P1 || PH == PH_P2 || PH == PH_P1G || PH == PH_P2G;
  static constexpr bool erows = PH == PH_POST || PH == PH_P2E || PH == PH_P3E || PH == PH_HF1;
  static constexpr bool wide = PH == PH_ETA || PH == PH_UF;                    // cells / edges in the wide chunks
  static constexpr bool untiled = wide || PH == PH_CS || PH == PH_D;           // of the untiled stacks only
};
static_assert(SUB_WC == 1, "the untiled stacks' wide cell chunks are also their plain ones");

template <int PH>
__host__ __device__ inline int cell_chunks(const Sched &sc) { return Dom<PH>::untiled ? sc.nwcell : sc.ncell; }
template <int PH>
__host__ __device__ inline int edge_chunks(const Sched &sc) { return Dom<PH>::wide ? sc.nwedge : Dom<PH>::untiled ? sc.nuedge : sc.nedge; }

// Blocks of a phase over a schedule.
template <int PH>
inline int phase_blocks(const Sched &sc) {
  return (Dom<PH>::cell ? cell_chunks<PH>(sc) : 0) + (Dom<PH>::edge ? edge_chunks<PH>(sc) : 0) + (Dom<PH>::vert ? sc.nvert : 0) +
         (Dom<PH>::rows ? sc.nrows : 0) + (Dom<PH>::grows ? sc.ngrows : 0) + (Dom<PH>::erows ? sc.nerows : 0);
}

// The chunk of block b of a phase and its kind (0 cell, 1 edge, 2 vertex, 3 (tracer, cell), 4 (tracer, edge)), or -1.
template <int PH>
__device__ __forceinline__ int phase_chunk(const Sched &sc, int b, Chunk &ch) {
  if (Dom<PH>::cell) {
    const int n = cell_chunks<PH>(sc);
    if (b < n) { ch = (Dom<PH>::untiled ? sc.wcell : sc.cell)[b]; return 0; }
    b -= n;
  }
  if (Dom<PH>::edge) {
    const int n = edge_chunks<PH>(sc);
    if (b < n) { ch = (Dom<PH>::wide ? sc.wedge : Dom<PH>::untiled ? sc.uedge : sc.edge)[b]; return 1; }
    b -= n;
  }
  if (Dom<PH>::vert) { if (b < sc.nvert) { ch = sc.vert[b]; return 2; } b -= sc.nvert; }
  if (Dom<PH>::grows) { if (b < sc.ngrows) { ch = sc.grows[b]; return 3; } b -= sc.ngrows; }
  if (Dom<PH>::rows) { if (b < sc.nrows) { ch = sc.rows[b]; return 3; } b -= sc.nrows; }
  if (Dom<PH>::erows) { if (b < sc.nerows) { ch = sc.erows[b]; return 4; } }
  return -1;
}


constexpr size_t S_STAGE_MAX = 64 * 1024;   // the slow tendency's staged neighbour records: at most this per block

void launch_phase_mixed(int ph, int lmax, int nb, cudaStream_t st, bool pdl, size_t smem, const StackDesc *desc,
                        const Sched &sc, int stage, int j);
void slow_phase_smem_mixed(size_t bytes);
const void *fast_grid_kernel_mixed();
void launch_fast_grid_mixed(const cudaLaunchConfig_t &cfg, const StackDesc *desc, const Sched &sc, int stage, int nsub,
                            GridBarrier *bar, BatchStatus *status, long long timeout_ns);

// The tiled fast loop (fast_tiles.cu): the kernel of a form (0 FP64, 1 mixed, 2 FP64 with walls) and capacity
// for `bps` tile blocks per SM, its block size, and its launch.
const void *fast_tiles_kernel(int bps, int cap, int form);
int fast_tiles_threads(int bps);
void launch_fast_tiles(int bps, int cap, int form, const cudaLaunchConfig_t &cfg, const StackDesc *desc, const TileRef *refs, int stage,
                       unsigned *flags, BatchStatus *status, long long timeout_ns, int fault_block);

}  // namespace bt
}  // namespace isw
