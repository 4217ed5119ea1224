// The batched step's kernels for stacks in the mixed form (layers_mixed.cuh, transport_mixed.cuh): the same phase list,
// chunk tables and tiles as the plain FP64 kernels in batch.cu, compiled with fused multiply-adds (this file alone).
#include "batch.cuh"
#include "layers_mixed.cuh"
#include "mixed_stage.cuh"
#include "transport_mixed.cuh"

namespace isw {
namespace bt {
namespace {

// The grid-wide sub-step passes over a wide chunk: PH_ETA's cells (sub-step 0 item by item, as it also forms the slot
// coefficients), PH_UF's edges (also forming the layer fluxes on the stack's last sub-step).
template <int PH>
__device__ __forceinline__ void substep_chunk(const StackDesc &d, int st, int j, const Chunk &ch) {
  if (j >= d.n[st]) return;
  const LayersDev &M = d.M;
  const float tau = (float)d.tau[st];
  const int first = ch.begin + (int)threadIdx.x;
  if (PH == PH_ETA) {
    if (j == 0)
      for (int i = first; i < ch.end; i += THREADS) mixed::bt_eta_cell(M, tau, 0, d.n[st], i);
    else
      mixed::bt_eta_cells<SUB_WC>(M, tau, j, d.n[st], first, ch.end);
  } else {
    mixed::bt_u_edges(M, tau, j, d.n[st], first, ch.end);
    if (j == d.n[st] - 1) {
      const mixed::MStageArgs a = mixed::mstage_args(d, st);
      for (int i = first; i < ch.end; i += THREADS) mixed::flux_edge(M, a, M.acc[i], i);
    }
  }
}

template <int PH, int LMAXK, int MINB = 0>
__global__ void __launch_bounds__(THREADS, MINB) k_phase_m(const StackDesc *__restrict__ S, const Sched sc, int st, int j) {
  Chunk ch{0, 0, 0};
  const int kind = phase_chunk<PH>(sc, blockIdx.x, ch);
  if (kind < 0) return;
  const StackDesc &d = stage_desc(S, ch.s);
  pdl_wait();
  pdl_trigger();
  if (Dom<PH>::wide) {                       // the grid-wide sub-step passes: a wide chunk, SUB_W items a thread
    substep_chunk<PH>(d, st, j, ch);
    return;
  }
  const int i = ch.begin + (int)threadIdx.x;
  if (PH == PH_S && d.s_stage) {             // the block stages its rows' distinct neighbour records, then computes
    extern __shared__ __align__(16) float4 stg4[];
    const mixed::MStageArgs a = mixed::mstage_args(d, st);
    ISW_BATCH_L(d.L, LMAXK, mixed::stage_pk4<LL>(d.M, ch.begin / THREADS, stg4));
    __syncthreads();
    if (i < ch.end) ISW_BATCH_L(d.L, LMAXK, (mixed::slow_edge<LL, true>(d.M, a.cdt, i, stg4)));
    return;
  }
  if (i >= ch.end) return;
  const LayersDev &M = d.M;
  if (PH == PH_INIT) {
    if (kind == 0) {
      ISW_BATCH_L(d.L, LMAXK, fp64::eta0_cell<LL>(M, d.h, i));
      if (M.nu4 != 0) ISW_BATCH_L(d.L, LMAXK, (mixed::div_cell<LL, double>(M, d.u, i)));
    } else if (kind == 1) {
      ISW_BATCH_L(d.L, LMAXK, mixed::ubar0_edge<LL>(M, d.h, d.u, i));
    } else if (M.nu4 != 0) {
      ISW_BATCH_L(d.L, LMAXK, (mixed::curl_vertex<LL, double>(M, d.u, i)));
    }
  } else if (PH == PH_LAPE1 || PH == PH_LAPE2) {
    if (M.nu4 != 0) ISW_BATCH_L(d.L, LMAXK, mixed::lap_edge<LL>(M, PH == PH_LAPE1 ? M.L1f : M.L2f, i));
  } else if (PH == PH_LAPCV) {
    if (M.nu4 != 0) {
      if (kind == 0) ISW_BATCH_L(d.L, LMAXK, (mixed::div_cell<LL, float>(M, M.L1f, i)));
      else ISW_BATCH_L(d.L, LMAXK, (mixed::curl_vertex<LL, float>(M, M.L1f, i)));
    }
  } else if (PH == PH_A) {
    const mixed::MStageArgs a = mixed::mstage_args(d, st);
    if (kind == 0) ISW_BATCH_L(d.L, LMAXK, mixed::bern_cell<LL>(M, a.hs, a.us, i));
    else ISW_BATCH_L(d.L, LMAXK, mixed::pv_vertex<LL>(M, a.hs, a.us, i));
  } else if (PH == PH_E) {
    const mixed::MStageArgs a = mixed::mstage_args(d, st);
    ISW_BATCH_L(d.L, LMAXK, mixed::edge_hq<LL>(M, a.hs, a.us, i));
  } else if (PH == PH_S) {
    const mixed::MStageArgs a = mixed::mstage_args(d, st);
    ISW_BATCH_L(d.L, LMAXK, mixed::slow_edge<LL>(M, a.cdt, i));
  } else if (PH == PH_CS) {
    const mixed::MStageArgs a = mixed::mstage_args(d, st);
    ISW_BATCH_L(d.L, LMAXK, mixed::scale_sum_cell<LL>(M, a, i));
  } else if (PH == PH_D) {
    const mixed::MStageArgs a = mixed::mstage_args(d, st);
    if (kind == 0) {
      ISW_BATCH_L(d.L, LMAXK, mixed::h_cell<LL>(M, a, i));
      if (st == 2) check_finite_column(d.h, M.g.N, d.L, i, sc.status);
    } else {
      ISW_BATCH_L(d.L, LMAXK, mixed::u_edge<LL>(M, a, i));
    }
  } else if (PH == PH_VMIX) {
    if ((M.vmix != 0 || M.vmix_cd != 0) && d.L > 1) ISW_BATCH_L(d.L, LMAXK, fp64::vmix_edge<LL, false>(M, d.h, d.u, d.dt, i));
  } else if (PH == PH_HF1) {
    const EdgeRow r = edge_row(d, i);
    ISW_BATCH_L(d.L, LMAXK, mixed::tr_hf_edge<LL>(d.T, d.tr, 1, r.j0, r.j1, r.e));
  } else if (PH == PH_POST) {
    if (kind == 1) {
      if ((M.vmix != 0 || M.vmix_cd != 0) && d.L > 1) ISW_BATCH_L(d.L, LMAXK, fp64::vmix_edge<LL, false>(M, d.h, d.u, d.dt, i));
    } else {
      const EdgeRow r = edge_row(d, i);
      ISW_BATCH_L(d.L, LMAXK, mixed::tr_hf_edge<LL>(d.T, d.tr, 1, r.j0, r.j1, r.e));
    }
  } else if (PH == PH_P1) {
    ISW_BATCH_L(d.L, LMAXK, mixed::tr_c1<LL>(d.T, d.tr, i / M.g.N, i % M.g.N));
  } else if (PH == PH_P2E) {
    const EdgeRow r = edge_row(d, i);
    ISW_BATCH_L(d.L, LMAXK, mixed::tr_hf_edge<LL>(d.T, d.tr, 2, r.j0, r.j1, r.e));
  } else if (PH == PH_P2) {
    ISW_BATCH_L(d.L, LMAXK, mixed::tr_c2<LL>(d.T, d.tr, i / M.g.N, i % M.g.N));
  } else if (PH == PH_P3E) {
    const EdgeRow r = edge_row(d, i);
    ISW_BATCH_L(d.L, LMAXK, mixed::tr_a_edge<LL>(d.T, d.tr, r.j0, r.j1, r.e));
  } else if (PH == PH_P3) {
    ISW_BATCH_L(d.L, LMAXK, mixed::tr_c3<LL>(d.T, d.tr, i / M.g.N, i % M.g.N));
  } else if (PH == PH_P4) {
    const int jj = i / M.g.N, c = i % M.g.N;
    ISW_BATCH_L(d.L, LMAXK, mixed::tr_p4<LL>(d.T, d.tr, jj, c));
    if (jj == 0)
      for (int l = 0; l < d.L; l++) d.Mm[(size_t)l * M.g.N + c] = d.tr.M1[(size_t)l * M.g.N + c];
  }
}

template <int PH>
void launch_m(int lmax, int nb, cudaStream_t st, bool pdl, size_t smem, const StackDesc *desc, const Sched &sc, int stage,
              int j) {
  constexpr int MB3 = phase_blocks_an_sm(PH, 3, true), MB8 = phase_blocks_an_sm(PH, 8, true);
  switch (lmax) {
    case 2: launch_kernel(k_phase_m<PH, 2>, nb, st, pdl, smem, desc, sc, stage, j); break;
    case 3: launch_kernel(more_blocks(nb, MB3) ? k_phase_m<PH, 3, MB3> : k_phase_m<PH, 3>, nb, st, pdl, smem, desc, sc, stage, j); break;
    case 5: launch_kernel(k_phase_m<PH, 5>, nb, st, pdl, smem, desc, sc, stage, j); break;
    default: launch_kernel(more_blocks(nb, MB8) ? k_phase_m<PH, 8, MB8> : k_phase_m<PH, 8>, nb, st, pdl, smem, desc, sc, stage, j); break;
  }
}

}  // namespace

void slow_phase_smem_mixed(size_t bytes) {
  for (const void *fn : {(const void *)k_phase_m<PH_S, 2>, (const void *)k_phase_m<PH_S, 3>, (const void *)k_phase_m<PH_S, 5>,
                         (const void *)k_phase_m<PH_S, 8>, (const void *)k_phase_m<PH_S, 8, phase_blocks_an_sm(PH_S, 8, true)>})
    ISW_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

void launch_phase_mixed(int ph, int lmax, int nb, cudaStream_t st, bool pdl, size_t smem, const StackDesc *desc,
                        const Sched &sc, int stage, int j) {
  switch (ph) {
    case PH_INIT: launch_m<PH_INIT>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_LAPE1: launch_m<PH_LAPE1>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_LAPCV: launch_m<PH_LAPCV>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_LAPE2: launch_m<PH_LAPE2>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_A: launch_m<PH_A>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_E: launch_m<PH_E>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_S: launch_m<PH_S>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_ETA: launch_m<PH_ETA>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_UF: launch_m<PH_UF>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_CS: launch_m<PH_CS>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_D: launch_m<PH_D>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_POST: launch_m<PH_POST>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_P2: launch_m<PH_P2>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_P3: launch_m<PH_P3>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_P4: launch_m<PH_P4>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_P1: launch_m<PH_P1>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_P2E: launch_m<PH_P2E>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_P3E: launch_m<PH_P3E>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_VMIX: launch_m<PH_VMIX>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    case PH_HF1: launch_m<PH_HF1>(lmax, nb, st, pdl, smem, desc, sc, stage, j); break;
    default: break;
  }
}

namespace {

// The grid-wide fast loop of stage `st` for the untiled mixed stacks as one cooperative launch (batch.cu's k_fast_grid
// with the mixed form's per-item arithmetic: PH_ETA's and PH_UF's of k_phase_m).
__global__ void __launch_bounds__(THREADS) k_fast_grid_m(const StackDesc *__restrict__ S, const Sched sc, int st, int nsub,
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
      if (i < ch.end && j < d.n[st]) mixed::bt_eta_cell(d.M, (float)d.tau[st], j, d.n[st], i);
    }
    if (!grid_sync(bar, status, timeout_ns)) return;
    for (int c = blockIdx.x; c < sc.nuedge; c += gridDim.x) {
      const Chunk ch = sc.uedge[c];
      select(ch.s);
      const int i = ch.begin + (int)threadIdx.x;
      if (i < ch.end && j < d.n[st]) {
        mixed::bt_u_edge(d.M, (float)d.tau[st], j, d.n[st], i);
        if (j == d.n[st] - 1) mixed::flux_edge(d.M, mixed::mstage_args(d, st), d.M.acc[i], i);
      }
    }
    if (!grid_sync(bar, status, timeout_ns)) return;
  }
}

}  // namespace

const void *fast_grid_kernel_mixed() { return (const void *)k_fast_grid_m; }

void launch_fast_grid_mixed(const cudaLaunchConfig_t &cfg, const StackDesc *desc, const Sched &sc, int stage, int nsub,
                            GridBarrier *bar, BatchStatus *status, long long timeout_ns) {
  ISW_CUDA(cudaLaunchKernelEx(&cfg, k_fast_grid_m, desc, sc, stage, nsub, bar, status, timeout_ns));
}

}  // namespace bt
}  // namespace isw
