// The mixed form's stage arguments from a stack's descriptor (shared by the grid-wide passes and the tiles).
#pragma once
#include "batch.cuh"
#include "layers_mixed.cuh"

namespace isw {
namespace mixed {

__device__ __forceinline__ MStageArgs mstage_args(const bt::StackDesc &d, int st) {
  const LayersDev &M = d.M;
  MStageArgs a;
  a.h0 = d.h;
  a.u0 = d.u;
  a.u0f = M.u32;
  a.hs = st == 0 ? d.h : st == 1 ? M.h1 : M.h2;
  a.us = st == 0 ? M.u32 : st == 1 ? M.u1f : M.u2f;
  a.hn = st == 0 ? M.h1 : st == 1 ? M.h2 : d.h;
  a.un = st == 2 ? d.u : nullptr;
  a.unf = st == 0 ? M.u1f : st == 1 ? M.u2f : nullptr;
  a.Fm = st == 2 ? d.Fm : nullptr;
  a.cdt = d.cdt[st];
  a.dt = d.dt;
  a.tau = (float)d.tau[st];
  a.inv_n = d.inv_n[st];
  a.n = d.n[st];
  return a;
}

}  // namespace mixed
}  // namespace isw
