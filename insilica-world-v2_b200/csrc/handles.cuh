// Library-side definitions of the Layers and Transport handles (shared by the per-call path and the batched step).
#pragma once
#include <list>
#include <vector>

#include "common.cuh"
#include "transport_fp64.cuh"

struct GraphEntry {
  const double *h, *u, *Fm, *theta;
  double dt;
  int nfast;
  cudaGraphExec_t exec;
};

struct isw_batch;
extern "C" void isw_batch_set_check(isw_batch *b, int on);   // whether its steps look for non-finite thicknesses (default 1)
extern "C" int isw_batch_pending(const isw_batch *b);        // the status code its next step would be refused with

struct isw_layers {
  isw_grid *grid;
  int device = 0;                   // the grid's device (kept here so that destroy reads nothing of the grid)
  isw::LayersDev d;
  std::vector<void *> allocs;
  cudaStream_t cap;                 // private stream the step graphs are captured on
  std::list<GraphEntry> graphs;     // most recent first
  int colmax_blocks;
  int *nonfinite;
  double nu4dt = 0;                 // nu4 dt of the last step (the exchange books the step's nabla^4 loss as heat)
  int version = 0;                  // bumped when an option is set: batches holding the stack rebuild its descriptor
  GraphEntry last_key{};            // option stacks: the arguments of the last direct step and the option version it saw
  int last_version = -1;
  int repeats = 0;                  // calls in a row that repeated the one before
  int solo_wait = 1;                // repeats before the private batch is built for them, and the steps the last build served
  int solo_steps = 0;
  bool percall = false;             // FP64: step with the per-call kernels instead of the private batch
  // the private one-stack batch (its step graph and tiles) that direct calls step through
  isw_batch *solo = nullptr;
  int solo_slot = -1;
  int solo_version = -1;            // the option version its descriptor was last stepped with
  GraphEntry solo_key{};
  double *solo_Fm = nullptr;        // Fm when the caller passes none
};

struct isw_transport {
  isw_grid *grid;
  int device = 0;                   // the grid's device (kept here so that destroy reads nothing of the grid)
  isw::TransportDev d;
  int L, T, precision;
  double beta;
  std::vector<void *> allocs;
};
