// Shared-memory tiles for the barotropic fast loop.
//
// The fast loop (reference layers.cu:366-388, driven by layers.py:168-175) alternates a cell pass (eta) and an edge pass
// (ubar) ceil(c nfast) times per stage. Each tile owns a compact region of cells (grown breadth-first from a seed, the
// smallest region growing first, so regions are compact and within a few cells of equal size) and the edges whose eI
// cell it owns; it holds on chip its cells out to k rings (ring 0 = owned) and every edge of those cells. It
// can then advance k sub-steps with no grid-wide sync: sub-step m (1..k) updates eta on cells of ring <= k - m + 1
// and ubar on edges whose nearer cell has ring <= k - m, which is exactly what the owned values after k sub-steps
// depend on. Tiles exchange owned eta and ubar through global memory every k sub-steps (double-buffered; a tile waits
// for the tiles whose cells it holds, not for the grid). Arithmetic is the reference's, per cell and edge, in the same gather order.
//
// Local numbering: cells in ring order, edges in order of their nearer cell's ring with the owned edges first, so
// "ring <= r" is a prefix and the owned edges are [0, eown).
#pragma once
#include <stdint.h>

#include <vector>

namespace isw {

// What one tile may hold: thread t of a block of NT keeps the state of cells t, t + NT, ... and edges t, t + NT, ... in
// registers (80 a thread), so a tile has at most C x NT cells, E x NT edges and A x NT edges of its own cells, whose
// sub-step sums are kept. Two capacities: the small one keeps all of it in registers but for 4 bytes a thread (48 in the
// mixed form), the large one (which lets a level-7 stack of 163,842 cells fill 148 SMs) spills some 100. The stage's end
// holds the fluxes and limiter factors of all layers at once where they fit in shared memory; where they do not (level 7 on
// 148 SMs: five FP64 layers, six mixed ones) the large capacity's other kernel takes them in groups of layers.
struct TileCap {
  int C, E, A;
  bool groups;
};
constexpr TileCap TILE_CAP[3] = {{2, 5, 3, false}, {2, 7, 5, false}, {2, 7, 5, true}};
// Threads of a tile block when one or two tiles share an SM.
constexpr int TILE_NT1 = 768, TILE_NT2 = 384;
constexpr int TILE_FLAG_STRIDE = 8;            // a tile's exchange flag has a 32-byte sector of its own

struct TileSetHost {
  int P = 0, k = 0;
  std::vector<int32_t> cell_off, edge_off;     // P + 1 offsets
  std::vector<int32_t> cells, edges;           // global ids, tile by tile, local order
  std::vector<int32_t> ncnt, ecnt;             // per tile k + 1 prefix counts: cells of ring <= r, edges of ring <= r
  std::vector<int32_t> eown;                   // per tile: owned edges (eI owned), the first of the local edges
  // per local cell its six slots, 2 x local edge + (1 where the cell is the edge's eJ side), padded with 2 x the tile's
  // edges, and its global id as the last two halves of the 16-byte word: in cellEdge order and in ascending edge order
  std::vector<uint16_t> cedge, casc;
  std::vector<int32_t> eix;                    // per local edge (global id, local cells eI | eJ << 16; 0x7fff outside)
  std::vector<int32_t> nbr_off, nbrs;          // per tile: the tiles it exchanges with (symmetric)
};

// Shared memory of a tile of nc cells (nc1 within one ring) and ne edges (ne0 of its own cells) whose stage's end holds L
// layers at once (groups: of more): the global ids (and the FP64 form's areas), then the fast loop's arrays, which the stage's
// end reuses. Fast loop, per edge and cell: FP64 the flux l_e H_e ub, l_e H_e, (G, d_e); Y. Mixed the flux and its negative,
// (G, 1/d_e); Y. One flux more, zero, for padded slots. Stage's end: the layer fluxes of the own cells' edges and the limiter
// factors, 8 bytes each, in groups also the edges' mean barotropic wind.
inline size_t tile_smem_bytes(size_t nc, size_t ne, size_t nc1, size_t ne0, size_t L, bool groups, bool mixed) {
  const size_t ids = (ne + nc + 1) / 2 * 8 + (mixed ? 0 : 8 * nc);
  const size_t loop = mixed ? (2 * (ne + 1) + 2 * ne + nc) * 4 : (4 * ne + 2 + nc) * 8;
  const size_t end = 8 * (L * (ne0 + nc1) + (groups ? ne0 : 0));
  return ids + 16 + (loop > end ? loop : end);   // (16: the loop's arrays start on a 16-byte boundary)
}

// Compact balanced partition of the N cells into P regions (owner per cell).
std::vector<int32_t> partition_cells(int N, const int32_t *nbr, int P);

// Build the tiles of a partition over a grid (neighbour table nbr (N x 6, pads -1), cellEdge and cellSign (N x 6),
// eI, eJ (E)).
TileSetHost build_tiles(int N, int E, const int32_t *nbr, const int32_t *cellEdge, const int8_t *cellSign, const int32_t *eI,
                        const int32_t *eJ, const std::vector<int32_t> &owner, int P, int k);

}  // namespace isw
