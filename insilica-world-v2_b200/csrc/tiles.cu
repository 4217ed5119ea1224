// Host-side construction of the fast-loop tiles (see tiles.cuh).
#include <algorithm>
#include <utility>

#include "common.cuh"
#include "tiles.cuh"

namespace isw {
namespace {

// A grid's first step plans on several tilings, each partitioned and built on the host: 0.26 s in all at level 6 and 0.39 at
// level 7 (0.68 and 1.05 with a heap in the growth and the local ids in hash tables, of which the tables took two thirds).
constexpr int PARTITION_ROUNDS = 12;

// Grow P regions from their seeds, the smallest region first (ties: the lower region id), one cell at a time,
// breadth-first within a region: regions are connected and within a few cells of equal size. A region takes one cell a
// turn and drops out when its frontier is empty, so "the smallest first" is turns in order of the region's id.
std::vector<int32_t> grow_regions(int N, const int32_t *nbr, const std::vector<int> &seed) {
  const int P = (int)seed.size();
  std::vector<int32_t> owner(N, -1);
  std::vector<std::vector<int>> frontier(P);     // its cells so far, taken ones and those reached since by others included
  std::vector<size_t> head(P, 0);
  std::vector<int> growing(P);
  for (int p = 0; p < P; p++) {
    frontier[p].reserve((size_t)4 * (N / P + 1));
    frontier[p].push_back(seed[p]);
    growing[p] = p;
  }
  while (!growing.empty()) {
    size_t keep = 0;
    for (const int p : growing) {
      auto &q = frontier[p];
      size_t &at = head[p];
      while (at < q.size() && owner[q[at]] >= 0) at++;
      if (at == q.size()) continue;
      const int c = q[at++];
      owner[c] = p;
      for (int s = 0; s < 6; s++) {
        const int j = nbr[(size_t)c * 6 + s];
        if (j >= 0 && owner[j] < 0) q.push_back(j);
      }
      growing[keep++] = p;
    }
    growing.resize(keep);
  }
  for (int c = 0; c < N; c++)
    if (owner[c] < 0) fail(ISW_EINVAL, "tiles: a cell no region reached");
  return owner;
}

// The worst region's work: cells within two rings of it (what a tile exchanging every other sub-step holds).
int worst_region(int N, const int32_t *nbr, const std::vector<int32_t> &owner, int P) {
  std::vector<std::vector<int>> own(P);
  for (int c = 0; c < N; c++) own[owner[c]].push_back(c);
  std::vector<int> mark(N, -1);
  int worst = 0;
  for (int p = 0; p < P; p++) {
    std::vector<int> held = own[p];
    for (int c : held) mark[c] = p;
    for (size_t r = 0, head = 0; r < 2; r++) {
      const size_t stop = held.size();
      for (; head < stop; head++)
        for (int s = 0; s < 6; s++) {
          const int j = nbr[(size_t)held[head] * 6 + s];
          if (j >= 0 && mark[j] != p) { mark[j] = p; held.push_back(j); }
        }
    }
    worst = std::max(worst, (int)held.size());
  }
  return worst;
}

}  // namespace

std::vector<int32_t> partition_cells(int N, const int32_t *nbr, int P) {
  if (P < 1 || P > N) fail(ISW_EINVAL, "tiles: P outside 1..N");
  // seeds spread along the cell numbering (Hilbert order: spread over the sphere), then moved to their regions' centres
  // (the cell farthest from the region's border) and grown again: regions grown from the first seeds are long where the
  // numbering turns, and a long region holds more halo. The round with the smallest worst region is kept.
  std::vector<int> seed(P);
  for (int p = 0; p < P; p++) seed[p] = (int)(((int64_t)p * N + N / 2) / P);
  std::vector<int32_t> best = grow_regions(N, nbr, seed), owner = best;
  int least = worst_region(N, nbr, best, P);
  for (int it = 0; it < PARTITION_ROUNDS && P > 1; it++) {
    std::vector<int> depth(N, -1), queue;
    queue.reserve(N);
    for (int c = 0; c < N; c++)
      for (int s = 0; s < 6; s++) {
        const int j = nbr[(size_t)c * 6 + s];
        if (j >= 0 && owner[j] != owner[c]) { depth[c] = 0; queue.push_back(c); break; }
      }
    for (size_t head = 0; head < queue.size(); head++) {
      const int c = queue[head];
      for (int s = 0; s < 6; s++) {
        const int j = nbr[(size_t)c * 6 + s];
        if (j >= 0 && depth[j] < 0 && owner[j] == owner[c]) { depth[j] = depth[c] + 1; queue.push_back(j); }
      }
    }
    for (int c : queue) seed[owner[c]] = c;      // the last cell reached of each region
    owner = grow_regions(N, nbr, seed);
    const int w = worst_region(N, nbr, owner, P);
    if (w < least) { least = w; best = owner; }
  }
  return best;
}

TileSetHost build_tiles(int N, int E, const int32_t *nbr, const int32_t *cellEdge, const int8_t *cellSign, const int32_t *eI,
                        const int32_t *eJ, const std::vector<int32_t> &owner, int P, int k) {
  if (P < 1 || k < 1) fail(ISW_EINVAL, "tiles: P and k must be positive");
  TileSetHost t;
  t.P = P;
  t.k = k;
  t.cell_off.push_back(0);
  t.edge_off.push_back(0);
  std::vector<std::vector<int>> own(P);
  for (int c = 0; c < N; c++) own[owner[c]].push_back(c);
  std::vector<int> ring(N, -1);                  // of the present tile, and its local ids (-1 outside it)
  std::vector<int> touched;
  std::vector<int> lc(N, -1), le(E, -1);
  std::vector<std::vector<int>> peers(P);        // tiles whose owned cells or edges a tile holds, made symmetric
  std::vector<int> met(P, -1);                   // met[o] == p: tile p has o among its peers
  auto meet = [&](int p, int o) {
    if (o == p || met[o] == p) return;
    met[o] = p;
    peers[p].push_back(o);
    peers[o].push_back(p);
  };
  for (int p = 0; p < P; p++) {
    std::vector<int> order = own[p];
    for (int c : order) { ring[c] = 0; touched.push_back(c); }
    size_t head = 0;
    std::vector<int> ring_end(k + 1, 0);
    ring_end[0] = (int)order.size();
    for (int r = 1; r <= k; r++) {
      const size_t stop = order.size();
      for (; head < stop; head++) {
        const int c = order[head];
        for (int s = 0; s < 6; s++) {
          const int j = nbr[(size_t)c * 6 + s];
          if (j < 0 || ring[j] >= 0) continue;
          ring[j] = r;
          order.push_back(j);
          touched.push_back(j);
        }
      }
      ring_end[r] = (int)order.size();
    }
    for (int r = 0; r <= k; r++) {
      const int a = r == 0 ? 0 : ring_end[r - 1], b = ring_end[r];
      std::sort(order.begin() + a, order.begin() + b);
    }
    for (size_t q = 0; q < order.size(); q++) lc[order[q]] = (int)q;
    // edges of the local cells, keyed by (ring of the nearer cell, not owned, id): owned edges first within ring 0
    std::vector<std::vector<int>> part(2 * (size_t)(k + 1));   // 2 ring + (not owned)
    size_t nedges = 0;
    for (int c : order)
      for (int s = 0; s < 6; s++) {
        const int e = cellEdge[(size_t)c * 6 + s];
        if (e < 0 || le[e] >= 0) continue;
        le[e] = 0;
        const int ra = ring[eI[e]] >= 0 ? ring[eI[e]] : k + 1, rb = ring[eJ[e]] >= 0 ? ring[eJ[e]] : k + 1;
        part[2 * (size_t)std::min(ra, rb) + (owner[eI[e]] == p ? 0 : 1)].push_back(e);
        nedges++;
      }
    std::vector<int> ev;
    ev.reserve(nedges);
    int eown = 0;
    std::vector<int> edge_end(k + 1, 0);
    for (int r = 0; r <= k; r++)
      for (int f = 0; f < 2; f++) {
        auto &v = part[2 * (size_t)r + f];
        std::sort(v.begin(), v.end());
        ev.insert(ev.end(), v.begin(), v.end());
        if (f == 0) eown += (int)v.size();
        edge_end[r] = (int)ev.size();
      }
    for (size_t q = 0; q < ev.size(); q++) le[ev[q]] = (int)q;
    if (order.size() > 32000 || ev.size() > 32000) fail(ISW_EINVAL, "tiles: a tile outgrows 16-bit local ids");
    for (int r = 0; r <= k; r++) {
      t.ncnt.push_back(ring_end[r]);
      t.ecnt.push_back(edge_end[r]);
    }
    t.eown.push_back(eown);
    const int pad = 2 * (int)ev.size();        // a padded slot reads the value after the last edge's, kept zero
    auto put = [](std::vector<uint16_t> &v, const int *slot, int id) {
      for (int s = 0; s < 6; s++) v.push_back((uint16_t)slot[s]);
      v.push_back((uint16_t)((uint32_t)id & 0xffffu));
      v.push_back((uint16_t)((uint32_t)id >> 16));
    };
    for (int c : order) {
      t.cells.push_back(c);
      meet(p, owner[c]);
      int slot[6];
      std::pair<int, int> asc[6];
      for (int s = 0; s < 6; s++) {
        const int e = cellEdge[(size_t)c * 6 + s];
        slot[s] = e < 0 ? pad : 2 * le[e] + (cellSign[(size_t)c * 6 + s] < 0 ? 1 : 0);
        asc[s] = std::make_pair(e < 0 ? E : e, slot[s]);
      }
      put(t.cedge, slot, c);
      std::sort(asc, asc + 6);
      for (int s = 0; s < 6; s++) slot[s] = asc[s].second;
      put(t.casc, slot, c);
    }
    for (const int e : ev) {
      t.edges.push_back(e);
      meet(p, owner[eI[e]]);
      const int a = lc[eI[e]], b = lc[eJ[e]];
      t.eix.push_back(e);
      t.eix.push_back((int32_t)((a < 0 ? 0x7fffu : (uint32_t)a) | (b < 0 ? 0x7fffu : (uint32_t)b) << 16));
    }
    t.cell_off.push_back((int32_t)t.cells.size());
    t.edge_off.push_back((int32_t)t.edges.size());
    for (int c : touched) ring[c] = lc[c] = -1;
    for (int e : ev) le[e] = -1;
    touched.clear();
  }
  t.nbr_off.push_back(0);
  for (int p = 0; p < P; p++) {
    std::sort(peers[p].begin(), peers[p].end());
    peers[p].erase(std::unique(peers[p].begin(), peers[p].end()), peers[p].end());
    t.nbrs.insert(t.nbrs.end(), peers[p].begin(), peers[p].end());
    t.nbr_off.push_back((int32_t)t.nbrs.size());
  }
  return t;
}

}  // namespace isw
