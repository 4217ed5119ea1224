// Host-side construction of the fast-loop tiles (see tiles.cuh).
#include <algorithm>
#include <deque>
#include <queue>
#include <set>
#include <tuple>
#include <unordered_map>

#include "common.cuh"
#include "tiles.cuh"

namespace isw {
namespace {

constexpr int PARTITION_ROUNDS = 12;


// Grow P regions from their seeds, the smallest region first (ties: the lower region id), one cell at a time,
// breadth-first within a region: regions are connected and within a few cells of equal size.
std::vector<int32_t> grow_regions(int N, const int32_t *nbr, const std::vector<int> &seed) {
  const int P = (int)seed.size();
  std::vector<int32_t> owner(N, -1);
  std::vector<std::deque<int>> frontier(P);
  std::vector<int> size(P, 0);
  for (int p = 0; p < P; p++) frontier[p].push_back(seed[p]);
  using Item = std::pair<int, int>;
  std::priority_queue<Item, std::vector<Item>, std::greater<Item>> heap;
  for (int p = 0; p < P; p++) heap.push({0, p});
  while (!heap.empty()) {
    const int p = heap.top().second;
    heap.pop();
    auto &q = frontier[p];
    while (!q.empty() && owner[q.front()] >= 0) q.pop_front();
    if (q.empty()) continue;
    const int c = q.front();
    q.pop_front();
    owner[c] = p;
    size[p]++;
    for (int s = 0; s < 6; s++) {
      const int j = nbr[(size_t)c * 6 + s];
      if (j >= 0 && owner[j] < 0) q.push_back(j);
    }
    heap.push({size[p], p});
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
  std::vector<int> ring(N, -1);
  std::vector<int> touched;
  std::vector<std::set<int>> peers(P);           // tiles whose owned cells or edges a tile holds, made symmetric
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
    std::unordered_map<int, int> lc;
    lc.reserve(order.size() * 2);
    for (size_t q = 0; q < order.size(); q++) lc[order[q]] = (int)q;
    // edges of the local cells, keyed by (ring of the nearer cell, not owned, id): owned edges first within ring 0
    std::vector<std::tuple<int, int, int>> ev;
    std::unordered_map<int, int> seen;
    seen.reserve(order.size() * 4);
    int eown = 0;
    for (int c : order)
      for (int s = 0; s < 6; s++) {
        const int e = cellEdge[(size_t)c * 6 + s];
        if (e < 0 || seen.count(e)) continue;
        seen[e] = 1;
        const int ra = ring[eI[e]] >= 0 ? ring[eI[e]] : k + 1, rb = ring[eJ[e]] >= 0 ? ring[eJ[e]] : k + 1;
        const int owned = owner[eI[e]] == p ? 0 : 1;
        if (!owned) eown++;
        ev.push_back(std::make_tuple(std::min(ra, rb), owned, e));
      }
    std::sort(ev.begin(), ev.end());
    std::unordered_map<int, int> le;
    le.reserve(ev.size() * 2);
    for (size_t q = 0; q < ev.size(); q++) le[std::get<2>(ev[q])] = (int)q;
    if (order.size() > 32000 || ev.size() > 32000) fail(ISW_EINVAL, "tiles: a tile outgrows 16-bit local ids");
    for (int r = 0; r <= k; r++) {
      t.ncnt.push_back(ring_end[r]);
      int ne = 0;
      while (ne < (int)ev.size() && std::get<0>(ev[ne]) <= r) ne++;
      t.ecnt.push_back(ne);
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
      if (owner[c] != p) { peers[p].insert(owner[c]); peers[owner[c]].insert(p); }
      int slot[6];
      std::pair<int, int> asc[6];
      for (int s = 0; s < 6; s++) {
        const int e = cellEdge[(size_t)c * 6 + s];
        slot[s] = e < 0 ? pad : 2 * le.at(e) + (cellSign[(size_t)c * 6 + s] < 0 ? 1 : 0);
        asc[s] = std::make_pair(e < 0 ? E : e, slot[s]);
      }
      put(t.cedge, slot, c);
      std::sort(asc, asc + 6);
      for (int s = 0; s < 6; s++) slot[s] = asc[s].second;
      put(t.casc, slot, c);
    }
    for (auto &tu : ev) {
      const int e = std::get<2>(tu);
      t.edges.push_back(e);
      const int o = owner[eI[e]];
      if (o != p) { peers[p].insert(o); peers[o].insert(p); }
      auto a = lc.find(eI[e]), b = lc.find(eJ[e]);
      t.eix.push_back(e);
      t.eix.push_back((int32_t)((a == lc.end() ? 0x7fffu : (uint32_t)a->second) | (b == lc.end() ? 0x7fffu : (uint32_t)b->second) << 16));
    }
    t.cell_off.push_back((int32_t)t.cells.size());
    t.edge_off.push_back((int32_t)t.edges.size());
    for (int c : touched) ring[c] = -1;
    touched.clear();
  }
  t.nbr_off.push_back(0);
  for (int p = 0; p < P; p++) {
    t.nbrs.insert(t.nbrs.end(), peers[p].begin(), peers[p].end());
    t.nbr_off.push_back((int32_t)t.nbrs.size());
  }
  return t;
}

}  // namespace isw
