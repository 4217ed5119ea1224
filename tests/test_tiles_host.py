"""The host side of the fast loop's tiles (csrc/tiles.cu), built alone and run on the CPU: the partition equals a plain
restatement of its rule, the tiles hold what the kernel indexes, and building them allocates per tile and not per cell or
edge (node containers took two thirds of the first step on a new grid)."""
import heapq
import os
import subprocess
from collections import deque

import numpy as np
import pytest

from conftest import PKG

MAIN = r'''
#include "tiles.cu"
#include <cstdio>
#include <cstdlib>
extern long long g_news;
namespace isw { void fail(int, const std::string &m) { std::fprintf(stderr, "%s\n", m.c_str()); std::exit(3); } }
template <class T> std::vector<T> get(FILE *f, size_t n) { std::vector<T> v(n); if (fread(v.data(), sizeof(T), n, f) != n) std::exit(4); return v; }
template <class T> void put(FILE *f, const std::vector<T> &v) { long long n = v.size(); fwrite(&n, 8, 1, f); for (T x : v) { int y = (int)x; fwrite(&y, 4, 1, f); } }
int main(int, char **a) {
  FILE *f = fopen(a[1], "rb");
  auto h = get<int>(f, 4);
  const int N = h[0], E = h[1], P = h[2], k = h[3];
  auto nbr = get<int>(f, 6 * (size_t)N), ce = get<int>(f, 6 * (size_t)N);
  auto cs = get<signed char>(f, 6 * (size_t)N);
  auto eI = get<int>(f, E), eJ = get<int>(f, E);
  auto owner = isw::partition_cells(N, nbr.data(), P);
  const long long before = g_news;
  auto t = isw::build_tiles(N, E, nbr.data(), ce.data(), (const int8_t *)cs.data(), eI.data(), eJ.data(), owner, P, k);
  const long long news = g_news - before;
  FILE *o = fopen(a[2], "wb");
  put(o, std::vector<int>{(int)news});
  put(o, owner); put(o, t.cell_off); put(o, t.edge_off); put(o, t.cells); put(o, t.edges); put(o, t.ncnt); put(o, t.ecnt);
  put(o, t.eown); put(o, t.cedge); put(o, t.casc); put(o, t.eix); put(o, t.nbr_off); put(o, t.nbrs);
  fclose(o);
  return 0;
}
'''
NEWS = r'''
#include <cstdlib>
#include <new>
long long g_news = 0;
void *operator new(std::size_t n) { g_news++; return std::malloc(n ? n : 1); }
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }
'''
NAMES = ('news owner cell_off edge_off cells edges ncnt ecnt eown cedge casc eix nbr_off nbrs').split()


@pytest.fixture(scope='module')
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp('tiles')
    (d / 'main.cu').write_text(MAIN)
    (d / 'news.cpp').write_text(NEWS)
    nvcc = os.environ.get('NVCC', '/usr/local/cuda/bin/nvcc')
    subprocess.run([nvcc, '-std=c++17', '-O1', '-gencode', 'arch=compute_100a,code=sm_100a', f'-I{PKG / "csrc"}',
                    str(d / 'main.cu'), str(d / 'news.cpp'), '-o', str(d / 'main')], check=True)

    def run(g, P, k):
        with open(d / 'in', 'wb') as f:
            np.array([g.N, g.E, P, k], np.int32).tofile(f)
            for a, dt in ((g.nbr, np.int32), (g.cellEdge, np.int32), (g.cellSign, np.int8), (g.eI, np.int32), (g.eJ, np.int32)):
                np.ascontiguousarray(a, dtype=dt).tofile(f)
        subprocess.run([str(d / 'main'), str(d / 'in'), str(d / 'out')], check=True)
        raw, out, at = (d / 'out').read_bytes(), {}, 0
        for name in NAMES:
            n = int(np.frombuffer(raw, np.int64, 1, at)[0])
            out[name] = np.frombuffer(raw, np.int32, n, at + 8)
            at += 8 + 4 * n
        return out
    return run


def grow(nbr, seeds):
    """The smallest region first (ties: the lower id), one cell at a time, breadth-first within a region."""
    owner, front = [-1] * len(nbr), [deque([s]) for s in seeds]
    heap = [(0, p) for p in range(len(seeds))]
    while heap:
        size, p = heapq.heappop(heap)
        q = front[p]
        while q and owner[q[0]] >= 0:
            q.popleft()
        if not q:
            continue
        c = q.popleft()
        owner[c] = p
        q.extend(j for j in nbr[c] if owner[j] < 0)
        heapq.heappush(heap, (size + 1, p))
    return owner


def within_two(nbr, owner, P):
    worst = 0
    for p in range(P):
        held = {c for c, o in enumerate(owner) if o == p}
        for _ in range(2):
            held |= {j for c in held for j in nbr[c]}
        worst = max(worst, len(held))
    return worst


def partition(nbr, P):
    """Twelve rounds: each region's seed moves to the cell farthest from the region's border (the last one a breadth-first
    walk from all borders reaches); the round whose worst region holds the fewest cells within two rings is kept."""
    N = len(nbr)
    seeds = [(p * N + N // 2) // P for p in range(P)]
    owner = best = grow(nbr, seeds)
    least = within_two(nbr, best, P)
    for _ in range(12):
        queue = [c for c in range(N) if any(owner[j] != owner[c] for j in nbr[c])]
        seen = set(queue)
        for c in queue:
            for j in nbr[c]:
                if j not in seen and owner[j] == owner[c]:
                    seen.add(j)
                    queue.append(j)
        for c in queue:
            seeds[owner[c]] = c
        owner = grow(nbr, seeds)
        w = within_two(nbr, owner, P)
        if w < least:
            least, best = w, owner
    return best


@pytest.mark.parametrize('P,k', [(2, 8), (37, 3), (160, 1)])
def test_tiles_of_a_grid(program, grid4, P, k):
    g = grid4
    nbr = [[int(j) for j in row if j >= 0] for row in g.nbr]
    t = program(g, P, k)
    assert t['owner'].tolist() == partition(nbr, P)
    assert t['news'][0] < 400 * P + 400        # (growing arrays of a tile: far fewer than its cells and edges in all)
    owner, sl = t['owner'], lambda name, off, p: t[name][t[off][p]:t[off][p + 1]]
    peers = [set() for _ in range(P)]
    for p in range(P):
        ring = {int(c): 0 for c in np.flatnonzero(owner == p)}
        layer = list(ring)
        order = sorted(layer)
        counts = [len(order)]
        for r in range(1, k + 1):
            layer = sorted({j for c in layer for j in nbr[c]} - set(ring))
            ring.update((j, r) for j in layer)
            order += layer
            counts.append(len(order))
        assert sl('cells', 'cell_off', p).tolist() == order
        assert t['ncnt'][p * (k + 1):(p + 1) * (k + 1)].tolist() == counts
        near = {}
        for c in order:
            for e in g.cellEdge[c]:
                if e >= 0:
                    a, b = int(g.eI[e]), int(g.eJ[e])
                    near[int(e)] = (min(ring.get(a, k + 1), ring.get(b, k + 1)), owner[a] != p, int(e))
        edges = [e for _, _, e in sorted(near.values())]
        assert sl('edges', 'edge_off', p).tolist() == edges
        assert t['ecnt'][p * (k + 1):(p + 1) * (k + 1)].tolist() == [sum(v[0] <= r for v in near.values()) for r in range(k + 1)]
        assert t['eown'][p] == sum(not v[1] for v in near.values())
        at_c, at_e, ne = {c: i for i, c in enumerate(order)}, {e: i for i, e in enumerate(edges)}, len(edges)
        for table in ('cedge', 'casc'):
            rows = t[table].reshape(-1, 8)[t['cell_off'][p]:t['cell_off'][p + 1]]
            for c, row in zip(order, rows):
                assert row[6] + (row[7] << 16) == c
                es = sorted((int(e), int(s)) for e, s in zip(g.cellEdge[c], g.cellSign[c]) if e >= 0)
                want = [2 * at_e[e] + (s < 0) for e, s in es]
                got = [int(v) for v in row[:6]]
                assert (got if table == 'casc' else sorted(got)) == (want if table == 'casc' else sorted(want)) + [2 * ne] * (6 - len(es))
        eix = t['eix'].reshape(-1, 2)[t['edge_off'][p]:t['edge_off'][p + 1]]
        assert eix[:, 0].tolist() == edges
        v = eix[:, 1].astype(np.uint32)
        assert (v & 0xffff).tolist() == [at_c.get(int(g.eI[e]), 0x7fff) for e in edges]
        assert (v >> 16).tolist() == [at_c.get(int(g.eJ[e]), 0x7fff) for e in edges]
        for o in {int(owner[c]) for c in order} | {int(owner[g.eI[e]]) for e in edges}:
            if o != p:
                peers[p].add(o)
                peers[o].add(p)
    for p in range(P):
        assert sl('nbrs', 'nbr_off', p).tolist() == sorted(peers[p])
