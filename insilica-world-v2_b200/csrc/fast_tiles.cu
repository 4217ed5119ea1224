// The barotropic fast loop of a stage over tiles (tiles.cuh; reference layers.cu:366-388, layers.py:168-175): one block per
// tile, every tile of a launch resident at once (cooperative launch). A kernel per precision form.
//
// A thread keeps the state of its cells and edges (t, t + NT, ...) in registers for the whole stage: eta, ub, the sub-step
// sums of its own cells' edges, the local ids. Shared memory holds the stage's constants (l_e H_e, the force, the metric;
// read by their own thread, conflict-free) and what other threads read: per edge the flux l_e H_e ub, which its two
// cells sum, and per cell Y = Gc (eta + gamma (eta - eta_prev)), which its edges difference. A thread issues the gathers
// of all its items before the arithmetic.
//
// The stage ends here too (phases C and D of the grid-wide path): a tile holds every edge of its own cells, so it forms
// their layer fluxes and its cells' limiter factors from the sums in registers, exchanges the factors once, and writes the
// stage's thicknesses and winds. This takes two launches and the sums' round trip through memory out of every stage.
//
// Tiles exchange owned values through global memory every k sub-steps, double-buffered by round. A tile raises its own
// flag after publishing and waits for its neighbours' flags only; a flag counts rounds and is never reset between
// launches (every tile of a stack raises it as often as the others), so a launch starts from its own flag's value. Two
// buffers suffice: a tile publishes round r + 2 only after its neighbours raised round r + 1, which they do after reading
// round r.
//
// What bounds it: a sub-step is 1.9 us FP64 (1.1 mixed) on tiles of 553 cells, of whose 3,600 cycles some 2,300 move
// shared-memory wavefronts (a third of them bank conflicts of the gathers); an exchange 3 us, staging 7, the stage's end 15.
// Before (constants in shared memory, a grid barrier an exchange, C and D as launches of their own) a level-6 member took
// 0.589 ms FP64 and 0.447 mixed, with this kernel 0.497 and 0.371 (nothing else changed).
//
// The FP64 form's values are the grid-wide passes' bit for bit: a cell sums +-(l_e H_e ub), rounded once per edge, in its
// slot order (rounding is symmetric in sign, and a sum that started from +0 is unchanged by the padded slot's zero); the
// limiter sums in ascending edge order. Compiled with
// -fmad=false; the mixed form's fused multiply-adds are written out.
#include "batch.cuh"
#include "mixed_stage.cuh"
#include "tiles.cuh"

namespace isw {
namespace bt {
namespace {

constexpr int FLAG_STRIDE = TILE_FLAG_STRIDE;

// Raise this tile's flag to `value` (the block's writes before it are visible to whoever reads the flag), then wait until
// every neighbour's reached it. False when a wait ran out, here or in another block.
__device__ __forceinline__ bool tile_exchange(const TileSetDev &T, int p, unsigned *flags, unsigned value, BatchStatus *status,
                                              long long timeout_ns, bool skip) {
  __syncthreads();
  if (threadIdx.x == 0 && !skip) {
    __threadfence();
    cuda::atomic_ref<unsigned, cuda::thread_scope_device>(flags[(size_t)p * FLAG_STRIDE]).store(value, cuda::memory_order_release);
  }
  const int n0 = T.nbr_off[p], n1 = T.nbr_off[p + 1];
  int ok = 1;
  cuda::atomic_ref<int, cuda::thread_scope_device> st(status->code);
  for (int q = n0 + (int)threadIdx.x; q < n1 && ok; q += blockDim.x) {
    cuda::atomic_ref<unsigned, cuda::thread_scope_device> f(flags[(size_t)T.nbrs[q] * FLAG_STRIDE]);
    unsigned it = 0;
    long long t0 = 0;
    while ((int)(f.load(cuda::memory_order_acquire) - value) < 0) {
      ++it;
      if ((it & 63) == 0) {
        if (it == 64) t0 = globaltimer();
        if (st.load(cuda::memory_order_relaxed) == ISW_ETIMEOUT) { ok = 0; break; }
        if (globaltimer() - t0 > timeout_ns) {
          raise_status(status, ISW_ETIMEOUT);
          ok = 0;
          break;
        }
      }
      if (it > (1u << 30)) { ok = 0; break; }
    }
  }
  return __syncthreads_and(ok) != 0;
}

template <class W>
__device__ __forceinline__ unsigned slot_of(const W &w, int q) {
  const unsigned v = q < 2 ? w.x : q < 4 ? w.y : w.z;
  return (q & 1) ? v >> 16 : v & 0xffffu;
}

// A slot's flux, outward positive: the FP64 form keeps one value per edge and flips its sign, the mixed one keeps both.
__device__ __forceinline__ double slot_flux(const double *fl, unsigned v) {
  const double x = fl[v >> 1];
  return __hiloint2double(__double2hiint(x) ^ (int)(v << 31), __double2loint(x));
}
__device__ __forceinline__ float slot_flux(const float *fl, unsigned v) { return fl[v]; }

// Bit 15 of an edge's local cells: a thin wall closes it (tiles have at most 32000 cells).
constexpr unsigned CLOSED = 0x8000u;

// What leaves a cell through its edges in one layer, for the limiter: each edge's value F l_e cdt, rounded as the grid-wide
// pass rounds it, in ascending edge order.
__device__ __forceinline__ double leaving(const double *F, uint4 w, const double lq[6], double cdt, unsigned pad) {
  double out = 0;
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const unsigned v = slot_of(w, q);
    if (v == pad) continue;                                    // a padded slot
    const double x = F[v >> 1] * lq[q] * cdt;
    if (!(v & 1u)) { if (x > 0) out += x; }
    else if (!(x > 0)) out -= x;
  }
  return out;
}

// The divergence of a cell's limited fluxes in one layer.
__device__ __forceinline__ double outflow(const double *F, uint3 w, unsigned pad) {
  double div = 0;
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const unsigned v = slot_of(w, q);
    if (v != pad) div += slot_flux(F, v);
  }
  return div;
}

// The stage's end of a stack whose layers do not fit in shared memory together: phases C and D for d.lg layers at a time, one
// exchange each, with the values of the register forms below. It walks the tile's edges instead of keeping them in registers
// (mean: the edges' mean barotropic wind, in shared memory; their barotropic change in global memory), because state kept in
// registers from group to group spilled. A step of one level-7 stack, grid-wide / groups with state in registers / this:
// 6 mixed layers 1.056 / 1.103 / 0.987 ms, 8 mixed 1.789 / 1.857 / 1.715, 5 FP64 1.302 / 1.383 / 1.301, 8 FP64 1.618 /
// 1.662 / 1.583; four level-6 stacks of 8 layers in one batch 1.595 -> 1.516 FP64, 1.770 -> 1.638 mixed.
template <int NT, bool MIXED, bool WALL>
__device__ __forceinline__ void end_in_groups(const StackDesc &d, int p, int st, unsigned *flags, unsigned turn, BatchStatus *status,
                                              long long timeout_ns, bool skip, const int *eid, const int *cid, double *mean,
                                              const int *cnt) {
  const LayersDev &M = d.M;
  const TileSetDev &T = d.tiles;
  const int t = threadIdx.x, N = M.g.N, E = M.g.E, c0 = T.cell_off[p], e0 = T.edge_off[p];
  const int nown = cnt[0], nc1 = cnt[1], eown = T.eown[p], ering = cnt[FAST_KMAX + 1];
  const unsigned pad = 2u * (T.edge_off[p + 1] - e0);
  const StageArgs a = stage_args(d, st);
  const mixed::MStageArgs am = mixed::mstage_args(d, st);
  double *F = mean + ering, *sc = F + (size_t)d.lg * ering;
  bool finite = true;
  for (int l0 = 0; l0 < d.L; l0 += d.lg) {
    const int L = min(d.lg, d.L - l0);
    if (l0 > 0) __syncthreads();                               // the layers before are done with F and sc
    for (int e = t; e < ering; e += NT) {
      const int2 x = T.eix[e0 + e];
      const double m = mean[e];
      if (MIXED) {
        const double *ha = am.hs + (size_t)l0 * N + cid[x.y & 0xffff], *hb = am.hs + (size_t)l0 * N + cid[(unsigned)x.y >> 16];
        const float *us = am.us + (size_t)l0 * E + x.x, ubs = M.ubs32[x.x];
#pragma unroll 4
        for (int l = 0; l < L; l++)
          F[l * ering + e] = (0.5 * (ha[(size_t)l * N] + hb[(size_t)l * N])) * ((double)(us[(size_t)l * E] - ubs) + m);
      } else {
        const bool closed = WALL && M.wall && M.wall[x.x] == 0;
        const double *he = M.hedge + (size_t)l0 * E + x.x, *us = a.us + (size_t)l0 * E + x.x, ubs = M.ubs[x.x];
#pragma unroll 4
        for (int l = 0; l < L; l++) {
          const double h = he[(size_t)l * E];
          F[l * ering + e] = closed ? 0.0 : h * (us[(size_t)l * E] - ubs) + h * m;
        }
      }
    }
    __syncthreads();
    for (int c = t; c < nown; c += NT) {
      const uint4 w = T.casc[c0 + c];
      double lq[6];
#pragma unroll
      for (int q = 0; q < 6; q++) {
        const unsigned v = slot_of(w, q);
        lq[q] = v == pad ? 0.0 : T.el[e0 + (v >> 1)].x;
      }
      const double ar = T.aarea[c0 + c];
      for (int l = 0; l < L; l++) {
        const size_t o = (size_t)(l0 + l) * N + cid[c];
        const double avail = a.h0[o] - M.floor_, out = leaving(F + l * ering, w, lq, a.cdt, pad);
        const double cap = (avail > 0 ? avail : 0.0) * ar;
        if (MIXED) {
          const float s = out > cap ? __double2float_rz(cap / out) : 1.f;
          sc[l * nc1 + c] = (double)s;
          __stcg(M.scale32 + o, s);
        } else {
          const double s = out > cap ? cap / out : 1.0;
          sc[l * nc1 + c] = s;
          __stcg(M.scale + o, s);
        }
      }
    }
    if (!tile_exchange(T, p, flags, ++turn, status, timeout_ns, skip)) return;
    for (int q = nown + t; q < nc1; q += NT)
      for (int l = 0; l < L; l++) {
        const size_t o = (size_t)(l0 + l) * N + cid[q];
        sc[l * nc1 + q] = MIXED ? (double)__ldcg(M.scale32 + o) : __ldcg(M.scale + o);
      }
    __syncthreads();
    for (int e = t; e < ering; e += NT) {
      const int2 x = T.eix[e0 + e];
      const int i = x.y & 0xffff, j = (unsigned)x.y >> 16;
      const double le = MIXED ? M.g.le[x.x] : T.el[e0 + e].x;
      const bool own = e < eown, closed = !MIXED && WALL && M.wall && M.wall[x.x] == 0;
      const double dub = own && !MIXED ? M.ub[x.x] : 0.0;
      const float dubf = own && MIXED ? M.dub[x.x] : 0.f;
#pragma unroll 4
      for (int l = 0; l < L; l++) {
        const size_t o = (size_t)(l0 + l) * E + x.x;
        double f = F[l * ering + e];
        if (MIXED) {                                           // the FP32 flux and factor, their product in FP64
          const float ff = (float)f;
          f = (double)ff * sc[l * nc1 + (ff > 0.f ? i : j)] * le;
        } else {
          f *= sc[l * nc1 + (f > 0 ? i : j)];
          f = f * le;
        }
        F[l * ering + e] = f;
        if (!own) continue;
        if (!MIXED) {
          if (a.Fm) a.Fm[o] = f * a.dt;
          a.un[o] = closed ? 0.0 : a.u0[o] + a.cdt * M.Tp[o] + dub;
        } else if (am.un) {
          if (am.Fm) am.Fm[o] = f * am.dt;
          am.un[o] = am.u0[o] + __fma_rn(am.cdt, (double)M.Tp32[o], (double)dubf);
        } else {
          am.unf[o] = am.u0f[o] + __fmaf_rn((float)am.cdt, M.Tp32[o], dubf);
        }
      }
    }
    __syncthreads();
    for (int c = t; c < nown; c += NT) {
      const uint4 w = T.cedge[c0 + c];
      const double ar = MIXED ? M.g.rA[cid[c]] : T.aarea[c0 + c];
      for (int l = 0; l < L; l++) {
        const size_t o = (size_t)(l0 + l) * N + cid[c];
        const double h0 = a.h0[o], div = outflow(F + l * ering, make_uint3(w.x, w.y, w.z), pad);
        const double h = MIXED ? __fma_rn(-(a.cdt * div), ar, h0) : h0 - (a.cdt * div) / ar;
        a.hn[o] = h;
        finite = finite && isfinite(h);
      }
    }
  }
  if (st == 2 && !finite && d.check) raise_status(status, ISW_ENOTFINITE);
}

template <int NT, int CAP, bool WALL>
__device__ __forceinline__ void tile_fp64(const StackDesc &d, int p, int st, unsigned *flags, BatchStatus *status,
                                          long long timeout_ns, bool skip, unsigned char *smem, const int *cnt) {
  constexpr int CM = TILE_CAP[CAP].C, EM = TILE_CAP[CAP].E, AM = TILE_CAP[CAP].A;
  const LayersDev &M = d.M;
  const TileSetDev &T = d.tiles;
  const int k = T.k, n = d.n[st], t = threadIdx.x;
  const int c0 = T.cell_off[p], nc = T.cell_off[p + 1] - c0;
  const int e0 = T.edge_off[p], ne = T.edge_off[p + 1] - e0;
  const int nown = cnt[0], eown = T.eown[p], ering = cnt[FAST_KMAX + 1];   // ering: the edges of the own cells
  const double tau = d.tau[st], gam = M.div_damp, grav = M.grav;
  int *eid = reinterpret_cast<int *>(smem), *cid = eid + ne;
  double *area = reinterpret_cast<double *>(smem) + (ne + nc + 1) / 2;
  unsigned char *work = smem + (((size_t)((ne + nc + 1) / 2 + nc) * 8 + 15) & ~(size_t)15);
  double2 *GD = reinterpret_cast<double2 *>(work);            // (G, d_e)
  double *lh = reinterpret_cast<double *>(GD + ne);           // l_e H_e
  double *fl = lh + ne;                                        // ne + 1 (+ 1 to keep the count even)
  double *Y = fl + ne + 2;
  double eta[CM], ub[EM], acc[AM];
  uint3 sl[CM];
  unsigned ij[EM];
  {                                            // the tables, then what they index, then the shared arrays
    int2 x[EM];
    double2 m[EM];
#pragma unroll
    for (int j = 0; j < EM; j++) {
      const int e = t + j * NT;
      x[j] = make_int2(0, 0);
      if (e < ne) {
        x[j] = T.eix[e0 + e];
        m[j] = T.el[e0 + e];
      }
    }
#pragma unroll
    for (int j = 0; j < EM; j++) {
      const int e = t + j * NT;
      if (j < AM) acc[j < AM ? j : 0] = 0.0;
      ub[j] = 0.0;
      ij[j] = (unsigned)x[j].y;
      if (e < ne) {
        const double H = M.He[x[j].x], G = M.G[x[j].x];
        ub[j] = M.ub0[x[j].x];
        eid[e] = x[j].x;
        if (WALL && M.wall && M.wall[x[j].x] == 0) ij[j] |= CLOSED;
        const double l = m[j].x * H;
        GD[e] = make_double2(G, m[j].y);
        lh[e] = l;
        fl[e] = l * ub[j];
      }
    }
  }
#pragma unroll
  for (int j = 0; j < CM; j++) {
    const int c = t + j * NT;
    eta[j] = 0.0;
    sl[j] = make_uint3(0u, 0u, 0u);
    if (c < nc) {
      const uint4 w = T.cedge[c0 + c];
      sl[j] = make_uint3(w.x, w.y, w.z);
      cid[c] = (int)w.w;
      eta[j] = M.eta0[w.w];
      area[c] = T.aarea[c0 + c];
    }
  }
  if (t == 0) fl[ne] = 0.0;                                    // the padded slots' flux
  unsigned turn = flags[(size_t)p * FLAG_STRIDE];
  for (int r = 0, done = 0; done < n; r++, done += k) {
    const int K = min(k, n - done);
    if (r > 0) {
      if (!tile_exchange(T, p, flags, ++turn, status, timeout_ns, skip)) return;
      const double *xe = (r & 1) ? M.eta : M.eta_prev;        // what round r - 1 published
      const double *xu = (r & 1) ? M.ub2 : M.cw;
#pragma unroll
      for (int j = 0; j < EM; j++) {
        const int e = t + j * NT;
        if (e >= eown && e < ne) ub[j] = __ldcg(xu + eid[e]);
      }
#pragma unroll
      for (int j = 0; j < CM; j++) {
        const int c = t + j * NT;
        if (c >= nown && c < nc) eta[j] = __ldcg(xe + cid[c]);
      }
#pragma unroll
      for (int j = 0; j < EM; j++) {
        const int e = t + j * NT;
        if (e >= eown && e < ne) fl[e] = lh[e] * ub[j];
      }
    }
    __syncthreads();
    for (int m = 1; m <= K; m++) {
      const int cn = cnt[K - m + 1];
#pragma unroll
      for (int j = 0; j < CM; j++) {
        const int c = t + j * NT;
        if (c < cn) {
          double f[6];
#pragma unroll
          for (int q = 0; q < 6; q++) f[q] = slot_flux(fl, slot_of(sl[j], q));
          double div = 0;
#pragma unroll
          for (int q = 0; q < 6; q++) div += f[q];
          const double e0v = eta[j], en = e0v - (tau * div) / area[c];
          eta[j] = en;
          Y[c] = grav * (en + gam * (en - e0v));
        }
      }
      __syncthreads();
      const int en = cnt[FAST_KMAX + 1 + K - m];
      double dy[EM];
#pragma unroll
      for (int j = 0; j < EM; j++) {
        dy[j] = 0.0;
        if (t + j * NT < en) dy[j] = -(Y[ij[j] >> 16] - Y[ij[j] & 0x7fffu]);
      }
#pragma unroll
      for (int j = 0; j < EM; j++) {
        const int e = t + j * NT;
        if (e < en) {
          const double v = ub[j];
          const double2 gd = GD[e];
          if (j < AM && e < ering) acc[j < AM ? j : 0] += v;
          double nv = v + tau * (dy[j] / gd.y + gd.x);
          if (WALL && (ij[j] & CLOSED)) nv = 0.0;              // walls (its wind starts from zero, so its sum is zero too)
          ub[j] = nv;
          fl[e] = lh[e] * nv;
        }
      }
      __syncthreads();
    }
    if (done + K < n) {                        // publish the owned values for the neighbours' next round
      double *xe = (r & 1) ? M.eta_prev : M.eta;
      double *xu = (r & 1) ? M.cw : M.ub2;
#pragma unroll
      for (int j = 0; j < CM; j++) {
        const int c = t + j * NT;
        if (c < nown) __stcg(xe + cid[c], eta[j]);
      }
#pragma unroll
      for (int j = 0; j < AM; j++) {
        const int e = t + j * NT;
        if (e < eown) __stcg(xu + eid[e], ub[j]);
      }
    }
  }
  if (TILE_CAP[CAP].groups) {
    double *mean = reinterpret_cast<double *>(work);
#pragma unroll
    for (int j = 0; j < AM; j++) {
      const int e = t + j * NT;
      if (e < ering) mean[e] = acc[j] * d.inv_n[st];
      if (e < eown) M.ub[eid[e]] = ub[j] - M.ub0[eid[e]];
    }
    end_in_groups<NT, false, WALL>(d, p, st, flags, turn, status, timeout_ns, skip, eid, cid, mean, cnt);
    return;
  }
  // ---- phase C: the layer fluxes of the own cells' edges and the limiter factors of the own cells ----
  const StageArgs a = stage_args(d, st);
  const int L = d.L, N = M.g.N, E = M.g.E, nc1 = cnt[1];
  double *F = reinterpret_cast<double *>(work), *sc = F + (size_t)L * ering;   // every layer's, where the fast loop's arrays lay
  double le[AM];
  {
    double ubs[AM];
#pragma unroll
    for (int j = 0; j < AM; j++) {
      const int e = t + j * NT;
      acc[j] *= a.inv_n;
      if (e < ering) {
        ubs[j] = M.ubs[eid[e]];
        le[j] = T.el[e0 + e].x;
      }
    }
    for (int l = 0; l < L; l++) {
      double he[AM], us[AM];
#pragma unroll
      for (int j = 0; j < AM; j++) {
        const int e = t + j * NT;
        if (e < ering) {
          const size_t o = (size_t)l * E + eid[e];
          he[j] = M.hedge[o];
          us[j] = a.us[o];
        }
      }
#pragma unroll
      for (int j = 0; j < AM; j++)
        if (t + j * NT < ering) F[l * ering + t + j * NT] = WALL && (ij[j] & CLOSED) ? 0.0 : he[j] * (us[j] - ubs[j]) + he[j] * acc[j];
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < CM; j++) {
    const int c = t + j * NT;
    if (c < nown) {
      const uint4 w = T.casc[c0 + c];
      double lq[6];
#pragma unroll
      for (int q = 0; q < 6; q++) {
        const unsigned v = slot_of(w, q);
        lq[q] = v == 2u * ne ? 0.0 : T.el[e0 + (v >> 1)].x;
      }
      const double ar = area[c];
      for (int l = 0; l < L; l++) {
        const size_t o = (size_t)l * N + cid[c];
        const double avail = a.h0[o] - M.floor_;
        const double out = leaving(F + l * ering, w, lq, a.cdt, 2u * ne);
        const double cap = (avail > 0 ? avail : 0.0) * ar;
        const double s = out > cap ? cap / out : 1.0;
        sc[l * nc1 + c] = s;
        __stcg(M.scale + o, s);
      }
    }
  }
  if (!tile_exchange(T, p, flags, ++turn, status, timeout_ns, skip)) return;
  // ---- phase D: the limited fluxes, the own cells' thicknesses, the owned edges' winds ----
  for (int q = nown + t; q < nc1; q += NT)
    for (int l = 0; l < L; l++) sc[l * nc1 + q] = __ldcg(M.scale + (size_t)l * N + cid[q]);
  __syncthreads();
  double dub[AM];
#pragma unroll
  for (int j = 0; j < AM; j++)
    if (t + j * NT < eown) dub[j] = ub[j] - M.ub0[eid[t + j * NT]];
  for (int l = 0; l < L; l++) {
    double u0[AM], tp[AM];
#pragma unroll
    for (int j = 0; j < AM; j++)
      if (t + j * NT < eown) {
        const size_t o = (size_t)l * E + eid[t + j * NT];
        u0[j] = a.u0[o];
        tp[j] = M.Tp[o];
      }
#pragma unroll
    for (int j = 0; j < AM; j++) {
      const int e = t + j * NT;
      if (e < ering) {
        double f = F[l * ering + e];
        f *= sc[l * nc1 + (f > 0 ? ij[j] & 0x7fffu : ij[j] >> 16)];
        const double x = f * le[j];
        F[l * ering + e] = x;
        if (e < eown) {
          const size_t o = (size_t)l * E + eid[e];
          if (a.Fm) a.Fm[o] = x * a.dt;
          a.un[o] = WALL && (ij[j] & CLOSED) ? 0.0 : u0[j] + a.cdt * tp[j] + dub[j];
        }
      }
    }
  }
  __syncthreads();
  bool finite = true;
#pragma unroll
  for (int j = 0; j < CM; j++) {
    const int c = t + j * NT;
    if (c < nown) {
      for (int l = 0; l < L; l++) {
        const size_t o = (size_t)l * N + cid[c];
        const double h0 = a.h0[o];
        const double div = outflow(F + l * ering, sl[j], 2u * ne);
        const double h = h0 - (a.cdt * div) / area[c];
        a.hn[o] = h;
        finite = finite && isfinite(h);
      }
    }
  }
  if (st == 2 && !finite && d.check) raise_status(status, ISW_ENOTFINITE);
}

// The mixed form: deviations deta = eta - eta0 and dub = ub - ub0 from zero in FP32, ub0's divergence c0 formed once per
// cell, the edges' sums of dub in FP64; the layer fluxes, thicknesses and final winds in FP64.
template <int NT, int CAP>
__device__ __forceinline__ void tile_mixed(const StackDesc &d, int p, int st, unsigned *flags, BatchStatus *status,
                                           long long timeout_ns, bool skip, unsigned char *smem, const int *cnt) {
  constexpr int CM = TILE_CAP[CAP].C, EM = TILE_CAP[CAP].E, AM = TILE_CAP[CAP].A;
  const LayersDev &M = d.M;
  const TileSetDev &T = d.tiles;
  const int k = T.k, n = d.n[st], t = threadIdx.x;
  const int c0 = T.cell_off[p], nc = T.cell_off[p + 1] - c0;
  const int e0 = T.edge_off[p], ne = T.edge_off[p + 1] - e0;
  const int nown = cnt[0], eown = T.eown[p], ering = cnt[FAST_KMAX + 1];
  const float tau = (float)d.tau[st], gam = (float)M.div_damp, grav = (float)M.grav;
  int *eid = reinterpret_cast<int *>(smem), *cid = eid + ne;
  unsigned char *work = smem + (((size_t)((ne + nc + 1) / 2) * 8 + 15) & ~(size_t)15);
  float2 *pair = reinterpret_cast<float2 *>(work);             // (flux, -flux), ne + 1 of them
  const float *fl = reinterpret_cast<const float *>(pair);
  float2 *GD = pair + ne + 1;                                  // (G, 1 / d_e)
  float *Y = reinterpret_cast<float *>(GD + ne);
  float deta[CM], rA[CM], cz[CM], lh[EM], dub[EM];
  double acc[AM];
  uint3 sl[CM];
  unsigned ij[EM];
  {                                            // the tables, then what they index, then the shared arrays
    int2 x[EM];
    float2 m[EM];
#pragma unroll
    for (int j = 0; j < EM; j++) {
      const int e = t + j * NT;
      x[j] = make_int2(0, 0);
      if (e < ne) {
        x[j] = T.eix[e0 + e];
        m[j] = T.el32[e0 + e];
      }
    }
#pragma unroll
    for (int j = 0; j < EM; j++) {
      const int e = t + j * NT;
      if (j < AM) acc[j < AM ? j : 0] = 0.0;
      lh[j] = dub[j] = 0.f;
      ij[j] = (unsigned)x[j].y;
      if (e < ne) {
        const float H = M.He32[x[j].x], G = M.G32[x[j].x], u0 = (float)M.ub0[x[j].x];
        eid[e] = x[j].x;
        lh[j] = m[j].x * H;
        GD[e] = make_float2(G, m[j].y);
        const float f = lh[j] * u0;                            // ub0's flux for c0, then zero
        pair[e] = make_float2(f, -f);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < CM; j++) {
    const int c = t + j * NT;
    deta[j] = rA[j] = cz[j] = 0.f;
    sl[j] = make_uint3(0u, 0u, 0u);
    if (c < nc) {
      const uint4 w = T.cedge[c0 + c];
      sl[j] = make_uint3(w.x, w.y, w.z);
      cid[c] = (int)w.w;
      rA[j] = T.arA32[c0 + c];
    }
  }
  if (t == 0) pair[ne] = make_float2(0.f, 0.f);                // the padded slots' flux
  __syncthreads();
#pragma unroll
  for (int j = 0; j < CM; j++) {
    if (t + j * NT < nc) {
#pragma unroll
      for (int q = 0; q < 6; q++) cz[j] += slot_flux(fl, slot_of(sl[j], q));
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < EM; j++)
    if (t + j * NT < ne) pair[t + j * NT] = make_float2(0.f, 0.f);
  unsigned turn = flags[(size_t)p * FLAG_STRIDE];
  for (int r = 0, done = 0; done < n; r++, done += k) {
    const int K = min(k, n - done);
    if (r > 0) {
      if (!tile_exchange(T, p, flags, ++turn, status, timeout_ns, skip)) return;
      const float *xe = M.xeta[(r - 1) & 1];
      const float *xu = M.xdub[(r - 1) & 1];
#pragma unroll
      for (int j = 0; j < EM; j++) {
        const int e = t + j * NT;
        if (e >= eown && e < ne) dub[j] = __ldcg(xu + eid[e]);
      }
#pragma unroll
      for (int j = 0; j < CM; j++) {
        const int c = t + j * NT;
        if (c >= nown && c < nc) deta[j] = __ldcg(xe + cid[c]);
      }
#pragma unroll
      for (int j = 0; j < EM; j++) {
        const int e = t + j * NT;
        const float f = lh[j] * dub[j];
        if (e >= eown && e < ne) pair[e] = make_float2(f, -f);
      }
    }
    __syncthreads();
    for (int m = 1; m <= K; m++) {
      const int cn = cnt[K - m + 1];
      float f[CM][6];
#pragma unroll
      for (int j = 0; j < CM; j++) {
#pragma unroll
        for (int q = 0; q < 6; q++) f[j][q] = 0.f;
        if (t + j * NT < cn) {
#pragma unroll
          for (int q = 0; q < 6; q++) f[j][q] = slot_flux(fl, slot_of(sl[j], q));
        }
      }
#pragma unroll
      for (int j = 0; j < CM; j++) {
        const int c = t + j * NT;
        if (c < cn) {
          float div = cz[j];
#pragma unroll
          for (int q = 0; q < 6; q++) div += f[j][q];
          const float d0 = deta[j], dn = mixed::bt_eta_new(d0, tau, div * rA[j]);
          deta[j] = dn;
          Y[c] = mixed::bt_y_new(grav, gam, dn, d0);
        }
      }
      __syncthreads();
      const int en = cnt[FAST_KMAX + 1 + K - m];
      float yi[EM], yj[EM];
#pragma unroll
      for (int j = 0; j < EM; j++) {
        yi[j] = yj[j] = 0.f;
        if (t + j * NT < en) {
          yi[j] = Y[ij[j] & 0xffffu];
          yj[j] = Y[ij[j] >> 16];
        }
      }
#pragma unroll
      for (int j = 0; j < EM; j++) {
        const int e = t + j * NT;
        if (e < en) {
          const float v = dub[j];
          const float2 gd = GD[e];
          if (j < AM && e < ering) acc[j < AM ? j : 0] += (double)v;
          const float nv = mixed::bt_u_new(v, tau, gd.x, yi[j], yj[j], gd.y);
          dub[j] = nv;
          const float fn = lh[j] * nv;
          pair[e] = make_float2(fn, -fn);
        }
      }
      __syncthreads();
    }
    if (done + K < n) {
      float *xe = M.xeta[r & 1];
      float *xu = M.xdub[r & 1];
#pragma unroll
      for (int j = 0; j < CM; j++) {
        const int c = t + j * NT;
        if (c < nown) __stcg(xe + cid[c], deta[j]);
      }
#pragma unroll
      for (int j = 0; j < AM; j++) {
        const int e = t + j * NT;
        if (e < eown) __stcg(xu + eid[e], dub[j]);
      }
    }
  }
  if (TILE_CAP[CAP].groups) {
    double *mean = reinterpret_cast<double *>(work);
#pragma unroll
    for (int j = 0; j < AM; j++) {
      const int e = t + j * NT;
      if (e < ering) mean[e] = __fma_rn(acc[j], d.inv_n[st], M.ub0[eid[e]]);
      if (e < eown) M.dub[eid[e]] = dub[j];
    }
    end_in_groups<NT, true, false>(d, p, st, flags, turn, status, timeout_ns, skip, eid, cid, mean, cnt);
    return;
  }
  // ---- phase C ----
  const mixed::MStageArgs a = mixed::mstage_args(d, st);
  const int L = d.L, N = M.g.N, E = M.g.E, nc1 = cnt[1];
  double *F = reinterpret_cast<double *>(work), *sc = F + (size_t)L * ering;
  double le[AM];
  {
    float ubs[AM];
#pragma unroll
    for (int j = 0; j < AM; j++) {
      const int e = t + j * NT;
      if (e < ering) {
        const int ge = eid[e];
        acc[j] = __fma_rn(acc[j], a.inv_n, M.ub0[ge]);         // the mean barotropic wind
        ubs[j] = M.ubs32[ge];
        le[j] = M.g.le[ge];
      }
    }
    for (int l = 0; l < L; l++) {
      double ha[AM], hb[AM];
      float us[AM];
#pragma unroll
      for (int j = 0; j < AM; j++) {
        const int e = t + j * NT;
        if (e < ering) {
          ha[j] = a.hs[(size_t)l * N + cid[ij[j] & 0xffffu]];
          hb[j] = a.hs[(size_t)l * N + cid[ij[j] >> 16]];
          us[j] = a.us[(size_t)l * E + eid[e]];
        }
      }
#pragma unroll
      for (int j = 0; j < AM; j++)
        if (t + j * NT < ering) F[l * ering + t + j * NT] = (0.5 * (ha[j] + hb[j])) * ((double)(us[j] - ubs[j]) + acc[j]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < CM; j++) {
    const int c = t + j * NT;
    if (c < nown) {
      const uint4 w = T.casc[c0 + c];
      double lq[6];
#pragma unroll
      for (int q = 0; q < 6; q++) {
        const unsigned v = slot_of(w, q);
        lq[q] = v == 2u * ne ? 0.0 : T.el[e0 + (v >> 1)].x;
      }
      const double ar = T.aarea[c0 + c];
      for (int l = 0; l < L; l++) {
        const size_t o = (size_t)l * N + cid[c];
        const double avail = a.h0[o] - M.floor_;
        const double out = leaving(F + l * ering, w, lq, a.cdt, 2u * ne);
        const double cap = (avail > 0 ? avail : 0.0) * ar;
        const float s = out > cap ? __double2float_rz(cap / out) : 1.f;   // rounded toward zero
        sc[l * nc1 + c] = (double)s;
        __stcg(M.scale32 + o, s);
      }
    }
  }
  if (!tile_exchange(T, p, flags, ++turn, status, timeout_ns, skip)) return;
  // ---- phase D: each edge's limited flux is one value, used by both cells and by Fm ----
  for (int q = nown + t; q < nc1; q += NT)
    for (int l = 0; l < L; l++) sc[l * nc1 + q] = (double)__ldcg(M.scale32 + (size_t)l * N + cid[q]);
  __syncthreads();
  for (int l = 0; l < L; l++) {
    double u0[AM];
    float u0f[AM], tp[AM];
#pragma unroll
    for (int j = 0; j < AM; j++)
      if (t + j * NT < eown) {
        const size_t o = (size_t)l * E + eid[t + j * NT];
        if (a.un) u0[j] = a.u0[o];
        else u0f[j] = a.u0f[o];
        tp[j] = M.Tp32[o];
      }
#pragma unroll
    for (int j = 0; j < AM; j++) {
      const int e = t + j * NT;
      if (e < ering) {
        const float f = (float)F[l * ering + e];               // the FP32 flux and factor, their product in FP64
        const double x = (double)f * sc[l * nc1 + (f > 0.f ? ij[j] & 0xffffu : ij[j] >> 16)] * le[j];
        F[l * ering + e] = x;
        if (e < eown) {
          const size_t o = (size_t)l * E + eid[e];
          if (a.un) {
            if (a.Fm) a.Fm[o] = x * a.dt;
            a.un[o] = u0[j] + __fma_rn(a.cdt, (double)tp[j], (double)dub[j]);
          } else {
            a.unf[o] = u0f[j] + __fmaf_rn((float)a.cdt, tp[j], dub[j]);
          }
        }
      }
    }
  }
  __syncthreads();
  bool finite = true;
#pragma unroll
  for (int j = 0; j < CM; j++) {
    const int c = t + j * NT;
    if (c < nown) {
      const double rAd = M.g.rA[cid[c]];
      for (int l = 0; l < L; l++) {
        const size_t o = (size_t)l * N + cid[c];
        const double h0 = a.h0[o];
        const double div = outflow(F + l * ering, sl[j], 2u * ne);
        const double h = __fma_rn(-(a.cdt * div), rAd, h0);
        a.hn[o] = h;
        finite = finite && isfinite(h);
      }
    }
  }
  if (st == 2 && !finite) raise_status(status, ISW_ENOTFINITE);
}

// FORM: 0 FP64, 1 mixed, 2 FP64 with thin walls.
template <int NT, int CAP, int FORM>
__global__ void __launch_bounds__(NT, TILE_NT1 / NT) k_fast_tiles(const StackDesc *__restrict__ S, const TileRef *__restrict__ refs,
                                                              int st, unsigned *flags, BatchStatus *status, long long timeout_ns,
                                                              int fault_block) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int cnt[2 * (FAST_KMAX + 1)];     // the tile's prefix counts: cells of ring <= r, then edges
  const TileRef tr = refs[blockIdx.x];
  const StackDesc &d = S[tr.s];
  const TileSetDev &T = d.tiles;
  if ((int)threadIdx.x <= T.k) {
    cnt[threadIdx.x] = T.ncnt[(size_t)tr.p * (T.k + 1) + threadIdx.x];
    cnt[FAST_KMAX + 1 + threadIdx.x] = T.ecnt[(size_t)tr.p * (T.k + 1) + threadIdx.x];
  }
  __syncthreads();
  const bool skip = (int)blockIdx.x == fault_block;
  unsigned *own = flags + (size_t)d.tile_base * FLAG_STRIDE;
  if (FORM == 1) tile_mixed<NT, CAP>(d, tr.p, st, own, status, timeout_ns, skip, smem, cnt);
  else tile_fp64<NT, CAP, FORM == 2>(d, tr.p, st, own, status, timeout_ns, skip, smem, cnt);
}

using Kernel = void (*)(const StackDesc *, const TileRef *, int, unsigned *, BatchStatus *, long long, int);

template <int NT, int CAP>
Kernel kernel_for(int form) {
  return form == 0 ? k_fast_tiles<NT, CAP, 0> : form == 1 ? k_fast_tiles<NT, CAP, 1> : k_fast_tiles<NT, CAP, 2>;
}

Kernel kernel_for(int bps, int cap, int form) {
  if (bps == 2) return cap == 0 ? kernel_for<TILE_NT2, 0>(form) : cap == 1 ? kernel_for<TILE_NT2, 1>(form) : kernel_for<TILE_NT2, 2>(form);
  return cap == 0 ? kernel_for<TILE_NT1, 0>(form) : cap == 1 ? kernel_for<TILE_NT1, 1>(form) : kernel_for<TILE_NT1, 2>(form);
}

}  // namespace

const void *fast_tiles_kernel(int bps, int cap, int form) { return (const void *)kernel_for(bps, cap, form); }

int fast_tiles_threads(int bps) { return bps == 2 ? TILE_NT2 : TILE_NT1; }

void launch_fast_tiles(int bps, int cap, int form, const cudaLaunchConfig_t &cfg, const StackDesc *desc, const TileRef *refs, int stage,
                       unsigned *flags, BatchStatus *status, long long timeout_ns, int fault_block) {
  ISW_CUDA(cudaLaunchKernelEx(&cfg, kernel_for(bps, cap, form), desc, refs, stage, flags, status, timeout_ns, fault_block));
}

}  // namespace bt
}  // namespace isw
