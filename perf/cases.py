"""The work that users of this core have it do, as cases that can be timed and checked.

Each case is one pass through the public entry points (`Layers.step`, `Layers.exchange`, `Transport.mass_after`,
`Transport.step_many`, `dsum`, `Batch.step`), on the grids (levels 4 to 7), layer counts (1 to 8), tracer counts (up to
16) and precision forms that the configurations, the tests and the benchmark of this repository use. Grids and a batch's
tuned layout are made once per process and kept, as a program keeps them; states come from the seed.

`exact` is the same pass in plain torch, 64 bits throughout, written from the equations: whole-array operations on the
grid's tables, none of this repository's kernels.

Time steps are at most half of the stacked workloads' (`isw.cases.stack_dt`), so that a state stays regular over the
thousands of passes that timing takes; the work of a pass does not depend on the step.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'insilica-world-v2_b200'))

from isw import cases as C  # noqa: E402
from isw import gpu  # noqa: E402
from isw import grid as G  # noqa: E402
from isw.batch import Batch  # noqa: E402
from isw.layers import Layers  # noqa: E402
from isw.transport import Transport  # noqa: E402
from isw.workload import fp64_stack_kinds, planet_grid  # noqa: E402

F64 = torch.float64
GRAV = C.GRAV
AIR = dict(cp=1004.6, kappa=287.04 / 1004.6, rd=287.04)
P0 = 1.0e5
FLOOR = 1.0
AIR_FLOOR = 10.0
SHELF = 50.0
CD_BOT = 2.5e-3
BETA = 0.25
DAMP = 0.1
THIN = 2.0
DAY_DRAG = 21600.0


# ---------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------

def listed():
    return [
        # one shallow-water layer on the coarse grid (the analytic single-layer tests): the smallest call there is
        dict(name='shallow-l4', kind='step', level=4, layers=1, tracers=0, nfast=4, form='double'),
        # one layer on the fine grid with the few fast sub-steps that it needs (the barotropic jet's configuration)
        dict(name='jet-l7-mixed', kind='step', level=7, layers=1, tracers=0, nfast=2, form='mixed'),
        # the reference model's own sequence of a tick, call by call: step, masses, transport, the exchange between layers
        # and a tracer's budget
        dict(name='world-l5', kind='world', level=5, layers=3, tracers=3, nfast=20, form='double'),
        # a deeper stack call by call in the mixed form, its tracers moved by the per-call transport
        dict(name='deep-l6-mixed', kind='step', level=6, layers=5, tracers=2, nfast=20, form='mixed'),
        # the benchmark's member (air 3 + ocean 2 layers, 3 tracers each) in one batch, in both forms, and on the fine grid
        dict(name='member-l6', kind='batch', levels='6', tracers=3, nfast=20, form='double'),
        dict(name='member-l6-mixed', kind='batch', levels='6', tracers=3, nfast=20, form='mixed'),
        dict(name='member-l7', kind='batch', levels='7', tracers=3, nfast=20, form='double'),
        # eight members in one batch (the throughput configuration)
        dict(name='batch8-l6-mixed', kind='batch', levels='6,6,6,6,6,6,6,6', tracers=3, nfast=20, form='mixed'),
        # an ensemble of several grid levels, as the forecast server's mix holds
        dict(name='ensemble-mixed', kind='batch', levels='5,5,5,5,6,6,7', tracers=2, nfast=20, form='mixed'),
        # transport alone with many tracers (a chemistry step on a given flow)
        dict(name='tracers-l6', kind='transport', level=6, layers=5, tracers=8, order=3, form='double'),
        # the atmosphere with its own thermodynamics (h = mass per area, potential temperature per layer)
        dict(name='air-l5', kind='air', level=5, layers=3, nfast=12, form='double'),
        # the ocean with its option branches (walls, shelf, per-cell buoyancy, tide, bottom drag) and a tracer
        dict(name='ocean-l6', kind='ocean', level=6, layers=2, tracers=1, nfast=20, form='double'),
    ]


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(['step', 'step', 'world', 'batch', 'batch', 'transport', 'air', 'ocean'])
    form = rng.choice(['double', 'mixed'])
    if kind == 'batch':
        most = 1.2e6                                     # cells x layers of the whole batch, below the largest listed one's
        levels, room = [], most
        for _ in range(rng.randint(1, 7)):
            n = rng.choice([4, 5, 6, 7])
            if 5 * _cells(n) <= room:
                levels.append(n)
                room -= 5 * _cells(n)
        return dict(kind=kind, levels=','.join(str(n) for n in sorted(levels or [4])), tracers=rng.randint(1, 3),
                    nfast=rng.randint(4, 24), form=form)
    level = rng.choice([4, 5, 6, 7])
    top = 8 if level < 7 else 5
    if kind == 'transport':
        L = rng.randint(1, top)
        T = min(rng.randint(1, 16), max(1, int(1.2e7 // (_cells(level) * L))))
        return dict(kind=kind, level=level, layers=L, tracers=T, order=rng.choice([1, 3, 3]), form=form)
    if kind == 'air':
        return dict(kind=kind, level=min(level, 6), layers=rng.randint(2, 6), nfast=rng.randint(6, 24), form='double')
    if kind == 'ocean':
        return dict(kind=kind, level=level, layers=rng.randint(2, 4), tracers=rng.randint(1, 3), nfast=rng.randint(6, 24), form='double')
    if kind == 'world':
        return dict(kind=kind, level=min(level, 6), layers=rng.randint(2, 6), tracers=rng.randint(1, 4), nfast=rng.randint(4, 24),
                    form='double')
    return dict(kind=kind, level=level, layers=rng.randint(1, top), tracers=rng.randint(0, 4 if level < 7 else 2),
                nfast=rng.randint(4, 24), form=form)


# ---------------------------------------------------------------------------------------------------------------------
# grids and inputs
# ---------------------------------------------------------------------------------------------------------------------

def _cells(n):
    return 10 * 4 ** n + 2


@functools.lru_cache(maxsize=None)
def _host_grid(level):
    return planet_grid(G.build(level, device=0 if level >= 5 else 'cpu'))


@functools.lru_cache(maxsize=None)
def _device_grid(level, form):
    before = gpu.PRECISION
    gpu.set_precision(form)
    try:
        return gpu.DeviceGrid(_host_grid(level), device=0)
    finally:
        gpu.set_precision(before)


def _dev():
    return torch.device('cuda', 0)


def _up(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device=_dev())


@functools.lru_cache(maxsize=None)
def _points(level):
    g = _host_grid(level)
    return _up(g.pos), _up(g.xm), _up(g.ne)


def _smooth(level, gen, rows, waves=24):
    """`rows` smooth random fields of about unit RMS at the cells: sums of plane waves of 500 km and longer."""
    pos, _, _ = _points(level)
    k = torch.randn(rows, waves, 3, generator=gen, dtype=F64, device=_dev()) * 6.0
    phase = torch.rand(rows, waves, 1, generator=gen, dtype=F64, device=_dev()) * (2 * math.pi)
    return torch.stack([torch.cos(k[r] @ pos.T + phase[r]).sum(0) for r in range(rows)]) * math.sqrt(2.0 / waves)


def _swirl(level, gen, rows, speed):
    """Normal winds of `rows` solid-body rotations about random axes."""
    _, xm, ne = _points(level)
    axis = torch.randn(rows, 3, generator=gen, dtype=F64, device=_dev())
    axis = axis / axis.norm(dim=1, keepdim=True) * speed
    return torch.stack([(torch.linalg.cross(axis[r].expand_as(xm), xm) * ne).sum(1) for r in range(rows)])


@functools.lru_cache(maxsize=None)
def _climate(level, kind, L):
    """A balanced stack without noise: the benchmark's air (3 layers) and ocean (2) stacks, else L even layers of 10 km
    in all under one 20 m/s jet. Device tensors h, u, b and the stack's constants."""
    g = _host_grid(level)
    if kind in ('air', 'ocean'):
        c = C.STACKS[kind]
        if c.get('flat'):
            b = np.full(g.N, c['base'])
        else:
            b = C.compress_peaks(C.topography(g, 0, device=_dev()), c['knee'], c['cap'])
        h, u = C.balanced_layers(g, c['H'], [C.jet_profile(U) for U in c['U']], c['gprime'], b, c['floor'], C.OMEGA_EARTH)
        par = dict(gprime=list(c['gprime']), stress=list(c['stress']), nu4=C.visc4(g, c['visc4_U']), vmix=c['vmix'], vmix_cd=c['vmix_cd'])
    else:
        b = np.zeros(g.N)
        gp = [1.0 / L] * (L - 1)
        h, u = C.balanced_layers(g, [10000.0 / L] * L, [C.jet_profile(20.0)] * L, gp, b, FLOOR, C.OMEGA_EARTH)
        par = dict(gprime=gp, stress=[0.0] * (L - 1) + [1e-4], nu4=C.visc4(g, 20.0), vmix=5e-4, vmix_cd=1e-3)
        if L == 1:
            par.update(vmix=0.0, vmix_cd=0.0, stress=[0.0])
    return _up(h), _up(u), _up(b), par


def _kind_of(L):
    return {2: 'ocean', 3: 'air'}.get(L, 'even')


def _stack_input(level, kind, L, gen, T):
    h, u, b, par = _climate(level, kind, L)
    N = h.shape[1]
    h = torch.clamp(h * (1 + 0.005 * _smooth(level, gen, L)), min=FLOOR).contiguous()
    rand = lambda: torch.rand(L, N, generator=gen, dtype=F64, device=_dev())
    tracers = []
    for j in range(T):                                   # potential temperature, vapour, gases
        if j == 0:
            tracers.append(250.0 + 60.0 * rand())
        elif j == 1:
            tracers.append(5e-3 * torch.exp(0.5 * torch.randn(L, N, generator=gen, dtype=F64, device=_dev())))
        else:
            tracers.append(rand())
    A = _up(_host_grid(level).areaCell)
    return dict(level=level, L=L, h=h, u=u.clone(), b=b, M=(h * A).contiguous(), tracers=tracers, floor=FLOOR, par=dict(par))


def _inputs(case, seed):
    """The seed's inputs as device tensors, the same for `prepare` and `exact`: a list of stacks (one but for a batch)."""
    gen = torch.Generator(device=_dev())
    gen.manual_seed(int(seed))
    kind = case['kind']
    if kind == 'batch':
        out = []
        for n in (int(x) for x in case['levels'].split(',')):
            for k, L in (('air', 3), ('ocean', 2)):
                s = _stack_input(n, k, L, gen, case['tracers'])
                s.update(kind=k, dt=C.stack_dt(n) / 2, nfast=case['nfast'])
                out.append(s)
        return out
    level, L = case['level'], case['layers']
    g = _host_grid(level)
    if kind in ('step', 'world'):
        s = _stack_input(level, _kind_of(L), L, gen, case['tracers'])
        s.update(dt=C.stack_dt(level) / (2 if level > 5 else 4), nfast=case['nfast'])
        if kind == 'world':
            s['wx'] = (1e-3 * _smooth(level, gen, L - 1)).contiguous()      # metres a tick across each interface
        return [s]
    A = _up(g.areaCell)
    if kind == 'transport':
        s = _stack_input(level, 'even', L, gen, case['tracers'])
        un = _swirl(level, gen, L, 40.0)
        s['Fm'] = (un * _up(g.le) * 2000.0 * (C.stack_dt(level) / 2)).contiguous()
        return [s]
    if kind == 'air':
        share = torch.linspace(1.0, 1.6, L, dtype=F64, device=_dev())
        mu = 101300.0 / GRAV * share / share.sum()
        h = (mu[:, None] * (1 + 0.002 * _smooth(level, gen, L))).contiguous()
        theta = (torch.linspace(395.0, 295.0, L, dtype=F64, device=_dev())[:, None] + 1.0 * _smooth(level, gen, L)).contiguous()
        par = dict(gprime=[0.0] * (L - 1), stress=[0.0] * (L - 1) + [0.0177], nu4=C.visc4(g, 20.0), vmix=5e-3, vmix_cd=0.0)
        return [dict(level=level, L=L, h=h, u=_swirl(level, gen, L, 5.0).contiguous(), theta=theta, b=torch.zeros(g.N, dtype=F64, device=_dev()),
                     M=None, tracers=[], floor=AIR_FLOOR, par=par, dt=C.stack_dt(level) / 4, nfast=case['nfast'])]
    # the ocean with its options: a basin floor with relief that pinches the lower layers out, a continent behind walls
    f = _smooth(level, gen, 4)
    b = -4000.0 + 1200.0 * torch.clamp(f[0], min=0.0)
    H = [100.0] + [3900.0 / (L - 1)] * (L - 1)
    top = torch.zeros_like(b)
    h = []
    for k in range(L):
        bottom = -sum(H[:k + 1]) * torch.ones_like(b) + 5.0 * f[1] if k + 1 < L else b
        bottom = torch.maximum(bottom, b + FLOOR * (L - 1 - k))
        h.append(torch.clamp(top - bottom, min=FLOOR))
        top = top - h[-1]
    h = torch.stack(h).contiguous()
    eI, eJ = (torch.as_tensor(np.asarray(x), dtype=torch.int64, device=_dev()) for x in (g.eI, g.eJ))
    land = f[2] > 0.9
    wall = (~(land[eI] | land[eJ])).to(F64).contiguous()
    sig = torch.stack([torch.zeros_like(b)] + [0.016 / k * (1 + 0.05 * f[3]) for k in range(1, L)]).contiguous()
    par = dict(gprime=[0.016] * (L - 1), stress=[0.0] * (L - 1) + [2.5e-4], nu4=C.visc4(g, 0.5), vmix=5e-4, vmix_cd=1e-3)
    tracers = [torch.rand(L, g.N, generator=gen, dtype=F64, device=_dev()) for _ in range(case['tracers'])]
    return [dict(level=level, L=L, h=h, u=(_swirl(level, gen, L, 0.3) * wall).contiguous(), b=b, M=(h * A).contiguous(), tracers=tracers,
                 floor=FLOOR, par=par, dt=C.stack_dt(level) / 2, nfast=case['nfast'], wall=wall, sig=sig, tide=(0.3 * f[1]).contiguous(),
                 cbot=(1e-4 * torch.rand(g.E, generator=gen, dtype=F64, device=_dev())).contiguous())]


# ---------------------------------------------------------------------------------------------------------------------
# the measured pass
# ---------------------------------------------------------------------------------------------------------------------

_TUNED = {}                                              # a case's batch layout, tuned once and kept by the program


def _objects(case, s, precision=None):
    dg = _device_grid(s['level'], case['form'])
    L, p = s['L'], s['par']
    kw = dict(b=s['b'], gprime=p['gprime'], stress=p['stress'], nu4=p['nu4'], floor=s['floor'], vmix=p['vmix'], vmix_cd=p['vmix_cd'])
    if 'theta' in s:
        kw['air'] = dict(AIR, t_ref=288.0)
    if 'wall' in s:
        kw.update(wall=s['wall'], shelf=SHELF, shelf_bed=True)
    core = Layers(dg, L, precision=precision, **kw)
    if 'sig' in s:
        core.sig, core.zm = s['sig'], torch.zeros_like(s['sig'])
        core.tide, core.cd_bot, core.cbot = s['tide'], CD_BOT, s['cbot']
    T = len(s['tracers'])
    tr = Transport(dg, layers=L, tracers=T, precision=precision) if T else None
    s.update(core=core, tr=tr)
    if 'Fm' not in s:
        s['Fm'] = torch.zeros_like(s['u'])
    if s['M'] is not None:
        s['M1'] = torch.zeros_like(s['M'])
    return s


def prepare(case, seed):
    stacks = _inputs(case, seed)
    if case['kind'] != 'batch':
        return dict(case=case, stack=_objects(case, stacks[0]))
    # members of one level and kind share one allocation, so that their results come back whole
    groups = {}
    for s in stacks:
        groups.setdefault((s['level'], s['kind']), []).append(s)
    out = {}
    for (level, kind), ss in groups.items():
        for name in ('h', 'u', 'M'):
            a = torch.stack([s[name] for s in ss])
            out[f'{kind}{level}.{name}'] = a
            for m, s in enumerate(ss):
                s[name] = a[m]
        a = torch.zeros_like(out[f'{kind}{level}.u'])
        out[f'{kind}{level}.Fm'] = a
        for m, s in enumerate(ss):
            s['Fm'] = a[m]
        for j in range(case['tracers']):
            a = torch.stack([s['tracers'][j] for s in ss])
            out[f'{kind}{level}.tr{j}'] = a
            for m, s in enumerate(ss):
                s['tracers'][j] = a[m]
    batch = Batch(0)
    for s in stacks:
        fp64 = case['form'] == 'mixed' and s['kind'] in fp64_stack_kinds(s['level'])
        _objects(case, s, precision='double' if fp64 else None)
        batch.add(s['core'], s['h'], s['u'], s['Fm'], tr=s['tr'], M=s['M'], M1=s['M1'], tracers=s['tracers'], dt=s['dt'], nfast=s['nfast'])
    key = tuple(sorted((k, v) for k, v in case.items() if k != 'name'))
    if key not in _TUNED:
        _TUNED[key], _ = batch.autotune(steps=5)
    batch.config(**_TUNED[key])
    return dict(case=case, batch=batch, stacks=stacks, out=out)


def _transport(s, order=3):
    s['tr'].mass_after(s['M'], s['Fm'], s['M1'])
    s['tr'].step_many(s['M'], s['M1'], s['Fm'], s['tracers'], order=order)


def run(state):
    case = state['case']
    kind = case['kind']
    if kind == 'batch':
        state['batch'].step()
        return state['out']
    s = state['stack']
    if kind == 'transport':
        _transport(s, case['order'])
        return dict(M1=s['M1'], tracers=s['tracers'])
    if kind == 'air':
        s['core'].step(s['h'], s['u'], s['dt'], s['nfast'], s['Fm'], theta=s['theta'])
        return dict(h=s['h'], u=s['u'], theta=s['theta'], Fm=s['Fm'])
    s['core'].step(s['h'], s['u'], s['dt'], s['nfast'], s['Fm'])
    out = dict(h=s['h'], u=s['u'], Fm=s['Fm'])
    if s['tr'] is not None:
        _transport(s)
        s['M'], s['M1'] = s['M1'], s['M']
        if kind == 'world':
            s['core'].exchange(s['wx'], s['h'], s['u'], s['M'], s['tracers'][0])
            out['budget'] = gpu.dsum(s['tracers'][0], s['M'])
        out.update(M=s['M'], tracers=s['tracers'])
    return out


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how close another implementation comes
# ---------------------------------------------------------------------------------------------------------------------

def _sizes(level):
    N = _cells(level)
    return N, 3 * N - 6, 2 * N - 4


def _grid_bytes(level, step, tr):
    """The grid's tables, read once: index tables 4 bytes, geometry 8."""
    N, E, NV = _sizes(level)
    b = N * (24 + 6 + 8) + E * (8 + 16)                   # cells' edges and signs, areas; edges' cells, l_e, d_e
    if step:
        b += E * (8 + 10 * 12) + NV * (3 * 9 + 16) + N * 48   # vertices of edges, TRiSK rows; vertices; kites
    if tr:
        b += N * 24 + E * (32 + 64)                       # neighbours, the transport's stencil
    return b


def _stack_work(level, L, T, nfast, step=True, air=False):
    N, E, NV = _sizes(level)
    b = f = 0
    if step:
        b += 8 * (2 * L * N + 3 * L * E + N)              # h, u in and out, Fm out, the bottom
        n = sum(max(1, math.ceil(c * nfast)) for c in (1 / 3, 1 / 2, 1.0))
        f += 3 * (L * E * 90 + L * N * 60 + L * NV * 20) + n * (22 * N + 8 * E) * (L if air else 1)
        if air:
            b += 16 * L * N
    if T:
        b += 8 * (2 * L * N + 2 * T * L * N) + (0 if step else 8 * L * E)
        f += T * L * (E * 75 + N * 90)
    return b, f


def work(case):
    kind = case['kind']
    if kind == 'batch':
        levels = [int(x) for x in case['levels'].split(',')]
        b = sum(_grid_bytes(n, True, True) for n in set(levels))
        f = 0
        for n in levels:
            for L in (3, 2):
                x = _stack_work(n, L, case['tracers'], case['nfast'])
                b, f = b + x[0], f + x[1]
        return {'bytes': b, 'flops': f}
    level, L, T = case['level'], case['layers'], case.get('tracers', 0)
    step = kind != 'transport'
    b, f = _stack_work(level, L, T, case.get('nfast', 0), step, kind == 'air')
    if kind == 'transport' and case['order'] == 1:
        f //= 4
    if kind == 'world':
        b += 8 * (L - 1) * _cells(level)
    return {'bytes': b + _grid_bytes(level, step, T > 0), 'flops': f}


def tolerance(case):
    """64-bit passes agree to the rounding of sums and of exp and pow (measured against `exact`: at most 1.2e-14); the
    mixed form's momentum, operators and fluxes are 32 bits (measured: at most 6.9e-8, the layer fluxes)."""
    if case['form'] == 'mixed' and case['kind'] != 'transport':
        return {'rel': 3e-7}
    return {'rel': 1e-13}


# ---------------------------------------------------------------------------------------------------------------------
# the same pass in 64 bits, in plain torch
# ---------------------------------------------------------------------------------------------------------------------

class _Tables:
    """A grid's tables as torch tensors."""

    def __init__(self, g):
        I = lambda a: torch.as_tensor(np.asarray(a).astype(np.int64), device=_dev())
        self.N, self.E, self.NV = g.N, g.E, g.NV
        ce = I(g.cellEdge).reshape(g.N, 6)
        self.ok = (ce >= 0).to(F64)
        self.ce = ce.clamp(min=0)
        self.sign = I(g.cellSign).reshape(g.N, 6).to(F64) * self.ok
        nb = I(g.nbr).reshape(g.N, 6)
        self.nb = torch.where(nb >= 0, nb, torch.arange(g.N, device=_dev())[:, None])
        self.eI, self.eJ, self.v1, self.v2 = I(g.eI), I(g.eJ), I(g.ev1), I(g.ev2)
        self.le, self.de, self.A, self.Av, self.fV = _up(g.le), _up(g.de), _up(g.areaCell), _up(g.areaV), _up(g.fV)
        self.vE, self.vC = I(g.vEdge).reshape(-1, 3), I(g.vCell).reshape(-1, 3)
        self.vS = I(g.vEdgeSign).reshape(-1, 3).to(F64)
        self.kw = _up(g.kite).reshape(-1)[self.vC * 6 + I(g.vSlot).reshape(-1, 3)]
        start = I(g.eoeStart)
        n = start[1:] - start[:-1]
        at = torch.arange(10, device=_dev())[None]
        real = at < n[:, None]
        pos = torch.where(real, start[:-1, None] + at, torch.zeros_like(start[:-1, None]))
        self.row, self.rw = I(g.eoe)[pos], _up(g.w)[pos] * real
        # second derivatives along an edge at each of its ends: cell, other cell, the two cells opposite
        deg, dist = I(g.deg), _up(g.dist).reshape(g.N, 6)
        self.side = []
        for c, k in ((self.eI, I(g.eKi)), (self.eJ, I(g.eKj))):
            m = deg[c]
            six = m == 6
            ka, kb = torch.where(six, (k + 3) % 6, (k + 2) % m), torch.where(six, (k + 3) % 6, (k + 3) % m)
            d1, d2 = dist[c, k], torch.where(six, dist[c, (k + 3) % 6], 0.5 * (dist[c, ka] + dist[c, kb]))
            s = 2 / (d1 + d2) * self.de ** 2 / 12
            self.side.append((c, nb[c, k], nb[c, ka], nb[c, kb], s / d1, s / d2))

    def out(self, f):
        """Each cell's sum of an edge field (rows, E), outward positive."""
        return (self.sign * f[:, self.ce]).sum(-1)

    def edge_sum(self, f):
        return (self.ok * f[:, self.ce]).sum(-1)

    def div(self, u):
        return self.out(self.le * u) / self.A

    def curl(self, u):
        return (self.vS * (self.de * u)[:, self.vE]).sum(-1) / self.Av

    def grad(self, c):
        return (c[..., self.eJ] - c[..., self.eI]) / self.de

    def lap(self, u):
        z = self.curl(u)
        return self.grad(self.div(u)) - (z[:, self.v2] - z[:, self.v1]) / self.le

    def mean(self, c):
        return 0.5 * (c[..., self.eI] + c[..., self.eJ])


@functools.lru_cache(maxsize=None)
def _tables(level):
    return _Tables(_host_grid(level))


def _step64(t, s):
    """One time-split RK3 step of a stack: (h, u, Fm, theta)."""
    h0, u0, dt, L = s['h'], s['u'], s['dt'], s['L']
    par, floor, b = s['par'], s['floor'], s['b']
    air, theta = 'theta' in s, s.get('theta')
    wall = s.get('wall')
    opt = 'sig' in s
    open_ = wall if wall is not None else 1.0
    cp, kap = AIR['cp'], AIR['kappa']
    up = lambda a: torch.flip(torch.cumsum(torch.flip(a, [0]), 0), [0])      # sums from the bottom layer
    eta0 = b + h0.sum(0)
    if opt:                                               # layers squeezed onto the bed
        bed = torch.zeros_like(h0)
        below = torch.zeros_like(h0[0])
        for k in range(L - 1, -1, -1):
            both = (h0[k] < 2 * floor) & (h0[k + 1] < 2 * floor) if k + 1 < L else torch.zeros_like(below, dtype=torch.bool)
            bed[k] = ((below <= (L - 1 - k) * 2 * floor) | both).to(F64)
            below = below + h0[k]
        shelf = SHELF * ((bed[:, t.eI] > 0) | (bed[:, t.eJ] > 0)).to(F64)

    def edge_h(h):
        m = t.mean(h)
        if opt:
            low = torch.minimum(h[:, t.eI], h[:, t.eJ])
            m = torch.where((shelf > 0) & (low < shelf), low, m)
        return m
    he0 = edge_h(h0)
    ub0 = open_ * (he0 * u0).sum(0) / he0.sum(0)
    lap4 = t.lap(t.lap(u0)) if par['nu4'] else torch.zeros_like(u0)
    col = lambda v: torch.as_tensor(v, dtype=F64, device=h0.device)[:, None]
    if air:                                               # the column's stiffness
        p = GRAV * torch.cumsum(h0, 0)
        jump = theta - torch.cat([theta[1:], torch.zeros_like(theta[:1])])
        S = torch.where(jump > 0, jump * GRAV * kap * cp * (p / P0) ** kap / p, torch.zeros_like(p))
    hs, us = h0, u0
    for c in (1 / 3, 1 / 2, 1.0):
        n = max(1, math.ceil(c * s['nfast']))
        cdt, tau = c * dt, c * dt / n
        ke = t.edge_sum(0.25 * t.le * t.de * us ** 2) / t.A
        if air:
            p = GRAV * torch.cumsum(hs, 0)
            pt = torch.cat([torch.zeros_like(p[:1]), p[:-1]])
            x = (p / P0) ** kap
            xt = torch.where(pt > 0, (pt / P0) ** kap, torch.zeros_like(pt))
            pibar = cp * (p * x - pt * xt) / ((kap + 1) * (p - pt))
            mont = [GRAV * b + theta[L - 1] * cp * x[L - 1]]
            for k in range(L - 2, -1, -1):
                mont.insert(0, mont[0] + (theta[k] - theta[k + 1]) * cp * x[k])
            B = torch.stack(mont) - up(S * torch.cumsum(hs, 0)) + ke
        else:
            z = b + up(hs)
            if opt:
                P = torch.cumsum(s['sig'] * hs, 0) - s['sig'] * hs
                B = P + s['sig'] * z + ke - s['tide']
                zm = z - 0.5 * hs
            else:
                B = ke.clone()
                for k in range(1, L):
                    B[k:] += par['gprime'][k - 1] * z[k]
        q = (t.curl(us) + t.fV) / ((t.kw * hs[:, t.vC]).sum(-1) / t.Av)
        qe = 0.5 * (q[:, t.v1] + q[:, t.v2])
        he = edge_h(hs)
        Q = torch.zeros_like(us)
        vt = torch.zeros_like(us)
        for j in range(10):
            r, w = t.row[:, j], t.rw[:, j]
            Q += w * torch.minimum(he[:, r], THIN * he) * us[:, r] * 0.5 * (qe + qe[:, r])
            vt += w * us[:, r]
        sq = 1.0
        if opt:
            fade = torch.clamp((he - 2 * floor) / (shelf - 2 * floor), min=0.0)
            sq = torch.where((shelf > 0) & (he < shelf), fade, torch.ones_like(he))
        T = Q - sq * t.grad(B)
        if opt:
            T = T - (1 - sq) / DAY_DRAG * us
        ck = col(par['stress']).expand(L, t.E).clone()
        if opt:
            ck[L - 1] += CD_BOT * torch.sqrt(us[L - 1] ** 2 + vt[L - 1] ** 2) + s['cbot']
        r = ck / torch.clamp(he, min=floor)
        T = T - torch.where(r * cdt > 1e-8, -torch.expm1(-r * cdt) / cdt, r) * us
        if air:
            T = T + t.mean(pibar) * t.grad(theta)
        if opt:
            T = T + sq * t.mean(zm) * t.grad(s['sig'])
        T = T - par['nu4'] * lap4
        H = he.sum(0)
        force = (he * T).sum(0) / H
        Tp = T - force
        if air:
            mu, uf, acc = h0, u0, torch.zeros_like(u0)
            for _ in range(n):
                new = mu - tau * t.div(he * uf)
                phi = up(S * torch.cumsum(new + DAMP * (new - mu), 0))
                mu = new
                acc = acc + uf
                uf = uf + tau * (-t.grad(phi) + Tp + force)
            F = he * acc / n
        else:
            ubs = (he * us).sum(0) / H
            eta, ub, acc = eta0, ub0, torch.zeros_like(ub0)
            for _ in range(n):
                new = eta - tau * t.div((H * ub)[None])[0]
                acc = acc + ub
                ub = open_ * (ub + tau * (-t.grad(GRAV * (new + DAMP * (new - eta))) + force))
                eta = new
            F = open_ * he * (us - ubs + open_ * acc / n)
        f = F * t.le * cdt                                # the floor limiter
        leaving = t.ok * torch.clamp(t.sign * f[:, t.ce], min=0.0)
        leaving = leaving.sum(-1)
        cap = torch.clamp(h0 - floor, min=0.0) * t.A
        scale = torch.where(leaving > cap, cap / leaving, torch.ones_like(cap))
        F = F * torch.where(F > 0, scale[:, t.eI], scale[:, t.eJ])
        hs = h0 - cdt * t.div(F)
        us = uf if air else open_ * (u0 + cdt * Tp + (ub - ub0))
    h, u, Fm = hs, us, F * t.le * dt
    if (par['vmix'] or par['vmix_cd']) and L > 1:         # the stress between layers
        u = u.clone()
        m = t.mean(h)
        diss = torch.zeros_like(u[0])
        for k in range(L - 1):
            ha, hb = m[k], m[k + 1]
            inv = 1 / ha + 1 / hb
            mid = (ha * u[k] + hb * u[k + 1]) / (ha + hb)
            d0 = u[k] - u[k + 1]
            d1 = d0 * torch.exp(-par['vmix'] * inv * dt) / (1 + par['vmix_cd'] * d0.abs() * inv * dt)
            u[k], u[k + 1] = mid + hb / (ha + hb) * d1, mid - ha / (ha + hb) * d1
            diss = diss + 0.5 * ha * hb / (ha + hb) * (d0 ** 2 - d1 ** 2)
        u = open_ * u
        if air:
            warm = t.edge_sum((0.5 * t.le * t.de * diss)[None])[0] / t.A
            p = GRAV * torch.cumsum(h, 0)
            pt = torch.cat([torch.zeros_like(p[:1]), p[:-1]])
            x, xt = (p / P0) ** kap, torch.where(pt > 0, (pt / P0) ** kap, torch.zeros_like(pt))
            pib = cp * (p * x - pt * xt) / ((kap + 1) * (p - pt))
            theta = theta + warm / (h.sum(0) * pib)
    return h, u, Fm, theta


def _transport64(t, M0, Fm, tracers, order):
    """The masses after the step and each tracer moved by third-order fluxes under Zalesak's limiter (order 1: upwind)."""
    M1 = M0 - t.out(Fm)
    moved = []
    for psi in tracers:
        low = torch.where(Fm >= 0, psi[:, t.eI], psi[:, t.eJ]) * Fm
        td = (M0 * psi - t.out(low)) / M1
        if order == 1:
            moved.append(td)
            continue

        def high(p):
            d = [-(w1 + w2) * p[:, c] + w1 * p[:, j] + 0.5 * w2 * (p[:, o1] + p[:, o2]) for c, j, o1, o2, w1, w2 in t.side]
            return Fm * (t.mean(p) - (d[0] + d[1])) + Fm.abs() * ((d[1] - d[0]) * BETA)
        p = psi
        for frac in (1 / 3, 1 / 2):
            p = (M0 * psi - frac * t.out(high(p))) / (M0 - frac * t.out(Fm))
        A = high(p) - low
        far = t.sign * A[:, t.ce]
        lose, gain = torch.clamp(far, min=0.0).sum(-1), torch.clamp(-far, min=0.0).sum(-1)
        hi, lo = torch.maximum(psi, td), torch.minimum(psi, td)
        top, bot = torch.maximum(hi, hi[:, t.nb].amax(-1)), torch.minimum(lo, lo[:, t.nb].amin(-1))
        zero = torch.zeros_like(td)
        Rp = torch.where(gain > 0, torch.clamp((top - td) * M1 / gain, max=1.0), zero)
        Rm = torch.where(lose > 0, torch.clamp((td - bot) * M1 / lose, max=1.0), zero)
        c = torch.where(A > 0, torch.minimum(Rp[:, t.eJ], Rm[:, t.eI]), torch.minimum(Rp[:, t.eI], Rm[:, t.eJ]))
        moved.append((td * M1 - t.out(c * A)) / M1)
    return M1, moved


def _exchange64(t, wx, h, u, M, psi, floor):
    """Thickness wx moved up across each interface (down where negative), with its tracer and momentum."""
    L = h.shape[0]
    vol = wx * t.A
    load = vol * torch.where(wx > 0, psi[1:], psi[:-1])
    none = torch.zeros_like(vol[:1])
    net = lambda f: torch.cat([f, none]) - torch.cat([none, f])
    M2 = M + net(vol)
    psi2 = (M * psi + net(load)) / M2
    h2 = h + net(vol) / t.A
    v = t.mean(wx)
    thick = [x for x in t.mean(h)]
    mom = [a * b for a, b in zip(thick, u)]

    def move(k, w):                                       # w moved up across interface k, where it is not zero
        d = (w > 0)
        td, md, u0 = torch.where(d, thick[k + 1], thick[k]), torch.where(d, mom[k + 1], mom[k]), torch.where(d, u[k + 1], u[k])
        carried = w * torch.where(td > floor, md / td, u0)
        mom[k], mom[k + 1] = mom[k] + carried, mom[k + 1] - carried
        thick[k], thick[k + 1] = thick[k] + w, thick[k + 1] - w
    for k in range(L - 2, -1, -1):
        move(k, torch.clamp(v[k], min=0.0))
    for k in range(L - 1):
        move(k, torch.clamp(v[k], max=0.0))
    return h2, torch.stack([m / a for m, a in zip(mom, thick)]), M2, psi2


def exact(case, seed):
    stacks = _inputs(case, seed)
    kind = case['kind']
    if kind == 'batch':
        parts = {}
        for s in stacks:
            t = _tables(s['level'])
            h, u, Fm, _ = _step64(t, s)
            M1, moved = _transport64(t, s['M'], Fm, s['tracers'], 3)
            for name, a in [('h', h), ('u', u), ('M', M1), ('Fm', Fm)] + [(f'tr{j}', x) for j, x in enumerate(moved)]:
                parts.setdefault(f"{s['kind']}{s['level']}.{name}", []).append(a)
        return {k: torch.stack(v) for k, v in parts.items()}
    s = stacks[0]
    t = _tables(s['level'])
    if kind == 'transport':
        M1, moved = _transport64(t, s['M'], s['Fm'], s['tracers'], case['order'])
        return dict(M1=M1, tracers=moved)
    h, u, Fm, theta = _step64(t, s)
    if kind == 'air':
        return dict(h=h, u=u, theta=theta, Fm=Fm)
    out = dict(h=h, u=u, Fm=Fm)
    if s['tracers']:
        M1, moved = _transport64(t, s['M'], Fm, s['tracers'], 3)
        if kind == 'world':
            h, u, M1, moved[0] = _exchange64(t, s['wx'], h, u, M1, moved[0], s['floor'])
            out.update(h=h, u=u, budget=float((moved[0] * M1).sum()))
        out.update(M=M1, tracers=moved)
    return out
