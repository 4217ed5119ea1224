"""Layer and tracer counts the golden cases do not reach (1, 5 and 8 layers; 1 to 16 tracers), against the oracle
(oracle/model.py over the C restatement), bit for bit: the FCT fields are stored with an item's layers side by side,
padded to an even count, so odd counts and the largest count take their own load and store paths. No stress terms,
so no exp() enters and the FP64 form must match exactly.
  - Transport.step_many call by call, orders 1 and 3
  - the batched step (dynamics, receiving masses and FCT of every stack in one graph) at 5 and 8 layers, tiled and
    grid-wide
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def dev():
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    return torch.device('cuda:0')


def _T(a, dev):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)


def _masses_and_fluxes(grid, L, seed):
    """Layer masses of ~300 m layers and a random edge flux small enough that no cell empties."""
    rng = np.random.default_rng(seed)
    h = 300.0 + 20.0 * rng.random((L, grid.N))
    M0 = h * np.asarray(grid.areaCell)[None]
    Fm = 2e-3 * float(M0.min()) * (rng.random((L, grid.E)) - 0.5)
    return M0, Fm


@pytest.mark.parametrize('L,ntr', [(1, 16), (5, 3), (8, 2)])
@pytest.mark.parametrize('order', [1, 3])
def test_transport_layer_counts(dev, grid4, oracle_lib, L, ntr, order):
    from isw import gpu, transport
    gpu.set_precision('double')
    O = oracle_lib
    dg, og = gpu.DeviceGrid(grid4), O.OracleGrid(grid4)
    tr, otr = transport.Transport(dg, layers=L, tracers=ntr), O.Transport(og, layers=L, tracers=ntr)
    M0, Fm = _masses_and_fluxes(grid4, L, 10 * L + ntr)
    rng = np.random.default_rng(L * 100 + ntr)
    psi = [rng.random((L, grid4.N)) + 0.5 * k for k in range(ntr)]
    gM, gM1, gF = _T(M0, dev), torch.zeros(L, grid4.N, dtype=torch.float64, device=dev), _T(Fm, dev)
    gpsi = [_T(p, dev) for p in psi]
    oM, oM1 = M0.copy(), np.zeros_like(M0)
    for _ in range(3):
        tr.mass_after(gM, gF, gM1)
        tr.step_many(gM, gM1, gF, gpsi, order=order)
        gM, gM1 = gM1, gM
        otr.mass_after(oM, Fm, oM1)
        otr.step_many(oM, oM1, Fm, psi, order=order)
        oM, oM1 = oM1, oM
    torch.cuda.synchronize()
    assert np.array_equal(gM.cpu().numpy(), oM)
    for k in range(ntr):
        assert np.array_equal(gpsi[k].cpu().numpy(), psi[k]), k


@pytest.mark.parametrize('L', [5, 8])
@pytest.mark.parametrize('tiles', [True, False])
def test_batched_step_layer_counts(dev, grid4, oracle_lib, L, tiles):
    """One stack of L layers with 2 tracers, 3 batched steps (nabla^4, drag, 4 fast sub-steps per stage) against the
    oracle's Layers.step + mass_after + step_many, bit for bit in h, u, Fm, M and the tracers."""
    from isw import gpu, transport
    from isw.batch import Batch
    from isw.layers import Layers
    gpu.set_precision('double')
    O = oracle_lib
    dg, og = gpu.DeviceGrid(grid4), O.OracleGrid(grid4)
    rng = np.random.default_rng(L)
    N, E = grid4.N, grid4.E
    h0 = 300.0 + 10.0 * rng.random((L, N))
    b = -300.0 * L + 50.0 * rng.random(N)
    u0 = 0.5 * (rng.random((L, E)) - 0.5)
    psi = [rng.random((L, N)), 1.0 + rng.random((L, N))]
    kw = dict(b=b, gprime=[0.05] * (L - 1), drag=1e-6, nu4=1e14)
    dt, nfast = 900.0, 4
    core, tr = Layers(dg, L, **kw), transport.Transport(dg, layers=L, tracers=2)
    oc, otr = O.Layers(og, L, **kw), O.Transport(og, layers=L, tracers=2)
    h, u, Fm = _T(h0, dev), _T(u0, dev), torch.zeros(L, E, dtype=torch.float64, device=dev)
    M = _T(h0 * np.asarray(grid4.areaCell)[None], dev)
    M1 = torch.zeros_like(M)
    gpsi = [_T(p, dev) for p in psi]
    batch = Batch(0)
    batch.config(tiles=tiles)
    batch.add(core, h, u, Fm, tr=tr, M=M, M1=M1, tracers=gpsi, dt=dt, nfast=nfast)
    oh, ou, oF = h0.copy(), u0.copy(), np.zeros((L, E))
    oM, oM1 = h0 * np.asarray(grid4.areaCell)[None], np.zeros((L, N))
    for _ in range(3):
        batch.step()
        oc.step(oh, ou, dt, nfast, oF)
        otr.mass_after(oM, oF, oM1)
        otr.step_many(oM, oM1, oF, psi)
        oM, oM1 = oM1, oM
    torch.cuda.synchronize()
    assert batch.status() == 0
    assert (batch.info()['tiles'] > 0) == tiles
    for name, a, ref in (('h', h, oh), ('u', u, ou), ('Fm', Fm, oF), ('M', M, oM), ('tr0', gpsi[0], psi[0]),
                         ('tr1', gpsi[1], psi[1])):
        assert np.array_equal(a.cpu().numpy(), ref), name


def _stack(dg, L, seed, T):
    rng = np.random.default_rng(seed)
    N, E = dg.host.N, dg.host.E
    dev = 'cuda:0'
    h = _T(300.0 + 10.0 * rng.random((L, N)), dev)
    u = _T(0.5 * (rng.random((L, E)) - 0.5), dev)
    M = (h * _T(np.asarray(dg.host.areaCell)[None], dev)).contiguous()
    return h, u, torch.zeros_like(u), M, torch.zeros_like(M), [_T(rng.random((L, N)), dev) for _ in range(T)]


@pytest.mark.parametrize('L', [7, 8])
@pytest.mark.parametrize('form', ['double', 'mixed'])
def test_many_blocks_equal_few(dev, grid4, form, L):
    """A launch with more blocks than fit the SMs takes the passes' instances with a launch bound (batched P1 and P4, the
    mixed S, the per-call P1): ten stacks of 16 tracers in one batch equal one of them alone with its tracers eight at a
    time, and 16 tracers by first order equal two calls of eight, bit for bit."""
    from isw import gpu, transport
    from isw.batch import Batch
    from isw.layers import Layers
    dg = gpu.DeviceGrid(grid4)
    kw = dict(gprime=[0.05] * (L - 1), floor=1.0, precision=form)

    def run(stacks, T, first):
        b, keep = Batch(0), []
        for q in range(stacks):
            core, tr = Layers(dg, L, **kw), transport.Transport(dg, layers=L, tracers=T, precision=form)
            h, u, Fm, M, M1, ps = _stack(dg, L, 5, 16)
            ps = ps[first:first + T]
            b.add(core, h, u, Fm, tr=tr, M=M, M1=M1, tracers=ps, dt=600.0, nfast=3)
            keep.append((core, tr, h, u, Fm, M, M1, ps))
        b.step()
        b.step()
        torch.cuda.synchronize()
        assert b.status() == 0
        return keep[-1]
    many, one, two = run(10, 16, 0), run(1, 8, 0), run(1, 8, 8)
    for a, x, y in zip(many[2:6], one[2:6], two[2:6]):
        assert torch.equal(a, x) and torch.equal(a, y)
    assert all(torch.equal(a, x) for a, x in zip(many[7], one[7] + two[7]))
    h, u, Fm, M, M1, ps = _stack(dg, L, 6, 16)
    tr = transport.Transport(dg, layers=L, tracers=16, precision=form)
    Fm = 1e-4 * float(M.min()) * u
    tr.mass_after(M, Fm, M1)
    apart = [p.clone() for p in ps]
    tr.step_many(M, M1, Fm, ps, 1)
    tr.step_many(M, M1, Fm, apart[:8], 1)
    tr.step_many(M, M1, Fm, apart[8:], 1)
    torch.cuda.synchronize()
    assert all(torch.equal(a, x) for a, x in zip(ps, apart))


def test_eight_layers_call_by_call_at_level6(dev):
    """Eight layers call by call on the 122,880 edges of level 6 (the slow tendency's instance with a launch bound) equal the
    batched step bit for bit."""
    from isw import gpu
    from isw import grid as G
    from isw.batch import Batch
    from isw.layers import Layers
    from isw.workload import planet_grid
    dg = gpu.DeviceGrid(planet_grid(G.build(6, device=0)))
    kw = dict(gprime=[0.05] * 7, floor=1.0, precision='double')
    h, u, Fm, *_ = _stack(dg, 8, 7, 0)
    h2, u2, Fm2 = h.clone(), u.clone(), Fm.clone()
    core, direct, b = Layers(dg, 8, **kw), Layers(dg, 8, batched=False, **kw), Batch(0)
    b.add(core, h, u, Fm, dt=100.0, nfast=3)
    for _ in range(2):
        b.step()
        direct.step(h2, u2, 100.0, 3, Fm2)
    torch.cuda.synchronize()
    assert b.status() == 0
    for x, y in ((h, h2), (u, u2), (Fm, Fm2)):
        assert torch.equal(x, y)
