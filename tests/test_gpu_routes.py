"""The step's routes for option stacks on a B200: through the private one-stack batch (its fast loop in tiles, walls
included) once calls repeat the one before them, call by call otherwise; every mix equals the call-by-call
kernels bit for bit."""
from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / 'golden'


def T(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device='cuda:0')


def golden(name):
    with np.load(GOLDEN / f'{name}.npz') as z:
        return {k: z[k] for k in z.files}


@pytest.mark.parametrize('options', ['all', 'walls', 'fields'])
def test_option_routes_equal_per_call(grid4, options):
    """Repeated calls, two sets of arrays in turn, an option set between calls, Fm given and not: h, u and Fm equal the
    per-call kernels' after every step; a NaN thickness is stepped, not refused, as before."""
    from isw.gpu import DeviceGrid
    from isw.layers import Layers
    z = golden('options_n4')
    dg = DeviceGrid(grid4)
    dt, nfast = float(z['dt']), int(z['nfast'])
    cores = []
    for batched in (True, False):
        kw = dict(wall=z['wall']) if options != 'fields' else {}
        if options == 'all':
            kw.update(shelf=50.0, shelf_bed=True)
        core = Layers(dg, 2, b=z['b'], gprime=[0.02], stress=[0.0, 2.5e-4], nu4=float(z['nu4']), floor=1.0, batched=batched, **kw)
        if options != 'walls':
            core.sig, core.cd_bot, core.cbot = T(z['sig']), 2.5e-3, T(z['cbot'])
        cores.append(core)
    wall = T(z['wall']) if options != 'fields' else 1.0
    sets = [[dict(h=T(z['h0']) * s, u=T(z['u0']) * wall, Fm=torch.zeros_like(T(z['u0']))) for s in (1.0, 1.001)] for _ in cores]
    order = [(0, True), (0, True), (0, True), (1, True), (0, True), (1, True), (1, True), (1, False), (1, False), (0, True),
             (0, True)]
    tide = T(np.linspace(-0.3, 0.3, dg.N))
    for n, (which, with_fm) in enumerate(order):
        for core, ss in zip(cores, sets):
            if n in (3, 9):
                core.tide = tide if n == 3 else None
            a = ss[which]
            core.step(a['h'], a['u'], dt, nfast, a['Fm'] if with_fm else None)
        torch.cuda.synchronize()
        for name in ('h', 'u', 'Fm'):
            x, y = (ss[which][name] for ss in sets)
            assert torch.equal(x, y), (n, name)
    for ss in sets:
        ss[0]['h'][0, 7] = float('nan')
    for _ in range(3):
        for core, ss in zip(cores, sets):
            core.step(ss[0]['h'], ss[0]['u'], dt, nfast, ss[0]['Fm'])
    torch.cuda.synchronize()
    assert all(core.status() == 0 for core in cores)
    assert torch.equal(*(torch.nan_to_num(ss[0]['h'], nan=-1.0) for ss in sets))


def test_timed_out_option_stack_is_refused(grid4):
    """A wait of the tile kernel that runs out on an option stack: every later step is refused with ISW_ETIMEOUT (a call
    that repeats the one before it, one with other arguments, one after an option was set, one inside a capture), and
    after a reset the stack steps on equal to the call-by-call kernels bit for bit (the launch that timed out wrote
    scratch only)."""
    from isw._lib import ISW_ETIMEOUT, IswError
    from isw.gpu import DeviceGrid
    from isw.layers import Layers
    z = golden('options_n4')
    dg = DeviceGrid(grid4)
    dt, nfast = float(z['dt']), int(z['nfast'])
    cores, states = [], []
    for batched in (True, False):
        cores.append(Layers(dg, 2, b=z['b'], gprime=[0.02], floor=1.0, batched=batched, wall=z['wall']))
        states.append((T(z['h0']), T(z['u0']) * T(z['wall']), torch.zeros_like(T(z['u0']))))

    def step(which, n=nfast):
        h, u, Fm = states[which]
        cores[which].step(h, u, dt, n, Fm)
    for _ in range(2):                                  # the second goes through the private batch
        step(0)
        step(1)
    core = cores[0]
    core.fault_test(timeout_s=0.05)
    torch.cuda.synchronize()
    assert core.status() == ISW_ETIMEOUT

    def refused(n=nfast):
        with pytest.raises(IswError) as err:
            step(0, n)
        assert err.value.status == ISW_ETIMEOUT
    refused()
    refused(nfast + 1)
    core.cd_bot = 2.5e-3
    refused()
    core.cd_bot = 0.0
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            refused()
    torch.cuda.synchronize()
    assert core.status(reset=True) == ISW_ETIMEOUT and core.status() == 0
    for _ in range(3):
        step(0)
        step(1)
    torch.cuda.synchronize()
    for x, y in zip(*states):
        assert torch.equal(x, y)


@pytest.mark.parametrize('order', ['pairs', 'option'])
def test_unpaid_builds_stop(grid4, order):
    """Orders in which building the private batch does not pay (two sets of arrays in pairs of calls; an option set before
    every other call) take no longer than the call-by-call kernels: host time per call in turns, the best of several. With
    a build in every pair they took 1.5 to 2 times as long."""
    import time
    from isw.gpu import DeviceGrid
    from isw.layers import Layers
    z = golden('options_n4')
    dg = DeviceGrid(grid4)
    cores = [Layers(dg, 2, b=z['b'], gprime=[0.02], floor=1.0, batched=batched, wall=z['wall']) for batched in (True, False)]
    sets = [[(T(z['h0']), T(z['u0']) * T(z['wall']), torch.zeros_like(T(z['u0']))) for _ in range(2)] for _ in cores]
    tide = T(np.linspace(-0.3, 0.3, dg.N))

    def calls(which, n):
        for i in range(n):
            if order == 'option' and i % 2 == 0:
                cores[which].tide = tide if i % 4 == 0 else None
            h, u, Fm = sets[which][i // 2 % 2 if order == 'pairs' else 0]
            cores[which].step(h, u, float(z['dt']) / 4, 2, Fm)
        torch.cuda.synchronize()
    times = [[], []]
    for turn in range(8):
        for which in (0, 1):
            t0 = time.perf_counter()
            calls(which, 80)
            if turn > 0:
                times[which].append(time.perf_counter() - t0)
    assert min(times[0]) < 1.25 * min(times[1]), times
    for x, y in zip(*(s[0] + s[1] for s in sets)):
        assert torch.equal(x, y)
