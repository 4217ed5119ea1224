"""The tile kernel where its tiles are large: more own edges than the small capacity holds, and stacks whose stage's end
does not fit in shared memory for all layers at once (it then takes them in groups)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def T(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device='cuda:0')


def stack(dg, L, seed):
    """h, u, Fm: thin enough layers beside thick ones that the floor limiter acts."""
    rng = np.random.default_rng(seed)
    N, E = dg.host.N, dg.host.E
    h = 200.0 + 20.0 * rng.random((L, N))
    h[:, rng.random(N) < 0.05] = 1.5
    return T(h), T(2.0 * (rng.random((L, E)) - 0.5)), torch.zeros(L, E, dtype=torch.float64, device='cuda:0')


@pytest.mark.parametrize('form', ['double', 'walls', 'mixed'])
@pytest.mark.parametrize('L,k', [(3, 2), (8, 1), (8, 2)])
def test_large_tiles(grid4, form, L, k):
    """Six tiles of 427 cells, two an SM (384 threads: more than 3 x 384 own edges, so the large capacity). Three
    layers end their stage at once; eight, of 1,281 edges and 427 cells or more a tile, need more than the 112 KB a block has
    beside its ids, and end it in groups. FP64: the call-by-call kernels' values bit for bit; mixed: those of small tiles (the batch's own choice)."""
    from isw.batch import Batch
    from isw.gpu import DeviceGrid
    from isw.layers import Layers
    dg = DeviceGrid(grid4)
    kw = dict(gprime=[0.02] * (L - 1), floor=1.0, nu4=1e14, precision='mixed' if form == 'mixed' else 'double')
    if form == 'walls':
        kw['wall'] = (np.random.default_rng(1).random(grid4.E) > 0.1).astype(np.float64)
    large, small = Batch(0), Batch(0)
    large.config(layout='packed', tile_cells=512, blocks_per_sm=2, tile_k=k)
    core, (h, u, Fm) = Layers(dg, L, **kw), stack(dg, L, L)
    large.add(core, h, u, Fm, dt=300.0, nfast=5)
    info = large.info()
    assert (info['tiles'], info['tile_k'], info['blocks_per_sm']) == (6, k, 2)
    assert L == 3 or info['smem'] < 8 * L * (1281 + 427)
    other, (h2, u2, Fm2) = Layers(dg, L, batched=False, **kw), stack(dg, L, L)
    if form == 'mixed':
        small.add(other, h2, u2, Fm2, dt=300.0, nfast=5)
        assert small.info()['tiles'] > 6
    for _ in range(3):
        large.step()
        if form == 'mixed':
            small.step()
        else:
            other.step(h2, u2, 300.0, 5, Fm2)
    torch.cuda.synchronize()
    assert large.status() == 0
    for x, y in ((h, h2), (u, u2), (Fm, Fm2)):
        assert torch.equal(x, y)


@pytest.mark.parametrize('form', ['double', 'mixed'])
def test_deep_stack_tiled_at_level7(form):
    """Eight layers on the 163,842 cells of level 7 step in tiles of the whole GPU, at every exchange interval that a
    one-layer stack has; FP64: the grid-wide passes' values bit for bit."""
    from isw import grid as G
    from isw.batch import Batch
    from isw.gpu import DeviceGrid
    from isw.layers import Layers
    from isw.workload import planet_grid
    dg = DeviceGrid(planet_grid(G.build(7, device=0)))
    states, intervals = [], []
    for tiles, L in ((True, 8), (False, 8), (True, 1)):
        b = Batch(0)
        b.config(tiles=tiles, layout='shared', blocks_per_sm=1)
        core, s = Layers(dg, L, gprime=[0.02] * (L - 1), floor=1.0, precision=form), stack(dg, L, 3)
        b.add(core, *s, dt=30.0, nfast=5)
        if L == 8:
            b.step()
            b.step()
            torch.cuda.synchronize()
            assert b.status() == 0
            states.append(s)
        assert (b.info()['tiles'] > 0) == tiles
        intervals.append(b.info()['tile_k'])
    assert intervals[0] == intervals[2] > 0
    if form == 'double':
        for x, y in zip(*states):
            assert torch.equal(x, y)
