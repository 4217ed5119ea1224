"""Deterministic sums from several threads and streams at once: each call leases its own scratch and result word."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [1, 2048, 2049, 122886, 33_000_001, 34_000_000])
def test_dsum_threads_and_streams(n):
    """Twelve threads on streams of their own (more than the leases kept) get the oracle's total, for sizes around one
    block, one pass, and the lease's capacity (beyond it the call allocates)."""
    from isw.gpu import dsum
    from oracle import model as M
    rng = np.random.default_rng(n)
    x, y = rng.standard_normal(n), rng.standard_normal(n)
    want = M.dsum(x, y)
    dx, dy = torch.as_tensor(x, device='cuda:0'), torch.as_tensor(y, device='cuda:0')
    torch.cuda.synchronize()
    got, threads = [], 12 if n < 1_000_000 else 2

    def work():
        st = torch.cuda.Stream()
        for _ in range(3):
            got.append(dsum(dx, dy, stream=st))
    ts = [threading.Thread(target=work) for _ in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert len(got) == 3 * threads and all(g == want for g in got)
