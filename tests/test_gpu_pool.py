"""The library's memory pool: what it keeps of freed instances is bounded, an
instance built from it starts from zeroed state, and threads share it."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEEP = 2 << 30


def _run(n, seed):
    import gop

    rng = np.random.default_rng(seed)
    xs = [gop.grid_uniform(m, 0.0, 1.0) for m in n]
    inst = gop.Instance(n, *xs, precision=seed % 2)
    W, B = np.ones(inst.shape(6)), np.full(inst.shape(3), 0.2)
    W[5] = 0.0
    W[1:4] = 0.1 * rng.standard_normal((3,) + inst.N)
    inst.upload(W, B)
    inst.prepare()
    inst.step(3)
    d = inst.download(("gas", "face_b"))
    inst.close()
    return d


def test_freed_memory_is_kept_up_to_a_bound():
    import gop
    import torch

    _run((16, 16, 16), 0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    insts = [gop.make(gop.PROBLEM_BLAST, (128, 128, 128)) for _ in range(4)]
    assert before - torch.cuda.mem_get_info()[0] > 3 * KEEP / 2
    for i in insts:
        i.close()
    _run((16, 16, 16), 0)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] <= KEEP + (256 << 20)


def test_threads_share_the_pool():
    grids = [(16, 16, 16), (24, 12, 8), (64, 64, 4), (33, 17, 5)]
    jobs = [(grids[k % 4], k) for k in range(16)]
    alone = [_run(*j) for j in jobs]
    with ThreadPoolExecutor(4) as ex:
        together = list(ex.map(lambda j: _run(*j), jobs))
    for a, b in zip(alone, together):
        for f in ("gas", "face_b"):
            np.testing.assert_array_equal(a[f], b[f])
