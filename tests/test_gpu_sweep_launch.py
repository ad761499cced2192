"""The sweeps' launch forms: the tiles of the three axes in one launch, or the
flux of each axis in its own where a grid has very many tiles.  Both must give
what the per-point kernels give, at sizes with one tile, partly filled tiles
and more tiles than blocks.

Tolerance as in test_gpu_sweep.py: the same operations in the same order,
1e-13 relative L1 for a multiply-add contracted differently.
"""
import numpy as np
import pytest

from conftest import NG, rel_l1

pytestmark = pytest.mark.gpu

TOL = 1e-13


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,bc", [((4, 16, 10000), "pppppp"),  # each axis on its own
                                  ((4, 4, 4), "pppppp"), ((33, 17, 5), "eesspp"),
                                  ((64, 40, 9), "pppppp"), ((32, 15, 31), "eeeeee")])
def test_launch_forms_equal_the_per_point_kernels(n, bc, prec):
    import gop

    rng = np.random.default_rng(sum(n) + prec)
    xs = [gop.grid_uniform(m, 0.0, m / 64.0) for m in n]
    N = tuple(m + 2 * NG + 1 for m in n)
    W, B = np.zeros((6,) + N), np.zeros((3,) + N)
    W[0] = 1.0 + 0.2 * rng.random(N)
    W[4] = 1.0 + 0.2 * rng.random(N)
    W[1:4] = 0.3 * rng.standard_normal((3,) + N)
    B[:] = 0.5 + 0.1 * rng.standard_normal((3,) + N)
    out = []
    for sweep in (True, False):
        inst = gop.Instance(n, *xs, bc=bc, precision=prec)
        inst.set_sweep(sweep)
        inst.upload(W, B)
        inst.prepare()
        inst.step(3)
        out.append(inst.download(("gas", "face_b")))
        inst.close()
    for f in ("gas", "face_b"):
        for m in range(out[0][f].shape[0]):
            assert rel_l1(out[0][f][m], out[1][f][m]) <= TOL, f"{f}[{m}]"
