"""FP64 steps of grids whose theta range starts at the pole, where the limiter's
coefficients are infinite: the tile-staged kernels (compiled with the look at pole
faces for such grids) against the per-point ones, and the row of cells at the pole,
whose face field takes the mean EMF on the pole, against golden values
(golden/ring_pole0.npz: the velocities after one step of the same start, computed
with the clamp and the limiter term by term -- fmin, fmax, signs -- before they were
rewritten).

Tolerance: one step takes each value through fewer than a thousand roundings of
1.1e-16 whose amplification is below ten: 1e-12 relative L1; 1e-13 between the two
forms, as elsewhere."""
import math

import numpy as np
import pytest

from conftest import NG, load_golden, rel_l1

pytestmark = pytest.mark.gpu


def _step(n, top, bc, sweep, steps):
    import gop

    rng = np.random.default_rng(sum(n))
    xs = [gop.grid_uniform(n[0], 1.0, 2.0), gop.grid_uniform(n[1], 0.0, top), gop.grid_uniform(n[2], 0.0, 2.0 * math.pi)]
    N = tuple(m + 2 * NG + 1 for m in n)
    W, B = np.zeros((6,) + N), np.zeros((3,) + N)
    W[0], W[4] = 1.0 + 0.2 * rng.random(N), 1.0 + 0.2 * rng.random(N)
    W[1:4] = 0.3 * rng.standard_normal((3,) + N)
    B[:] = 0.5 + 0.1 * rng.standard_normal((3,) + N)
    inst = gop.Instance(n, *xs, coord=gop.COORD_SPHERICAL, bc=bc, ring_average=True)
    inst.set_sweep(sweep)
    inst.upload(W, B)
    inst.prepare()
    inst.step(steps)
    d = inst.download(("gas", "face_b"))
    inst.close()
    return d


@pytest.mark.parametrize("n,top,bc", [((8, 16, 32), math.pi, "eeoopp"), ((33, 12, 64), 0.5 * math.pi, "eeoepp")])
def test_forms_agree(n, top, bc):
    a, b = _step(n, top, bc, True, 3), _step(n, top, bc, False, 3)
    for f in a:
        for m in range(a[f].shape[0]):
            assert rel_l1(a[f][m], b[f][m]) <= 1e-13, f"{f}[{m}]"


@pytest.mark.parametrize("sweep", [True, False])
@pytest.mark.parametrize("key,n,top,bc", [("sphere", (8, 16, 32), math.pi, "eeoopp"),
                                          ("hemisphere", (8, 16, 32), 0.5 * math.pi, "eeoepp")])
def test_row_at_the_pole(key, n, top, bc, sweep):
    v = _step(n, top, bc, sweep, 1)["gas"][1:4, NG:NG + n[0], NG, NG:NG + n[2]]
    g = load_golden("ring_pole0")[key]
    for m in range(3):
        assert rel_l1(v[m], g[m]) <= 1e-12, f"v{m + 1}"
