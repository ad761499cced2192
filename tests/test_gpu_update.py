"""The Cartesian update from shared-memory tiles against the per-cell kernel:
the same arithmetic on the same values, so the states agree to the rounding of
a multiply-add contracted differently (1e-13 relative L1, as for the flux and
EMF sweeps).  Grids large enough for the tiles (6 a resident block) whose last
tiles are partly filled on every axis, in both precisions, and one with a
background field."""
import numpy as np
import pytest

from conftest import NG, rel_l1

pytestmark = pytest.mark.gpu

TOL = 1e-13


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,bg", [((64, 96, 96), False), ((97, 99, 83), False), ((4, 250, 401), False),
                                  ((72, 90, 81), True)])
def test_tiled_update_equals_the_per_cell_update(n, bg, prec):
    import gop

    rng = np.random.default_rng(sum(n) + prec)
    xs = [gop.grid_uniform(m, 1.0, 1.0 + m / 64.0) for m in n]
    N = tuple(m + 2 * NG + 1 for m in n)
    W, B = np.zeros((6,) + N), np.zeros((3,) + N)
    W[0] = 1.0 + 0.2 * rng.random(N)
    W[4] = 1.0 + 0.2 * rng.random(N)
    W[1:4] = 0.3 * rng.standard_normal((3,) + N)
    B[:] = 0.5 + 0.1 * rng.standard_normal((3,) + N)
    out = []
    for sweep in (True, False):
        inst = gop.Instance(n, *xs, bc="eeeeee", precision=prec)
        if bg:
            inst.set_background_device(gop.BG_DIPOLE, moment=0.2)
        inst.set_sweep(sweep)
        inst.upload(W, B)
        inst.prepare()
        inst.step(2)
        out.append((inst.download(("gas", "face_b")), inst.stats()))
        inst.close()
    (a, sa), (b, sb) = out
    for f in ("gas", "face_b"):
        for m in range(a[f].shape[0]):
            assert rel_l1(a[f][m], b[f][m]) <= TOL, f"{f}[{m}]"
    assert abs(sa["dt"] - sb["dt"]) <= 1e-13 * sb["dt"]
    assert abs(sa["divb_max"] - sb["divb_max"]) <= 1e-11 * sb["divb_max"]
