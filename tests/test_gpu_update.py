"""The update from shared-memory tiles against the per-cell kernel:
the same arithmetic on the same values, so the states agree to the rounding of
a multiply-add contracted differently (1e-13 relative L1, as for the flux and
EMF sweeps).  Grids large enough for the tiles (6 a resident block) whose last
tiles are partly filled on every axis, in both precisions, and one with a
background field; spherical shells in FP64 (the mixed path has the per-cell
kernel only)."""
import math

import numpy as np
import pytest

from conftest import NG, rel_l1

pytestmark = pytest.mark.gpu

TOL = 1e-13


GRIDS = [((64, 96, 96), False), ((97, 99, 83), False), ((4, 250, 401), False), ((72, 90, 81), True)]
SHELLS = [((64, 56, 64), False), ((33, 59, 61), False), ((40, 61, 66), True)]
CASES = [(n, bg, p, 0) for n, bg in GRIDS for p in (0, 1)] + [(n, bg, 0, 2) for n, bg in SHELLS]


@pytest.mark.parametrize("n,bg,prec,coord", CASES)
def test_tiled_update_equals_the_per_cell_update(n, bg, prec, coord):
    import gop

    rng = np.random.default_rng(sum(n) + prec)
    dom = ((1.0, 2.0), (0.25 * math.pi, 0.75 * math.pi), (-0.8, 0.8))
    xs = [gop.grid_uniform(m, *(dom[a] if coord else (1.0, 1.0 + m / 64.0))) for a, m in enumerate(n)]
    N = tuple(m + 2 * NG + 1 for m in n)
    W, B = np.zeros((6,) + N), np.zeros((3,) + N)
    W[0] = 1.0 + 0.2 * rng.random(N)
    W[4] = 1.0 + 0.2 * rng.random(N)
    W[1:4] = 0.3 * rng.standard_normal((3,) + N)
    B[:] = 0.5 + 0.1 * rng.standard_normal((3,) + N)
    out = []
    for sweep in (True, False):
        inst = gop.Instance(n, *xs, coord=coord, bc="eeeeee", precision=prec)
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
