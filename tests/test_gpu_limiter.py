"""The PDM limiter's corner cases, on the device, against the checker.

States of a few whole-number values put the limiter on its ties: equal
neighbours at the face (the clamp leaves one value), equal cells on one side
(the slope term vanishes and the reference's factor |sgn + sgn| is one),
extrema and steps.  One step from them is compared, by the tile-staged sweeps
and by the per-point kernels, at sizes with partial tiles and at the smallest
grid.

Tolerance: one step takes each value through fewer than a thousand roundings
of 1.1e-16 whose amplification, by cell-centred cancellation, is below 10:
1e-12 relative L1.  On the spherical grid the limiter jumps where a slope is
exactly zero (its two coefficients do not cancel there), so a rounding in the
face field or in the edge velocities may move the EMF and through it the
velocity; rho and p, whose ties are exact on both sides, are compared there.
"""
import math

import numpy as np
import pytest

from conftest import NG, rel_l1

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.mark.parametrize("sweep", [True, False])
@pytest.mark.parametrize("n,coord", [((4, 4, 4), 0), ((33, 9, 7), 0), ((64, 8, 16), 0),
                                     ((20, 17, 9), 2), ((32, 8, 8), 2)])
def test_ties_match_the_checker(oracle_mod, n, coord, sweep):
    import gop

    rng = np.random.default_rng(sum(n) + coord)
    dom = ((1.0, 2.0, 0.25 * math.pi, 0.75 * math.pi, -0.25 * math.pi, 0.25 * math.pi) if coord
           else (0.0, 1.0, 0.0, 1.0, 0.0, 1.0))
    bc = "eeeeee" if coord else "pppppp"
    xs = [gop.grid_uniform(n[a], dom[2 * a], dom[2 * a + 1]) for a in range(3)]
    N = tuple(m + 2 * NG + 1 for m in n)
    W = np.zeros((6,) + N)
    B = np.zeros((3,) + N)
    act = tuple(slice(NG, NG + m) for m in n)
    W[(0,) + act] = rng.integers(1, 4, n)
    W[(4,) + act] = rng.integers(1, 4, n)
    for m in (1, 2, 3):
        W[(m,) + act] = rng.integers(-1, 2, n)
    for c in range(3):
        if coord:  # no ties in the field
            B[c] = 0.1 * (1.0 + c) + 0.01 * rng.standard_normal(N)
        else:
            s = list(act)
            s[c] = slice(NG, NG + n[c] + 1)
            B[(c,) + tuple(s)] = rng.integers(-1, 2, [m + (a == c) for a, m in enumerate(n)])
    ref = oracle_mod.Oracle(n, *xs, coord=coord, bc=bc)
    ref.set_state(W, B)
    ref.prepare()
    ref.run(1)
    r = ref.state()
    inst = gop.Instance(n, *xs, coord=coord, bc=bc)
    inst.set_sweep(sweep)
    inst.upload(W, B)
    inst.prepare()
    inst.step(1)
    d = inst.download(("gas", "face_b"))
    inst.close()
    for m in ((0, 4) if coord else range(5)):
        assert rel_l1(d["gas"][m][act], r["W"][m][act]) <= TOL, f"W{m}"
    if not coord:
        for c in range(3):
            s = list(act)
            s[c] = slice(NG, NG + n[c] + 1)
            assert rel_l1(d["face_b"][c][tuple(s)], r["B"][c][tuple(s)]) <= TOL, f"B{c}"


@pytest.mark.parametrize("b", [0.0, 5.0, 30.0])
def test_negative_density_is_reported(b):
    """Faces between cells of negative density have no signal speed, however
    strong the field (b^2 below and above ca^2 |rho|): the step reports it."""
    import gop

    n = (16, 12, 8)
    xs = [gop.grid_uniform(m, 0.0, 1.0) for m in n]
    N = tuple(m + 2 * NG + 1 for m in n)
    W, B = np.zeros((6,) + N), np.zeros((3,) + N)
    W[0], W[4], B[0] = 1.0, 1.0, b
    W[0, NG + 4:NG + 8, NG + 4:NG + 8, NG + 2:NG + 6] = -1.0
    inst = gop.Instance(n, *xs)
    inst.upload(W, B)
    inst.prepare()
    with pytest.raises(gop.GopError) as e:
        inst.step(2)
    assert e.value.code == -34
    inst.close()
