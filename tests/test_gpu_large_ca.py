"""A Boris speed of light far above every signal (no limit in effect, as a user
asks for who wants the plain Alfven speed).

Against the oracle, which evaluates the reference's separate roots, on Cartesian
grids: the state after two steps, their time, and the CFL step of the same state in
device memory.  Tolerance: as for one step of states without ties (fewer than a
thousand roundings of 1.1e-16, amplified less than tenfold: 1e-12 relative L1),
twice.  (On a spherical grid the limiter jumps where a slope is zero, so rough
states differ from the oracle's by more than roundings.)

Against itself, on either kind of grid: above about 1e20 nothing is left of the
limit in 53 bits, so powers of two give the same bits."""
import ctypes as C
import math

import numpy as np
import pytest

from conftest import NG, rel_l1

pytestmark = pytest.mark.gpu

TOL = 2e-12




def _case(n, coord):
    import gop

    rng = np.random.default_rng(sum(n) + coord)
    dom = ((1.0, 2.0), (0.25 * math.pi, 0.75 * math.pi), (-0.8, 0.8)) if coord else ((0.0, 1.0),) * 3
    xs = [gop.grid_uniform(m, *dom[a]) for a, m in enumerate(n)]
    N = tuple(m + 2 * NG + 1 for m in n)
    W, B = np.zeros((6,) + N), np.zeros((3,) + N)
    W[0], W[4] = 1.0 + 0.2 * rng.random(N), 1.0 + 0.2 * rng.random(N)
    W[1:4] = 0.3 * rng.standard_normal((3,) + N)
    B[:] = 0.5 + 0.1 * rng.standard_normal((3,) + N)
    return xs, W, B


def _run(n, coord, ca, sweep):
    """State and statistics after two steps, the first CFL step, and that of
    gop_cfl_dt_noalloc."""
    import gop
    import torch

    xs, W, B = _case(n, coord)
    inst = gop.Instance(n, *xs, coord=coord, bc="eeeeee" if coord else "pppppp", ca=ca)
    inst.set_sweep(sweep)
    inst.upload(W, B)
    inst.prepare()
    dt0 = inst.stats()["dt0"]
    L = gop.lib()
    L.gop_cfl_dt_noalloc.argtypes = [C.POINTER(gop.Desc)] + [C.c_void_p] * 6
    d = inst.download(("gas", "face_b"))  # (with the ghosts filled)
    dev = [torch.from_numpy(d[k]).cuda() for k in ("gas", "face_b")]
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.gop_cfl_dt_noalloc(C.byref(inst.desc), *[C.c_void_p(t.data_ptr()) for t in dev], None, None,
                                C.c_void_p(out.data_ptr()), stream) == 0
    inst.step(2)
    d, st = inst.download(("gas", "face_b")), inst.stats()
    inst.close()
    return d, st, dt0, float(out[0])


@pytest.mark.parametrize("sweep", [True, False])
@pytest.mark.parametrize("n", [(16, 12, 9), (64, 56, 64)])
@pytest.mark.parametrize("ca", [10.0, 1e30, 1e80, 1e100, 1e150])
def test_as_the_oracle(oracle_mod, ca, n, sweep):
    xs, W, B = _case(n, 0)
    ref = oracle_mod.Oracle(n, *xs, ca=ca)
    ref.set_state(W, B)
    ref.prepare()
    ref.run(2)
    r = ref.state()
    d, st, dt0, dt_noalloc = _run(n, 0, ca, sweep)
    act = tuple(slice(NG, NG + m) for m in n)
    for m in range(5):
        assert rel_l1(d["gas"][m][act], r["W"][m][act]) <= TOL, f"W{m}"
    for c in range(3):
        s = list(act)
        s[c] = slice(NG, NG + n[c] + 1)
        assert rel_l1(d["face_b"][c][tuple(s)], r["B"][c][tuple(s)]) <= TOL, f"B{c}"
    assert math.isclose(st["time"], r["time"], rel_tol=TOL)
    assert math.isclose(dt_noalloc, dt0, rel_tol=TOL)


@pytest.mark.parametrize("sweep", [True, False])
@pytest.mark.parametrize("n,coord", [((16, 12, 9), 0), ((20, 17, 9), 2), ((64, 40, 44), 2)])
def test_the_same_however_large(n, coord, sweep):
    d, *rest = _run(n, coord, 2.0**100, sweep)
    for e in (260, 333, 511):
        dl, *restl = _run(n, coord, 2.0**e, sweep)
        assert restl == rest
        for f in d:
            np.testing.assert_array_equal(dl[f], d[f])
