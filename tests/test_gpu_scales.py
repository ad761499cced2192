"""States in units far from one (densities and pressures of 1e-99 to 1e99): the products
under the FP64 speeds' roots, of fourth order in the density, leave the range of a
double where the reference's separate quotients do not.  Against the oracle: the
state after two steps, its time, and the CFL step of the same state in device
memory.

Tolerance: as for one step of states without ties (fewer than a thousand
roundings of 1.1e-16, amplified less than tenfold: 1e-12 relative L1), twice."""
import ctypes as C
import math

import numpy as np
import pytest

from conftest import NG, rel_l1

pytestmark = pytest.mark.gpu

TOL = 2e-12


@pytest.mark.parametrize("sweep", [True, False])
@pytest.mark.parametrize("n", [(16, 12, 9), (64, 56, 64)])
@pytest.mark.parametrize("power", [-330, -240, -80, 0, 80, 240, 330])
def test_units_far_from_one(oracle_mod, power, n, sweep):
    import gop
    import torch

    s = 2.0**power
    rng = np.random.default_rng(sum(n))
    N = tuple(m + 2 * NG + 1 for m in n)
    xs = [gop.grid_uniform(m, 0.0, 1.0) for m in n]
    W, B = np.zeros((6,) + N), np.zeros((3,) + N)
    W[0], W[4] = s * (1.0 + 0.2 * rng.random(N)), s * (1.0 + 0.2 * rng.random(N))
    W[1:4] = 0.3 * rng.standard_normal((3,) + N)
    B[:] = math.sqrt(s) * (0.5 + 0.1 * rng.standard_normal((3,) + N))
    floors = dict(rho_floor=1e-3 * s, p_floor=1e-4 * s)
    ref = oracle_mod.Oracle(n, *xs, **floors)
    ref.set_state(W, B)
    ref.prepare()
    ref.run(2)
    r = ref.state()
    inst = gop.Instance(n, *xs, **floors)
    inst.set_sweep(sweep)
    inst.upload(W, B)
    inst.prepare()
    dt0 = inst.stats()["dt0"]
    d = inst.download(("gas", "face_b"))  # (with the ghosts filled)
    L = gop.lib()
    L.gop_cfl_dt_noalloc.argtypes = [C.POINTER(gop.Desc)] + [C.c_void_p] * 6
    dev = [torch.from_numpy(d[k]).cuda() for k in ("gas", "face_b")]
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    assert L.gop_cfl_dt_noalloc(C.byref(inst.desc), *[C.c_void_p(t.data_ptr()) for t in dev], None, None,
                                C.c_void_p(out.data_ptr()),
                                C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    inst.step(2)
    d, st = inst.download(("gas", "face_b")), inst.stats()
    inst.close()
    act = tuple(slice(NG, NG + m) for m in n)
    for m in range(5):
        assert rel_l1(d["gas"][m][act] / r["W"][m][act].max(), r["W"][m][act] / r["W"][m][act].max()) <= TOL, f"W{m}"
    for c in range(3):
        f = list(act)
        f[c] = slice(NG, NG + n[c] + 1)
        ref_b = r["B"][c][tuple(f)]
        assert rel_l1(d["face_b"][c][tuple(f)] / ref_b.max(), ref_b / ref_b.max()) <= TOL, f"B{c}"
    assert math.isclose(st["time"], r["time"], rel_tol=TOL)
    assert math.isclose(float(out[0]), dt0, rel_tol=TOL)
