"""States the step must report (GOP_ENUMERIC): a signal speed that is no number
in the reference's form, sqrt(gamma p / rho) and sqrt(b^2 / rho) by themselves
(src/solver_func.c:1005-1018, 875-902), may not become one because the
library evaluates it over a common denominator.  In both precisions, by the
tile-staged sweeps and by the per-point kernels, and with the field on either
side of the value where the denominator changes sign."""
import numpy as np
import pytest

from conftest import NG

pytestmark = pytest.mark.gpu

N3 = (16, 12, 8)
PATCH = tuple(slice(NG + 2, NG + m - 2) for m in N3)


def _state(rho, p, b):
    N = tuple(m + 2 * NG + 1 for m in N3)
    W, B = np.zeros((6,) + N), np.zeros((3,) + N)
    W[0], W[4], B[0] = rho, p, b
    return W, B


def _step(W, B, history, prec, sweep):
    """The code of one step from this state (0 or a GOP_E* code)."""
    import gop

    inst = gop.Instance(N3, *[gop.grid_uniform(m, 0.0, 1.0) for m in N3], precision=prec)
    inst.set_sweep(sweep)
    inst.upload(W, B, *(history or ()), dt0=1e-3 if history else 0.0)
    inst.prepare(restart=bool(history))
    code = 0
    try:
        inst.step(1)
    except gop.GopError as e:
        code = e.code
    flags = inst.stats()["flags"]
    inst.close()
    assert flags == (1 if code else 0)
    return code


@pytest.mark.parametrize("sweep", [True, False])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("b", [0.0, 1.0, 3.0, 30.0])
def test_negative_density_around_an_edge(b, prec, sweep):
    """Half-step densities are extrapolated in time and nothing holds them above
    zero: in a patch that was ten times denser they are about -1 or lower here.
    Without a field the edge's speed is that of the gas alone and the step goes
    on; with one it has no speed, below and above b^2 = ca^2 |rho|."""
    W, B = _state(0.1, 1.0, b)
    Wp = W.copy()
    Wp[(0,) + PATCH] = 1.0
    assert _step(W, B, (Wp, B), prec, sweep) == (0 if b == 0.0 else -34)


@pytest.mark.parametrize("sweep", [True, False])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("rho,p", [(1.0, -0.5), (-1.0, 1.0), (-1.0, -0.5), (0.0, 1.0)])
@pytest.mark.parametrize("b", [0.0, 0.3, 5.0, 30.0])
def test_states_without_a_signal_speed(b, rho, p, prec, sweep):
    """A patch of negative pressure (in a field strong enough, the common
    denominator's numerator is positive there), of negative density, of both,
    of no density."""
    W, B = _state(1.0, 1.0, b)
    W[(0,) + PATCH], W[(4,) + PATCH] = rho, p
    assert _step(W, B, None, prec, sweep) == -34


@pytest.mark.parametrize("b", [0.0, 0.3, 5.0, 30.0])
@pytest.mark.parametrize("prec", [0, 1])
def test_cells_without_a_signal_speed_set_no_time_step(b, prec):
    """The CFL minimum of the prepared state skips a cell of negative pressure."""
    import gop

    W, B = _state(1.0, 1.0, b)
    dt = []
    for bad in (False, True):
        if bad:  # would be the fastest cell by far
            W[0, NG + 3, NG + 3, NG + 3], W[4, NG + 3, NG + 3, NG + 3] = 1e-6, -1e-9
        inst = gop.Instance(N3, *[gop.grid_uniform(m, 0.0, 1.0) for m in N3], precision=prec)
        inst.upload(W, B)
        inst.prepare()
        dt.append(inst.stats()["dt0"])
        inst.close()
    assert dt[0] == dt[1]


@pytest.mark.parametrize("rho,p", [(1.0, -0.5), (-1.0, 1.0), (-1.0, -0.5), (0.0, 1.0), (-1e-4, -1.0)])
@pytest.mark.parametrize("b", [0.0, 0.3, 30.0])
def test_the_device_states_step_is_the_instances(b, rho, p):
    """gop_cfl_dt_noalloc skips and counts the cells that gop_prepare does (-rho and
    -p without a field have the speed of rho and p).  Tolerance: some twenty
    roundings of 1.1e-16 on either side."""
    import ctypes as C

    import gop
    import torch

    W, B = _state(1.0, 1.0, b)
    W[(0,) + PATCH], W[(4,) + PATCH] = rho, p
    inst = gop.Instance(N3, *[gop.grid_uniform(m, 0.0, 1.0) for m in N3])
    inst.upload(W, B)
    inst.prepare()
    L = gop.lib()
    L.gop_cfl_dt_noalloc.argtypes = [C.POINTER(gop.Desc)] + [C.c_void_p] * 6
    dev = [torch.from_numpy(a).cuda() for a in (W, B)]
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    assert L.gop_cfl_dt_noalloc(C.byref(inst.desc), *[C.c_void_p(t.data_ptr()) for t in dev], None, None,
                                C.c_void_p(out.data_ptr()),
                                C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    dt0 = inst.stats()["dt0"]
    inst.close()
    assert abs(float(out[0]) - dt0) <= 1e-14 * dt0
