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
