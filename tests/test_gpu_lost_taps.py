"""A half-step value that is no number (an uploaded AB2 history with one): fmin and
fmax of the reference's clamp leave the larger neighbour in the place of the
interpolated value, on either side of a face.  That is the same seen from either
end of the axis, so a state that is its own mirror image stays one.

Tolerance: one step takes each value through fewer than a thousand roundings of
1.1e-16 (6e-8 on the mixed path) whose amplification is below ten: 1e-12 (6e-4)
of the largest value."""
import numpy as np
import pytest

from conftest import NG

pytestmark = pytest.mark.gpu


def _wrapped(a):
    """Active cells with their periodic ghosts (and an upper point each)."""
    return np.pad(a, ((NG, NG + 1),) * 3, mode="wrap")


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("sweep", [True, False])
@pytest.mark.parametrize("prec", [0, 1])
def test_mirror_images_stay_mirror_images(axis, prec, sweep):
    import gop

    n = (16, 10, 12)
    rng = np.random.default_rng(axis)
    flip = lambda a: np.flip(a, axis)

    def fields(scale):
        W = np.zeros((6,) + n)
        W[0], W[4] = 1.0 + scale * rng.random(n), 1.0 + scale * rng.random(n)
        W[1:4] = scale * rng.standard_normal((3,) + n)
        sign = [1, 1, 1, 1, 1, 1]
        sign[1 + axis] = -1
        return np.stack([0.5 * (w + s * flip(w)) for w, s in zip(W, sign)]), sign

    W, sign = fields(0.3)
    Wp = W + 0.1 * fields(0.3)[0]
    at = [4, 3, 5]
    mirrored = list(at)
    mirrored[axis] = n[axis] - 1 - at[axis]
    Wp[4][tuple(at)] = Wp[4][tuple(mirrored)] = np.nan
    full = lambda V: np.stack([_wrapped(v) for v in V])
    inst = gop.Instance(n, *[gop.grid_uniform(m, 0.0, 1.0) for m in n], precision=prec)
    inst.set_sweep(sweep)
    B = np.zeros(inst.shape(3))
    inst.upload(full(W), B, full(Wp), B, dt0=2e-3)
    inst.prepare(restart=True)
    inst.step(1)
    d = inst.download(("gas",))["gas"]
    inst.close()
    act = tuple(slice(NG, NG + m) for m in n)
    tol = 6e-4 if prec else 1e-12
    for m in range(5):
        a = d[m][act]
        assert np.isfinite(a).all()
        assert np.abs(a - sign[m] * flip(a)).max() <= tol * np.abs(a).max(), f"W{m}"
