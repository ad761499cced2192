"""A field of 1e-165 to 1e-140, as it is a few cells away from a field loop: its
square and what is multiplied with it underflow.  The Alfven speed is nothing
beside the gas, and the step is that without a field."""
import numpy as np
import pytest

from conftest import NG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sweep", [True, False])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("rho", [0.004, 1.0, 50.0])
@pytest.mark.parametrize("ca", [0.1, 1.0, 10.0, 1e4])
def test_tiny_fields_do_nothing(ca, rho, prec, sweep):
    import gop

    n = (24, 12, 9)
    xs = [gop.grid_uniform(m, 0.0, 1.0) for m in n]
    rng = np.random.default_rng(3)
    out = []
    for field in (True, False):
        inst = gop.Instance(n, *xs, ca=ca, precision=prec)
        inst.set_sweep(sweep)
        W, B = np.zeros(inst.shape(6)), np.zeros(inst.shape(3))
        W[0], W[4] = rho, 1.0
        W[1:4] = 0.1 * np.random.default_rng(4).standard_normal(W[1:4].shape)
        if field:  # every power of ten, along the first axis
            B[:] = (10.0 ** -np.arange(165.0, 140.0, -25.0 / B.shape[1]))[:B.shape[1], None, None]
            B *= rng.uniform(1.0, 3.0, B.shape)
        inst.upload(W, B)
        inst.prepare()
        inst.step(3)
        out.append(inst.download(("gas",))["gas"])
        assert inst.stats()["flags"] == 0
        inst.close()
    np.testing.assert_array_equal(out[0], out[1])
