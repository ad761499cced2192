"""A restart from an AB2 history whose periodic ghost layers do not repeat its
active cells (a history kept without its ghosts, say): gop_prepare fills the
ghosts of the state, not of the history, so the first step takes what was
uploaded, as the reference does.  Against the oracle; and by the launches of a
step, that a history with its ghosts filled costs no more than none.

Tolerance: one step takes each value through fewer than a thousand roundings of
1.1e-16 whose amplification is below ten: 1e-12 relative L1; two steps, twice."""
import numpy as np
import pytest

from conftest import NG, rel_l1

pytestmark = pytest.mark.gpu


def _case(n, bc, filled):
    rng = np.random.default_rng(sum(n) + ord(bc[0]) + ord(bc[4]))
    N = tuple(m + 2 * NG + 1 for m in n)

    def state():
        W, B = np.zeros((6,) + N), np.zeros((3,) + N)
        W[0], W[4] = 1.0 + 0.2 * rng.random(N), 1.0 + 0.2 * rng.random(N)
        W[1:4] = 0.3 * rng.standard_normal((3,) + N)
        B[:] = 0.5 + 0.1 * rng.standard_normal((3,) + N)
        return W, B

    (W, B), (Wp, Bp) = state(), state()
    if filled:
        act = tuple(slice(NG, NG + m) for m in n)
        for t in (*Wp, *Bp):
            t[:] = np.pad(t[act], ((NG, NG + 1),) * 3, mode="wrap")
    return W, B, 0.9 * W + 0.1 * Wp if not filled else Wp, Bp


@pytest.mark.parametrize("steps", [1, 2])
@pytest.mark.parametrize("sweep", [True, False])
@pytest.mark.parametrize("n", [(16, 12, 9), (33, 5, 4)])
@pytest.mark.parametrize("bc", ["pppppp", "ppeeee", "eeppss", "sseepp"])
def test_uploaded_history_is_taken_as_it_is(oracle_mod, bc, n, sweep, steps):
    import gop

    W, B, Wp, Bp = _case(n, bc, False)
    xs = [gop.grid_uniform(m, 0.0, 1.0) for m in n]
    ref = oracle_mod.Oracle(n, *xs, bc=bc)
    ref.set_state(W, B, Wp, Bp, time=0.5, dt0=4e-3)
    ref.prepare(restart=True)
    ref.run(steps)
    r = ref.state()
    inst = gop.Instance(n, *xs, bc=bc)
    inst.set_sweep(sweep)
    inst.upload(W, B, Wp, Bp, time=0.5, dt0=4e-3)
    inst.prepare(restart=True)
    batch = gop.Batch([inst])
    batch.step([steps])
    d = inst.download(("gas", "face_b"))
    batch.close()
    inst.close()
    act = tuple(slice(NG, NG + m) for m in n)
    for m in range(5):
        assert rel_l1(d["gas"][m][act], r["W"][m][act]) <= steps * 1e-12, f"W{m}"
    for c in range(3):
        s = list(act)
        s[c] = slice(NG, NG + n[c] + 1)
        assert rel_l1(d["face_b"][c][tuple(s)], r["B"][c][tuple(s)]) <= steps * 1e-12, f"B{c}"


def test_a_filled_history_costs_nothing():
    """Launches of three steps: without a history, with a filled one, with one that
    is not, and without one again."""
    import gop

    n = (16, 12, 9)
    inst = gop.Instance(n, *[gop.grid_uniform(m, 0.0, 1.0) for m in n])
    count = []
    for history, filled in ((False, True), (True, True), (True, False), (False, True)):
        W, B, Wp, Bp = _case(n, "pppppp", filled)
        inst.upload(W, B, *((Wp, Bp) if history else ()), dt0=4e-3)
        inst.prepare(restart=history)
        before = gop.kernel_launches()
        inst.step(3)
        count.append(gop.kernel_launches() - before)
    inst.close()
    assert count[0] == count[1] == count[3] == count[2] - 3
