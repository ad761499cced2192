"""gop_autotune and the update's two forms: where the tiles apply they are timed
against the per-cell launch and reported (GOP_TUNE_SWEEP), where they do not the
reported shape is the one that runs.  On a 128^3 FP64 grid the tiles take 139 us
and the per-cell launch 171."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SWEEP = 14


@pytest.mark.parametrize("n,prec,tiles", [((128, 128, 128), 0, True), ((24, 20, 16), 0, False),
                                          ((24, 20, 16), 1, False)])
def test_the_reported_update_is_the_one_that_runs(n, prec, tiles):
    import gop

    out = []
    for tune in (True, False):
        inst = gop.make(gop.PROBLEM_BLAST, n, precision=prec)
        inst.prepare()
        if tune:
            chosen = inst.autotune(reps=5)
            assert (chosen["update"] == SWEEP) == tiles
            assert all(chosen[f"c2c_{a}"] == 0 for a in "ijk")
        inst.step(3)
        out.append(inst.download(("gas", "face_b")))
        inst.close()
    for f in out[0]:  # (a multiply-add contracted differently in another form)
        np.testing.assert_allclose(out[0][f], out[1][f], rtol=0, atol=1e-13 if prec == 0 else 1e-6)
