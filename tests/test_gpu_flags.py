"""Steps of an instance whose error flag says that a pipeline wait has timed out
(the flag is written from outside; nothing waits): the tile-staged launches leave
without work, every block counts itself so that the tile counters end at zero
even if they did not begin so, the step reports the timeout and nothing else, and
the instance is whole again after an upload."""
import json
import os
import subprocess
import sys
import textwrap

import pytest

from conftest import ROOT
from test_host_order import _scalars

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def blocks(tmp_path_factory):
    so = tmp_path_factory.mktemp("blocks") / "libdevice_blocks.so"
    subprocess.run(["gcc", "-std=gnu99", "-O1", "-fPIC", "-shared", str(ROOT / "tests/fake/device_blocks.c"),
                    "-o", str(so), "-ldl"], check=True)
    return so


PROG = textwrap.dedent("""
    import ctypes as C, json, sys
    sys.path.insert(0, sys.argv[1])
    import numpy as np, gop
    A = json.loads(sys.argv[2])
    sc, n = A["sc"], A["n"]
    gop.lib()
    F = C.CDLL(None)
    F.block_of.restype = C.c_void_p
    F.block_of.argtypes = [C.c_size_t]
    copy = C.CDLL("libcudart.so.12").cudaMemcpy
    copy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
    inst = gop.Instance(n, *[gop.grid_uniform(m, 0.0, 1.0) for m in n], precision=A["prec"])
    at = F.block_of(8 * sc["NSCAL"])
    def put(name, v):
        v = np.array([v])
        assert copy(at + 8 * sc[name], v.ctypes.data, 8, 1) == 0
    def get(name):
        v = np.zeros(1)
        assert copy(v.ctypes.data, at + 8 * sc[name], 8, 2) == 0
        return float(v[0])
    def code_of_a_step():
        try:
            inst.step(1)
        except gop.GopError as e:
            return e.code
        return 0
    def start(bad):
        W, B = np.ones(inst.shape(6)), np.full(inst.shape(3), 0.2)
        W[5] = 0.0
        W[1:4] = 0.1 * np.random.default_rng(1).standard_normal((3,) + inst.N)
        if bad:
            W[4, 8, 8, 8] = np.nan
        inst.upload(W, B)
        inst.prepare()
    out = {}
    start(False)
    out["clean"] = code_of_a_step()
    first = inst.download(("gas", "face_b"))
    start(A["nan"])
    put("S_TILE", np.array([7, 0], np.uint32).view(np.float64)[0])
    put("S_FLAGS", 2.0)
    out["flagged"] = code_of_a_step()
    out["flags"] = inst.stats()["flags"]
    out["counters"] = get("S_TILE")
    start(False)
    out["again"] = code_of_a_step()
    d = inst.download(("gas", "face_b"))
    out["same"] = all(bool(np.array_equal(d[f], first[f])) for f in d)
    print(json.dumps(out))
    """)


def _run(blocks, n, prec, nan):
    r = subprocess.run([sys.executable, "-c", PROG, str(ROOT / "gamera-op_b200"),
                        json.dumps(dict(sc=_scalars(), n=n, prec=prec, nan=nan))],
                       capture_output=True, text=True, timeout=300, env=dict(os.environ, LD_PRELOAD=str(blocks)))
    assert r.returncode == 0, r.stderr
    return json.loads(r.stdout.splitlines()[-1])


# the per-cell update, and the update from tiles
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [(32, 24, 20), (64, 96, 96)])
def test_flagged_steps_leave_the_counters_at_zero(blocks, n, prec):
    out = _run(blocks, n, prec, False)
    assert out == dict(clean=0, flagged=-5, flags=2, counters=0.0, again=0, same=True)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [(32, 24, 20), (64, 96, 96)])
def test_a_timed_out_step_is_not_taken_for_a_bad_state(blocks, n, prec):
    """The per-cell update runs on what the sweeps have left undone and finds a
    state that is no number."""
    out = _run(blocks, n, prec, True)
    assert out == dict(clean=0, flagged=-5, flags=2, counters=0.0, again=0, same=True)
