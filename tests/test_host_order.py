"""What the host copies of gop_upload, gop_set_background and gop_download wait
for, on a stand-in for the CUDA runtime (fake/fake_cuda.c) that writes down
every call: the journal is read as a graph (an operation follows the one before
it on its stream, a wait the event's record) and the order of two operations
is what the graph says.  Fields below and above the size from which they travel
on a stream of their own."""
import json
import os
import re
import subprocess
import sys
import textwrap

import pytest

from conftest import ROOT

SIZES = [(16, 16, 16), (100, 100, 100)]  # 0.1 and 10 MB a field


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = tmp_path_factory.mktemp("fake") / "libfake_cuda.so"
    subprocess.run(["gcc", "-std=gnu99", "-O1", "-fPIC", "-shared", str(ROOT / "tests/fake/fake_cuda.c"),
                    "-o", str(so)], check=True)
    return so


def _run(fake, body, **args):
    """Runs body (with gop, np, F = the stand-in, and args) in a process of its
    own; returns what it leaves in `out`."""
    prog = textwrap.dedent("""
        import ctypes as C, json, sys
        sys.path.insert(0, sys.argv[1])
        import numpy as np, gop
        A = json.loads(sys.argv[2])
        F = C.CDLL(None)
        F.fake_journal.restype = C.c_char_p
        F.fake_block.restype = C.c_void_p
        F.fake_block.argtypes = [C.c_size_t]
        F.fake_note.argtypes = [C.c_char_p, C.c_void_p]
        def instance(n):
            return gop.Instance(n, *[gop.grid_uniform(m, 0.0, 1.0) for m in n])
        def journal():
            return [l.split() for l in F.fake_journal().decode().splitlines()]
        out = None
        """) + textwrap.dedent(body) + "\nprint(json.dumps(out))\n"
    env = dict(os.environ, LD_PRELOAD=str(fake))
    r = subprocess.run([sys.executable, "-c", prog, str(ROOT / "gamera-op_b200"), json.dumps(args)],
                       capture_output=True, text=True, env=env, timeout=300)
    assert r.returncode == 0, r.stderr
    return json.loads(r.stdout.splitlines()[-1])


def _order(ops):
    """before[k]: the operations known to have ended when operation k starts;
    at the end, those a host wait has seen end."""
    last, event, before, done = {}, {}, [], set()
    for k, (op, stream, other) in enumerate(ops):
        b = set(last.get(stream, set())) | done
        if op == "wait":
            b |= event.get(other, set())
        if op == "record":
            event[other] = set(b)
        if op == "sync":
            done |= b
        before.append(b)
        last[stream] = b | {k}
    return before, done


@pytest.mark.parametrize("call", ["upload", "restart", "background"])
@pytest.mark.parametrize("n", SIZES)
def test_host_arrays_are_read_in_the_callers_stream_order(fake, n, call):
    """Work the caller has enqueued on the stream given to gop_set_stream (a copy
    into the array, say) ends before the library reads a host array."""
    ops = _run(fake, """
        inst = instance(A["n"])
        inst.set_stream(0x77770)
        W, B, E = np.zeros(inst.shape(6)), np.zeros(inst.shape(3)), np.zeros(inst.shape(9))
        for _ in range(2):  # (the second call finds the staging slots used before)
            F.fake_clear()
            F.fake_note(b"caller", 0x77770)
            if A["call"] == "background":
                inst.set_background(dict(b0=B, lorentz=B, b0_face=E, b0_edge=E))
            else:
                inst.upload(W, B, *((W, B) if A["call"] == "restart" else ()))
        out = journal()
        """, n=n, call=call)
    assert ops[0][0] == "caller"
    before, _ = _order(ops)
    reads = [k for k, o in enumerate(ops) if o[0] == "h2d"]
    assert reads and all(0 in before[k] for k in reads)


@pytest.mark.parametrize("copy", [1, 2, 4, 8])
@pytest.mark.parametrize("call", ["upload", "background", "get_background", "download"])
@pytest.mark.parametrize("n", SIZES)
def test_a_failed_call_leaves_no_copy_of_the_callers_arrays_running(fake, n, call, copy):
    """A call that returns with an error has waited for the copies it had
    started: the arrays are the caller's again."""
    code, ops = _run(fake, """
        inst = instance(A["n"])
        W, B, E = np.zeros(inst.shape(6)), np.zeros(inst.shape(3)), np.zeros(inst.shape(9))
        bg = dict(b0=B, lorentz=B, b0_face=E, b0_edge=E)
        if A["call"] == "get_background":
            inst.set_background(bg)
        F.fake_clear()
        F.fake_fail_copy(A["copy"])
        code = 0
        try:
            if A["call"] == "upload":
                inst.upload(W, B, W, B)
            elif A["call"] == "background":
                inst.set_background(bg)
            elif A["call"] == "get_background":
                inst.get_background()
            else:
                inst.download(("gas", "face_b", "gas_p", "face_b_p"))
        except gop.GopError as e:
            code = e.code
        out = [code, journal()]
        """, n=n, call=call, copy=copy)
    if "failed" not in [o[0] for o in ops]:  # the call makes fewer copies
        assert code == 0
        return
    assert code == -5
    _, done = _order(ops)
    assert all(k in done for k, o in enumerate(ops) if o[0] in ("h2d", "d2h"))


def _scalars():
    """Places of the instance's device scalars by name (and their number)."""
    src = (ROOT / "gamera-op_b200/csrc/gop_device.cuh").read_text()
    body = re.sub(r"//[^\n]*", "", re.search(r"enum Scal : int \{(.*?)\}", src, re.S).group(1))
    return {m.split("=")[0].strip(): k for k, m in enumerate(x for x in body.split(",") if x.strip())}


@pytest.mark.parametrize("restart", [False, True])
def test_prepare_clears_what_a_failed_step_left(fake, restart):
    """A step whose pipeline gave up may leave its tile counters above zero: a
    prepared instance starts from clear flags and counters all the same."""
    sc = _scalars()
    left = _run(fake, """
        inst = instance((16, 16, 16))
        inst.upload(np.zeros(inst.shape(6)), np.zeros(inst.shape(3)))
        s = (C.c_double * A["count"]).from_address(F.fake_block(8 * A["count"]))
        for k in A["names"]:
            s[k] = 3.0
        try:
            inst.prepare(restart=A["restart"])
        except gop.GopError:  # (no kernel has set a time step)
            pass
        out = [s[k] for k in A["names"]]
        """, names=[sc[k] for k in ("S_STOP", "S_STEPS", "S_FLAGS", "S_PAR", "S_TILE")], count=sc["NSCAL"],
        restart=restart)
    assert left == [0.0] * 5


@pytest.mark.parametrize("n,code", [((1000, 1000, 500), 0), ((1000, 1000, 540), -12), ((1280, 1280, 1280), -12),
                                    ((4, 4, 2**25), -12)])
@pytest.mark.parametrize("prec", [0, 1])
def test_fields_beyond_the_kernels_offsets_are_refused(fake, n, code, prec):
    """The kernels index a field by 32-bit byte offsets: 2^29 points, ghosts and row
    padding included, are too many, on a GPU with any memory."""
    got = _run(fake, """
        try:
            gop.Instance(A["n"], *[np.linspace(1.0, 2.0, m + 9) for m in A["n"]], precision=A["prec"])
            out = 0
        except gop.GopError as e:
            out = e.code
        """, n=n, prec=prec)
    assert got == code
