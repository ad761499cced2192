"""The points each launch of a step covers, by slot.  The three centre-to-edge
slots are one launch of a fixed shape and no grid of their own: nothing to launch
there (in a process of its own, for what a slot out of range would write)."""
import json
import subprocess
import sys
import textwrap

from conftest import ROOT

PROG = textwrap.dedent("""
    import ctypes as C, json, sys
    sys.path.insert(0, sys.argv[1])
    import gop
    class Dim3(C.Structure):
        _fields_ = [(a, C.c_uint) for a in "xyz"]
    f = gop.lib()._ZN3gop12launch_spaceERKNS_6ParamsEi
    f.restype, f.argtypes = Dim3, [C.c_void_p, C.c_int]
    P = (C.c_int * 1024)(*[5, 7, 11], *[14, 16, 20])  # n, N
    out = [f(C.addressof(P), slot) for slot in range(gop.Instance.TUNE_SLOTS.index("update") + 2)]
    print(json.dumps([[d.x, d.y, d.z] for d in out]))
    """)


def test_launch_space():
    r = subprocess.run([sys.executable, "-c", PROG, str(ROOT / "gamera-op_b200")], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stderr
    none = [0, 0, 0]
    assert json.loads(r.stdout) == [[14, 16, 20], none, none, none,  # ab2, c2c
                                    [5, 8, 12], [6, 7, 12], [6, 8, 11],  # emf
                                    [6, 7, 11], [5, 8, 11], [5, 7, 12],  # flux
                                    [5, 7, 11], none]  # update, no slot
