"""gop_release_memory: what the library kept of closed instances is the device's
again, live instances are untouched, and the next instance is made as ever."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_kept_memory_is_given_back():
    import gop
    import torch

    gop.release_memory()  # (none made yet, or another test's)
    live = gop.make(gop.PROBLEM_BLAST, (32, 32, 32))
    live.prepare()
    live.step(2)
    torch.cuda.synchronize()
    gop.release_memory()
    before = torch.cuda.mem_get_info()[0]
    states = []
    for _ in range(2):
        inst = gop.make(gop.PROBLEM_BLAST, (96, 96, 96))
        inst.prepare()
        inst.step(2)
        states.append(inst.download(("gas",))["gas"])
        held = inst.stats()["device_bytes"]
        inst.close()
        torch.cuda.synchronize()
        assert before - torch.cuda.mem_get_info()[0] > held // 2  # kept
        gop.release_memory()
        assert before - torch.cuda.mem_get_info()[0] <= 64 << 20  # (mapped in blocks of 32 MB)
    np.testing.assert_array_equal(*states)
    live.step(2)
    assert live.stats()["steps"] == 4 and live.stats()["flags"] == 0
    live.close()
