"""An upload in the order of the caller's stream, on the device: the pinned array
is still being filled by a copy on that stream, behind a delay, when gop_upload
is called.  Fields below and above 8 MB (from there on they travel on a stream
of their own)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(16, 16, 16), (100, 100, 101)])
def test_upload_follows_the_callers_copy_into_the_array(n):
    import gop
    import torch

    inst = gop.Instance(n, *[gop.grid_uniform(m, 0.0, 1.0) for m in n], bc="nnnnnn")
    gen = torch.Generator(device="cuda").manual_seed(n[2])
    stream = torch.cuda.Stream()
    inst.set_stream(stream.cuda_stream)
    src = [1.0 + torch.rand(inst.shape(nf), generator=gen, dtype=torch.float64, device="cuda") for nf in (6, 3)]
    host = [torch.zeros(inst.shape(nf), dtype=torch.float64).pin_memory() for nf in (6, 3)]
    torch.cuda.synchronize()
    for _ in range(2):  # (the second time the staging slots have been used)
        for h in host:
            h.zero_()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(100_000_000)  # about 50 ms
            for h, s in zip(host, src):
                h.copy_(s, non_blocking=True)
        inst.upload(host[0].numpy(), host[1].numpy())
        d = inst.download(("gas", "face_b"))
        np.testing.assert_array_equal(d["gas"], src[0].cpu().numpy())
        np.testing.assert_array_equal(d["face_b"], src[1].cpu().numpy())
    inst.close()
