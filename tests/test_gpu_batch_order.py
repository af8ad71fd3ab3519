"""A batch's upload and download come behind the work of the legacy default
stream that writes or reads the same page-locked buffer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DELAY = 200_000_000   # cycles: about a tenth of a second


def test_upload_and_download_follow_the_default_stream():
    import torch

    from lsmlib_b200 import batched, gpu
    lib = gpu.load()
    b = batched.Batch([(40, 36, 30), (20, 44, 18)], [(0.1, 0.1, 0.1)] * 2, 8)
    rng = np.random.default_rng(3)
    want = rng.standard_normal(b.total)
    old = rng.standard_normal(b.total)
    g = torch.from_numpy(want).cuda()
    g2 = torch.zeros_like(g)
    host = torch.zeros(b.total, dtype=torch.float64, pin_memory=True)
    torch.cuda.synchronize()
    # the buffer is still being written when the upload is called
    torch.cuda._sleep(DELAY)
    host.copy_(g, non_blocking=True)
    assert lib.lsmgpu_batch_upload(b.h, host.data_ptr()) == 0
    got = np.zeros(b.total)
    assert lib.lsmgpu_batch_download(b.h, got.ctypes.data) == 0
    assert np.array_equal(got, want)
    # and still being read when the download is called
    host.copy_(torch.from_numpy(old))
    torch.cuda._sleep(DELAY)
    g2.copy_(host, non_blocking=True)
    assert lib.lsmgpu_batch_download(b.h, host.data_ptr()) == 0
    torch.cuda.synchronize()
    assert np.array_equal(g2.cpu().numpy(), old)
    assert np.array_equal(host.numpy(), want)
