"""Large host copies in pieces: every byte, at lengths around the pieces' and the
plain copy's limits, from several threads at once, after the slots were
handed back, and from pinned memory."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def batch_of(nbytes):
    """A one-grid batch whose packed buffer has about nbytes (x, y extents fixed)."""
    from lsmlib_b200 import batched
    nz = max(2, round(nbytes / 8 / (58 * 50)) - 6)
    return batched.Batch([(52, 44, nz)], [(0.1, 0.1, 0.1)], 8)


def roundtrip(b, seed, out):
    rng = np.random.default_rng(seed)
    f = np.asfortranarray(rng.standard_normal(b.shape(0)))
    b.upload([f])
    out.append(np.array_equal(b.download()[0], f))


@pytest.mark.parametrize("nbytes", [MB, 8 * MB - 30000, 8 * MB + 30000, 10 * MB, 16 * MB + 23000,
                                    33 * MB])
def test_roundtrip(nbytes):
    from lsmlib_b200 import gpu
    out = []
    b = batch_of(nbytes)
    roundtrip(b, 1, out)
    assert gpu.load().lsmgpu_release_scratch() == 0
    roundtrip(b, 2, out)
    assert out == [True, True]


def test_threads():
    out = []
    batches = [batch_of(12 * MB + 50000 * q) for q in range(4)]
    threads = [threading.Thread(target=roundtrip, args=(b, q, out))
               for q, b in enumerate(batches)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert out == [True] * 4


def test_pinned_destination():
    import ctypes

    from lsmlib_b200 import gpu
    b = batch_of(12 * MB)
    out = []
    roundtrip(b, 5, out)
    lib = gpu.load()
    p = lib.lsmgpu_host_alloc(b.total * 8)
    try:
        assert lib.lsmgpu_batch_download(b.h, p) == 0
        got = np.ctypeslib.as_array((ctypes.c_double * b.total).from_address(p))
        assert np.array_equal(b.unpack(got)[0], b.download()[0]) and out == [True]
    finally:
        lib.lsmgpu_host_free(p)
