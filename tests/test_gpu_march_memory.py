"""The march's memory: its scratch per point, and lists longer than its threads,
whose results wait in the output array: every point of the output is still
written, front points and points outside the mask among them."""
import ctypes

import numpy as np
import pytest

import oracle
from test_gpu_distance import gpu_distance, lib, same_bits  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2])
def test_lists_longer_than_the_threads(lib, order):  # noqa: F811
    # a wavy front across a wide, flat grid: some 90,000 points a step, for
    # 148 x 512 (order 1) or 148 x 384 threads
    nz, ny, nx = 20, 280, 330
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    phi = z - 9.3 + 0.9 * np.sin(0.11 * x) * np.cos(0.07 * y)
    mask = np.where((x - 200) ** 2 + (y - 100) ** 2 < 900, -1.0, 1.0)
    want = oracle.oracle_fmm(ordered=True)(phi, order, [1.0, 1.0, 1.0], mask)
    got, _ = gpu_distance(lib, phi, order, [1.0, 1.0, 1.0], mask)
    assert same_bits(got, want)


def test_scratch_per_point(lib):  # noqa: F811
    import torch

    n = 224
    ax = np.arange(n) - 0.45 * n
    phi = np.sqrt(ax[:, None, None] ** 2 + ax[None, :, None] ** 2 + ax[None, None, :] ** 2) - 60
    src = torch.from_numpy(phi).cuda()
    out = torch.empty_like(src)
    dims = (ctypes.c_int * 3)(n, n, n)
    h = (ctypes.c_double * 3)(1.0, 1.0, 1.0)
    torch.cuda.synchronize()
    assert lib.lsmgpu_release_scratch() == 0
    assert lib.lsmgpu_distance_function3d(out.data_ptr(), src.data_ptr(), None, 1, dims, h,
                                          None) == 0   # (modules loaded, buffers made)
    torch.cuda.synchronize()
    assert lib.lsmgpu_release_scratch() == 0
    free = torch.cuda.mem_get_info()[0]
    assert lib.lsmgpu_distance_function3d(out.data_ptr(), src.data_ptr(), None, 1, dims, h,
                                          None) == 0
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]   # freed scratch stays mapped up to 8 GiB
    assert lib.lsmgpu_release_scratch() == 0
    # 82 bytes a point, eleven buffers in the pool's units of at most 32 MB
    assert 40 * n ** 3 < used < 82 * n ** 3 + (64 << 20)
