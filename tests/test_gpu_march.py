"""The march kernel at the limits of its choices, bit for bit against the heap
march that pops ties by index: grids on both sides of the one-cluster limit
and of the longer threshold step, lists shorter than a warp, tied keys (a
plane front: every point of a plane ties), and spacings at which the quadratic's
terms are tiny or huge."""
import numpy as np
import pytest

import oracle
from test_fmm_golden import seeded_mask, seeded_spheres
from test_gpu_distance import gpu_distance, lib, same_bits  # noqa: F401

pytestmark = pytest.mark.gpu

# 39^3 fits one cluster, 40^3 does not; 72^3 takes the longer step at order 1,
# 88^3 the shorter; one row, one column, two planes
SHAPES = [(39, 39, 39), (40, 40, 40), (72, 72, 72), (88, 88, 88), (1, 1, 40), (1, 50, 1),
          (2, 90, 30), (1, 200, 33)]


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_distance_sizes(lib, shape, order):  # noqa: F811
    phi, dx = seeded_spheres(shape, sum(shape))
    mask = seeded_mask(shape, sum(shape)) if shape[0] == 40 else None
    want = oracle.oracle_fmm(ordered=True)(phi, order, dx, mask)
    got, _ = gpu_distance(lib, phi, order, dx, mask)
    assert same_bits(got, want)


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("scale", [1e-9, 1.0, 1e7])
def test_distance_ties_and_scales(lib, scale, order):  # noqa: F811
    z, y, x = np.meshgrid(*[np.arange(m, dtype=float) for m in (14, 18, 22)], indexing="ij")
    for phi in (x - 7.3, np.maximum(x - 7.25, y - 9.25)):
        want = oracle.oracle_fmm(ordered=True)(phi * scale, order, [scale] * 3, None)
        got, _ = gpu_distance(lib, phi * scale, order, [scale] * 3)
        assert same_bits(got, want)
