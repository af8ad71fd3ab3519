"""The pair kernels' tiling -- narrow last columns (rows of 8 or 4 pairs), slabs
of few planes, ragged edges -- against the one-cell strict kernels, which are
pinned to the oracle: every fill-box cell of one stage, and no cell beside
the fill box written."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# x extents around the narrow columns' limits (1, 8, 9, 16, 17 columns left),
# y extents around 8, 16 and 32 rows, z extents of few and several slabs
SIZES = [(33, 33, 5), (8, 31, 9), (9, 33, 4), (40, 32, 3), (41, 17, 7), (16, 16, 12),
         (48, 9, 23), (49, 8, 6), (17, 7, 3), (64, 24, 2), (1, 65, 1), (31, 3, 40)]
ADVECT, NORMAL, REINIT = 0, 1, 2


@pytest.mark.parametrize("precision", [8, 4])
@pytest.mark.parametrize("n", SIZES)
def test_stage_matches_one_cell_kernels(n, precision):
    from lsmlib_b200 import gpu, integrator
    dt = np.float64 if precision == 8 else np.float32
    rng = np.random.default_rng(sum(n))
    g = 3
    shape = tuple(m + 2 * g for m in n)
    gb = tuple(v for m in n for v in (-g, m - 1 + g))
    fb = tuple(v for m in n for v in (0, m - 1))
    x = np.meshgrid(*[np.arange(s) * 0.1 for s in shape], indexing="ij")
    phi = np.sin(x[0]) * np.cos(0.7 * x[1]) + 0.3 * x[2] + 0.02 * rng.standard_normal(shape) - 0.4
    dev = [gpu.DeviceArray.from_host(np.asfortranarray(a.astype(dt))) for a in
           (phi, phi + 0.01, 1 + 0.5 * np.sin(x[1]), np.cos(x[0] + x[2]), np.sin(x[2]) - 0.2)]
    prev = integrator.get_fp_mode()
    try:
        for kind, aux in ((ADVECT, dev[2:5]), (NORMAL, [dev[2]]), (REINIT, [])):
            out = []
            for mode in (integrator.FP_FAST, integrator.FP_STRICT):
                integrator.set_fp_mode(mode)
                o = gpu.DeviceArray.from_host(np.full(shape, 7.0, dtype=dt, order="F"))
                integrator.stage(kind, precision, o, dev[0], dev[1], aux, gb, fb,
                                 (0.1, 0.11, 0.12), 0.02, 33, bc_mask=0)
                out.append(o.download().astype(np.float64))
            inner = tuple(slice(g, g + m) for m in n)
            # the bound of the fused parity tests, and FP32's: its faces carry
            # up to ~20 roundings of values of the size of phi / dx
            tol = 1e-12 if precision == 8 else 1e-5
            scale = np.max(np.abs(out[1][inner]))
            assert np.max(np.abs(out[0][inner] - out[1][inner])) <= tol * scale
            out[0][inner] = 7.0
            assert np.all(out[0] == 7.0)
    finally:
        integrator.set_fp_mode(prev)
