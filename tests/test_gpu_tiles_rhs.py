"""The pair kernels' tiling, right-hand sides and CFL speeds alone: both
precisions against the FP64 one-cell strict kernels on the same (FP32) inputs.
A stage with a huge dt returns dt times its right-hand side."""
import numpy as np
import pytest

from test_gpu_tiles import ADVECT, NORMAL, REINIT, SIZES

pytestmark = pytest.mark.gpu

G = 3
DX = (0.1, 0.11, 0.12)


def setup(n):
    shape = tuple(m + 2 * G for m in n)
    gb = tuple(v for m in n for v in (-G, m - 1 + G))
    fb = tuple(v for m in n for v in (0, m - 1))
    x = np.meshgrid(*[np.arange(s) * 0.1 for s in shape], indexing="ij")
    phi = np.sin(x[0]) * np.cos(0.7 * x[1]) + 0.3 * x[2] - 0.4
    vel = (1 + 0.5 * np.sin(x[1]), np.cos(x[0] + x[2]), np.sin(x[2]) - 0.2)
    return gb, fb, [a.astype(np.float32) for a in (phi,) + vel]


def upload(a, precision):
    from lsmlib_b200 import gpu
    return gpu.DeviceArray.from_host(
        np.asfortranarray(a.astype(np.float64 if precision == 8 else np.float32)))


@pytest.mark.parametrize("n", SIZES)
def test_right_hand_sides(n):
    from lsmlib_b200 import integrator
    gb, fb, arrays = setup(n)
    inner = tuple(slice(G, G + m) for m in n)
    phi = arrays[0].astype(np.float64)
    steep = max(float(np.max(np.abs(np.diff(phi, axis=d)))) / DX[d] for d in range(3))
    big = 2.0 ** 40
    prev = integrator.get_fp_mode()
    try:
        for kind, aux, lipschitz in ((ADVECT, arrays[1:], 4.0), (NORMAL, arrays[1:2], 3.0),
                                     (REINIT, [], 3.0)):
            out = {}
            for mode, precision in ((integrator.FP_STRICT, 8), (integrator.FP_FAST, 8),
                                    (integrator.FP_FAST, 4)):
                integrator.set_fp_mode(mode)
                src = upload(arrays[0], precision)
                o = upload(np.full(phi.shape, 7.0), precision)
                integrator.stage(kind, precision, o, src, src,
                                 [upload(a, precision) for a in aux], gb, fb, DX, big, 1,
                                 bc_mask=0)
                got = o.download().astype(np.float64)
                out[mode, precision] = got[inner] / big
                got[inner] = 7.0
                assert np.all(got == 7.0)
            want = out[integrator.FP_STRICT, 8]
            # FP32: a weight's relative error is at most 8 u D^2 / (S + eps), the
            # candidates it moves between lie within sqrt(S) of each other, and
            # eps = 1e-6 D^2: 2.4e-4 D / dx at worst (S = eps) for a derivative
            tol = {8: 1e-12, 4: 2.5e-4}
            for precision in (8, 4):
                err = np.max(np.abs(out[integrator.FP_FAST, precision] - want))
                assert err <= tol[precision] * steep * lipschitz, (kind, precision, err)
    finally:
        integrator.set_fp_mode(prev)


@pytest.mark.parametrize("precision", [8, 4])
@pytest.mark.parametrize("n", [n for n in SIZES if min(n) > 1])   # what the driver takes
def test_cfl_speed_of_every_column(n, precision):
    """dt follows the fastest cell, at either end of the box, and no slower value
    of an earlier call is left in the blocks without work."""
    from lsmlib_b200 import integrator
    gb, fb, arrays = setup(n)
    prev = integrator.get_fp_mode()
    try:
        for peak in (tuple(G for _ in n), tuple(G + m - 1 for m in n)):
            dts = []
            for mode, prec in ((integrator.FP_STRICT, 8), (integrator.FP_FAST, precision)):
                integrator.set_fp_mode(mode)
                ws = integrator.Workspace(gb, prec)
                F = np.ones(arrays[0].shape, dtype=np.float32)
                ws.normal(upload(arrays[0], prec), upload(1e4 * F, prec), fb, DX)
                F[peak] = 50.0
                ws.set_time(0.0)
                ws.normal(upload(arrays[0], prec), upload(F, prec), fb, DX)
                dts.append(ws.time()[1])
                ws.close()
            # the speed is a ratio of derivatives: their relative error, 2.4e-4
            # of the largest in FP32, three times over
            assert abs(dts[1] - dts[0]) <= (1e-12 if precision == 8 else 1e-3) * dts[0]
    finally:
        integrator.set_fp_mode(prev)
