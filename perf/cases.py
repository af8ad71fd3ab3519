"""The workloads whose speed is tracked: what programs have this library do.

Every case goes through the public entry points: ``pylsmlib`` on torch
tensors (level set time stepping, reinitialization, the adjoint, the fast
marching routines), ``lsmlib_b200.batched`` (many small grids) and
``lsmlib_b200.gpu.toolbox()`` (the reference-compatible routines on device
arrays).  Inputs are unions of spheres as in ``lsmlib_b200.workloads``, drawn
from the seed.

``exact`` holds an independent FP64 formulation in plain torch: HJ-WENO5,
Godunov and upwind right-hand sides, TVD-RK3, the CFL conditions, the face
ghost cells, the batched and adjoint models, and the first-order fast
marching fixed point.
"""
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import pylsmlib
from lsmlib_b200 import adjoint, batched, gpu, integrator
from lsmlib_b200.toolbox import Field

TINY, ZERO_TOL = 1e-99, 1e-11
DTYPES = {"float64": torch.float64, "float32": torch.float32}


def listed():
    return [
        # A small grid stepped with reinitialization, as examples and tests do:
        # a chain of short launches.
        {"name": "normal_32", "kind": "normal", "nx": 32, "ny": 32, "nz": 32,
         "dtype": "float64", "boundary": "linear", "steps": 10},
        # The benchmark configuration: 256^3 FP64, ten steps and the 20
        # reinitialization pseudo-steps after them.
        {"name": "normal_256", "kind": "normal", "nx": 256, "ny": 256, "nz": 256,
         "dtype": "float64", "boundary": "linear", "steps": 10},
        # The FP32 form on a ragged grid with Neumann faces.
        {"name": "normal_f32_ragged", "kind": "normal", "nx": 211, "ny": 163, "nz": 150,
         "dtype": "float32", "boundary": "copy", "steps": 10},
        # Reinitialization alone, the sign from phi0, on a ragged mid-size grid.
        {"name": "reinit_odd", "kind": "reinit", "nx": 129, "ny": 97, "nz": 131,
         "dtype": "float64", "boundary": "linear", "steps": 20},
        # Passive transport by velocity arrays in a periodic box (a flow solver's
        # interface tracking).
        {"name": "external_periodic", "kind": "external", "nx": 160, "ny": 144, "nz": 130,
         "dtype": "float64", "boundary": "periodic", "steps": 10},
        # The deformation benchmark's grid (512^3 FP64): the largest fields.
        {"name": "deformation_512", "kind": "deformation", "nx": 512, "ny": 512, "nz": 512,
         "dtype": "float64", "boundary": "linear", "steps": 4},
        # The same flow in FP32 with the tiles near the interface in FP64.
        {"name": "deformation_band", "kind": "deformation", "nx": 192, "ny": 176, "nz": 160,
         "dtype": "float32", "boundary": "linear", "steps": 10},
        # Many uneven grids advanced together and read back (a parameter study).
        {"name": "batch_48", "kind": "batch", "grids": 48, "lo": 24, "hi": 96,
         "dtype": "float64", "boundary": "periodic", "steps": 50},
        # One gradient of an inverse problem: forward model and reverse sweep.
        {"name": "adjoint_80", "kind": "adjoint", "nx": 80, "ny": 72, "nz": 64,
         "lattice": 8, "steps": 24},
        # Re-distancing of host arrays by fast marching, second order.
        {"name": "distance_3d", "kind": "march", "solver": "distance", "nx": 128, "ny": 112,
         "nz": 120, "order": 2},
        # Extension velocities on a 2D slice, first order (latency bound).
        {"name": "extension_2d", "kind": "march", "solver": "extension", "nx": 301, "ny": 237,
         "nz": 1, "order": 1},
        # A host code's own Runge-Kutta stage through the drop-in routines.
        {"name": "toolbox_stage", "kind": "toolbox", "nx": 160, "ny": 128, "nz": 120},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["normal", "normal", "reinit", "external", "deformation", "batch",
                       "adjoint", "march", "march", "toolbox"])
    boundary = rng.choice(["linear", "linear", "copy", "periodic"])
    dtype = rng.choice(["float64", "float64", "float32"])

    def dims(lo, hi):
        return {"nx": _log(rng, lo, hi), "ny": _log(rng, lo, hi), "nz": _log(rng, lo, hi)}
    if kind in ("normal", "external"):
        return {"kind": kind, **dims(24, 256), "dtype": dtype, "boundary": boundary, "steps": 10}
    if kind == "reinit":
        return {"kind": kind, **dims(24, 256), "dtype": dtype, "boundary": boundary, "steps": 20}
    if kind == "deformation":
        return {"kind": kind, **dims(32, 384), "dtype": dtype, "boundary": "linear",
                "steps": rng.randint(3, 8)}
    if kind == "batch":
        lo = rng.randint(12, 40)
        return {"kind": kind, "grids": _log(rng, 6, 48), "lo": lo,
                "hi": rng.randint(lo + 8, 96), "dtype": dtype, "boundary": boundary,
                "steps": rng.randint(10, 50)}
    if kind == "adjoint":
        return {"kind": kind, **dims(24, 96), "lattice": rng.randint(4, 9),
                "steps": rng.randint(6, 20)}
    if kind == "march":
        flat = rng.random() < 0.5
        d = dims(64, 512) if flat else dims(32, 128)
        return {"kind": kind, "solver": rng.choice(["distance", "extension", "eikonal"]),
                "nx": d["nx"], "ny": d["ny"], "nz": 1 if flat else d["nz"],
                "order": rng.choice([1, 2])}
    return {"kind": kind, **dims(24, 192)}


# -- inputs -------------------------------------------------------------------------
def _spheres(seed, extent, coords):
    """min_l |x - c_l| - r_l of six spheres drawn for a box of half-widths ``extent``."""
    rng = np.random.default_rng(seed)
    phi = None
    used = [e for e in extent if e > 0]
    for _ in range(6):
        c = rng.uniform(-0.6, 0.6, size=3) * np.asarray(extent)
        r = float(rng.uniform(0.1, 0.3)) * min(used)
        d = torch.zeros((), dtype=torch.float64, device="cuda")
        for a in range(3):
            d = d + (coords[a] - float(c[a])) ** 2
        d = torch.sqrt(d) - r
        phi = d if phi is None else torch.minimum(phi, d)
    return phi


def _grid(case, unit=False):
    """Isotropic spacing, the longest axis 2 long around 0 (1 long from 0: ``unit``)."""
    n = (case["nx"], case["ny"], case["nz"])
    h = (1.0 if unit else 2.0) / max(n)
    lo = [0.0 if unit else -0.5 * v * h for v in n]
    hi = [a + v * h for a, v in zip(lo, n)]
    return pylsmlib.Grid.set_grid_dims(n, lo, hi, "VERY_HIGH")


def _axes(g):
    """x, y, z of the grid points, broadcastable to g.shape."""
    out = []
    for a in range(3):
        t = g.x_lo_ghostbox[a] + g.dx[a] * torch.arange(g.grid_dims_ghostbox[a], device="cuda",
                                                        dtype=torch.float64)
        out.append(t.reshape([-1 if b == 2 - a else 1 for b in range(3)]))
    return out


def _fields(case, seed):
    """The grid and the FP64 inputs of a time-stepping case."""
    kind = case["kind"]
    g = _grid(case, unit=kind == "deformation")
    x, y, z = _axes(g)
    rng = np.random.default_rng(seed + 1)
    s = [float(v) for v in rng.uniform(0.0, 2 * math.pi, size=6)]
    if kind == "deformation":
        c = [0.35 * n * h + float(v) for n, h, v in
             zip(g.grid_dims, g.dx, rng.uniform(-0.02, 0.02, size=3))]
        m = min(n * h for n, h in zip(g.grid_dims, g.dx))
        phi = torch.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) - 0.15 * m
        return g, phi, []
    half = [0.5 * n * h for n, h in zip(g.grid_dims, g.dx)]
    phi = _spheres(seed, half, (x, y, z))
    if kind == "reinit":   # not a distance function: a smooth factor, same zero level set
        phi = phi * (1.2 + 0.5 * torch.sin(3 * x + s[0]) * torch.sin(2 * y + s[1])
                     * torch.cos(z + s[2]))
        return g, phi, []
    if kind == "external":
        u = 0.8 + 0.4 * torch.sin(math.pi * y + s[0]) * torch.cos(math.pi * z + s[1]) + 0 * phi
        v = -0.3 + 0.6 * torch.sin(math.pi * z + s[2]) * torch.cos(math.pi * x + s[3]) + 0 * phi
        w = 0.5 * torch.cos(math.pi * x + s[4]) * torch.cos(math.pi * y + s[5]) + 0 * phi
        return g, phi, [u, v, w]
    f = 1.0 + 0.2 * (torch.sin(4 * math.pi * x + s[0]) * torch.sin(4 * math.pi * y + s[1])
                     * torch.sin(4 * math.pi * z + s[2]))
    return g, phi, [f]


def _batch_inputs(case, seed):
    rng = np.random.default_rng([case["grids"], case["lo"], case["hi"]])   # sizes by case
    sizes = [tuple(int(v) for v in rng.integers(case["lo"], case["hi"] + 1, size=3))
             for _ in range(case["grids"])]
    dx = [tuple(2.0 / v for v in n) for n in sizes]
    rng = np.random.default_rng(seed)
    vel = [tuple(float(v) for v in rng.uniform(-1, 1, size=3)) for _ in sizes]
    npdt = np.float64 if case["dtype"] == "float64" else np.float32
    fields = []
    for k, (n, h) in enumerate(zip(sizes, dx)):
        ax = [(-1 + (torch.arange(-3, n[a] + 3, device="cuda", dtype=torch.float64) + 0.5) * h[a])
              .reshape([-1 if b == 2 - a else 1 for b in range(3)]) for a in range(3)]
        phi = _spheres(seed * 1000 + k, (1.0, 1.0, 1.0), ax)
        fields.append(np.asfortranarray(phi.cpu().numpy().T.astype(npdt)))
    return sizes, dx, vel, fields


def _adjoint_inputs(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    h = 2.0 / max(n)
    lo = tuple(-0.5 * v * h for v in n)
    rng = np.random.default_rng(seed)
    m = case["lattice"]
    theta = rng.normal(0.0, 0.5, size=(3, m, m, m))
    ax = [lo[a] + (np.arange(-3, n[a] + 3) + 0.5) * h for a in range(3)]
    x, y, z = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    e = [0.5 * v * h for v in n]
    c = rng.uniform(-0.05, 0.05, size=3)
    r = 0.3 * min(e)
    phi0 = np.asfortranarray(np.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) - r)
    target = np.asfortranarray(
        (np.sqrt((x / 0.4) ** 2 + (y / 0.3) ** 2 + (z / 0.25) ** 2) - 1.0) * 0.25)
    return n, (h, h, h), lo, theta, phi0, target, 1.5 * h


def _march_inputs(case, seed):
    """phi (C order, (nz, ny, nx) or (ny, nx)), per-axis dx, and the sources or speed."""
    n = (case["nx"], case["ny"], case["nz"])
    h = 2.0 / (max(n) - 1)
    half = [0.5 * (v - 1) * h for v in n]
    ax = [(-half[a] + h * torch.arange(n[a], device="cuda", dtype=torch.float64))
          .reshape([-1 if b == 2 - a else 1 for b in range(3)]) for a in range(3)]
    x, y, z = ax
    phi = _spheres(seed, half, ax)
    s = [float(v) for v in np.random.default_rng(seed + 1).uniform(0, 2 * math.pi, size=3)]
    phi = phi * (1.2 + 0.5 * torch.sin(3 * x + s[0]) * torch.sin(2 * y + s[1])
                 * torch.cos(3 * z + s[2]))
    extra = []
    if case["solver"] == "extension":
        extra = [1.0 + 0.3 * torch.sin(4 * x + s[1]) * torch.cos(3 * y + s[2]) + 0 * phi,
                 torch.cos(2 * x + s[0]) + 0.5 * torch.sin(5 * y + z + s[1]) + 0 * phi]
    elif case["solver"] == "eikonal":
        extra = [1.0 + 0.4 * torch.sin(4 * x + s[1]) * torch.cos(3 * y + s[2] + z) + 0 * phi]
    drop = (lambda t: t[0]) if n[2] == 1 else (lambda t: t)
    return (drop(phi).contiguous().cpu().numpy(), h,
            [drop(t).contiguous().cpu().numpy() for t in extra])


class _View:
    """A torch tensor as the data of a toolbox Field (x fastest)."""

    def __init__(self, t):
        self.tensor, self.ptr = t, t.data_ptr()
        self.shape = tuple(reversed(t.shape))


PM = ("phi_x_plus", "phi_y_plus", "phi_z_plus", "phi_x_minus", "phi_y_minus", "phi_z_minus")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sizes, dx, vel, fields = _batch_inputs(case, seed)
        b = batched.Batch(sizes, dx, 8 if case["dtype"] == "float64" else 4)
        b.upload(fields)
        b.set_velocity(vel, 0.5)
        b.set_bc({"linear": batched.BC_LINEAR, "copy": batched.BC_COPY,
                  "periodic": batched.BC_PERIODIC}[case["boundary"]])
        b.autotune(report=False)
        return {"kind": kind, "batch": b, "steps": case["steps"]}
    if kind == "adjoint":
        n, dx, lo, theta, phi0, target, eps = _adjoint_inputs(case, seed)
        p = adjoint.AdvectionAdjoint(n, dx, lo, case["lattice"], case["steps"],
                                     max(1, int(math.ceil(math.sqrt(case["steps"])))))
        p.set_theta(theta)
        p.set_dt(p.cfl_dt(0.5))
        p.set_fields(phi0, target, eps)
        return {"kind": kind, "problem": p, "theta": torch.tensor(theta, requires_grad=True),
                "phi0": torch.tensor(phi0, requires_grad=True)}
    if kind == "march":
        phi, dx, extra = _march_inputs(case, seed)
        return {"kind": kind, "phi": phi, "dx": dx, "extra": extra, "solver": case["solver"],
                "order": case["order"]}
    g, phi, extra = _fields(case if kind != "toolbox" else {**case, "kind": "normal"}, seed)
    if kind == "toolbox":
        lo = (0, 0, 0)
        names = PM + ("lse_rhs", "u_stage1", "D1")
        f = {k: Field(_View(torch.zeros(g.shape, device="cuda", dtype=torch.float64)), lo)
             for k in names}
        f["phi"] = Field(_View(phi.contiguous()), lo)
        f["vel_n"] = Field(_View(extra[0].contiguous()), lo)
        return {"kind": kind, "tb": gpu.toolbox(), "grid": g, "fields": f}
    dt = DTYPES[case["dtype"]]
    phi = phi.to(dt).contiguous()
    policy = None
    if kind == "deformation" and dt == torch.float32:
        policy = integrator.FP64_SIGN | integrator.STOCH_ROUND | integrator.FP64_BAND
    integ = pylsmlib.LevelSetIntegrator(g, dtype=dt, boundary=case["boundary"],
                                        use_phi0_for_sgn=kind == "reinit", fp32_policy=policy)
    return {"kind": kind, "integ": integ, "phi0": phi, "phi": phi.clone(),
            "extra": [t.to(dt).contiguous() for t in extra], "steps": case["steps"]}


def run(s):
    kind = s["kind"]
    if kind == "batch":
        s["batch"].advect(s["steps"])
        return s["batch"].download()
    if kind == "adjoint":
        th, ph = s["theta"], s["phi0"]
        th.grad = ph.grad = None
        loss = pylsmlib.advection_loss(th, ph, s["problem"])
        loss.backward()
        return {"loss": loss.detach(), "theta": th.grad, "phi0": ph.grad}
    if kind == "march":
        if s["solver"] == "distance":
            return [pylsmlib.computeDistanceFunction(s["phi"], s["dx"], s["order"])]
        if s["solver"] == "extension":
            return list(pylsmlib.computeExtensionFields(s["phi"], np.stack(s["extra"]), s["dx"],
                                                        s["order"]))
        return [pylsmlib.solveEikonalEquation(s["phi"], s["extra"][0], s["dx"], s["order"])]
    if kind == "toolbox":
        return _toolbox_stage(s)
    # the program's level set starts from its initial state in every pass
    s["phi"].copy_(s["phi0"])
    if kind == "normal":
        s["integ"].advance_normal(s["phi"], s["extra"][0], nsteps=s["steps"])
    elif kind == "reinit":
        s["integ"].reinitialize(s["phi"], iters=s["steps"])
    elif kind == "external":
        s["integ"].advance_external(s["phi"], s["extra"], nsteps=s["steps"])
    else:
        s["integ"].advance_deformation(s["phi"], period=3.0, t_end=3.0, nsteps=s["steps"])
    return s["phi"]


def _toolbox_stage(s):
    tb, g, f = s["tb"], s["grid"], s["fields"]
    d = dict(zip(("dx", "dy", "dz"), g.dx))

    def pick(*names):
        return {k: f[k] for k in names}
    tb.LSM3D_HJ_WENO5(pick("phi", "D1", *PM), g.fb, **d)
    tb.LSM3D_ZERO_OUT_LEVEL_SET_EQN_RHS(pick("lse_rhs"))
    tb.LSM3D_ADD_NORMAL_VEL_TERM_TO_LSE_RHS(pick("lse_rhs", "vel_n", *PM), g.fb)
    dt = tb.LSM3D_COMPUTE_STABLE_NORMAL_VEL_DT(pick("vel_n", *PM), g.fb, cfl_number=0.5, **d)["dt"]
    tb.LSM3D_TVD_RK3_STAGE1({"u_stage1": f["u_stage1"], "u_cur": f["phi"], "rhs": f["lse_rhs"]},
                            g.fb, dt=dt)
    for face in range(6):
        tb.LSM3D_LINEAR_EXTRAPOLATION({"phi": f["u_stage1"]}, g.fb, bdry_location_idx=face)
    out = {k: f[k].data.tensor for k in PM + ("lse_rhs", "u_stage1")}
    out["dt"] = dt
    return out


def work(case):
    """Bytes a pass reads or writes once and the operations of the scheme.

    A WENO5 side is 65 operations (smoothness indicators, weights, candidates),
    the two sides of a face sharing their indicators 100; upwind kinds take one
    side per axis, two-sided kinds a face per axis."""
    kind = case["kind"]
    if kind == "batch":
        cells = case["grids"] * (0.5 * (case["lo"] + case["hi"])) ** 3
        w = 8 if case["dtype"] == "float64" else 4
        return {"bytes": cells * w * 8 * case["steps"], "flops": cells * 3 * 205 * case["steps"]}
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "adjoint":   # forward, recomputation and transpose of every stage
        return {"bytes": cells * 8 * 3 * case["steps"] * (6 + 6 + 12),
                "flops": cells * 3 * case["steps"] * (205 + 205 + 900)}
    if kind == "march":
        arrays = {"distance": 2, "extension": 6, "eikonal": 3}[case["solver"]]
        return {"bytes": cells * 8 * arrays, "flops": cells * 60 * case["order"]}
    if kind == "toolbox":
        return {"bytes": cells * 8 * (1 + 6 + 1 + 1 + 1), "flops": cells * (3 * 130 + 60)}
    w = 8 if case["dtype"] == "float64" else 4
    if kind == "reinit":
        return {"bytes": cells * w * 8 * case["steps"], "flops": cells * 3 * 330 * case["steps"]}
    if kind == "external":
        return {"bytes": cells * w * 17 * case["steps"], "flops": cells * 3 * 205 * case["steps"]}
    if kind == "deformation":
        return {"bytes": cells * w * 8 * case["steps"], "flops": cells * 3 * 215 * case["steps"]}
    # normal: three stages a step, the reinitialization after every tenth
    per, re = 3 * 330, 20 * (case["steps"] // 10)
    return {"bytes": cells * w * (11 * case["steps"] + 8 * re),
            "flops": cells * (per * case["steps"] + 3 * 330 * re)}


# -- FP64 values in plain torch ----------------------------------------------------------
def _side(v1, v2, v3, v4, v5):
    s1 = 13.0 / 12.0 * (v1 - 2 * v2 + v3) ** 2 + 0.25 * (v1 - 4 * v2 + 3 * v3) ** 2
    s2 = 13.0 / 12.0 * (v2 - 2 * v3 + v4) ** 2 + 0.25 * (v2 - v4) ** 2
    s3 = 13.0 / 12.0 * (v3 - 2 * v4 + v5) ** 2 + 0.25 * (3 * v3 - 4 * v4 + v5) ** 2
    m = torch.maximum(torch.maximum(torch.maximum(v1 * v1, v2 * v2),
                                    torch.maximum(v3 * v3, v4 * v4)), v5 * v5)
    eps = 1e-6 * m + TINY
    a1, a2, a3 = 0.1 / (s1 + eps) ** 2, 0.6 / (s2 + eps) ** 2, 0.3 / (s3 + eps) ** 2
    p1 = v1 / 3 - 7 * v2 / 6 + 11 * v3 / 6
    p2 = -v2 / 6 + 5 * v3 / 6 + v4 / 3
    p3 = v3 / 3 + 5 * v4 / 6 - v5 / 6
    return (a1 * p1 + a2 * p2 + a3 * p3) / (a1 + a2 + a3)


def _box(fb):
    """Slices (z, y, x) of the fill box."""
    return tuple(slice(fb[2 * a], fb[2 * a + 1] + 1) for a in (2, 1, 0))


def _pm(phi, fb, axis, h):
    """phi^+ and phi^- of one axis (0 = x) over the fill box."""
    d = 2 - axis
    idx = list(_box(fb))
    lo, n = fb[2 * axis], fb[2 * axis + 1] - fb[2 * axis] + 1
    idx[d] = slice(lo - 3, lo + n + 3)
    v = torch.diff(phi[tuple(idx)], dim=d) / h   # v[m]: between cells lo-3+m and lo-2+m
    w = [v.narrow(d, m, n) for m in range(6)]
    return _side(w[5], w[4], w[3], w[2], w[1]), _side(w[0], w[1], w[2], w[3], w[4])


def _face_ghosts(phi, fb, boundary):
    """The three ghost layers beyond each face of the fill box, written in place."""
    for axis in range(3):
        d = 2 - axis
        lo, hi = fb[2 * axis], fb[2 * axis + 1]
        n = hi - lo + 1

        def at(i):
            idx = list(_box(fb))
            idx[d] = i
            return tuple(idx)
        for q in (1, 2, 3):
            if boundary == "periodic":
                phi[at(lo - q)] = phi[at(lo - q + n)]
                phi[at(hi + q)] = phi[at(hi + q - n)]
            elif boundary == "copy":
                phi[at(lo - q)] = phi[at(lo)]
                phi[at(hi + q)] = phi[at(hi)]
            else:
                phi[at(lo - q)] = phi[at(lo)] + (phi[at(lo)] - phi[at(lo + 1)]) * q
                phi[at(hi + q)] = phi[at(hi)] + (phi[at(hi)] - phi[at(hi - 1)]) * q


def _rk3(phi, rhs, fb, boundary, dt, c=(0.0, 1.0, 0.5)):
    """One TVD-RK3 step in place; rhs(array, stage time fraction)."""
    b = _box(fb)
    _face_ghosts(phi, fb, boundary)
    p1 = phi.clone()
    p1[b] = phi[b] + dt * rhs(phi, c[0])
    _face_ghosts(p1, fb, boundary)
    p2 = phi.clone()
    p2[b] = 0.75 * phi[b] + 0.25 * (p1[b] + dt * rhs(p1, c[1]))
    _face_ghosts(p2, fb, boundary)
    phi[b] = phi[b] / 3 + 2.0 / 3.0 * (p2[b] + dt * rhs(p2, c[2]))


def _normal_rhs(phi, f, fb, h):
    g = 0
    for a in range(3):
        p, m = _pm(phi, fb, a, h[a])
        g = g + torch.where(f > 0, torch.maximum(torch.clamp(m, min=0) ** 2,
                                                 torch.clamp(p, max=0) ** 2),
                            torch.maximum(torch.clamp(m, max=0) ** 2,
                                          torch.clamp(p, min=0) ** 2))
    return torch.where(f.abs() >= ZERO_TOL, -f * torch.sqrt(g), torch.zeros_like(f))


def _normal_dt(phi, f, fb, h, cfl=0.5):
    n2, s = max(h) ** 2, 0
    for a in range(3):
        p, m = _pm(phi, fb, a, h[a])
        c = torch.maximum(p.abs(), m.abs())
        n2, s = n2 + c * c, s + c / h[a]
    return cfl / ((f.abs() / torch.sqrt(n2) * s).max() + TINY)


def _reinit(phi, fb, boundary, h, iters, use_phi0):
    b = _box(fb)
    s0 = phi[b].clone()
    dxs = max(h) ** 2

    def rhs(u, _):
        c = s0 if use_phi0 else u[b]
        n2 = 0
        for a in range(3):
            p, m = _pm(u, fb, a, h[a])
            n2 = n2 + torch.where(c > 0,
                                  torch.maximum(torch.clamp(-p, min=0), torch.clamp(m, min=0)),
                                  torch.maximum(torch.clamp(p, min=0),
                                                torch.clamp(-m, min=0))) ** 2
        sgn = c / torch.sqrt(c * c + (dxs if use_phi0 else n2 * dxs))
        return torch.where(c.abs() >= ZERO_TOL, sgn * (1 - torch.sqrt(n2)),
                           torch.zeros_like(c))
    for _ in range(iters):
        _rk3(phi, rhs, fb, boundary, 0.5 * min(h))


def _advect_rhs(phi, vel, fb, h):
    out = 0
    for a in range(3):
        p, m = _pm(phi, fb, a, h[a])
        g = torch.where(vel[a] > 0, m, p)
        out = out - vel[a] * torch.where(vel[a].abs() < ZERO_TOL, torch.zeros_like(g), g)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind == "march":
        return _exact_march(case, seed)
    if kind == "toolbox":
        return _exact_toolbox(case, seed)
    g, phi, extra = _fields(case, seed)
    dt_in = DTYPES[case["dtype"]]
    phi = phi.to(dt_in).double().contiguous()
    extra = [t.to(dt_in).double() for t in extra]
    fb, h, bc, b = g.fb, g.dx, case["boundary"], _box(g.fb)
    if kind == "reinit":
        _reinit(phi, fb, bc, h, case["steps"], True)
    elif kind == "normal":
        f = extra[0][b]
        for s in range(case["steps"]):
            _face_ghosts(phi, fb, bc)
            dt = _normal_dt(phi, f, fb, h)
            _rk3(phi, lambda u, c: _normal_rhs(u, f, fb, h), fb, bc, dt)
            if (s + 1) % 10 == 0:
                _reinit(phi, fb, bc, h, 20, False)
    elif kind == "external":
        v = [t[b] for t in extra]
        dt = 0.5 / (sum(t.abs() / e for t, e in zip(v, h)).max() + TINY)
        for _ in range(case["steps"]):
            _rk3(phi, lambda u, c: _advect_rhs(u, v, fb, h), fb, bc, dt)
    else:
        x, y, z = [t[tuple(q if t.shape[e] > 1 else slice(None) for e, q in enumerate(b))]
                   for t in _axes(g)]
        sx, sy, sz = [torch.sin(math.pi * t) for t in (x, y, z)]
        tx, ty, tz = [torch.sin(2 * math.pi * t) for t in (x, y, z)]
        base = [2 * sx * sx * ty * tz, -tx * sy * sy * tz, -tx * ty * sz * sz]
        speed = sum(t.abs() / e for t, e in zip(base, h)).max()
        t = 0.0
        for _ in range(case["steps"]):
            dt = float(0.5 / (speed * abs(math.cos(math.pi * t / 3.0)) + TINY))
            dt = min(dt, 3.0 - t)
            _rk3(phi, lambda u, c: math.cos(math.pi * (t + c * dt) / 3.0)
                 * _advect_rhs(u, base, fb, h), fb, bc, dt)
            t += dt
    return phi


def _exact_batch(case, seed):
    sizes, dx, vel, fields = _batch_inputs(case, seed)
    out = []
    if case["steps"] * sum(n[0] * n[1] * n[2] for n in sizes) > 1.5e9 or \
            case["steps"] * len(sizes) > 3000:
        return None   # minutes of small torch launches
    for n, h, v, f in zip(sizes, dx, vel, fields):
        phi = torch.tensor(np.ascontiguousarray(f.T), device="cuda").double()
        fb = (3, n[0] + 2, 3, n[1] + 2, 3, n[2] + 2)
        dt = 0.5 / (sum(abs(a) / b for a, b in zip(v, h)) + TINY)

        def rhs(u, _):
            g = 0
            for a in range(3):
                p, m = _pm(u, fb, a, h[a])
                g = g - v[a] * (m if v[a] > 0 else p)
            return g
        for _ in range(case["steps"]):
            _rk3(phi, rhs, fb, case["boundary"], dt)
        out.append(phi.cpu().numpy().T)
    return out


def _linear_pad(u):
    """u with three linearly extrapolated ghost layers per face (corners unused)."""
    for d in range(3):
        n = u.shape[d]
        a, b = u.narrow(d, 0, 1), u.narrow(d, 1, 1)
        y, z = u.narrow(d, n - 1, 1), u.narrow(d, n - 2, 1)
        u = torch.cat([a + (a - b) * q for q in (3, 2, 1)] + [u]
                      + [y + (y - z) * q for q in (1, 2, 3)], dim=d)
    return u


def _exact_adjoint(case, seed):
    n, h, lo, theta, phi0, target, eps = _adjoint_inputs(case, seed)
    m = case["lattice"]
    th = torch.tensor(theta, device="cuda", requires_grad=True)
    start = torch.tensor(phi0, device="cuda")[3:-3, 3:-3, 3:-3].permute(2, 1, 0).contiguous()
    start.requires_grad_(True)
    goal = torch.tensor(target, device="cuda")[3:-3, 3:-3, 3:-3].permute(2, 1, 0)
    hats = []
    for a in range(3):
        r = (torch.arange(n[a], device="cuda", dtype=torch.float64) + 0.5) * (m - 1) / n[a]
        j = torch.arange(m, device="cuda", dtype=torch.float64)
        hats.append(torch.clamp(1 - (r[:, None] - j[None, :]).abs(), min=0))
    vel = [torch.einsum("zyx,Kz,Jy,Ix->KJI", th[c], hats[2], hats[1], hats[0])
           for c in range(3)]
    with torch.no_grad():
        dt = float(0.5 / (sum(v.abs() / e for v, e in zip(vel, h)).max() + TINY))
    fb = (3, n[0] + 2, 3, n[1] + 2, 3, n[2] + 2)

    def rhs(u, v):
        return _advect_rhs(_linear_pad(u), v, fb, h)

    def step(u, v0, v1, v2):
        v = (v0, v1, v2)
        p1 = u + dt * rhs(u, v)
        p2 = 0.75 * u + 0.25 * (p1 + dt * rhs(p1, v))
        return u / 3 + 2.0 / 3.0 * (p2 + dt * rhs(p2, v))

    def heaviside(x):
        s = 0.5 * (1 + x / eps + torch.sin(math.pi * x / eps) / math.pi)
        return torch.where(x < -eps, torch.zeros_like(x),
                           torch.where(x > eps, torch.ones_like(x), s))
    u = start
    for _ in range(case["steps"]):
        u = checkpoint(step, u, *vel, use_reentrant=False)
    loss = ((heaviside(u) - heaviside(goal)) ** 2).sum() * (h[0] * h[1] * h[2])
    loss.backward()
    gp = torch.zeros(tuple(v + 6 for v in n), dtype=torch.float64)
    gp[3:-3, 3:-3, 3:-3] = start.grad.permute(2, 1, 0).cpu()
    return {"loss": loss.detach().cpu(), "theta": th.grad.cpu(), "phi0": gp}


def _exact_toolbox(case, seed):
    g, phi, extra = _fields({**case, "kind": "normal"}, seed)
    phi = phi.contiguous()
    fb, h, b = g.fb, g.dx, _box(g.fb)
    out = {k: torch.zeros(g.shape, device="cuda", dtype=torch.float64)
           for k in PM + ("lse_rhs", "u_stage1")}
    for a, x in enumerate("xyz"):
        out["phi_%s_plus" % x][b], out["phi_%s_minus" % x][b] = _pm(phi, fb, a, h[a])
    f = extra[0][b]
    out["lse_rhs"][b] = _normal_rhs(phi, f, fb, h)
    dt = float(_normal_dt(phi, f, fb, h))
    u = out["u_stage1"]
    u[b] = phi[b] + dt * out["lse_rhs"][b]
    for face in range(6):   # over the whole ghost box, face by face
        axis, hi = face // 2, face % 2
        d = 2 - axis
        e = fb[2 * axis + hi]
        s = (u.select(d, e) - u.select(d, e + (-1 if hi else 1))).clone()
        for i in range(e + 1, u.shape[d]) if hi else range(0, e):
            u.select(d, i).copy_(u.select(d, e) + s * abs(i - e))
    out["dt"] = dt
    return out


# -- first-order fast marching as a fixed point ------------------------------------------
def _shift(u, d, side, fill):
    """The neighbour below (side 0) or above (side 1) along dimension d."""
    pad = torch.full_like(u.narrow(d, 0, 1), fill)
    n = u.shape[d]
    return torch.cat([pad, u.narrow(d, 0, n - 1)] if side == 0
                     else [u.narrow(d, 1, n - 1), pad], dim=d)


def _solve_quadratic(best, c):
    """Larger root of sum over the finite entries (u - best_d)^2 = c (isotropic spacing)."""
    use = torch.isfinite(best)
    v = torch.where(use, best, torch.zeros_like(best))
    a = use.sum(0).double()
    mean = v.sum(0) / torch.clamp(a, min=1)
    # about the mean: a (u - mean)^2 = c - sum (v - mean)^2
    var = (torch.where(use, (v - mean) ** 2, torch.zeros_like(v))).sum(0)
    disc = (c - var) / torch.clamp(a, min=1)
    root = mean + torch.sqrt(torch.clamp(disc, min=0))
    return torch.where((a > 0) & (disc >= 0), root, torch.full_like(root, math.inf))


def _march_update(u, front, c, dims):
    """The first-order update of every point: front neighbours first, then the
    free ones in ascending order while they precede the value so far."""
    inf = math.inf
    nb = torch.stack([_shift(u, d, s, inf) for d in dims for s in (0, 1)])
    isf = torch.stack([_shift(front, d, s, False) for d in dims for s in (0, 1)])
    axes = len(dims)

    def per_axis(mask):
        v = torch.where(mask, nb, torch.full_like(nb, inf))
        return torch.minimum(v[0::2], v[1::2])
    mask = isf.clone()
    cur = _solve_quadratic(per_axis(mask), c)
    order = torch.argsort(torch.where(isf, torch.full_like(nb, inf), nb), dim=0)
    go = torch.ones_like(front)
    for r in range(2 * axes):
        q = order[r:r + 1]
        v = torch.gather(torch.where(isf, torch.full_like(nb, inf), nb), 0, q)[0]
        go = go & (v < cur) & torch.isfinite(v)
        mask = mask.scatter(0, q, torch.gather(mask, 0, q) | go[None])
        new = _solve_quadratic(per_axis(mask), c)
        cur = torch.where(go & torch.isfinite(new), new, cur)
    return cur, per_axis(mask), mask, nb


def _exact_march(case, seed):
    if case["order"] == 2:
        # the second-order stencil depends on the order in which a heap accepts
        # the points, tied keys included: no formula gives it
        return None
    phi_h, h, extra_h = _march_inputs(case, seed)
    phi = torch.tensor(phi_h, device="cuda")
    dims = list(range(phi.dim()))
    extra = [torch.tensor(t, device="cuda") for t in extra_h]
    fields = []
    if case["solver"] == "eikonal":
        low = float(phi.min())
        front = phi <= 0
        u = torch.where(front, phi - low, torch.full_like(phi, math.inf))
        c = (h / extra[0]) ** 2
    else:
        inv, near = torch.zeros_like(phi), torch.zeros_like(phi, dtype=torch.bool)
        fsum = [torch.zeros_like(phi) for _ in extra]
        for d in dims[::-1]:
            best = torch.full_like(phi, math.inf)
            val = [torch.zeros_like(phi) for _ in extra]
            for s in (0, 1):
                q = _shift(phi, d, s, math.nan)
                cross = q * phi <= 0
                fr = phi / (phi - q)
                dist = torch.where(cross, fr * h, torch.full_like(phi, math.inf))
                take = dist < best if s else cross
                best = torch.where(take, dist, best)
                for k, e in enumerate(extra):
                    v = e + fr * (_shift(e, d, s, 0.0) - e)
                    val[k] = torch.where(take, v, val[k])
            hit = torch.isfinite(best)
            w = torch.where(hit, 1 / best ** 2, torch.zeros_like(best))
            near |= hit
            inv = inv + w
            for k in range(len(extra)):
                fsum[k] = fsum[k] + torch.where(hit, val[k] * w, torch.zeros_like(w))
        on = phi.abs() < ZERO_TOL
        front = near | on
        u = torch.where(on, torch.full_like(phi, ZERO_TOL),
                        torch.where(near, torch.sqrt(1 / inv), torch.full_like(phi, math.inf)))
        fields = [torch.where(on, e, torch.where(near, fs / inv, torch.full_like(e, -1.0)))
                  for e, fs in zip(extra, fsum)]
        c = torch.full_like(phi, h * h)
    if not bool(front.any()):
        return None
    for k in range(40 * max(phi.shape)):
        cur, _, _, _ = _march_update(u, front, c, dims)
        new = torch.where(front, u, cur)
        if k % 8 == 7 and torch.equal(new, u):
            break
        u = new
    if fields:
        cur, best, mask, nb = _march_update(u, front, c, dims)
        use = torch.isfinite(best)
        g = torch.where(use, u[None] - best, torch.zeros_like(best))
        plus = mask[1::2] & (~mask[0::2] | (nb[1::2] < nb[0::2]))
        for k in range(len(fields)):
            f = fields[k]
            for it in range(40 * max(phi.shape)):
                up = torch.stack([torch.where(plus[a], _shift(f, d, 1, 0.0), _shift(f, d, 0, 0.0))
                                  for a, d in enumerate(dims)])
                new = torch.where(front, f, (g * up).sum(0) / g.sum(0))
                if it % 8 == 7 and torch.equal(new, f):
                    break
                f = new
            fields[k] = f
    if case["solver"] == "eikonal":
        return [(u + low).cpu().numpy()]
    d = torch.where(phi > 0, u, -u).cpu().numpy()
    return [d] if case["solver"] == "distance" else [d, torch.stack(fields).cpu().numpy()]
