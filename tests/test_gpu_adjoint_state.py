"""The adjoint problem's final state keeps the caller's ghost cells over repeated
runs and new fields, and the problem holds no field more than its states need."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (20, 18, 17)


def fields(seed):
    rng = np.random.default_rng(seed)
    shape = tuple(m + 6 for m in N)
    x = np.meshgrid(*[np.linspace(-1, 1, s) for s in shape], indexing="ij")
    phi0 = np.asfortranarray(np.sqrt(sum(c * c for c in x)) - 0.5 - 0.01 * seed)
    edge = np.ones(shape, dtype=bool)
    edge[3:-3, 3:-3, 3:-3] = False
    phi0[edge] = rng.standard_normal(int(edge.sum()))   # never read, and kept
    return phi0, np.asfortranarray(phi0 + 0.05), edge


def test_final_state_keeps_the_ghost_cells():
    from lsmlib_b200 import adjoint
    p = adjoint.AdvectionAdjoint(N, (0.1,) * 3, (0.0,) * 3, lattice=4, nsteps=5,
                                 checkpoint_every=2)
    rng = np.random.default_rng(1)
    p.set_theta(rng.uniform(-0.3, 0.3, size=(3, 4, 4, 4)))
    p.set_dt(0.02)
    losses = []
    for seed in (1, 2, 1):
        phi0, target, edge = fields(seed)
        p.set_fields(phi0, target, 0.15)
        first = p.forward()
        for _ in range(2):
            got = p.phi_final()
            assert np.array_equal(got[edge], phi0[edge])
            assert np.all(np.isfinite(got)) and not np.array_equal(got, phi0)
            p.backward()
            assert p.forward() == first
        losses.append(first)
    assert losses[0] == losses[2] != losses[1]


def test_number_of_fields():
    import torch

    from lsmlib_b200 import adjoint
    n = (100, 100, 100)
    steps, every = 8, 3
    one = 10 << 20   # 106^3 doubles, 9.5 MB, in the driver's 2 MB units
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    p = adjoint.AdvectionAdjoint(n, (0.1,) * 3, (0.0,) * 3, lattice=4, nsteps=steps,
                                 checkpoint_every=every)
    used = free - torch.cuda.mem_get_info()[0]
    p.close()
    # velocity and its gradient, target, state, two stages, five sums of the
    # sweep; checkpoints; two sets of a segment's three states a step
    count = 3 + 3 + 1 + 1 + 2 + 5 + -(-steps // every) + 2 * 3 * every
    assert used < (count + 0.9) * one
