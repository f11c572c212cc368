"""GPU tests that a call repeated from the same inputs gives the same bits, on
states whose warps diverge most: particles thrown out of the fluid (densities of
zero and velocities that are not finite put some lanes of a batch on the exact
path and not others), and crowded cells in the reverse pass (some lanes have a
neighbour list and others too many neighbours for one).

A block's barrier that does not wait for a lane shows here as a sum of another
batch, in a few steps of a hundred, so the calls are repeated 300 times."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_small_steps import small_scene

pytestmark = pytest.mark.gpu

REPEATS = 300


def bits(tensors):
    import torch

    return [t.clone().view(torch.int32) for t in tensors]


def all_equal(a, b):
    import torch

    return all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("batch", [False, True])
def test_scattered_particles(pbf, cuda, order, batch):
    import torch

    n = 30011  # 938 batches of 32: more than the resident blocks' first ones
    rng = np.random.default_rng(n)
    pos, vel, box = small_scene(pbf, n, False, rng)
    p = pbf.scenes.scene_params()
    extra = pbf.scenes.lattice((8, 8, 8), (0.0, 0.0, 0.0), rng)
    if batch:
        pos, vel = np.concatenate([pos, extra]), np.concatenate([vel, np.zeros_like(extra)])
    zero = (0.0, 0.0, 0.0)
    first, scattered = None, False
    for r in range(REPEATS):
        st = pbf.ParticleState(pos, vel)
        sim = (pbf.Ensemble(p, [box, (0.8, 0.8, 0.8)], [zero] * 2, [n, len(extra)]) if batch
               else pbf.Simulator(p, box, zero, n))
        with sim:
            sim.set_tuning(dense_all=1, order=order)
            got = []
            for _ in range(4):
                st.step(sim)
                rho = sim.density() if batch else sim.density(n)
                got += bits((st.pos, st.vel, st.iid, rho))
        if first is None:
            first = got
            scattered = bool((~torch.isfinite(st.vel)).any()) and bool((~(rho > 0)).any())
        assert all_equal(first, got), f"run {r}"
    assert scattered  # the state the test is about


def test_crowded_reverse_pass(pbf, cuda):
    """133,952 particles (one lane each), a cloud of 600 of them crowded into
    cells of up to 150: adjoints and the walls' bitwise the same."""
    import torch

    rng = np.random.default_rng(9)
    cloud = pbf.scenes.lattice((9, 9, 9), (0.0, 0.0, 0.0), rng)[:600].copy()
    cloud[:, :3] = 0.002 + cloud[:, :3] * 0.6  # at the lower walls: some are clamped
    block = pbf.scenes.lattice((56, 52, 46), (1.6, 0.2, 0.2), rng)[600:]
    pos = np.concatenate([cloud, block])
    vel = rng.normal(0, 0.4, size=pos.shape).astype(np.float32)
    vel[:, 3] = 0
    n = len(pos)
    p = pbf.default_params()
    p.up[0], p.up[1], p.up[2] = 0.0, 1.0, 0.0
    p.niter = 2
    g = torch.from_numpy(rng.normal(size=(2, n, 4)).astype(np.float32)).cuda()
    first = None
    with pbf.Simulator(p, (6.4, 3.2, 3.2), (0.0, 0.0, 0.0), n) as sim:
        for r in range(REPEATS // 3):
            sim.tape(True)
            st = pbf.ParticleState(pos, vel)
            st.step(sim)
            got = bits(sim.backward(g[0], g[1]))
            first = got if first is None else first
            assert all_equal(first, got), f"run {r}"
