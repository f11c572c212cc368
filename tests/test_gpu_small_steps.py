"""GPU tests of small steps (every particle dense, fewer than 131,072): the
one-block sort and scan of the grid at their edges, and the cooperative
launches around the passes (followers, group tables, work list, buckets)
against the separate launches a large step uses.

A scene stepped alone takes the small path; the same scene in a batch whose
other scene makes it large takes the other.  Both sum every window in the same
parts in the same order, so the states must be bitwise equal."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_parity import compare_grid, ref_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 33, 8191, 8192, 8193])
@pytest.mark.parametrize("box", [(0.3, 0.1, 0.3), (1.0, 1.0, 1.2), (3.2, 3.2, 1.6), (12.8, 6.4, 6.4)])
def test_grid_edges(pbf, oracle, cuda, n, box):
    """Up to 8,192 particles sorted in one block by 1 to 3 digits of 7 bits; the
    cell scan in one block up to 8,192 entries (the second box has 1,201, the
    third 16,385, the last 524,289)."""
    rng = np.random.default_rng(n)
    xs = np.zeros((n, 4), np.float32)
    xs[:, :3] = rng.uniform(-0.05, 1.05, size=(n, 3)) * np.array(box)
    xs[: n // 3] = xs[0]  # a cell of many: ties keep input order
    compare_grid(pbf, oracle, ref_params(pbf), box, (0.0, 0.0, 0.0), xs)


def small_scene(pbf, n, piled, rng):
    """n particles of a jittered lattice, a third of them on two points if piled."""
    side = int(np.ceil(n ** (1 / 3)))
    pos = pbf.scenes.lattice((side, side, side), (0.0, 0.0, 0.0), rng)[:n].copy()
    if piled:
        pos[: n // 4, :3] = (0.13, 0.12, 0.11)
        pos[n // 4: n // 3, :3] = (0.13, 0.12, 0.115)
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(0, 0.3, size=(n, 3))
    return pos[rng.permutation(n)].copy(), vel, (2 * side * 0.05,) * 3


@pytest.mark.parametrize("n,piled", [(1, False), (511, False), (512, True), (1025, True), (4097, False), (4096, True),
                                     (20000, True), (30011, False)])
@pytest.mark.parametrize("which", ["scene", "reference"])
@pytest.mark.parametrize("order", [1, 0])
def test_small_and_large_launches_agree(pbf, cuda, n, piled, which, order):
    import torch

    rng = np.random.default_rng(n)
    pos, vel, box = small_scene(pbf, n, piled, rng)
    fill = pbf.scenes.lattice((64, 32, 64), (0.0, 0.0, 0.0), rng)  # 131,072 particles: the batch is large
    p = pbf.scenes.scene_params() if which == "scene" else ref_params(pbf)
    st = pbf.ParticleState(pos, vel)
    with pbf.Simulator(p, box, (0.0, 0.0, 0.0), n) as sim:
        sim.set_tuning(dense_all=1, order=order)
        for _ in range(4):
            st.step(sim)
        torch.cuda.synchronize()
        sim.check_device()
    alone = [t.cpu().numpy() for t in (st.pos, st.vel, st.iid[:n])]
    both = pbf.ParticleState(np.concatenate([pos, fill]), np.concatenate([vel, np.zeros_like(fill)]))
    with pbf.Ensemble(p, [box, (6.4, 3.2, 3.2)], [(0.0, 0.0, 0.0)] * 2, [n, len(fill)]) as ens:
        ens.set_tuning(dense_all=1, order=order)
        for _ in range(4):
            both.step(ens)
        torch.cuda.synchronize()
    for a, b in zip(alone, (both.pos, both.vel, both.iid)):
        assert a.tobytes() == b[:n].cpu().numpy().tobytes()
