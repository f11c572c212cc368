"""GPU tests of the reverse pass's neighbour lists: particles with a list, with
more neighbours than a list holds, and both in one warp; one lane per particle
(131,072 particles and more) against several.

A small cloud in the corner of a wide box is stepped alone (several lanes) and
beside a far block of particles that makes the step large (one lane).  No
window of the cloud holds a particle of the block and the forward's sums are
the same, so the cloud's adjoints differ by the order of FP32 sums only: of at
most 600 terms, 600 * 2^-24 = 4e-5 of the terms' size per sum, with headroom
for cancellation the 2e-3 of the largest adjoint that the reverse pass is held
to against the FP64 oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = 2e-3
BOX = ((6.4, 3.2, 3.2), (0.0, 0.0, 0.0))


def cloud(pbf, squeeze, n=600):
    """A jittered lattice squeezed towards its corner: 33 neighbours a particle
    at 1 (all listed), 33 / squeeze^3 inside it at less."""
    rng = np.random.default_rng(int(100 * squeeze))
    pos = pbf.scenes.lattice((9, 9, 9), (0.0, 0.0, 0.0), rng)[:n].copy()
    pos[:, :3] = 0.3 + pos[:, :3] * squeeze
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(0, 0.4, size=(n, 3))  # some pairs end up one-sided
    a, b = rng.normal(size=(2, n, 4)).astype(np.float32)
    a[:, 3] = b[:, 3] = 0
    p = pbf.default_params()
    p.up[0], p.up[1], p.up[2] = 0.0, 1.0, 0.0
    p.niter = 2
    return pos, vel, a, b, p


def adjoints(pbf, p, pos, vel, a, b, lanes=0):
    import torch

    n = len(pos)
    x, v = (torch.from_numpy(t.copy()).cuda() for t in (pos, vel))
    iid = torch.arange(n, dtype=torch.int32, device="cuda")
    npos, nvel = torch.empty_like(x), torch.empty_like(x)
    with pbf.Simulator(p, *BOX, n) as sim:
        sim.set_tuning(dense_all=0, bwd_lanes=lanes)
        sim.tape(True)
        sim.step(x, npos, v, nvel, iid, n)
        order = iid.long()
        g = [torch.from_numpy(t).cuda()[order].contiguous() for t in (a, b)]
        g_pos, g_vel, _ = sim.backward(*g)
        torch.cuda.synchronize()
    return g_pos.cpu().numpy()[:, :3], g_vel.cpu().numpy()[:, :3]


def close(got, want, what):
    scale = np.abs(want).max()
    err = np.abs(got - want).max()
    assert err <= REL * scale, f"{what}: max err {err:.3e} vs scale {scale:.3e}"


@pytest.mark.parametrize("squeeze", [1.0, 0.8, 0.6])
def test_one_lane_matches_several(pbf, cuda, squeeze):
    pos, vel, a, b, p = cloud(pbf, squeeze)
    rng = np.random.default_rng(3)
    block = pbf.scenes.lattice((56, 52, 46), (1.6, 0.2, 0.2), rng)  # 133,952 particles
    fill = np.zeros((len(block), 4), np.float32)
    big = adjoints(pbf, p, np.concatenate([pos, block]), np.concatenate([vel, fill]),
                   np.concatenate([a, fill]), np.concatenate([b, fill]))
    for lanes in (8, 16, 32):
        small = adjoints(pbf, p, pos, vel, a, b, lanes)
        for k, what in enumerate(("g_pos", "g_vel")):
            close(big[k][: len(pos)], small[k], f"{what}, {lanes} lanes")


@pytest.mark.parametrize("squeeze", [0.8, 0.6])
def test_crowded_matches_oracle(pbf, oracle, cuda, squeeze):
    pos, vel, a, b, p = cloud(pbf, squeeze)
    got = adjoints(pbf, p, pos, vel, a, b)
    iid = np.arange(len(pos), dtype=np.uint32)
    x, v = pos.astype(np.float64), vel.astype(np.float64)
    r = oracle.step(p, *BOX, x, v, iid, "f64")
    want = oracle.step_backward(p, *BOX, x, v, iid, a[r["iid"]].astype(np.float64), b[r["iid"]].astype(np.float64), "f64")
    close(got[0], want["pos"][:, :3], "g_pos")
    close(got[1], want["vel"][:, :3], "g_vel")
