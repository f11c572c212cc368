"""GPU test of the xsph pass over pairs of particles where some density is not
positive or some velocity not finite: the pass visits the neighbours as ever
and looks for what poisons a sum (the IEEE NaN of 0 * dv / (rho_i + rho_j)) in
the window's flagged cells only.  A step whose particles are not paired (grid
order) visits every candidate of such windows; both must give the same bits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["scene", "reference"])
@pytest.mark.parametrize("planted", ["none", "lost", "inf", "nan", "fast"])
def test_pairs_match_every_candidate(pbf, cuda, which, planted):
    import torch

    from test_gpu_parity import ref_params

    rng = np.random.default_rng(5)
    pos = pbf.scenes.lattice((64, 32, 65), (0.0, 0.0, 0.0), rng)  # 133,120 particles: paired
    n = len(pos)
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(0, 1.0, size=(n, 3))
    some = rng.choice(n, 40, replace=False)
    if planted == "lost":  # leave their windows within the step: density 0
        pos[some, :3] = rng.uniform(0.0, 3.0, size=(40, 3))
        vel[some, 0] = 400.0
    elif planted == "inf":
        vel[some[:20], 0], vel[some[20:], 2] = np.inf, -np.inf
    elif planted == "nan":
        pos[some[:20], 1] = np.nan
        vel[some[20:], 1] = np.nan
    elif planted == "fast":  # differences of finite velocities that overflow
        vel[some[:20], 0], vel[some[20:], 0] = 3e38, -3e38
    p = pbf.scenes.scene_params() if which == "scene" else ref_params(pbf)
    out = []
    for order in (1, 0):
        st = pbf.ParticleState(pos.copy(), vel.copy())
        with pbf.Simulator(p, (6.4, 3.2, 6.5), (0.0, 0.0, 0.0), n) as sim:
            sim.set_tuning(order=order)
            for _ in range(2):
                st.step(sim)
            torch.cuda.synchronize()
        out.append([t.cpu().numpy() for t in (st.pos, st.vel, st.iid[:n])])
    for a, b in zip(*out):
        if a.dtype == np.float32:
            a, b = (np.where(np.isnan(t), np.float32(np.nan), t).view(np.uint32) for t in (a, b))
        assert np.array_equal(a, b)
