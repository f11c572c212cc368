"""GPU test of paired slots beyond the hit lists (one particle in many cells:
more slots than 1.25 a particle): their particles walk the window in the delta_p
passes, with the bits of the listed ones.  Grid order pairs nothing and lists
every particle; which order the passes take changes no result."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_parity import ref_params

pytestmark = pytest.mark.gpu


# slots per particle at these spacings: 1.06, 1.35, 1.6 and more
@pytest.mark.parametrize("spacing", [0.05, 0.085, 0.095])
@pytest.mark.parametrize("piled", [False, True])
def test_orders_agree(pbf, cuda, spacing, piled):
    import torch

    rng = np.random.default_rng(int(1000 * spacing))
    pos = pbf.scenes.lattice((30, 31, 29), (0.0, 0.0, 0.0), rng, spacing=spacing)
    if piled:  # a grouped cell: one particle a pair
        pos[:700, :3] = pos[-1, :3]
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(0, 0.3, size=(len(pos), 3))
    box = (31 * spacing, 31 * spacing, 31 * spacing)
    out = []
    for order in (0, 1):
        st = pbf.ParticleState(pos, vel)
        with pbf.Simulator(ref_params(pbf), box, (0.0, 0.0, 0.0), len(pos)) as sim:
            sim.set_tuning(dense_all=0, order=order)
            for _ in range(3):
                st.step(sim)
            torch.cuda.synchronize()
        out.append([t.cpu().numpy().tobytes() for t in (st.pos, st.vel, st.iid)])
    assert out[0] == out[1]


@pytest.mark.parametrize("which", ["scene", "reference"])
def test_orders_agree_without_kernel_eps(pbf, cuda, which):
    """kernel_eps 0 leaves the sparse kernel no packed walk: one particle a thread
    in either order, the exact rules (scattered particles) included."""
    import torch

    from test_gpu_small_steps import small_scene

    rng = np.random.default_rng(11)
    pos, vel, box = small_scene(pbf, 9001, False, rng)
    p = pbf.scenes.scene_params() if which == "scene" else ref_params(pbf)
    p.kernel_eps = 0.0
    out = []
    for order in (0, 1):
        st = pbf.ParticleState(pos, vel)
        with pbf.Simulator(p, box, (0.0, 0.0, 0.0), len(pos)) as sim:
            sim.set_tuning(dense_all=0, order=order)
            for _ in range(4):
                st.step(sim)
            torch.cuda.synchronize()
        out.append([t.cpu().numpy().tobytes() for t in (st.pos, st.vel, st.iid)])
    assert out[0] == out[1]
