"""GPU tests of the dense kernel's hit queue where it is used: a step with grouped
cells, interleaved windows, staged ones.  Hits are visited in the order they were
queued, so its length changes nothing."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_parity import ref_params
from test_gpu_small_steps import small_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("piled,tuning", [(True, {}), (False, {"dense_interleave": 1}), (True, {"dense_interleave": 1}),
                                          (False, {"stage_dense": 1536})])
@pytest.mark.parametrize("which", ["scene", "reference"])
def test_queue_length_is_bitwise_neutral(pbf, cuda, piled, tuning, which):
    import torch

    rng = np.random.default_rng(17)
    pos, vel, box = small_scene(pbf, 6007, piled, rng)
    p = pbf.scenes.scene_params() if which == "scene" else ref_params(pbf)
    out = []
    for queue in (1, 2, 8):
        st = pbf.ParticleState(pos, vel)
        with pbf.Simulator(p, box, (0.0, 0.0, 0.0), len(pos)) as sim:
            sim.set_tuning(dense_all=1, queue_dense=queue, **tuning)
            for _ in range(4):
                st.step(sim)
            torch.cuda.synchronize()
            sim.check_device()
        out.append([t.cpu().numpy().tobytes() for t in (st.pos, st.vel, st.iid)])
    assert out[0] == out[1] == out[2]


def test_autotune_leaves_an_unused_queue_alone(pbf, cuda):
    import torch

    sc = pbf.scenes.dam_break(seed=4)
    st = pbf.ParticleState(sc.pos, sc.vel)
    with pbf.Simulator(ref_params(pbf), sc.ulim, sc.llim, sc.n) as sim:
        for _ in range(4):
            t = sim.autotune(st.pos, st.vel, st.iid, steps=1)
            assert t["queue_dense"] == 1 or t["dense_interleave"] == 1 or t["stage_dense"] > 0
            assert t["stage_sparse"] == 0 and t["queue_sparse"] == 1
        torch.cuda.synchronize()
