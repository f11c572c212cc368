"""GPU tests of a small step whose grid barrier gives up: with a limit of one
poll no block but the last to arrive waits long enough.  The step ends by
itself, the status says so, and the solver's next steps, from the same state
and with the default limit, are bitwise those of a solver that never failed
(the group tables that the failed step left half written are cleared)."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from test_gpu_small_steps import small_scene

pytestmark = pytest.mark.gpu


def steps(pbf, sim, pos, vel, count):
    import torch

    st = pbf.ParticleState(pos, vel)
    out = []
    for _ in range(count):
        st.step(sim)
        out += [t.clone().view(torch.int32) for t in (st.pos, st.vel, st.iid)]
    torch.cuda.synchronize()
    return out


# a third of the particles on two points: group tables, so barriers from the first iteration on
@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("n,order", [(20000, 1), (20000, 0), (4096, 1)])
def test_barrier_gives_up_and_recovers(pbf, cuda, n, order, batch):
    import torch

    rng = np.random.default_rng(n)
    pos, vel, box = small_scene(pbf, n, True, rng)
    p = pbf.scenes.scene_params()
    zero = (0.0, 0.0, 0.0)

    def make():
        sim = pbf.Ensemble(p, [box], [zero], [n]) if batch else pbf.Simulator(p, box, zero, n)
        sim.set_tuning(order=order)
        return sim

    with make() as sim:
        want = steps(pbf, sim, pos, vel, 2)
        sim.check_device()
    with make() as sim:
        for graphs in (True, False):
            sim.use_graphs(graphs)
            sim.set_wait_limit(1)
            steps(pbf, sim, pos, vel, 1)
            with pytest.raises(pbf.PbfError) as e:
                sim.check_device()
            assert e.value.status == pbf.PBF_ERR_TIMEOUT
            sim.check_device()  # reported once
            sim.set_wait_limit(0)
            got = steps(pbf, sim, pos, vel, 2)
            sim.check_device()
            assert all(torch.equal(a, b) for a, b in zip(want, got))
        # a step that fails between two good ones, nothing read in between
        sim.set_wait_limit(1)
        steps(pbf, sim, pos, vel, 2)
        sim.set_wait_limit(0)
        assert all(torch.equal(a, b) for a, b in zip(want, steps(pbf, sim, pos, vel, 2)))
        with pytest.raises(pbf.PbfError):
            sim.check_device()


def test_limits(pbf, cuda):
    p = pbf.default_params()
    with pbf.Simulator(p, (1.0, 1.0, 1.0), (0.0, 0.0, 0.0), 16) as sim:
        with pytest.raises(pbf.PbfError):
            sim.set_wait_limit(-1)
    assert pbf.lib().pbf_noalloc_check_device(ctypes.c_void_p(0)) == pbf.PBF_OK
