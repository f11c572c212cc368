"""GPU tests of a nearly full device: what an allocation that fails leaves behind.
A filler takes the device's memory up to a stated rest; a failing allocation is
an ordinary error."""
from __future__ import annotations

import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def device_with(rest):
    """Leaves about `rest` bytes of the device free."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - rest, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del filler
        torch.cuda.empty_cache()


def ref_params(pbf):
    p = pbf.default_params()
    p.up[0], p.up[1], p.up[2] = 0.0, 1.0, 0.0
    p.niter = 2
    return p


def test_tape_after_a_failed_enable(pbf, cuda):
    """1,048,576 particles: the reverse pass's scratch is ~620 MB in six
    allocations, of which 200 MB hold the first ones only.  The call fails; with
    memory again the next one allocates all of them, and the adjoints are those of
    a solver whose first call succeeded."""
    import torch

    rng = np.random.default_rng(1)
    pos = pbf.scenes.lattice((128, 64, 128), (0.0, 0.0, 0.0), rng)
    n = len(pos)
    p = ref_params(pbf)
    box = ((12.8, 6.4, 6.4), (0.0, 0.0, 0.0))
    g = torch.from_numpy(rng.normal(size=(2, n, 4)).astype(np.float32)).cuda()
    out = []
    for fail in (False, True):
        with pbf.Simulator(p, *box, n) as sim:
            if fail:
                with device_with(200 * MB):
                    with pytest.raises(pbf.PbfError) as e:
                        sim.tape(True)
                    assert e.value.status == pbf.PBF_ERR_CUDA
            sim.tape(True)
            x, v = torch.from_numpy(pos.copy()).cuda(), torch.zeros(n, 4, device="cuda")
            npos, nvel = torch.empty_like(x), torch.empty_like(x)
            iid = torch.arange(n, dtype=torch.int32, device="cuda")
            sim.step(x, npos, v, nvel, iid, n)
            out.append([t.view(torch.int32) for t in sim.backward(g[0], g[1])])
            torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(*out))


def two_steps(pbf, p, box, pos, rest=None):
    """The state after two steps of a solver created with `rest` bytes free."""
    import torch

    st = pbf.ParticleState(pos, np.zeros_like(pos))
    with contextlib.ExitStack() as stack:
        if rest is not None:
            stack.enter_context(device_with(rest))
        with pbf.Simulator(p, *box, len(pos)) as sim:
            st.step(sim)
            st.step(sim)
            torch.cuda.synchronize()
    return [t.clone().view(torch.int32) for t in (st.pos, st.vel, st.iid)]


def test_solver_without_room_for_its_hit_lists(pbf, cuda):
    """1,048,576 particles in 524,288 cells (a solver reserves four times those):
    ~330 MB of scratch without the hit lists, ~670 with.  In 450 MB the solver
    works without lists, bit for bit the same."""
    import torch

    rng = np.random.default_rng(2)
    pos = pbf.scenes.lattice((128, 64, 128), (0.0, 0.0, 0.0), rng)
    p = ref_params(pbf)
    box = ((12.8, 6.4, 6.4), (0.0, 0.0, 0.0))
    want = two_steps(pbf, p, box, pos)
    got = two_steps(pbf, p, box, pos, rest=450 * MB)
    assert all(torch.equal(a, b) for a, b in zip(want, got))


def test_tape_without_room_for_its_neighbour_lists(pbf, cuda):
    """The reverse pass of 1,048,576 particles takes ~530 MB with its tape, 268
    more with neighbour lists.  Without them its sums walk the windows: the same
    terms in another order, 33 of them at rest (600 * 2^-24 = 4e-5 of their size
    for 600, with headroom for cancellation 2e-3 of the largest adjoint)."""
    import torch

    rng = np.random.default_rng(3)
    pos = pbf.scenes.lattice((128, 64, 128), (0.0, 0.0, 0.0), rng)
    n = len(pos)
    p = ref_params(pbf)
    g = torch.from_numpy(rng.normal(size=(2, n, 4)).astype(np.float32)).cuda()
    out = []
    for rest in (None, 720 * MB):
        x, v = torch.from_numpy(pos.copy()).cuda(), torch.zeros(n, 4, device="cuda")
        npos, nvel = torch.empty_like(x), torch.empty_like(x)
        iid = torch.arange(n, dtype=torch.int32, device="cuda")
        with pbf.Simulator(p, (12.8, 6.4, 6.4), (0.0, 0.0, 0.0), n) as sim:
            with contextlib.ExitStack() as stack:
                if rest is not None:
                    stack.enter_context(device_with(rest))
                sim.tape(True)
                sim.step(x, npos, v, nvel, iid, n)
                out.append([t.cpu().numpy() for t in sim.backward(g[0], g[1])])
    for a, b, what in zip(*out, ("g_pos", "g_vel", "g_lim")):
        err, scale = np.abs(a - b).max(), np.abs(a).max()
        assert err <= 2e-3 * max(scale, 1e-30), f"{what}: {err:.3e} of {scale:.3e}"
    assert any((a != b).any() for a, b in zip(*out))  # the other path ran
