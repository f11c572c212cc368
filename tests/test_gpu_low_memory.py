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
