"""GPU test of small steps on a stream that holds part of the chip (a green
context): the cooperative launches need a resident block per 1,024 particles, so
a step with more of them than the stream has multiprocessors takes the separate
launches.  The results are bitwise those of the whole chip."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from test_gpu_small_steps import small_scene

pytestmark = pytest.mark.gpu


@pytest.fixture()
def part_of_the_chip(cuda):
    """A stream with 8 multiprocessors, through the driver API."""
    import torch

    torch.zeros(1, device="cuda")  # the primary context is up
    d = ctypes.CDLL("libcuda.so.1")
    dev, count = ctypes.c_int(), ctypes.c_uint(1)
    whole, part, rest = (ctypes.create_string_buffer(1024) for _ in range(3))  # CUdevResource
    desc, ctx, stream = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()

    def ok(status, what):
        if status == 801:  # CUDA_ERROR_NOT_SUPPORTED
            pytest.skip(f"{what}: not supported")
        assert status == 0, (what, status)

    ok(d.cuDeviceGet(ctypes.byref(dev), 0), "cuDeviceGet")
    ok(d.cuDeviceGetDevResource(dev, whole, 1), "cuDeviceGetDevResource")
    ok(d.cuDevSmResourceSplitByCount(part, ctypes.byref(count), whole, rest, 0, 8), "cuDevSmResourceSplitByCount")
    ok(d.cuDevResourceGenerateDesc(ctypes.byref(desc), part, 1), "cuDevResourceGenerateDesc")
    ok(d.cuGreenCtxCreate(ctypes.byref(ctx), desc, dev, 1), "cuGreenCtxCreate")
    ok(d.cuGreenCtxStreamCreate(ctypes.byref(stream), ctx, 1, 0), "cuGreenCtxStreamCreate")
    try:
        yield d, stream
    finally:
        d.cuStreamSynchronize(stream)
        d.cuStreamDestroy_v2(stream)
        d.cuGreenCtxDestroy(ctx)


@pytest.mark.parametrize("n", [4096, 30011])
@pytest.mark.parametrize("graphs", [False, True])
def test_step_on_part_of_the_chip(pbf, cuda, part_of_the_chip, n, graphs):
    import torch

    d, stream = part_of_the_chip
    rng = np.random.default_rng(n)
    pos, vel, box = small_scene(pbf, n, True, rng)
    out = []
    for where in (None, stream.value):
        st = pbf.ParticleState(pos, vel)
        with pbf.Simulator(pbf.scenes.scene_params(), box, (0.0, 0.0, 0.0), n) as sim:
            sim.use_graphs(graphs)
            torch.cuda.synchronize()
            for _ in range(3):
                st.step(sim, where)
            if where is not None:
                assert d.cuStreamSynchronize(stream) == 0
            torch.cuda.synchronize()
            sim.check_device(where)
        out.append([t.cpu().numpy().tobytes() for t in (st.pos, st.vel, st.iid)])
    assert out[0] == out[1]
