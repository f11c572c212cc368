"""GPU tests of the one-thread-per-particle kernels: the hit lists that the
lambda pass leaves for the delta_p passes, and the lambda and XSPH passes that
take two particles of one cell per thread in current-cell order.

Bars:
  * current-cell order (paired) and grid order (one particle per thread) give
    bitwise the same state: the same hits summed in the same order;
  * either matches the FP64 oracle within 1e-5 h for one iteration.

The cases sit at the edges of the kernels: one particle, odd cells, the last
group of four candidates at the buffer's end, lists over their 64 entries and
windows over the 12 queued chunks (denser lattices), windows of exactly the
dense window's size and one more, a particle far outside the box.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_parity import TOL_X, ref_params

pytestmark = pytest.mark.gpu


def step(pbf, params, ulim, pos, vel, **tuning):
    import torch

    n = len(pos)
    d = [torch.from_numpy(a.copy()).cuda() for a in (pos, vel)]
    iid = torch.arange(n, dtype=torch.int32, device="cuda")
    npos, nvel = torch.empty_like(d[0]), torch.empty_like(d[1])
    with pbf.Simulator(params, ulim, (0.0, 0.0, 0.0), n) as sim:
        sim.set_tuning(dense_all=0, **tuning)
        sim.step(d[0], npos, d[1], nvel, iid, n)
        torch.cuda.synchronize()
    return [t.cpu().numpy() for t in (npos, nvel, d[0], d[1], iid)]


CASES = [(1, 0.05, 2048), (2, 0.05, 2048), (3, 0.05, 2048), (33, 0.05, 2048), (129, 0.05, 2048), (1001, 0.05, 2048),
         (4095, 0.05, 512), (4097, 0.041, 2048), (5000, 0.03, 2048), (5000, 0.03, 700), (5000, 0.05, 216)]


@pytest.mark.parametrize("n,spacing,window", CASES)
@pytest.mark.parametrize("niter", [1, 4])
def test_paired_and_single_walks_agree(pbf, oracle, cuda, n, spacing, window, niter):
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    pos = pbf.scenes.lattice((side, side, side), (0.0, 0.0, 0.0), rng, spacing=spacing, jitter=spacing / 10)
    pos = pos[rng.permutation(len(pos))[:n]].copy()  # holes in the lattice: cells of every population
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(0, 0.3, size=(n, 3))
    if n > 100:
        pos[5, :3] = (-0.4, 3.0, 0.2)  # outside the box: clamped into an edge cell
    p = ref_params(pbf, niter)
    box = (2 * side * spacing,) * 3
    paired = step(pbf, p, box, pos, vel, dense_window=window, order=1)
    single = step(pbf, p, box, pos, vel, dense_window=window, order=0)
    for a, b in zip(paired, single):
        assert a.tobytes() == b.tobytes()
    if niter == 1:
        r = oracle.step(p, box, (0.0, 0.0, 0.0), pos, vel, np.arange(n, dtype=np.uint32), prec="f64")
        np.testing.assert_array_equal(paired[4].astype(np.uint32), r["iid"])
        assert np.abs(paired[0][:, :3] - r["npos"][:, :3]).max() <= TOL_X


@pytest.mark.parametrize("what", ["nan", "inf", "kernel_eps"])
def test_general_walk_agrees(pbf, cuda, what):
    """Steps that may not take the sign test: a non-finite position, and a
    kernel_eps of zero (a pair at distance zero then has a gradient)."""
    rng = np.random.default_rng(3)
    pos = pbf.scenes.lattice((9, 9, 9), (0.0, 0.0, 0.0), rng)
    vel = np.zeros_like(pos)
    p = ref_params(pbf, 3)
    if what == "kernel_eps":
        p.kernel_eps = 0.0
    else:
        pos[100, 1] = np.nan if what == "nan" else np.inf
    paired = step(pbf, p, (0.9, 0.9, 0.9), pos, vel, dense_window=2048, order=1)
    single = step(pbf, p, (0.9, 0.9, 0.9), pos, vel, dense_window=2048, order=0)
    for a, b in zip(paired, single):
        assert np.array_equal(np.isnan(a), np.isnan(b)) if a.dtype.kind == "f" else True
        assert np.nan_to_num(a).tobytes() == np.nan_to_num(b).tobytes()
