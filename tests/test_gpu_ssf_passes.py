"""GPU tests of the SSF kernels at the edges their launches depend on: the
splat's sprites per warp (by particle count) and its thickness width (by
radius), images that are not whole smoothing tiles, background blocks, and
several renders by one renderer (a render leaves the splat's images clear)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_ssf import assert_splat_exact, bits, dam_zup, gpu_render, params_for, random_cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 155647, 155649])
@pytest.mark.parametrize("radius", [0.05, 0.7])
def test_splat_bit_exact_counts_and_radii(pbf, oracle, cuda, n, radius):
    """8 sprites a warp below 155,648 particles, 32 from there on; 32-bit
    thickness below radius 0.4995."""
    pos = random_cloud(np.random.default_rng(n), n, [-0.5, -1.5, 0.0], [1.5, 0.5, 1.2])
    w, h = (96, 72) if n > 1000 else (320, 240)
    assert_splat_exact(pbf, oracle, params_for(pbf, w, h, eye=(2.6, -6.2, 2.8), radius=radius), pos)


@pytest.mark.parametrize("w,h", [(1, 1), (31, 15), (33, 17), (64, 48), (129, 50)])
@pytest.mark.parametrize("blur_option,kernel_r", [(0, 0), (0, 3), (1, 7), (0, 20)])
def test_smoothing_sizes(pbf, oracle, cuda, w, h, blur_option, kernel_r):
    """Tiles of 32 x 16 pixels, four rows a thread: the first pass from the
    splat's own image, against the float oracle's filter within 1e-5 |z|, the
    same background pixels (the bar of test_gpu_ssf)."""
    p = params_for(pbf, w, h, blur_option=blur_option, kernel_r=kernel_r, smooth_niter=1)
    pos = dam_zup(pbf)
    got = gpu_render(pbf, p, pos)
    want = oracle.ssf_render(p, pos, prec="f32")["depth"]
    assert np.array_equal(got["depth"] > 99, want > 99)
    assert (np.abs(got["depth"] - want) <= 1e-5 * np.abs(want)).all()


def test_renders_do_not_depend_on_earlier_ones(pbf, cuda):
    """The same frame alone, and after a frame of other particles, an empty one
    and one with other settings; with and without a colour image, profiled and
    not."""
    import torch

    p = params_for(pbf, 200, 120, smooth_niter=3)
    a = torch.from_numpy(dam_zup(pbf)).cuda()
    b = torch.from_numpy(random_cloud(np.random.default_rng(2), 3000, [-0.5, -1.5, 0.0], [1.5, 0.5, 1.2])).cuda()

    def frame(r):
        color = r.render(a)
        return [color.cpu().numpy()] + [v.cpu().numpy() for _, v in sorted(r.images().items())]

    with pbf.SSFRenderer(p) as r:
        want = frame(r)
    with pbf.SSFRenderer(p) as r:
        r.render(b)
        r.render(b, n=0)
        q = p.copy()
        q.smooth_niter, q.kernel_r = 2, 20
        r.load_params(q)
        r.render(b)
        r.load_params(p)
        got = frame(r)
        for x, y in zip(got, want):
            assert np.array_equal(bits(x), bits(y))
        r.profile_enable(True)
        for x, y in zip(frame(r), want):
            assert np.array_equal(bits(x), bits(y))
