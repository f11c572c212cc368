"""GPU test of the density grid (pbf_density_grid) at the edges of its kernel:
lattices that are not whole bricks of 4 x 8 x 8 nodes, particle counts around
the eight parts and the 1,024-particle batches, more bricks than a cluster
shares, particles outside the lattice and non-finite ones."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def reference(pos, lo, hi, dims, h):
    """Float64 poly6 density at the cell centres, and the particles within h of each."""
    axes = [np.float32(lo[a]) + (np.arange(dims[a], dtype=np.float32) + np.float32(0.5)) *
            ((np.float32(hi[a]) - np.float32(lo[a])) / np.float32(dims[a])) for a in range(3)]
    nodes = np.stack(np.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3).astype(np.float64)
    h = float(np.float32(h))
    out, hits = np.zeros(len(nodes)), np.zeros(len(nodes))
    p = pos[np.isfinite(pos[:, :3]).all(1), :3].astype(np.float64)
    for k, x in enumerate(nodes):
        w = h * h - ((p - x) ** 2).sum(1)
        w = w[w > 0]
        out[k], hits[k] = (w ** 3).sum(), len(w)
    return 315.0 / (64 * math.pi * h ** 9) * out.reshape(dims), hits.reshape(dims)


@pytest.mark.parametrize("n,dims", [(0, (3, 3, 3)), (1, (1, 1, 1)), (7, (5, 9, 3)), (8, (4, 8, 8)), (1023, (33, 17, 16)),
                                    (1025, (2, 31, 7)), (8191, (9, 9, 9)), (8193, (12, 16, 24)), (20011, (8, 8, 8)),
                                    (300, (4097, 1, 1))])
def test_density_grid_edges(pbf, cuda, n, dims):
    import torch

    rng = np.random.default_rng(n + dims[0])
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(-0.15, 1.15, size=(n, 3))
    pos[:, 3] = 7.0
    if n > 1000:
        pos[5, 0], pos[6, 1], pos[7, 2] = np.nan, np.inf, -np.inf
    lo, hi, h = (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), 0.11
    d = torch.from_numpy(pos).cuda()
    got = pbf.adjoint.density_grid(d, lo, hi, dims, h)
    again = pbf.adjoint.density_grid(d, lo, hi, dims, h)
    assert torch.equal(got, again)
    want, hits = reference(pos, lo, hi, dims, h)
    # a float term coef w^3, w = h^2 - q: w is off by at most 8 eps h^2 (coordinates up to 1.15 and the node's), the
    # term by 3 x that and 4 roundings; each addition adds one rounding of a sum of at most hits terms
    h32, eps = float(np.float32(h)), 2.0 ** -24
    w0 = 315.0 / (64 * math.pi * h32 ** 3)
    coord = 4 * eps * 1.15 * 2 * h32  # |dq| from the coordinates' own roundings, 2 |r| |dr|
    term = w0 * (3 * (8 * eps + coord / h32 ** 2) + 4 * eps)
    assert (np.abs(got.cpu().numpy() - want) <= hits * term + hits * hits * eps * w0).all()
