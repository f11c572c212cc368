"""GPU test of the cell prefix at the edges of its launches: one block up to
8,192 entries, the downsweep adding up the tiles before its own up to 4,096
tiles of 2,048 entries, a launch of its own for the tiles' prefix beyond.
Whole numbers: equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_parity import compare_grid, ref_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [
    (1.3, 1.8, 3.5),     # 8,191 entries: one block, its last round ragged
    (1.6, 1.6, 3.2),     # 8,193: 5 tiles, the last of one entry
    (3.3, 3.2, 3.2),     # 33,793: 17 tiles, the last of 1,025
    (12.8, 6.4, 6.3),    # 516,097: 253 tiles, the last of one entry
    (25.6, 25.6, 12.7),  # 8,323,073: 4,065 tiles
    (25.6, 25.6, 12.8),  # 8,388,609: 4,097 tiles
])
def test_cell_prefix(pbf, oracle, cuda, box):
    n = 20000
    rng = np.random.default_rng(n)
    xs = np.zeros((n, 4), np.float32)
    xs[:, :3] = rng.uniform(-0.01, 1.01, size=(n, 3)) * np.array(box)
    xs[: n // 4] = xs[0]
    compare_grid(pbf, oracle, ref_params(pbf), box, (0.0, 0.0, 0.0), xs)
