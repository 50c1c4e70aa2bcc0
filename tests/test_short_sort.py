"""The grid build's short and long sorts and its cell table against the
oracle (needs a GPU): sizes at the edges of tiles and of the ranges, one to
four digit passes, empty stretches of cells, all particles in one cell."""
import numpy as np
import pytest

import granular_gpu_gb300 as gg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 255, 256, 257, 1023, 1024, 1025, 4097, 131071, 131072, 131073, 262144, 262145, 524287, 524288, 524289]


@pytest.mark.parametrize("cells", [(1, 1, 1), (5, 6, 7), (255, 1, 1), (16, 16, 1), (40, 23, 31), (300, 250, 240)])
@pytest.mark.parametrize("shape", ["even", "one_cell", "far_corner", "outside"])
def test_build_matches_oracle(cells, shape):
    L = 0.0404
    span = np.array(cells, np.float32) * np.float32(L)
    sizes = SIZES if shape == "even" and cells == (40, 23, 31) else [1, 257, 5000, 70001]
    g = gg.Grid(max(sizes), cells, L)
    for n in sizes:
        rng = np.random.default_rng(n)
        if shape == "even":
            p = rng.uniform(-0.02, 1.02, (n, 3)) * span
        elif shape == "one_cell":
            p = np.full((n, 3), 0.3) * L
        elif shape == "far_corner":
            p = span - rng.uniform(0.0, 2.5 * L, (n, 3))
        else:
            p = rng.uniform(1.5, 2.0, (n, 3)) * span
        p = p.astype(np.float32)
        k, sk, pm, cst = g.build(p)
        ok, osk, opm, ocs = orc.grid_build(p, cells, L)
        assert np.array_equal(k, ok) and np.array_equal(sk, osk) and np.array_equal(pm, opm), n
        assert np.array_equal(cst, ocs), n
    g.close()
