"""Surface detection and contact lists by one thread to a particle against the
oracle (needs a GPU): candidate masks over partly filled and overfull chunks,
mixed masses, positions that are not numbers."""
import numpy as np
import pytest

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import workloads
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

FIELDS = (gg.FIELD_SURFACE, gg.FIELD_SURFACE_DISTANCE, gg.FIELD_REMOVE, gg.FIELD_POS, gg.FIELD_MASS)


def _check(side, spacing, heavy, bad, adaptive):
    r = 0.005
    d = workloads.box_drop(2, substeps=8, adaptive=adaptive)
    s = spacing * r
    length = np.float32(workloads.CELL_PER_RADIUS * r)
    space = (max(1.0, side * s + 0.1),) * 3
    walls, cells = workloads.box_walls(space, length)
    p = workloads.lattice((side,) * 3, s, (0.05, 0.05, 0.05), 0.2 * s, 3)
    n = len(p)
    rng = np.random.default_rng(5)
    masses = np.where(rng.uniform(size=n) < heavy, rng.choice([2.0, 4.0, 8.0], n), 1.0).astype(np.float32)
    d.update(particles=p, n_particles=n, masses=masses, boundary=walls, n_boundary=len(walls), space_size=space,
             cell_size=tuple(cells), cell_length=float(length), density=workloads.density_for_radius(r))
    d["params"].math_mode, d["params"].stab_iters, d["params"].iters = 1, 1, 2
    g = gg.GranularSystem(**workloads.system_kwargs(d), masses=masses, device=0)
    o = orc.OracleSystem(d, fp64=False)
    if bad:
        x = o.read(gg.FIELD_POS).copy()
        rows = rng.permutation(n)[:8]
        x[rows, np.arange(8) % 3] = np.nan
        g.write(gg.FIELD_POS, x)
        o.write(gg.FIELD_POS, x)
    g.step(1)
    o.step(1)
    for f in FIELDS if adaptive else (gg.FIELD_POS,):
        assert np.array_equal(g.read(f), o.read(f), equal_nan=True), f"field {f}"
    g.close()
    o.close()


@pytest.mark.parametrize("bad", [False, True])
@pytest.mark.parametrize("spacing,heavy", [(1.9, 0.0), (1.9, 0.2), (1.2, 0.05)])
def test_surface_of_a_large_system_matches_oracle(spacing, heavy, bad):
    _check(90, spacing, heavy, bad, 1)


@pytest.mark.parametrize("bad", [False, True])
@pytest.mark.parametrize("spacing,heavy", [(1.9, 0.0), (1.9, 0.2), (1.1, 0.05)])
def test_lists_built_by_threads_match_oracle(spacing, heavy, bad):
    _check(50, spacing, heavy, bad, 0)
