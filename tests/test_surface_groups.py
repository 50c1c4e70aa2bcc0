"""Surface detection with groups of lanes and with a thread to a particle
against the oracle (needs a GPU): sizes at partly filled groups and beside
the line between the two, mixed masses, more neighbours than a group lists."""
import numpy as np
import pytest

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import abi, workloads
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _check(n, spacing, heavy, radius=0.01):
    r = radius
    side = int(np.ceil(n ** (1 / 3)))
    d = workloads.box_drop(2, substeps=8, adaptive=1)
    s = spacing * r
    length = np.float32(workloads.CELL_PER_RADIUS * r)
    space = (max(1.0, side * s + 0.1),) * 3
    walls, cells = workloads.box_walls(space, length)
    p = workloads.lattice((side,) * 3, s, (0.05, 0.05, 0.05), 0.2 * s, 3)
    rng = np.random.default_rng(3)
    p = p[rng.permutation(len(p))[:n]]
    masses = np.where(rng.uniform(size=n) < heavy, rng.choice([2.0, 4.0, 8.0], n), 1.0).astype(np.float32)
    d.update(particles=p, n_particles=n, masses=masses, boundary=walls, n_boundary=len(walls), space_size=space,
             cell_size=tuple(cells), cell_length=float(length), density=workloads.density_for_radius(r))
    d["params"].math_mode, d["params"].stab_iters, d["params"].iters = 1, 0, 1
    g = gg.GranularSystem(**workloads.system_kwargs(d), masses=masses, device=0)
    o = orc.OracleSystem(d, fp64=False)
    for k in range(2):
        for f in (gg.FIELD_SURFACE, gg.FIELD_SURFACE_DISTANCE, gg.FIELD_REMOVE, gg.FIELD_POS, gg.FIELD_MASS):
            assert np.array_equal(g.read(f), o.read(f)), f"step {k}, field {f}"
        g.step(1)
        o.step(1)
    g.close()
    o.close()


@pytest.mark.parametrize("heavy", [0.0, 0.3])
@pytest.mark.parametrize("n,spacing", [(1, 2.0), (7, 2.0), (9, 1.5), (33, 2.0), (1000, 1.9), (9000, 0.9), (30000, 1.2)])
def test_groups_match_oracle(n, spacing, heavy):
    _check(n, spacing, heavy)


@pytest.mark.parametrize("n", [700000, 700001])
def test_both_sides_of_the_line_match_oracle(n):
    _check(n, 1.9, 0.1, radius=0.005)


@pytest.mark.parametrize("reach", [0.035, 0.02])
@pytest.mark.parametrize("n,spacing", [(1, 2.0), (9, 1.8), (257, 2.0), (4000, 1.9), (12000, 1.4)])
def test_merge_scan_groups_match_oracle(n, spacing, reach):
    """Partners and density of the merge: the radius inside the surface pass's
    reach and beyond it, equal distances (an unjittered lattice)."""
    r = workloads.REF_RADIUS
    side = int(np.ceil(n ** (1 / 3)))
    d = workloads.box_drop(2, substeps=8, adaptive=1)
    s = spacing * r
    p = workloads.lattice((side,) * 3, s, (0.2, 0.2, 0.2), 0.0 if spacing == 2.0 else 0.1 * s, 4)[:n]
    masses = np.full(n, 0.5, np.float32)
    d.update(particles=p, n_particles=n, masses=masses)
    d["params"].math_mode, d["params"].min_merge_mass, d["params"].merge_radius = 1, 0.1, reach
    d["params"].surface_dist_threshold = 0.0
    g = gg.GranularSystem(**workloads.system_kwargs(d), masses=masses, device=0)
    o = orc.OracleSystem(d, fp64=False)
    for k in range(3):
        for f in (gg.FIELD_REMOVE, gg.FIELD_MERGE, gg.FIELD_MERGE_VELOCITY, gg.FIELD_MASS, gg.FIELD_POS):
            assert np.array_equal(g.read(f), o.read(f)), f"step {k}, field {f}"
        g.step(1)
        o.step(1)
    g.close()
    o.close()
