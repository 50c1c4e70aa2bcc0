"""Merge detection with a thread to a particle, beyond the lines to the groups
of lanes (needs a GPU): against the oracle with mixed masses, past a first
marking, and its time beside systems a little larger."""
import numpy as np
import pytest

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import workloads
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _scene(n, spacing, reach, masses, jitter):
    r = workloads.REF_RADIUS
    side = int(np.ceil(n ** (1 / 3)))
    s = spacing * r
    length = np.float32(workloads.CELL_PER_RADIUS * r)
    space = (side * s + 0.1,) * 3
    walls, cells = workloads.box_walls(space, length)
    d = workloads.box_drop(2, substeps=8, adaptive=1)
    p = workloads.lattice((side,) * 3, s, (0.05,) * 3, jitter * s, 4)[:n]
    d.update(particles=p, n_particles=n, masses=masses, boundary=walls, n_boundary=len(walls), space_size=space,
             cell_size=tuple(cells), gravity=(0.0, 0.0, 0.0))
    pr = d["params"]
    pr.math_mode, pr.stab_iters, pr.iters = 1, 0, 1
    pr.min_merge_mass, pr.max_mass, pr.merge_radius, pr.surface_dist_threshold = 0.1, 3.0, reach, 0.0
    return d


# inside the surface pass's reach, beyond it, and (0.15) over the whole
# stencil; an unjittered lattice, whose partners lie at equal distances
@pytest.mark.parametrize("n,reach,jitter", [(500001, 0.02, 0.1), (500001, 0.06, 0.0), (2000001, 0.15, 0.1),
                                            (2000001, 0.15, 0.0)])
def test_thread_scan_matches_oracle(n, reach, jitter):
    masses = np.random.default_rng(5).choice([0.5, 1.0, 2.0], n).astype(np.float32)
    d = _scene(n, 1.9, reach, masses, jitter)
    g = gg.GranularSystem(**workloads.system_kwargs(d), masses=masses, device=0)
    o = orc.OracleSystem(d, fp64=False)
    removed = []
    for k in range(4):
        for f in (gg.FIELD_REMOVE, gg.FIELD_MERGE, gg.FIELD_MERGE_VELOCITY, gg.FIELD_MASS, gg.FIELD_POS):
            assert np.array_equal(g.read(f), o.read(f)), f"step {k}, field {f}"
        removed.append(int((g.read(gg.FIELD_REMOVE) != 0).sum()))
        g.step(1)
        o.step(1)
    assert max(removed) > 0
    g.close()
    o.close()


@pytest.mark.parametrize("kind,below,above", [("surface", 690000, 720000), ("merge", 1980000, 2020000)])
def test_threads_take_over_where_they_are_faster(kind, below, above):
    """Particles 2.6 r apart, which fill the chip with a thread each: a few
    percent more of them take about as much longer (and, two masses being too
    much for one, none merge)."""
    ms = []
    for n in (below, above):
        d = _scene(n, 2.6, 0.035, None, 0.1)
        d["params"].max_mass, d["params"].math_mode = 1.5, 0
        g = gg.GranularSystem(**workloads.system_kwargs(d), device=0)
        g.step(2)
        assert g.size() == n
        best = 1e9
        for _ in range(4):
            g.profile_begin()
            g.step(2)
            best = min(best, g.profile_end()[kind]["ms"])
        ms.append(best)
        g.close()
    assert ms[0] <= 1.15 * ms[1]


@pytest.mark.parametrize("n,reach", [(450000, 0.06), (500000, 0.06), (500000, 0.02)])
def test_one_particle_beyond_the_line_changes_nothing(n, reach):
    """CUDA's math functions, which the oracle matches to 4 ulp only: the
    same particles with one more far from them, which takes the system to the
    kernels beyond the line, keep their surface flags, distances and merges."""
    masses = np.random.default_rng(6).choice([0.5, 1.0, 2.0], n + 1).astype(np.float32)
    masses[n] = 1.0
    out = []
    for more in (0, 1):
        d = _scene(n + 1, 1.9, reach, None, 0.1)
        length, space = np.float32(d["cell_length"]), tuple(x + 0.4 for x in d["space_size"])
        walls, cells = workloads.box_walls(space, length)
        p = d["particles"].copy()
        p[n] = [x - 0.2 for x in space]  # behind all others in the cells' order
        d.update(boundary=walls, n_boundary=len(walls), space_size=space, cell_size=tuple(cells), particles=p[:n + more],
                 n_particles=n + more)
        d["params"].math_mode = 0
        g = gg.GranularSystem(**workloads.system_kwargs(d), masses=masses[:n + more], device=0)
        fields = []
        for _ in range(3):
            g.step(1)
            fields += [g.read(f)[:n] for f in (gg.FIELD_SURFACE, gg.FIELD_SURFACE_DISTANCE, gg.FIELD_REMOVE,
                                               gg.FIELD_MERGE, gg.FIELD_MASS, gg.FIELD_POS)]
        assert g.size() == n + more and (fields[2] != 0).any()
        out.append(fields)
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
