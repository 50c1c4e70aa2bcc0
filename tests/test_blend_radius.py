"""Radii during the merge blending against the oracle (needs a GPU): a whole
density, where both radius laws are one value, and fractional ones."""
import numpy as np
import pytest

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import workloads
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ledger", [0, 1])
@pytest.mark.parametrize("density", [238732.0, 238732.40625, 238732.984375])
def test_blending_radii_match_oracle(density, ledger):
    r = workloads.REF_RADIUS
    d = workloads.box_drop(2, substeps=8, adaptive=1)
    s = 2.0 * r
    p = workloads.lattice((10, 10, 10), s, (0.2, 0.2, 0.2), 0.1 * s, 4)
    masses = np.full(len(p), 0.5, np.float32)
    d.update(particles=p, n_particles=len(p), masses=masses, density=density)
    d["params"].math_mode, d["params"].min_merge_mass, d["params"].merge_radius = 1, 0.1, 0.035
    d["params"].surface_dist_threshold, d["params"].mass_ledger = 0.0, ledger
    g = gg.GranularSystem(**workloads.system_kwargs(d), masses=masses, device=0)
    o = orc.OracleSystem(d, fp64=False)
    for k in range(6):
        for f in (gg.FIELD_MASS, gg.FIELD_POS, gg.FIELD_SURFACE, gg.FIELD_SURFACE_DISTANCE, gg.FIELD_REMOVE):
            assert np.array_equal(g.read(f), o.read(f)), f"step {k}, field {f}"
        g.step(1)
        o.step(1)
    assert (o.read(gg.FIELD_REMOVE) == -1).any()
    g.close()
    o.close()
