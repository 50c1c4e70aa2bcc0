"""The contact sweep's thread kernels well above the line to the groups of
lanes (needs a GPU): both contact laws against the oracle over several kept
sweeps, and the residual summed by the sweeps against the residual kernel."""
import numpy as np
import pytest

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import learn, workloads
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spacing,law", [(400000, 1.9, 0), (400000, 1.9, 1), (400001, 1.4, 0), (400001, 1.4, 1),
                                           (500000, 1.7, 0), (500000, 1.7, 1), (1500001, 1.9, 1)])
def test_laws_match_oracle(n, spacing, law):
    r = 0.005 if n < 1000000 else 0.004
    side = int(np.ceil(n ** (1 / 3)))
    d = workloads.box_drop(2, substeps=8, configured=law == 1)
    p = workloads.lattice((side,) * 3, spacing * r, (0.02,) * 3, 0.2 * spacing * r, 1)
    p = p[np.random.default_rng(1).permutation(len(p))[:n]]
    length = np.float32(workloads.CELL_PER_RADIUS * r)
    walls, cells = workloads.box_walls((1.0, 1.0, 1.0), length)
    d.update(particles=p, n_particles=n, boundary=walls, n_boundary=len(walls), cell_size=tuple(cells),
             cell_length=float(length), density=workloads.density_for_radius(r))
    d["params"].math_mode, d["params"].stab_iters, d["params"].iters = 1, 1, 4
    s = gg.GranularSystem(**workloads.system_kwargs(d), device=0)
    o = orc.OracleSystem(d, fp64=False)
    s.step(1)
    o.step(1)
    for f in (gg.FIELD_CONTACTS, gg.FIELD_NUM_CONSTRAINTS, gg.FIELD_POS, gg.FIELD_VEL):
        assert np.array_equal(s.read(f), o.read(f)), f
    s.close()
    o.close()


@pytest.mark.parametrize("law", ["coulomb", "cap"])
def test_residual_from_the_sweeps(law):
    out = []
    for variant in (0, 1):
        d = learn.pile_scene(5, dims=(0.8, 0.65, 0.8), target_residual=1e-2 * learn.R, max_sweeps=10, law=law, drop=0.0)
        s = gg.GranularSystem(**workloads.system_kwargs(d), device=0)
        assert s.size() > 400000
        s.set_tuning(sweep_variant=variant)
        for _ in range(2):
            s.step(1)
            st = s.stats()
            out.append((st["last_sweeps"], st["last_residual"], st["last_residual_max"],
                        [s.read(f) for f in (gg.FIELD_POS, gg.FIELD_VEL, gg.FIELD_CONTACTS, gg.FIELD_NUM_CONSTRAINTS)]))
        s.close()
    for a, b in zip(out[:2], out[2:]):
        assert a[0] == b[0]
        # the same penetrations in other orders: 64 single-precision additions a thread at most
        assert abs(a[1] - b[1]) <= 64 * 2.0 ** -24 * abs(b[1])
        assert a[2] == b[2]
        for x, y in zip(a[3], b[3]):
            assert np.array_equal(x, y)
