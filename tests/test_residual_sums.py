"""Residual mode with the residual summed by the sweeps and decided on the
device, against the stencil sweep with its own residual kernel (needs a GPU):
the same sweeps and bits, at sizes of every sweep kernel, with both laws, a
target met at once, one met on the way, and a cap on the sweeps."""
import numpy as np
import pytest

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import learn, workloads

pytestmark = pytest.mark.gpu


def _run(law, dims, target, cap, variant, steps=3):
    d = learn.pile_scene(5, dims=dims, target_residual=target * learn.R, max_sweeps=cap, law=law, drop=0.0)
    s = gg.GranularSystem(**workloads.system_kwargs(d), device=0)
    s.set_tuning(sweep_variant=variant)
    out = []
    for _ in range(steps):
        s.step(1)
        st = s.stats()
        out.append((st["last_sweeps"], st["last_residual"], st["last_residual_max"], s.read(gg.FIELD_POS),
                    s.read(gg.FIELD_VEL), s.read(gg.FIELD_NUM_CONSTRAINTS), s.read(gg.FIELD_CONTACTS)))
    s.close()
    return out


@pytest.mark.parametrize("law", ["coulomb", "cap"])
@pytest.mark.parametrize("dims", [(0.08, 0.1, 0.09), (0.2, 0.3, 0.2), (0.35, 0.3, 0.3), (0.5, 0.45, 0.5)])
@pytest.mark.parametrize("target,cap", [(1e-2, 60), (1e-3, 7), (1e-3, 0), (0.9, 20)])
def test_residual_from_the_sweeps(law, dims, target, cap):
    if law == "cap" and dims[0] > 0.4:
        target, cap = max(target, 1e-2), min(cap, 10)
    for a, b in zip(_run(law, dims, target, cap, 0), _run(law, dims, target, cap, 1)):
        assert a[0] == b[0] <= cap
        # the same penetrations, added in other orders: 64 single-precision
        # additions a thread at most
        assert abs(a[1] - b[1]) <= 64 * 2.0 ** -24 * abs(b[1])
        assert a[2] == b[2]
        for x, y in zip(a[3:], b[3:]):
            assert np.array_equal(x, y)
