"""The profile of the residual mode (needs a GPU): the sweeps queued behind the
one that meets the target return at once and book no work."""
import pytest

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import learn, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(0.08, 0.1, 0.09), (0.5, 0.45, 0.5)])
@pytest.mark.parametrize("target,cap", [(1e-2, 200), (0.9, 20), (1e-9, 5)])
def test_units_are_the_sweeps_that_ran(dims, target, cap):
    d = learn.pile_scene(5, dims=dims, target_residual=target * learn.R, max_sweeps=cap, law="coulomb", drop=0.0)
    s = gg.GranularSystem(**workloads.system_kwargs(d), device=0)
    stab, n = d["params"].stab_iters, s.size()
    for _ in range(3):
        s.profile_begin()
        s.step(1)
        p = s.profile_end()
        sweeps = s.stats()["last_sweeps"]
        # the sweep that finds the target met runs, and applies nothing
        met = 1 if sweeps < cap else 0
        assert p["sweep"]["units"] == n * (stab + sweeps + met)
        assert p["apply"]["units"] == n * (stab + sweeps)
    s.close()
