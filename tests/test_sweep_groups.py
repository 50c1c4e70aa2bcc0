"""The contact sweep's groups of lanes against the oracle (needs a GPU): at
the sizes where the lanes to a particle change, at partly filled groups and
warps, with lists longer than a list holds, and with the rebuild queues of
systems that run a thread to a particle."""
import numpy as np
import pytest

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import abi, workloads
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _scene(n, spacing, law, seed=1):
    """n particles of radius 0.01 from a jittered lattice on the floor of a
    box, in no particular order; with spacings below 0.8 r a particle has
    more than 64 candidates."""
    r = workloads.REF_RADIUS
    side = int(np.ceil(n ** (1 / 3)))
    d = workloads.box_drop(2, substeps=8, configured=law == 1)
    s = spacing * r
    p = workloads.lattice((side,) * 3, s, (0.5 - side * s / 2, 0.02, 0.5 - side * s / 2), 0.2 * s, seed)
    rng = np.random.default_rng(seed)
    p = p[rng.permutation(len(p))[:n]]
    d.update(particles=p, n_particles=n)
    d["params"].math_mode = 1
    d["params"].stab_iters, d["params"].iters = 1, 3
    return d


def _check(d, steps):
    s = gg.GranularSystem(**workloads.system_kwargs(d), device=0)
    o = orc.OracleSystem(d, fp64=False)
    for k in range(steps + 1):
        if k:
            s.step(1)
            o.step(1)
        for f in (gg.FIELD_CONTACTS, gg.FIELD_NUM_CONSTRAINTS, gg.FIELD_POS, gg.FIELD_VEL):
            assert np.array_equal(s.read(f), o.read(f)), f"step {k}, field {f}"
    most = int(s.read(gg.FIELD_CONTACTS).max())
    s.close()
    o.close()
    return most


@pytest.mark.parametrize("law", [0, 1])
@pytest.mark.parametrize("n", [1, 3, 7, 8, 9, 31, 33, 257, 4095, 4096, 4097, 16384, 16385])
def test_group_sizes_match_oracle(n, law):
    _check(_scene(n, 1.5, law), 2)


@pytest.mark.parametrize("law", [0, 1])
@pytest.mark.parametrize("n,spacing", [(3000, 0.7), (9000, 0.6), (20000, 0.8)])
def test_overlong_lists_match_oracle(n, spacing, law):
    assert _check(_scene(n, spacing, law), 2) > 64


@pytest.mark.parametrize("law", [0, 1])
@pytest.mark.parametrize("n,spacing", [(100000, 1.9), (100001, 1.9), (110000, 0.8), (140000, 1.2)])
def test_thread_kernels_and_their_queues_match_oracle(n, spacing, law):
    most = _check(_scene(n, spacing, law), 2)
    assert most > 64 or spacing > 0.8


@pytest.mark.parametrize("law", [0, 1])
@pytest.mark.parametrize("n", [600, 9000, 30000, 101000])
@pytest.mark.parametrize("spacing", [1.3, 1.15, 0.95, 0.8])
def test_long_lists_match_oracle(n, spacing, law):
    """A skin of 1.2 r and spacings that list from about 60 to about 250
    candidates: lists of both kinds kept over the sweeps, long ones that stay
    long, and more than a long one holds."""
    d = _scene(n, spacing, law)
    d["params"].nlist_skin = 0.012
    d["params"].stab_iters, d["params"].iters = 1, 5
    _check(d, 1)


def test_long_lists_are_kept_and_run_out():
    """Fewer long lists than particles that want one: with room for two
    long lists (a capacity of 100 particles) the others scan every sweep."""
    d = _scene(100, 1.0, 0)
    d["params"].nlist_skin = 0.014
    d["params"].iters = 6
    d["max_particles"] = 100
    _check(d, 2)
    d = _scene(20000, 1.15, 0)
    d["params"].nlist_skin, d["params"].iters = 0.014, 6
    d["gravity"] = (0.0, 0.0, 0.0)
    s = gg.GranularSystem(**workloads.system_kwargs(d), device=0)
    s.profile_begin()
    s.step(1)
    built = s.profile_end()["_nlist_rebuilds"]
    assert built < 7 * 20000, "every sweep rebuilt every list"
    s.close()
