"""Few particles in a large grid (needs a GPU): the grid's extent changes no
result, and the per-sweep tables over its cells cost what clearing them costs."""
import numpy as np
import pytest
import torch

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import workloads

pytestmark = pytest.mark.gpu


def _scene(n, cells, adaptive=0):
    """n particles (r = 0.005) at 1.9 r in one corner of a cube of cells^3 cells."""
    r = 0.005
    side = int(np.ceil(n ** (1 / 3)))
    d = workloads.box_drop(2, substeps=8, adaptive=adaptive)
    length = np.float32(workloads.CELL_PER_RADIUS * r)
    space = (max(0.5, 1.9 * r * side + 0.1),) * 3
    walls, _ = workloads.box_walls(space, length)
    p = workloads.lattice((side,) * 3, 1.9 * r, (0.03,) * 3, 0.1 * r, 1)[:n]
    params = workloads.scaled_params(r, iters=4)
    params.merge_enabled, params.upsample_enabled = adaptive, 0
    d.update(particles=p, n_particles=n, boundary=walls, n_boundary=len(walls), space_size=space, cell_size=(cells,) * 3,
             cell_length=float(length), density=workloads.density_for_radius(r), params=params)
    return gg.GranularSystem(**workloads.system_kwargs(d), device=0)


# grids that the sweep's own threads clear, and 512 entries a thread and more
@pytest.mark.parametrize("n,small,large", [(300, 60, 180), (5000, 60, 400), (20000, 60, 450), (110000, 80, 400)])
def test_extent_changes_no_result(n, small, large):
    out = []
    for cells in (small, large):
        s = _scene(n, cells, adaptive=1)
        s.step(4)
        out.append([s.read(f) for f in (gg.FIELD_POS, gg.FIELD_VEL, gg.FIELD_MASS, gg.FIELD_NUM_CONSTRAINTS)])
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_sweeps_of_few_particles_cost_the_clear():
    """Seven sweeps of 300 particles over 100 M cells: at most seven clears of
    a table of that size and 50 us each."""
    s = _scene(300, 464)
    s.step(2)
    sweeps = clear = 1e9
    for _ in range(5):
        s.profile_begin()
        s.step(1)
        sweeps = min(sweeps, s.profile_end()["sweep"]["ms"])
    s.close()
    table = torch.empty(464 ** 3 + 1, dtype=torch.int32, device="cuda")
    for _ in range(5):
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        table.zero_()
        t1.record()
        torch.cuda.synchronize()
        clear = min(clear, t0.elapsed_time(t1))
    assert sweeps <= 7 * (clear + 0.05)
