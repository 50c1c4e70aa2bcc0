"""The per-particle passes that run launched chained, whose pointers are not
__restrict__: their loads must still be in flight together (needs a GPU)."""
import numpy as np
import pytest
import torch

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import workloads

pytestmark = pytest.mark.gpu

# bytes a particle: the permutation, both ways for position and velocity
# (float4) and for eight 4-byte fields
REORDER_BYTES = 4 + 2 * (16 + 16 + 8 * 4)


def _copy_rate(nbytes):
    a = torch.empty(nbytes // 2, dtype=torch.uint8, device="cuda")
    b = torch.empty_like(a)
    best = 1e9
    for _ in range(10):
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        b.copy_(a)
        t1.record()
        torch.cuda.synchronize()
        best = min(best, t0.elapsed_time(t1))
    return nbytes / best


def test_reorder_runs_at_the_copy_rate():
    """The reorder of 8 M particles moves its bytes at 85 % of the rate of a
    copy of as many at least (a lattice: its gathers are nearly in order)."""
    d = workloads.column_collapse((128, 256, 256), upsample_per=0, adaptive=0)
    n = d["n_particles"]
    s = gg.GranularSystem(**workloads.system_kwargs(d))
    best = 1e9
    for _ in range(5):
        s.profile_begin()
        s.step(1)
        best = min(best, s.profile_end()["reorder"]["ms"])
    s.close()
    assert n * REORDER_BYTES / best >= 0.85 * _copy_rate(n * REORDER_BYTES)
