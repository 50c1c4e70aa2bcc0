"""The profile's count of contact-list builds over graph replays (needs a GPU)."""
import pytest

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [7, 20, 50])  # a group of lanes to a particle, and a thread
def test_replays_count_their_builds(side):
    counts = []
    for graph in (False, True):
        s = gg.GranularSystem(**workloads.system_kwargs(workloads.box_drop(side, configured=True)), device=0)
        s.step(2)
        if graph:
            s.graph_capture(2)
        s.profile_begin()
        for _ in range(3):
            if graph:
                s.graph_launch()
            else:
                s.step(2)
        counts.append(s.profile_end()["_nlist_rebuilds"])
        s.close()
    assert counts[0] == counts[1] >= 6 * side ** 3
