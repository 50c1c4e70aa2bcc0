"""Which partner finds a particle, decided from the particle's window of
positions, against the oracle's division and truncation (needs a GPU).

Pairs in contact with one particle on a cell face or an ulp beside it, in
cells from the grid's first to its last, so that the partner's query cell is
one, two or no cells away from the particle's binning cell; no gravity, one
sweep, so x* stays where it is put."""
import numpy as np
import pytest

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import abi, workloads
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [0.01, 0.005, 0.002])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("skin", [-1.0, 0.0])
def test_counts_at_cell_faces_match_oracle(r, axis, skin):
    L = np.float32(workloads.CELL_PER_RADIUS * r)
    cells = (9, 8, 7)
    points = []
    row = 0
    for k in range(0, cells[axis] + 1):
        face = np.float32(k) * L
        for a in (np.nextafter(face, np.float32(-1)), face, np.nextafter(face, np.float32(9)), face - L, face + L):
            # (a partner in contact is nearer than a cell, so the far ends
            # of the window are met from the face one cell further)
            for off in (-1.9 * r, 0.3 * r, 1.9 * r):
                base = np.array([L * (1.5 + 2 * (row % 3)), L * 1.5, L * 1.5], np.float32)
                base[(axis + 1) % 3] = L * (0.7 + 0.03 * (row % 17))
                p, q = base.copy(), base.copy()
                p[axis] = a
                q[axis] = np.float32(a + off)
                points += [p, q]
                row += 1
    points = np.array(points, np.float32)
    # keep the pairs apart from each other along the third axis, scene by scene
    for chunk in range(0, len(points), 12):
        d = workloads.box_drop(2, substeps=4)
        p = points[chunk:chunk + 12].copy()
        third = (axis + 2) % 3
        for k in range(len(p) // 2):
            p[2 * k:2 * k + 2, third] = L * np.float32(0.6 + (k % 3) * 2.1)
        d.update(particles=p, n_particles=len(p), boundary=np.zeros((0, 3), np.float32), n_boundary=0,
                 cell_size=cells, cell_length=float(L), space_size=tuple(float(c * L) for c in cells),
                 gravity=(0.0, 0.0, 0.0), density=workloads.density_for_radius(r))
        d["params"].math_mode, d["params"].stab_iters, d["params"].iters = 1, 0, 1
        d["params"].nlist_skin = skin
        s = gg.GranularSystem(**workloads.system_kwargs(d), device=0)
        o = orc.OracleSystem(d, fp64=False)
        assert np.array_equal(s.read(gg.FIELD_CONTACTS), o.read(abi.FIELD_CONTACTS))
        assert np.array_equal(s.read(gg.FIELD_NUM_CONSTRAINTS), o.read(abi.FIELD_NUM_CONSTRAINTS))
        assert np.array_equal(s.read(gg.FIELD_POS), o.read(abi.FIELD_POS))
        s.close()
        o.close()
