"""The upsampling on packed pairs of candidates (needs a GPU): its square
root against sqrtf, and its render points against the oracle."""
import os
import subprocess

import numpy as np
import pytest

import granular_gpu_gb300 as gg
from granular_gpu_gb300 import abi, workloads
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")


def test_packed_square_root_equals_sqrtf_for_every_float(tmp_path):
    exe = str(tmp_path / "sqrt2_check")
    subprocess.run([NVCC, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-fmad=false", "-std=c++17",
                    os.path.join(HERE, "cpp", "sqrt2_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "differ: 0", r.stdout + r.stderr


@pytest.mark.parametrize("counts", [(1, 1, 1), (2, 1, 1), (3, 1, 1), (5, 7, 9), (12, 11, 13)])
@pytest.mark.parametrize("odd", ["", "coincident", "nan", "far"])
def test_whole_stencil_render_points_match_oracle(counts, odd):
    """The support covers the stencil (0.045 at cells of 0.00808); odd and
    even particle counts and columns; a render point on a particle, a NaN
    particle, a particle far from the cell it was binned in."""
    d = workloads.column_collapse(counts, adaptive=0, upsample_per=4, constants="reference", skip=True)
    d["params"].math_mode = 1
    p, u = d["particles"], d["upsampled"]
    if odd == "coincident":
        u[: len(p)] = p
        d["gravity"] = (0.0, 0.0, 0.0)
    s = gg.GranularSystem(**workloads.system_kwargs(d), device=0)
    o = orc.OracleSystem(d, fp64=False)
    if odd in ("nan", "far"):
        v = np.zeros_like(p)
        v[len(p) // 2] = np.nan if odd == "nan" else (40.0, 0.0, 0.0)
        s.write(gg.FIELD_VEL, v)
        o.write(abi.FIELD_VEL, v)
    for k in range(3):
        s.step(1)
        o.step(1)
        for f in (gg.FIELD_POS, gg.FIELD_VEL):
            a, b = s.read(f, gg.SET_UPSAMPLED), o.read(f, abi.SET_UPSAMPLED)
            assert np.array_equal(a, b, equal_nan=True), f"step {k}, field {f}"
        assert np.array_equal(s.read(gg.FIELD_POS), o.read(abi.FIELD_POS), equal_nan=True)
    s.close()
    o.close()
