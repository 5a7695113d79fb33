"""The range in which the branch-free projection's roots and divisors have to lie
(csrc/rounded.cuh argumentAndPositive): against the IEEE operators over every
float of it, and coarse, heavy and stiff cells and fine and light ones, whose
determinants lie near its ends and past them, against the oracle, bit for bit."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
INF = float("inf")


def test_every_float_of_the_range(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = tmp_path / "check"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-fmad=false",
                    str(ROOT / "tests" / "float_checks" / "check_positive_range.cu"), "-o", str(out)], check=True)
    run = subprocess.run([str(out)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout + run.stderr


# edge (m), density, Young's modulus, steps a second: determinants of 2^-21, 2^-29, 2^-47 and past the range
# (those cells are done over), 2^107 and past the range
@pytest.mark.parametrize("h,density,youngs,rate", [(1.0, 2000.0, 1e9, 60), (1.0, 2000.0, 2e11, 60),
                                                   (10.0, 2000.0, 1e9, 60), (60.0, 2000.0, 1e9, 60),
                                                   (2e-4, 1000.0, 1e5, 600), (2e-5, 1000.0, 1e5, 600)])
@pytest.mark.parametrize("dims", [(16, 4, 4), (70, 9, 8)])
def test_heavy_and_light_cells(vsimlib, gpu, dims, h, density, youngs, rate):
    import pyoracle
    import vsim.scenes as sc
    from vsim import Simulator

    mat = dict(sc.DEFAULT_MATERIAL, youngs_modulus=youngs, density=density, poisson_ratio=0.3)
    body = sc.Body(dims, (0.0, 0.0, 0.0), h, np.ones(int(np.prod(dims)), np.uint8), mat)
    scene = sc.Scene([body], ((-INF,) * 3, (INF,) * 3), step_duration=1 / rate, substeps=3, contact=False)
    rest = sc.rest_positions(body).astype(np.float64)
    off = rest + 0.03 * h * np.random.default_rng(4).standard_normal(rest.shape)
    pos = np.concatenate([off, np.zeros((len(off), 1))], 1).astype(np.float32)
    sim, orc = Simulator(scene), pyoracle.Oracle(scene, 32)
    zero = np.zeros_like(pos)
    sim.write_state(pos, pos, zero)
    orc.set_state(pos, pos, zero)
    for frame in range(3):
        sim.dispatch(3)
        orc.dispatch(3)
        for name, g, o in zip(("pos", "prev", "vel"), sim.read_state(), orc.state()):
            assert np.array_equal(g, o, equal_nan=True), f"frame {frame}: {name}"
    sim.destroy()
