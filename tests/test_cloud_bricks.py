"""The voxeliser's stamp in 4 x 4 x 4 bricks against the host restatement,
where its ways part: boxes of one and two bricks an axis and of more, at every
place in a brick; grids of one to five cells on an axis, where boxes leave the
grid; clouds whose every Gaussian float cannot decide; rotations off a 16-byte
boundary; more Gaussians than one round of a block, and fewer than a warp. And
the plain float frame's reach bracket on the host."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


def _cloud(n, half, reach, seed):
    rng = np.random.default_rng(seed)
    half = np.broadcast_to(np.asarray(half, float), 3)
    pos = (rng.uniform(-1, 1, (n, 3)) * half).astype(np.float32)
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    scale = reach * rng.uniform(0.2, 0.5, (n, 3))
    return pos, q.astype(np.float32), scale.astype(np.float32)


@pytest.fixture(scope="module")
def vz(vsimlib, gpu):
    from vsim import voxelize

    return voxelize


def _same(vz, cloud, element, **kw):
    host_stats, dev_stats = {}, {}
    host = vz.voxelize_cloud(*cloud, element, stats=host_stats, **kw)
    dev = vz.voxelize_cloud_on_device(*cloud, element, stats=dev_stats, **kw)
    assert dev.dims == host.dims and dev.origin == host.origin and dev.h == host.h
    assert np.array_equal(dev.occupancy, host.occupancy)
    assert dev_stats == host_stats


@pytest.mark.gpu
@pytest.mark.parametrize("cells", [0.3, 1.0, 2.0, 2.6, 4.0, 9.0])
@pytest.mark.parametrize("n", [5, 700])
def test_box_spans(vz, cells, n):
    # reaches of `cells` cells: one brick an axis, two, and three and more
    _same(vz, _cloud(n, 0.05, 0.004 * cells, seed=n), 0.004, fill=False)


@pytest.mark.gpu
@pytest.mark.parametrize("fill", [False, True])
@pytest.mark.parametrize("padding", [0, 1, 2])
@pytest.mark.parametrize("half", [(0.001, 0.03, 0.03), (0.03, 0.003, 0.03), (0.03, 0.03, 0.005), (0.001, 0.001, 0.03),
                                  (0.03, 0.002, 0.002), (0.001, 0.001, 0.001)])
def test_thin_grids(vz, half, padding, fill):
    _same(vz, _cloud(300, half, 0.0009, seed=3), 0.004, padding=padding, fill=fill)


@pytest.mark.gpu
@pytest.mark.parametrize("cells", [1.0, 6.0])
def test_out_of_float_range(vz, cells):
    # 2^42 times a cloud of 0.05 m: no edge or centre is decided in float
    pos, rot, scale = _cloud(400, 0.05, 0.004 * cells, seed=8)
    big = np.float32(2.0 ** 42)
    _same(vz, (pos * big, rot, scale * big), 0.004 * 2.0 ** 42)


@pytest.mark.gpu
@pytest.mark.parametrize("thin", [0.0, 1e-7, 1e-5])
@pytest.mark.parametrize("cells", [1.0, 7.0])
def test_surfels(vz, cells, thin):
    # an axis of no or next to no thickness: every sample goes to double
    pos, rot, scale = _cloud(300, 0.05, 0.004 * cells, seed=12)
    scale[::2, 1] = thin
    _same(vz, (pos, rot, scale), 0.004)


@pytest.mark.gpu
def test_rotations_off_a_boundary(vz):
    import torch

    cloud = _cloud(3000, 0.05, 0.006, seed=4)
    host = vz.voxelize_cloud(*cloud, 0.004)
    pos, rot, scale = (torch.from_numpy(a).cuda() for a in cloud)
    held = torch.empty(rot.numel() + 1, device="cuda")
    off = held[1:].view(rot.shape).copy_(rot)
    assert off.data_ptr() % 16 == 4
    dev = vz.voxelize_cloud_on_device(pos, off, scale, 0.004)
    assert dev.dims == host.dims and np.array_equal(dev.occupancy, host.occupancy)


CHECK = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include "float_bounds.cuh"
using namespace vsim;
int main() {
    std::mt19937_64 g(7);
    auto uni = [&] { return double(g() >> 11) * 0x1p-53; };
    long bad = 0, held = 0;
    for (long n = 0; n < 400000; n++) {
        float q[4], scale[3], rf[3], col[9], plain[9];
        double v[4], len = 0, r[3];
        for (int k = 0; k < 4; k++) { v[k] = uni() * 2 - 1; len += v[k] * v[k]; }
        // unit, nearly axis-aligned, or of any length
        if (n % 3 == 1) { v[n % 4] *= 1e-6; v[(n + 1) % 4] *= 1e-3; }
        const double by = n % 3 == 2 ? std::pow(10.0, uni() * 6 - 3) : 1 / std::sqrt(len);
        for (int k = 0; k < 4; k++) q[k] = float(v[k] * by);
        const double x = q[0], y = q[1], z = q[2], w = q[3];
        const double e[9] = {1.0 - 2.0 * (y * y + z * z), 2.0 * (x * y + z * w), 2.0 * (x * z - y * w),
                             2.0 * (x * y - z * w), 1.0 - 2.0 * (x * x + z * z), 2.0 * (y * z + x * w),
                             2.0 * (x * z + y * w), 2.0 * (y * z - x * w), 1.0 - 2.0 * (x * x + y * y)};
        for (int k = 0; k < 9; k++) col[k] = float(e[k]);
        const double sigma = 2.0;
        for (int a = 0; a < 3; a++) {
            scale[a] = float(std::pow(10.0, uni() * 6 - 5));  // axes up to a million to one
            r[a] = sigma * double(scale[a]);
            rf[a] = bounds::radiusEstimate(float(sigma), scale[a]);
        }
        bounds::frameInFloat(q[0], q[1], q[2], q[3], plain);
        const float slack = bounds::reachSlack(q[0], q[1], q[2], q[3], rf);
        for (int a = 0; a < 3; a++) {
            const float hf = bounds::reachEstimate(plain, rf, a);
            if (std::isnan(hf)) continue;
            const double exact = bounds::hypotV8(double(col[a]) * r[0], double(col[3 + a]) * r[1], double(col[6 + a]) * r[2]);
            const float narrow = hf * float(1.0 - bounds::kReachSlack) - slack;
            const float wide = hf * float(1.0 + bounds::kReachSlack) + slack;
            held++;
            if (!(double(narrow) <= exact && exact <= double(wide))) bad++;
        }
    }
    std::printf("%ld held, %ld bad\n", held, bad);
    return bad || held < 1000000;
}
"""


def test_reach_bracket_of_the_plain_frame(tmp_path):
    source = tmp_path / "check.cpp"
    source.write_text(CHECK)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "visionary-sim_gb300" / "csrc"),
                    str(source), "-o", str(tmp_path / "check")], check=True)
    run = subprocess.run([str(tmp_path / "check")], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
