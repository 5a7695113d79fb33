"""The voxeliser's stamp of grids with fewer than three cells on an axis
(csrc/cloud_volume.cu cloudStampLooseKernel and cloudStampLooseBoxKernel), where
boxes leave the grid and their indices wrap into other rows: one and two cells
on each axis, boxes of a cell, of what a warp shares and of more, surfels and
Gaussians that float cannot decide among them. Against the host restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("cells", [1, 2])
@pytest.mark.parametrize("reach", [0.4, 3.0, 12.0])  # cells
@pytest.mark.parametrize("odd", ["", "surfels", "far"])
def test_flat_clouds(vsimlib, gpu, axis, cells, reach, odd):
    from vsim import voxelize as vz

    rng = np.random.default_rng(axis + 10 * cells)
    h, n = 0.004, 900
    half = np.full(3, 0.07)
    half[axis] = 1e-4
    pos = rng.uniform(-1, 1, (n, 3)) * half
    scale = h * reach / 2 * rng.uniform(0.2, 1.0, (n, 3))
    rot = np.zeros((n, 4))
    rot[:, 3] = 1  # no turn: the flat axis keeps its reach
    turn = rng.uniform(0, 2 * np.pi, n)
    rot[:, axis], rot[:, 3] = np.sin(turn / 2), np.cos(turn / 2)  # about it: any
    scale[:, axis] = h * (0.2 if cells == 1 else 0.4)
    if odd == "surfels":
        scale[::3, axis] = 0.0
        scale[1::3, (axis + 1) % 3] = 1e-8
    if odd == "far":  # past what float decides
        pos, scale, h = pos * 2.0 ** 42, scale * 2.0 ** 42, h * 2.0 ** 42
    args = [a.astype(np.float32) for a in (pos, rot, scale)]
    host = vz.voxelize_cloud(*args, h, padding=0, fill=False)
    dev = vz.voxelize_cloud_on_device(*args, h, padding=0, fill=False)
    assert min(host.dims) < 3
    assert dev.dims == host.dims and dev.origin == host.origin
    assert np.array_equal(dev.occupancy, host.occupancy)
