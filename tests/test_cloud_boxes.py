"""The voxeliser's larger boxes (csrc/cloud_volume.cu cloudStampBoxKernel)
where warps meet at one brick: boxes that lie on one another, whose bricks fill
while others look at them, and blocks that hold boxes tested in float, brick by
brick, beside boxes tested in double, cell by cell. Against the host
restatement, several times over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thin", [0, 2, 3])  # every n-th a surfel of next to no thickness
@pytest.mark.parametrize("half", [0.01, 0.06])
def test_boxes_on_one_another(vsimlib, gpu, half, thin):
    from vsim import voxelize as vz

    rng = np.random.default_rng(5 + thin)
    n = 2500
    pos = rng.uniform(-half, half, (n, 3)).astype(np.float32)
    rot = rng.normal(size=(n, 4))
    rot = (rot / np.linalg.norm(rot, axis=1, keepdims=True)).astype(np.float32)
    scale = (0.02 * rng.uniform(0.4, 1.0, (n, 3))).astype(np.float32)  # boxes of about ten cells an axis
    if thin:
        scale[::thin, 1] = 1e-7
    host = vz.voxelize_cloud(pos, rot, scale, 0.004, fill=False)
    for _ in range(4):
        dev = vz.voxelize_cloud_on_device(pos, rot, scale, 0.004, fill=False)
        assert dev.dims == host.dims and np.array_equal(dev.occupancy, host.occupancy)
