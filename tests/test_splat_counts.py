"""The splat deformation's stores (whole words through a warp's share of
shared memory, csrc/splat_sort.cu storeXyz) against the oracle, bit for bit,
at the counts where warps and blocks end, and the reads into pinned and
pageable buffers and with outputs left out."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 63, 65, 255, 256, 257, 1000])
def test_counts(vsimlib, gpu, count):
    import pyoracle
    import torch
    import vsim.scenes as sc
    from vsim import Simulator

    scene = sc.noise_blob(n=9, seed=4, splats=count)
    sim, orc = Simulator(scene), pyoracle.Oracle(scene, 32)
    sim.dispatch(4)
    orc.dispatch(4)
    view = (0.2, -0.5, -0.84)
    m, q, s, *_ = scene.splats[0]
    om, oc, keys = orc.splat_deform(0, m, q, s, view)
    for axes in (False, True):
        (sim.deform_splats_axes if axes else sim.deform_splats)(view)
        sim.sort_splats()
        means, cov, order = sim.read_splats()
        assert np.array_equal(means, om) and np.array_equal(cov, oc)
        assert np.array_equal(order, pyoracle.stable_sort(keys))
    rot, scale = sim.read_splat_axes()
    orot, oscale = pyoracle.ellipsoid_axes_f32(oc)
    assert np.array_equal(rot, orot) and np.array_equal(scale, oscale)
    lib = vsimlib.lib()
    pinned = torch.zeros((count, 3), dtype=torch.float32, pin_memory=True)
    fp = C.POINTER(C.c_float)
    assert lib.vsim_splats_read(sim.handle, C.cast(pinned.data_ptr(), fp), None, None, count) == vsimlib.VSIM_OK
    assert np.array_equal(pinned.numpy(), om)
    assert lib.vsim_splats_read_axes(sim.handle, None, C.cast(pinned.data_ptr(), fp), count) == vsimlib.VSIM_OK
    assert np.array_equal(pinned.numpy(), oscale)
    sim.destroy()
