"""vsim_tune: a sweep where frames read the launch shape (a run of over 256 cells
sends them to the colour passes, as the four-lane form does), and the caller's
shape back at once where they do not; the state stays either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,lanes,sweeps", [(300, 1, True), (40, 4, True), (40, 1, False)])
def test_tune(vsimlib, gpu, nx, lanes, sweeps):
    import pyoracle
    import vsim.scenes as sc
    from vsim import Simulator

    dims = (nx, 3, 4)
    body = sc.Body(dims, (0.0, 0.02, 0.0), sc.H, np.ones(int(np.prod(dims)), np.uint8), dict(sc.DEFAULT_MATERIAL))
    scene = sc.Scene([body], ((-1.0, 0.0, -1.0), (6.0, 1.0, 1.0)), step_duration=1 / 600, substeps=5, contact=False)
    sim, orc = Simulator(scene), pyoracle.Oracle(scene, 32)
    sim.set_cell_lanes(lanes)
    sim.set_launch_shape(512, 8)
    sim.dispatch(5)
    orc.dispatch(5)
    before = sim.read_state()
    shape = sim.tune(1)
    if sweeps:
        assert shape[0] in (128, 256, 512) and shape[1] in (0, 4, 8)
    else:
        assert shape == (512, 8)
    for frame in range(2):
        for name, g, o in zip(("pos", "prev", "vel"), sim.read_state(), orc.state()):
            assert np.array_equal(g, o), f"frame {frame}: {name}"
        if frame == 0:
            for a, b in zip(before, sim.read_state()):
                assert np.array_equal(a, b)
        sim.dispatch(5)
        orc.dispatch(5)
    sim.destroy()
