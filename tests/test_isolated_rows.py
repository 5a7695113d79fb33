"""Isolated bodies' frames either side of where row passes pay (csrc/sim.cu
rowsPay): pools of up to a wave of groups, of more nearly empty ones (which take
the colours), and of more that are full enough, against the oracle; and a
server's ticks over a pool that takes the colours."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pool(count, dims):
    import vsim.scenes as sc

    rng = np.random.default_rng(count)
    bodies = []
    for b in range(count):
        occ = (rng.random(np.prod(dims)) < 0.9).astype(np.uint8)
        occ[0] = 1
        mat = dict(sc.DEFAULT_MATERIAL, youngs_modulus=float(rng.uniform(5e4, 4e5)))
        bodies.append(sc.Body(dims, (0.0, 0.01, 0.0), sc.H, occ, mat))
    return bodies, ((-0.5, 0.0, -0.5), (1.5, 1.5, 1.5))


@pytest.mark.parametrize("count,dims,passes", [(100, (2, 2, 2), 4), (456, (2, 2, 2), 4), (457, (2, 2, 2), 8),
                                               (600, (3, 2, 2), 8), (470, (9, 8, 8), 4), (460, (6, 6, 6), 8)])
def test_pools(vsimlib, gpu, count, dims, passes):
    import pyoracle
    import vsim.scenes as sc
    from vsim import Simulator

    bodies, tank = pool(count, dims)
    scene = sc.Scene(bodies, tank, step_duration=1 / 600, substeps=4, contact=True, self_contact=True, isolated=True)
    sim, orc = Simulator(scene), pyoracle.Oracle(scene, 32)
    sim.set_contact(False)
    assert sim.frame_launches(1) == 2 + passes
    sim.set_contact(True)
    for frame in range(2):
        sim.dispatch(4)
        orc.dispatch(4)
        for name, g, o in zip(("pos", "prev", "vel"), sim.read_state(), orc.state()):
            assert np.array_equal(g, o), f"frame {frame}: {name}"
    sim.destroy()


def test_ticks_of_a_pool_in_colours(vsimlib, gpu):
    import pyoracle
    import vsim.scenes as sc
    from vsim.server import Server

    bodies, tank = pool(500, (3, 2, 2))
    server = Server(bodies, tank)
    frames = {0: 2, 7: 1, 255: 3, 499: 1}
    for session, n in frames.items():
        server.submit(session, n)
    while server.stats()["pending"]:
        server.tick()
        server.poll()
    for session, n in frames.items():
        orc = pyoracle.Oracle(sc.Scene([bodies[session]], tank, step_duration=1 / 600, substeps=10, contact=True,
                                       self_contact=True, isolated=True), 32)
        for _ in range(n):
            orc.dispatch(10)
        assert np.array_equal(server.read_positions(session), orc.state()[0]), f"session {session}"
    server.destroy()
