"""The row pass (two colours a launch, csrc/step_kernels.cu elasticRowKernel)
against the oracle, bit for bit, at the sizes where its links, chains and
groups end: one to a few cells, a chain that fills a warp and one past it, a
chain that fills a group and one past it (which takes the colours one by
one), rows with gaps, several bodies whose chains share groups, the stretch
limit, and cells whose operands leave the branch-free arithmetic's ranges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(vsimlib, gpu):
    return vsimlib


def scene_of(rows, holes=0.0, seed=0, stretch=0.0):
    import vsim.scenes as sc

    rng = np.random.default_rng(seed)
    bodies = []
    for b, dims in enumerate(rows):
        occ = (rng.random(dims[0] * dims[1] * dims[2]) >= holes).astype(np.uint8)
        occ[0] = 1
        mat = dict(sc.DEFAULT_MATERIAL, max_stretch=stretch)
        bodies.append(sc.Body(tuple(dims), (0.0, 0.3 * b, 0.0), sc.H, occ, mat))
    inf = float("inf")
    return sc.Scene(bodies, ((-inf, -inf, -inf), (inf, inf, inf)), step_duration=1 / 600, substeps=3, contact=False)


def run(scene, pos, frames=2):
    import pyoracle
    from vsim import Simulator

    sim, orc = Simulator(scene), pyoracle.Oracle(scene, 32)
    vel = np.zeros_like(pos)
    sim.write_state(pos, pos, vel)
    orc.set_state(pos, pos, vel)
    for frame in range(frames):
        sim.dispatch(scene.substeps)
        orc.dispatch(scene.substeps)
        for name, g, o in zip(("pos", "prev", "vel"), sim.read_state(), orc.state()):
            bad = np.flatnonzero(np.any(g != o, axis=1))
            assert bad.size == 0, f"frame {frame}: {name} differs at {bad.size} nodes, first {bad[:5]}"
    launches = sim.frame_launches(1)
    sim.destroy()
    return launches


def strained(scene, seed=5, amount=0.15):
    import vsim.scenes as sc

    rng = np.random.default_rng(seed)
    rest = np.concatenate([sc.rest_positions(b) for b in scene.bodies]).astype(np.float64)
    moved = rest + amount * sc.H * rng.standard_normal(rest.shape)
    return np.concatenate([moved, np.zeros((len(rest), 1))], 1).astype(np.float32)


@pytest.mark.parametrize("nx", [1, 2, 3, 4, 63, 64, 65, 66, 127, 255, 256, 257, 258])
@pytest.mark.parametrize("holes", [0.0, 0.3])
def test_row_lengths(lib, nx, holes):
    scene = scene_of([(nx, 3, 2)], holes, seed=nx)
    launches = run(scene, strained(scene))
    if holes == 0.0:
        # a pass's two rows in one group: the frame in one launch; in two:
        # predict, close and the row passes; a run past a group: the colours
        assert launches == (1 if nx <= 128 else 6 if nx <= 256 else 10)


def test_bodies_share_groups(lib):
    scene = scene_of([(5, 4, 3), (64, 2, 2), (1, 1, 1), (130, 3, 3), (17, 9, 4)], 0.2, seed=3)
    run(scene, strained(scene))


def test_stretch_limit(lib):
    scene = scene_of([(70, 3, 3), (9, 5, 4)], 0.1, seed=4, stretch=1.08)
    run(scene, strained(scene, amount=0.2))


def test_operands_out_of_range(lib):
    """Elements collapsed to a point, to a line and blown up far past the
    ranges: those cells, even and odd, are done over with the IEEE operators."""
    import vsim.scenes as sc

    scene = scene_of([(70, 3, 3)], 0.0, seed=6)
    pos = strained(scene)
    nx, ny, nz = scene.bodies[0].node_dims
    grid = pos.reshape(nz, ny, nx, 4)
    grid[:, :, 4:7, :3] = grid[0, 0, 5, :3]            # an even and an odd cell, every node at one place
    grid[:, :, 21:23, :3] = grid[0, 0, 21, :3]         # one odd cell
    grid[:2, :2, 40:42, :3] *= np.float32(1e-12)       # tiny
    grid[1:, 1:, 50:52, :3] += np.float32(3e4) * sc.H  # enormous
    run(scene, pos, frames=1)


@pytest.mark.parametrize("rows,stretch", [([(171, 64, 90)], 0.0), ([(171, 64, 90)], 1.1),
                                          ([(31 + b % 7, 24, 25 - b % 5) for b in range(44)], 0.0)])
def test_many_groups(lib, rows, stretch):
    """Passes of more groups than three a multiprocessor, which a block takes
    in turn: one body with gaps, with the stretch limit, and bodies that
    change from group to group."""
    scene = scene_of(rows, 0.15, seed=8, stretch=stretch)
    scene.substeps = 2
    run(scene, strained(scene, amount=0.1), frames=1)


@pytest.mark.parametrize("longest", [40, 256, 257])
@pytest.mark.parametrize("stretch", [0.0, 1.05])
def test_rows_of_sessions_in_ticks(lib, longest, stretch):
    """Sessions stepped in shared frames, some of them at a time: each body's
    groups are its own, and a body with a run of 257 cells sends all of them
    the colours' way."""
    import pyoracle
    import vsim.scenes as sc
    from vsim.server import Server

    rng = np.random.default_rng(longest)
    bodies = []
    for dims in ((1, 1, 1), (3, 2, 1), (longest, 2, 3), (9, 7, 5), (130, 3, 2), (2, 40, 3)):
        occ = (rng.random(np.prod(dims)) >= 0.15).astype(np.uint8)
        occ[: dims[0]] = 1
        bodies.append(sc.Body(dims, (0.0, 0.02, 0.0), sc.H, occ, dict(sc.DEFAULT_MATERIAL, max_stretch=stretch)))
    tank = ((-1.0, 0.0, -1.0), (6.0, 3.0, 6.0))
    server = Server(bodies, tank)
    frames = [2, 1, 3, 2, 0, 3]
    for b, n in enumerate(frames):
        if n:
            server.submit(b, n, None)
    while server.stats()["pending"]:
        server.tick()
        server.poll()
    for b, n in enumerate(frames):
        orc = pyoracle.Oracle(sc.Scene([bodies[b]], tank, step_duration=1 / 600, substeps=10, contact=True,
                                       self_contact=True, isolated=True), 32)
        for _ in range(n):
            orc.dispatch(10)
        assert np.array_equal(server.read_positions(b), orc.state()[0]), f"session {b}"
    server.destroy()
