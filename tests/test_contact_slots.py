"""Contact in two launches (csrc/step_kernels.cu binSlotsKernel and
collideSlotsKernel) against the oracle, bit for bit, and against the five-launch
chain, where the buckets' slots, the records' lists and the groups of lanes
end: buckets of one to over 32 records (slots, then the overflow list, then
past what a bucket shows), records with more candidates than their list
holds, buckets at the grid's rim, bodies sitting a frame out, record counts
around a block's 24, and contact switched between the two chains."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(vsimlib, gpu):
    return vsimlib


def make(scene):
    import pyoracle
    from vsim import Simulator

    return Simulator(scene), pyoracle.Oracle(scene, 32)


def same(sim, orc, what):
    for name, g, o in zip(("pos", "prev", "vel"), sim.read_state(), orc.state()):
        bad = np.flatnonzero(np.any(g != o, axis=1))
        assert bad.size == 0, f"{what}: {name} differs at {bad.size} nodes, first {bad[:5]}"


def start(sim, orc, pos, vel=None):
    vel = np.zeros_like(pos) if vel is None else vel
    sim.write_state(pos, pos, vel)
    orc.set_state(pos, pos, vel)


# factor: how far the blob is squeezed about its centre -- at most a few
# records a bucket; most buckets past their slots; buckets past 32 records and
# records with hundreds of candidates
@pytest.mark.parametrize("factor", [0.8, 0.45, 0.3, 0.2, 0.12])
def test_crowded_buckets(lib, factor):
    import vsim.scenes as sc

    scene = sc.noise_blob(n=20, seed=5, splats=0)
    sim, orc = make(scene)
    pos = orc.state()[0]
    centre = pos[orc.inv_mass() > 0, :3].mean(axis=0)
    squeezed = pos.copy()
    squeezed[:, :3] = centre + (squeezed[:, :3] - centre) * np.float32(factor)
    start(sim, orc, squeezed)
    assert sim.frame_launches(1) < 10  # the two-launch chain
    for frame in range(3):
        sim.dispatch(scene.substeps)
        orc.dispatch(scene.substeps)
        same(sim, orc, f"factor {factor} frame {frame}")
    sim.destroy()


@pytest.mark.parametrize("side", [1, 2, 3, 5])
def test_small_bodies_in_a_corner(lib, side):
    """Two boxes overlapping in the tank's corner, their buckets at the
    grid's rim (and past it: nodes outside are binned at the rim)."""
    import vsim.scenes as sc

    ones = np.ones(side ** 3, np.uint8)
    a = sc.Body((side,) * 3, (0.0, 0.0, 0.0), sc.H, ones, dict(sc.DEFAULT_MATERIAL))
    b = sc.Body((side,) * 3, (0.006, 0.009, 0.004), sc.H, ones, dict(sc.DEFAULT_MATERIAL, friction=0.1, density=500.0))
    edge = side * sc.H
    scene = sc.Scene([a, b], ((0.0, 0.0, 0.0), (edge, edge, edge)), step_duration=1 / 1200, substeps=5)
    sim, orc = make(scene)
    pos = orc.state()[0]
    vel = np.zeros_like(pos)
    vel[:, :3] = [-1.0, -2.0, 1.5]
    start(sim, orc, pos, vel)
    for frame in range(4):
        sim.dispatch(scene.substeps)
        orc.dispatch(scene.substeps)
        same(sim, orc, f"frame {frame}")
    sim.destroy()


def test_chains_take_turns_and_bodies_sit_out(lib):
    """Frames of both chains on one simulator (the mapping forces the longer
    one), a contact census and a pair list between them, and a body left out
    of some frames: as the longer chain alone gives."""
    import vsim.scenes as sc
    from vsim import Simulator

    rng = np.random.default_rng(3)
    bodies = [sc.Body((6, 5, 7), (0.1 * b, 0.02, 0.02 * b), sc.H, (rng.random(210) < 0.8).astype(np.uint8),
                      dict(sc.DEFAULT_MATERIAL)) for b in range(3)]
    scene = sc.Scene(bodies, ((-0.3, 0.0, -0.3), (0.6, 1.0, 0.5)), step_duration=1 / 600, substeps=6, self_contact=True)
    mixed, plain = Simulator(scene), Simulator(scene)
    plain.set_gather_mapping("warp")
    rest = mixed.read_positions()
    rest[:, 0] *= np.float32(0.6)
    for sim in (mixed, plain):
        sim.write_state(rest, rest, np.zeros_like(rest))
    for frame in range(9):
        active = [True, frame % 3 != 1, True]
        mixed.set_gather_mapping(("auto", "thread", "auto", "warp")[frame % 4])
        for sim in (mixed, plain):
            sim.set_bodies_active(active)
            sim.dispatch(scene.substeps)
        if frame == 4:
            assert mixed.contact_census()["records"] > 0
            assert np.array_equal(mixed.contact_pairs(), plain.contact_pairs())
        for g, o in zip(mixed.read_state(), plain.read_state()):
            assert np.array_equal(g, o), f"frame {frame}"
    mixed.destroy()
    plain.destroy()


@pytest.mark.parametrize("factor", [0.3, 0.1, 0.02])
def test_crowded_buckets_in_order(lib, factor):
    """The five-launch chain's order of a crowded bucket: hundreds and
    thousands of records in one, starting at any place of the order."""
    import vsim.scenes as sc

    scene = sc.noise_blob(n=20, seed=5, splats=0)
    sim, orc = make(scene)
    sim.set_gather_mapping("thread")
    pos = orc.state()[0]
    inside = orc.inv_mass() > 0
    centre = pos[inside, :3].mean(axis=0)
    squeezed = pos.copy()
    squeezed[:, :3] = centre + (squeezed[:, :3] - centre) * np.float32(factor)
    # some where they were, so that the crowd's run starts at an odd place
    squeezed[::17] = pos[::17]
    start(sim, orc, squeezed)
    for frame in range(2):
        sim.dispatch(scene.substeps)
        orc.dispatch(scene.substeps)
        same(sim, orc, f"factor {factor} frame {frame}")
    sim.destroy()
