"""Contact in two launches (csrc/step_kernels.cu joinCrowd and collideFull) where
buckets are full: bodies whose cells differ in size, so that the finer one's
records share buckets of the coarser one's edge; heaps in the tank's outermost
buckets, of records a few past the 32 a bucket shows and of thousands; and
scenes that have gone NaN, whose records are all in the first bucket. Against
the oracle and the five-launch chain, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(scene, pos, frames=3, compare="oracle", short=True):
    """Frames from `pos` (`short`: of the two-launch chain); returns the last positions."""
    import pyoracle
    from vsim import Simulator

    steps = scene.substeps
    zero = np.zeros_like(pos)
    sim = Simulator(scene)
    sim.write_state(pos, pos, zero)
    longer = Simulator(scene)
    longer.set_gather_mapping("thread")
    longer.write_state(pos, pos, zero)
    others = [longer]
    if short is not None:
        assert (sim.frame_launches(1) < longer.frame_launches(1)) == short
    if compare == "oracle":
        orc = pyoracle.Oracle(scene, 32)
        orc.set_state(pos, pos, zero)
        others.append(orc)
    for frame in range(frames):
        sim.dispatch(steps)
        got = sim.read_state()
        for other in others:
            other.dispatch(steps)
            want = other.read_state() if other is longer else other.state()
            for name, g, o in zip(("pos", "prev", "vel"), got, want):
                same = (g == o) | (np.isnan(g) & np.isnan(o))
                bad = np.flatnonzero(~same.all(axis=1))
                assert bad.size == 0, f"frame {frame}: {name} differs from {type(other).__name__} at {bad.size} nodes"
    sim.destroy()
    longer.destroy()
    return got[0]


# squeeze: how far the finer body is squeezed. The coarser one's cells are `ratio`
# times its own; past two records a bucket at rest the scene takes the longer chain
@pytest.mark.parametrize("ratio,holes,squeeze,short", [
    (2, 0.0, 0.9, True), (2, 0.0, 0.6, True), (2, 0.0, 0.35, True), (2, 0.35, 0.7, False), (3, 0.0, 0.7, False),
    (3, 0.35, 0.7, False), (4, 0.0, 0.7, False)])
def test_cells_of_two_sizes(vsimlib, gpu, ratio, holes, squeeze, short):
    import vsim.scenes as sc

    rng = np.random.default_rng(ratio)
    dims = (30, 22, 28)
    fine = sc.Body(dims, (0.01, 0.004, 0.01), sc.H, (rng.random(np.prod(dims)) >= holes).astype(np.uint8),
                   dict(sc.DEFAULT_MATERIAL, density=800.0))
    coarse = sc.Body((6, 3, 5), (0.03, 22.5 * squeeze * sc.H, 0.0), ratio * sc.H, np.ones(90, np.uint8),
                     dict(sc.DEFAULT_MATERIAL))
    scene = sc.Scene([fine, coarse], ((-0.2, 0.0, -0.2), (0.8, 1.0, 0.8)), step_duration=1 / 600, substeps=4,
                     self_contact=True)
    pos = np.concatenate([sc.rest_positions(fine), sc.rest_positions(coarse)])
    pos = np.concatenate([pos, np.zeros((len(pos), 1), np.float32)], 1)
    pos[: fine.node_count, :3] *= np.float32(squeeze)  # it touches itself and the coarse one
    check(scene, pos, frames=2, short=short)


@pytest.mark.parametrize("records,far", [(31, 1), (32, 1), (33, 1), (34, 3), (64, 1), (65, 5), (2400, 1)])
def test_heaps_at_a_corner(vsimlib, gpu, records, far):
    """Nodes put past the tank's corner, out of reach of each other or nearly
    in one place: all in the corner's bucket, `records` of them surface
    records; `far` corners at once."""
    import vsim.scenes as sc

    n = 21
    body = sc.Body((n, n, n), (0.0, 0.1, 0.0), sc.H, np.ones(n ** 3, np.uint8), dict(sc.DEFAULT_MATERIAL))
    scene = sc.Scene([body], ((-0.1, 0.0, -0.1), (0.6, 0.6, 0.6)), step_duration=1 / 600, substeps=3, self_contact=True)
    rng = np.random.default_rng(records)
    pos = np.concatenate([sc.rest_positions(body), np.zeros((body.node_count, 1), np.float32)], 1)
    surface = rng.permutation(sc.surface_nodes(body))[: records]
    corner = np.arange(len(surface)) % far
    away = np.stack([np.where(corner & 1, 0.7, -0.2), np.where(corner & 2, 0.8, 0.75), np.where(corner & 4, 0.7, -0.2)], 1)
    pos[surface, :3] = away + rng.uniform(0, 0.05, (len(surface), 3))
    check(scene, pos, frames=2)


def test_a_whole_body_past_a_corner(vsimlib, gpu):
    import vsim.scenes as sc

    scene = sc.noise_blob(n=24, seed=5, splats=0)
    scene.substeps = 4
    body = scene.bodies[0]
    pos = np.concatenate([sc.rest_positions(body), np.zeros((body.node_count, 1), np.float32)], 1)
    pos[:, :3] += np.float32(2.0)
    check(scene, pos, frames=2)
    # and back among the common ones, on the same simulator: the crowds have gone
    pos[::2, :3] -= np.float32(2.0)
    check(scene, pos, frames=2)


def test_gone_nan(vsimlib, gpu):
    """Every position NaN, and one NaN node that spreads."""
    import vsim.scenes as sc

    scene = sc.noise_blob(n=16, seed=5, splats=0)
    scene.substeps = 3
    body = scene.bodies[0]
    pos = np.concatenate([sc.rest_positions(body), np.zeros((body.node_count, 1), np.float32)], 1)
    one = pos.copy()
    one[sc.surface_nodes(body)[40], 0] = np.nan
    check(scene, one, frames=4, compare="longer chain")
    pos[:, :3] = np.nan
    assert np.isnan(check(scene, pos, frames=2, compare="longer chain")).any()
