"""The two-launch contact's buffers (csrc/sim.cu makeSlots): held only once
contact can touch anything, and where the device has no room for them the frames
run all the same, in the longer chain, until there is."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def scene():
    """A small body in a tank of 34 million buckets."""
    import vsim.scenes as sc

    body = sc.Body((9, 8, 7), (0.0, 0.02, 0.0), sc.H, np.ones(504, np.uint8), dict(sc.DEFAULT_MATERIAL))
    edge = 323 * sc.H
    return sc.Scene([body], ((-0.1, 0.0, -0.1), (edge - 0.1, edge, edge - 0.1)), step_duration=1 / 600, substeps=4,
                    self_contact=False)


def folded(scene):
    import vsim.scenes as sc

    pos = np.concatenate([sc.rest_positions(scene.bodies[0]), np.zeros((scene.bodies[0].node_count, 1), np.float32)], 1)
    pos[:, 1] *= np.float32(0.6)
    return pos


def free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_held_when_contact_matters(vsimlib, gpu, scene):
    from vsim import Simulator

    buckets = 33e6
    Simulator(scene).destroy()  # what the library and the driver keep
    before = free()
    sim = Simulator(scene)
    alone = before - free()
    assert alone < 10 * buckets  # counts and starts
    assert sim.frame_launches(1) == 1  # nothing can touch: no contact, one launch
    sim.set_self_contact(True)
    assert before - free() > alone + 20 * buckets
    short = sim.frame_launches(1)
    sim.set_gather_mapping("thread")
    assert short < sim.frame_launches(1)
    sim.destroy()


def test_no_room(vsimlib, gpu, scene):
    import pyoracle
    import torch
    from vsim import Simulator

    # the oracle's tank ends nearer, past where the body goes
    near = replace(scene, tank=(scene.tank[0], (0.7, 0.7, 0.7)))
    sim, orc = Simulator(scene), pyoracle.Oracle(near, 32)
    torch.cuda.empty_cache()
    held = torch.empty(max(free() - (400 << 20), 1), dtype=torch.uint8, device="cuda")  # the slots alone need 520 MB
    sim.set_self_contact(True)
    orc.set_self_contact(True)
    pos = folded(scene)
    sim.write_state(pos, pos, np.zeros_like(pos))
    orc.set_state(pos, pos, np.zeros_like(pos))

    def frames():
        for frame in range(2):
            sim.dispatch(4)
            orc.dispatch(4)
            for name, g, o in zip(("pos", "prev", "vel"), sim.read_state(), orc.state()):
                assert np.array_equal(g, o), f"frame {frame}: {name}"
        return sim.frame_launches(1)

    longer = frames()
    del held
    torch.cuda.empty_cache()
    sim.set_self_contact(True)
    assert frames() < longer
    sim.destroy()
