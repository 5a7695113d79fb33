"""Whole scenes either side of the record count up to which contact takes two
launches (csrc/sim.cu kSlotRecordsPerSm): the frame each takes, and that it
equals the five-launch chain's, a thread a record, node for node."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,short", [(172, True), (180, False)])
def test_largest_scene_of_two_launches(vsimlib, gpu, n, short):
    import torch
    import vsim.scenes as sc
    from vsim import Simulator

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms != 152:
        pytest.skip("sized for 152 SMs")
    scene = sc.blob_and_sheet(n, splats=0)
    pos = np.concatenate([sc.rest_positions(b) for b in scene.bodies])
    pos = np.concatenate([pos, np.zeros((len(pos), 1), np.float32)], 1)
    blob = scene.bodies[0].node_count
    pos[:blob, 1] *= np.float32(0.8)          # folded onto itself
    pos[blob:, 1] -= np.float32(0.21 * n * sc.H)  # the sheet in the blob's top
    sims = [Simulator(scene), Simulator(scene)]
    sims[1].set_gather_mapping("thread")
    for sim in sims:
        sim.write_state(pos, pos, np.zeros_like(pos))
    assert (sims[0].stats()["contact_nodes"] <= 3200 * sms) == short
    assert (sims[0].frame_launches(1) < sims[1].frame_launches(1)) == short
    for _ in range(2):
        for sim in sims:
            sim.dispatch(5)
        for name, g, o in zip(("pos", "prev", "vel"), sims[0].read_state(), sims[1].read_state()):
            assert np.array_equal(g, o), name
    for sim in sims:
        sim.destroy()
