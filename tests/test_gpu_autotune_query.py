"""The autotuner of the discrete kinds: the query kernel takes no launch shape and no light budget, so it is
one candidate, not one per shape, and is reported with its own shape whatever the timings' noise."""
import pytest

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('kind', ['RobotToObs', 'ObsToRobot'])
def test_query_kernel_is_one_candidate(ctx, panda, kind):
    import torch
    robot = rtcd.Robot(ctx, panda)
    scene = rtcd.Scene.from_mesh(ctx, scenes.reference_scene('medium'))
    q = torch.from_numpy(scenes.uniform_poses(panda, 3000, seed=1)).cuda()
    torch.cuda.synchronize()
    picks = []
    for _ in range(4):
        best = rtcd.Detector(ctx, kind, robot, scene).autotune(q, 3000)
        if best['stage_b_form'] in (0, 3, 4):
            assert best['traverse_threads'] == 128 and best['light_steps'] == 0
            picks.append(best['traverse_blocks_per_sm'])
    assert len(picks) == 4 and len(set(picks)) == 1
