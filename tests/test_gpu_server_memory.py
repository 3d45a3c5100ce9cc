"""The server books for a launch what the launch allocates: at least its slot's growth of device memory
(but for fixed buffers of under 4 MB and the allocator's 2 MB pages), at most twice that and those."""
import pytest

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.mark.parametrize('kind,counts', [('RobotToObs', False), ('RobotToObs', True), ('ObsToRobot', False),
                                         ('Linear', False), ('Quadratic', False)])
def test_booked_bytes(ctx, panda, kind, counts):
    import torch
    robot = rtcd.Robot(ctx, panda, spheres=scenes.synth_spheres(panda))
    scene = rtcd.Scene.from_mesh(ctx, scenes.sweep_scene())
    det = rtcd.Detector(ctx, kind, robot, scene)
    if det.sweep:
        q, off = scenes.random_walk_trajectories(panda, 1000, 60, seed=1)
    else:
        q, off = scenes.uniform_poses(panda, 60000, seed=1), None
    det.check(q[:2 * 60], None if off is None else off[:3], counts=counts)  # the kernels are loaded
    srv = rtcd.Server(ctx, slots=1, max_batch_units=1 << 20)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    srv.wait(srv.submit(det, q, off, counts=counts))
    grown = free - torch.cuda.mem_get_info()[0]
    booked = srv.stats()['inflight_bytes_peak']
    srv.close()
    assert grown > 16 * MB
    pages = 14 * 2 * MB     # a page each for the workspace's buffers
    assert grown - 4 * MB - pages <= booked <= 2 * grown + 4 * MB, (booked / MB, grown / MB)
