"""A scene much smaller than the robot (one part on a bench): the clearance grid covers the part alone, and the
cull still drops the links that are far from it, and none in contact."""
import numpy as np
import pytest

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu


def _box(center, extent):
    v, t = scenes.box_mesh(center, extent)
    return scenes.Mesh(v, t, np.array([0, len(t)]))


@pytest.mark.parametrize('name', ['RobotToObs', 'ObsToRobot'])
@pytest.mark.parametrize('center,extent', [((0.5, 0.1, 0.4), (0.05, 0.05, 0.05)), ((0.3, -0.2, 0.6), (0.1, 0.002, 0.3)),
                                           ((0.0, 0.0, -0.05), (2.0, 2.0, 0.05)), ((1.5, 1.5, 0.5), (0.1, 0.1, 0.1))])
def test_small_scene(ctx, panda, name, center, extent):
    robot = rtcd.Robot(ctx, panda)
    det = rtcd.Detector(ctx, name, robot, rtcd.Scene.from_mesh(ctx, _box(center, extent)))
    n = 20000
    q = scenes.uniform_poses(panda, n, seed=11)
    a = det.check(q, counts=True)
    kept = det.stats()['work_items']
    b = det.check(q, counts=True, flags=rtcd.CHECK_NO_CULL)
    assert np.array_equal(a['flags'], b['flags']) and np.array_equal(a['counts'], b['counts'])
    assert kept < 0.1 * 7 * n       # all of them, without the distance to the grid
