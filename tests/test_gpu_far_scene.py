"""A cell far from the origin (a base frame in survey coordinates): the clearance grid's bound holds there,
where positions are rounded to more than its margins near the origin."""
import numpy as np
import pytest

from oracle import oracle as O
from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu


def _moved(panda, mesh, shift):
    model = dict(panda)
    base = np.array(panda['base_tf'], np.float32).copy()
    flat = base.reshape(-1)
    flat[[3, 7, 11]] += np.asarray(shift, np.float32)
    model['base_tf'] = base
    return model, scenes.Mesh(mesh.verts + np.asarray(shift, np.float32), mesh.tris, mesh.obstacle_tri_off)


@pytest.mark.parametrize('shift', [(800.0, -300.0, 40.0), (5000.0, 7000.0, 300.0), (-60000.0, 20000.0, 900.0)])
@pytest.mark.parametrize('scene', ['dust', 'shelf'])
def test_far_scene(ctx, panda, shift, scene):
    rng = np.random.default_rng(2)
    if scene == 'dust':
        c = rng.uniform([-0.8, -0.8, 0.0], [0.8, 0.8, 1.2], (200, 1, 3))
        mesh = scenes.Mesh((c + rng.normal(0, 0.01, (200, 3, 3))).reshape(-1, 3), np.arange(600).reshape(200, 3),
                           np.array([0, 200]))
    else:
        mesh = scenes.reference_scene('simple')
    model, mesh = _moved(panda, mesh, shift)
    robot = rtcd.Robot(ctx, model, spheres=scenes.synth_spheres(panda))
    sc = rtcd.Scene.from_mesh(ctx, mesh)
    q = scenes.uniform_poses(panda, 20000, seed=1)
    for name in ('RobotToObs', 'ObsToRobot'):
        det = rtcd.Detector(ctx, name, robot, sc)
        a, b = det.check(q, counts=True), det.check(q, counts=True, flags=rtcd.CHECK_NO_CULL)
        assert b['flags'].any()
        assert np.array_equal(a['flags'], b['flags']) and np.array_equal(a['counts'], b['counts']), name
