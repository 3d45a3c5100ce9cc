"""The clearance cull (k_prepare) loses no hit: flags and counts equal those without a cull, on
scenes whose cells are far larger or smaller than the robot's spheres, on slanted and degenerate
triangles, beside obstacles far outside the grid's reach, and for poses that are not finite."""
import numpy as np
import pytest

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu


def _slanted(rng, n, size):
    c = rng.uniform([-0.8, -0.8, 0.0], [0.8, 0.8, 1.2], (n, 1, 3))
    v = (c + rng.normal(0, size, (n, 3, 3))).reshape(-1, 3)
    return scenes.Mesh(v, np.arange(3 * n).reshape(n, 3), np.array([0, n]))


def _joined(a, b):
    return scenes.Mesh(np.concatenate([a.verts, b.verts]), np.concatenate([a.tris, b.tris + len(a.verts)]),
                       np.array([0, a.n_tris, a.n_tris + b.n_tris]))


def _scenes():
    rng = np.random.default_rng(3)
    far = _slanted(rng, 4, 1.0)
    far.verts[:] += np.float32(200.0)
    flat = _slanted(rng, 30, 0.3)
    flat.verts[:, 2] = np.float32(0.4)
    point = scenes.Mesh(np.full((3, 3), 0.3), np.array([[0, 1, 2]]), np.array([0, 1]))
    return {'one': _slanted(rng, 1, 0.5), 'slanted': _slanted(rng, 40, 0.4), 'dust': _slanted(rng, 3000, 0.004),
            'far': _joined(_slanted(rng, 20, 0.2), far), 'flat': flat, 'point': point,
            'shelf': scenes.reference_scene('simple'), 'small': scenes.discrete_small()}


@pytest.mark.parametrize('name', ['RobotToObs', 'ObsToRobot'])
@pytest.mark.parametrize('n', [1, 33, 2000])
def test_cull_loses_no_hit(ctx, panda, name, n):
    robot = rtcd.Robot(ctx, panda)
    q = scenes.uniform_poses(panda, n, seed=n)
    if n > 1:
        q[n // 2, 3], q[n - 1, 0] = np.nan, np.inf
    for label, mesh in _scenes().items():
        det = rtcd.Detector(ctx, name, robot, rtcd.Scene.from_mesh(ctx, mesh))
        for kw in ({}, {'counts': True}, {'flags': rtcd.CHECK_TWO_WAY}):
            more = dict(kw, flags=kw.get('flags', 0) | rtcd.CHECK_NO_CULL)
            a, b = det.check(q, **kw), det.check(q, **more)
            for k in a:
                assert np.array_equal(a[k], b[k]), (label, kw, k)
