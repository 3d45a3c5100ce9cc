"""Triangles without a usable normal in the clearance grid: corners on one line (a wire), two equal corners,
and slivers down to 1e-7 m wide, each alone in its scene.  Their edges are obstacles like any other: the
discrete checks agree with those without a cull, the sweeps with the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu
KINDS = ['same corner', 'on the line', 1e-7, 1e-6, 3e-6, 1e-5, 1e-3]


def _slivers(kind, count):
    rng = np.random.default_rng(KINDS.index(kind))
    for _ in range(count):
        a = rng.uniform([-0.6, -0.6, 0.1], [0.6, 0.6, 0.9])
        d = rng.normal(size=3)
        b = a + d / np.linalg.norm(d) * rng.uniform(0.3, 1.4)
        if kind == 'same corner':
            c = b.astype(np.float32)
        else:
            c = a + rng.uniform(0.2, 0.8) * (b - a)
            if kind != 'on the line':
                w = np.cross(b - a, rng.normal(size=3))
                c = c + kind * w / np.linalg.norm(w)
        yield scenes.Mesh(np.array([a, b, c]), np.array([[0, 1, 2]]), np.array([0, 1]))


@pytest.mark.parametrize('kind', KINDS)
def test_discrete(ctx, panda, kind):
    robot = rtcd.Robot(ctx, panda)
    q = scenes.uniform_poses(panda, 3000, seed=5)
    hits = 0
    for mesh in _slivers(kind, 8):
        scene = rtcd.Scene.from_mesh(ctx, mesh)
        for name in ('ObsToRobot', 'RobotToObs'):
            det = rtcd.Detector(ctx, name, robot, scene)
            a, b = det.check(q, counts=True), det.check(q, counts=True, flags=rtcd.CHECK_NO_CULL)
            assert np.array_equal(a['flags'], b['flags']) and np.array_equal(a['counts'], b['counts']), name
            hits += int(b['flags'].sum())
            det.close()
    assert hits > 20


@pytest.mark.parametrize('kind', KINDS)
@pytest.mark.parametrize('name', ['Linear', 'Quadratic'])
def test_sweeps(ctx, panda, kind, name):
    sph = scenes.synth_spheres(panda)
    robot, orob = rtcd.Robot(ctx, panda, spheres=sph), O.Robot(panda, spheres=sph)
    q, off = scenes.random_walk_trajectories(panda, 200, 8, seed=6)
    hits = 0
    for mesh in _slivers(kind, 6):
        det = rtcd.Detector(ctx, name, robot, rtcd.Scene.from_mesh(ctx, mesh))
        ref = O.sweep(name == 'Quadratic', orob, O.Scene(mesh), q, off)
        got = det.check(q, off, segments=True)
        assert not ((got['flags'] != ref['traj_hit']) & (ref['traj_band'] == 0)).any()
        assert not ((got['seg_flags'] != ref['seg_hit']) & (ref['seg_band'] == 0)).any()
        hits += int(ref['traj_hit'].sum())
        det.close()
    assert hits > 20
