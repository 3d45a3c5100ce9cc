"""Link boxes given by the caller (link_obbs): whatever boxes hold the meshes, also with axes that are not
unit vectors or not quite at right angles, the discrete checks agree with those without a cull."""
import ctypes as C

import numpy as np
import pytest

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu


def _robot(ctx, model, obbs):
    """rtcd.Robot with link_obbs (15 floats per link: centre, half sizes, axes)."""
    robot = rtcd.Robot.__new__(rtcd.Robot)
    create = rtcd.lib().rtcd_robot_create
    keep = np.ascontiguousarray(obbs, np.float32)

    class Lib:
        def rtcd_robot_create(self, c, d, out):
            d._obj.link_obbs = keep.ctypes.data_as(C.POINTER(C.c_float))
            return create(c, d, out)

        def __getattr__(self, name):
            return getattr(real, name)

    real, old = rtcd.lib(), rtcd.lib
    rtcd.lib = lambda: Lib()
    try:
        robot.__init__(ctx, model)
    finally:
        rtcd.lib = old
    return robot


@pytest.mark.parametrize('form', ['unit', 'long axes', 'short axes', 'sheared'])
def test_given_boxes(ctx, panda, form):
    obbs = []
    for l in range(len(panda['link_vert_off']) - 1):
        v = panda['link_verts'][panda['link_vert_off'][l]:panda['link_vert_off'][l + 1]].astype(np.float64)
        axes = np.eye(3)
        if form == 'long axes':
            axes = 1.3 * axes
        elif form == 'short axes':
            axes = 0.8 * axes
        elif form == 'sheared':
            axes[0, 1], axes[2, 0] = 0.15, -0.1
        # centre + sum of t_k h_k axes[k], |t_k| <= 1, holds every vertex, and so does the box that reads
        # the half sizes along the axes' directions
        c = 0.5 * (v.min(0) + v.max(0))
        t = np.maximum(np.abs((v - c) @ np.linalg.inv(axes)), np.abs((v - c) @ axes.T)).max(0)
        obbs.append(np.concatenate([c, 1.3 * t + 0.01, axes.ravel()]))
    robot = _robot(ctx, panda, np.stack(obbs))
    plain = rtcd.Robot(ctx, panda)
    q = scenes.uniform_poses(panda, 6000, seed=3)
    for mesh in (scenes.discrete_small(), scenes.reference_scene('simple')):
        sc = rtcd.Scene.from_mesh(ctx, mesh)
        for name in ('RobotToObs', 'ObsToRobot'):
            det = rtcd.Detector(ctx, name, robot, sc)
            a, b = det.check(q, counts=True), det.check(q, counts=True, flags=rtcd.CHECK_NO_CULL)
            assert np.array_equal(a['flags'], b['flags']) and np.array_equal(a['counts'], b['counts']), name
            if form == 'unit':
                c = rtcd.Detector(ctx, name, plain, sc).check(q, counts=True)
                assert np.array_equal(a['flags'], c['flags']) and np.array_equal(a['counts'], c['counts']), name
