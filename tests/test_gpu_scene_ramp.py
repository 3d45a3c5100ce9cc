"""A scene with one large oblique triangle (a ramp) is made in the time of any other: its cells of the
clearance grid, up to 16.7 million, are not one thread's work."""
import time

import numpy as np
import pytest

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu


def _time(ctx, mesh):
    times = []
    for _ in range(4):
        t = time.perf_counter()
        scene = rtcd.Scene.from_mesh(ctx, mesh)
        times.append(time.perf_counter() - t)
        scene.close()
    return min(times)


@pytest.mark.parametrize('ramp', [[[-0.9, -0.9, 0.0], [0.9, -0.2, 0.9], [-0.2, 0.9, 1.8]],
                                  [[-0.9, -0.9, 0.0], [0.9, -0.9, 0.0], [-0.9, 0.9, 1.8]]])
def test_ramp_is_made_quickly(ctx, panda, ramp):
    ramp = np.array(ramp)
    small = np.array([[-0.9, -0.9, 0.0], [-0.89, -0.9, 0.0], [-0.9, -0.89, 0.0], [0.9, 0.9, 1.8], [0.89, 0.9, 1.8],
                      [0.9, 0.89, 1.8]])
    a = _time(ctx, scenes.Mesh(ramp, np.array([[0, 1, 2]]), np.array([0, 1])))
    b = _time(ctx, scenes.Mesh(small, np.array([[0, 1, 2], [3, 4, 5]]), np.array([0, 2])))
    print('ramp %.1f ms, the same grid without it %.1f ms' % (1e3 * a, 1e3 * b))
    assert a < b + 0.1


def test_small_part_is_made_quickly(ctx, panda):
    """The grid of a part of a few centimetres is small (0.4 ms without a grid, 4.7 with 256 cells along it)."""
    v, t = scenes.box_mesh((0.5, 0.1, 0.4), (0.05, 0.03, 0.05))
    a = min(_time(ctx, scenes.Mesh(v, t, np.array([0, len(t)]))) for _ in range(4))
    print('small part %.2f ms' % (1e3 * a))
    assert a < 0.002
