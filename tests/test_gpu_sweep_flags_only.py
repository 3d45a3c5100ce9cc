"""Sweep batches without segment flags and counts in the staged light pass: a group of trajectories ends when
all of them are hit, and the quadratic pass takes smaller blocks.  The flags equal those of a call with
segment flags, for groups of one and of several trajectories, in scenes that hit all, some or none of them."""
import numpy as np
import pytest

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu


def _box(center, extent):
    v, t = scenes.box_mesh(center, extent)
    return scenes.Mesh(v, t, np.array([0, len(t)]))


@pytest.mark.parametrize('kind', ['Linear', 'Quadratic'])
@pytest.mark.parametrize('n,lo,hi', [(3600, 3, 6), (3601, 8, 24), (3602, 40, 40)])
def test_flags_only(ctx, panda, kind, n, lo, hi):
    robot = rtcd.Robot(ctx, panda, spheres=scenes.synth_spheres(panda))
    q, off = scenes.random_walk_trajectories(panda, n, scenes.log_uniform_counts(n, lo, hi, seed=n), seed=n)
    rates = []
    for mesh in (_box((0, 0, -0.05), (2, 2, 0.05)), scenes.sweep_scene_sparse(), _box((3, 3, 3), (0.1, 0.1, 0.1))):
        scene = rtcd.Scene.from_mesh(ctx, mesh)
        for kw in ({}, {'light_steps': 0xFFFFFFFF}, {'residency_percent': 30}):
            det = rtcd.Detector(ctx, kind, robot, scene, **kw)
            for surface in (False, True):
                a = det.check(q, off, surface=surface)['flags']
                assert kw.get('residency_percent') or det.stats()['path_flags'] & 1      # staged
                assert np.array_equal(a, det.check(q, off, segments=True, surface=surface)['flags'])
            rates.append(a.mean())
            det.close()
    assert max(rates) > 0.9 and min(rates) == 0.0
