"""The quadratic sweeps' default launch (256 threads, binary tree in the staged pass) against the other
trees and block sizes, and the batch size from which the staged pass is taken."""
import numpy as np
import pytest
import torch

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('surface', [False, True])
@pytest.mark.parametrize('below', [1, 0])
def test_quadratic_default_launch(ctx, panda, small_scene, surface, below):
    robot = rtcd.Robot(ctx, panda, spheres=scenes.synth_spheres(panda))
    sc = rtcd.Scene.from_mesh(ctx, small_scene)
    # the line of 128-thread blocks, 5 to an SM, four trajectories each; one below it is unstaged
    n = 20 * torch.cuda.get_device_properties(0).multi_processor_count - below
    q, off = scenes.random_walk_trajectories(panda, n, scenes.log_uniform_counts(n, 3, 9, seed=3), seed=3)
    want = None
    for cfg in ({}, {'stage_b_form': 1}, {'stage_b_form': 3}, {'traverse_threads': 128},
                {'traverse_threads': 128, 'stage_b_form': 3, 'sweep_descend_cap': 3}, {'sweep_group': 1}):
        det = rtcd.Detector(ctx, 'Quadratic', robot, sc, **cfg)
        got = det.check(q, off, segments=True, surface=surface)
        assert det.stats()['path_flags'] & 1 == 1 - below
        want = want or got
        for k in ('flags', 'seg_flags'):
            assert np.array_equal(want[k], got[k]), (cfg, k)
        det.close()
