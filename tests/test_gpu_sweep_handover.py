"""Units handed from the sweeps' light pass to the heavy pass: with every unit handed over after
one visit, from the 4-wide tree's stack or from the root (binary light pass), flags, segment
flags and counts equal those of a light pass that finishes every unit itself."""
import numpy as np
import pytest

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('kind', ['Linear', 'Quadratic'])
@pytest.mark.parametrize('surface', [False, True])
@pytest.mark.parametrize('n,lo,hi', [(1, 3, 3), (2, 40, 90), (75, 3, 9)])
def test_handed_over_units_keep_results(ctx, panda, small_scene, kind, surface, n, lo, hi):
    robot = rtcd.Robot(ctx, panda, spheres=scenes.synth_spheres(panda))
    q, off = scenes.random_walk_trajectories(panda, n, scenes.log_uniform_counts(n, lo, hi, seed=n), seed=n)
    for mesh in (small_scene, scenes.reference_scene('simple')):
        sc = rtcd.Scene.from_mesh(ctx, mesh)
        never = rtcd.Detector(ctx, kind, robot, sc, light_steps=0xFFFFFFFF)
        want = [never.check(q, off, segments=True, surface=surface),
                never.check(q, off, surface=surface),
                never.check(q, off, segments=True, counts=True, surface=surface)]
        for form, steps in ((0, 1), (0, 7), (1, 1)):
            det = rtcd.Detector(ctx, kind, robot, sc, light_steps=steps, stage_b_form=form)
            got = [det.check(q, off, segments=True, surface=surface), det.check(q, off, surface=surface),
                   det.check(q, off, segments=True, counts=True, surface=surface)]
            for w, g in zip(want, got):
                for k in ('flags', 'seg_flags', 'counts'):
                    if k in w:
                        assert np.array_equal(w[k], g[k]), (form, steps, k)
            det.close()
