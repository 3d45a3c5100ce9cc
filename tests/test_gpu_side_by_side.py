"""Launches that share work among their warps (csrc/share.cuh), several side by side on one GPU: blocks
of one start while warps of it already wait.  Each check's results equal those of the same check alone."""
import threading

import numpy as np
import pytest

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu


def _jobs(ctx, panda):
    robot = rtcd.Robot(ctx, panda, spheres=scenes.synth_spheres(panda))
    shelf = rtcd.Scene.from_mesh(ctx, scenes.reference_scene('medium'))
    small = rtcd.Scene.from_mesh(ctx, scenes.discrete_small())
    jobs = []
    for i, (kind, scene, n) in enumerate((('RobotToObs', shelf, 300), ('ObsToRobot', shelf, 900), ('RobotToObs', small, 40),
                                          ('Linear', shelf, 30), ('Quadratic', small, 60))):
        det = rtcd.Detector(ctx, kind, robot, scene, light_steps=4)
        q, off = ((scenes.uniform_poses(panda, n, seed=i), None) if not det.sweep else
                  scenes.random_walk_trajectories(panda, n, scenes.log_uniform_counts(n, 6, 24, seed=i), seed=i))
        jobs.append((det, q, off))
    return jobs


def test_results_side_by_side(ctx, panda):
    jobs = _jobs(ctx, panda)
    alone = [[det.check(q, off, counts=c) for c in (False, True)] for det, q, off in jobs]
    wrong = []

    def loop(i):
        det, q, off = jobs[i]
        for k in range(60):
            got, want = det.check(q, off, counts=bool(k & 1)), alone[i][k & 1]
            if not all(np.array_equal(got[f], want[f]) for f in ('flags', 'counts')[:1 + (k & 1)]):
                wrong.append((i, k))

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
