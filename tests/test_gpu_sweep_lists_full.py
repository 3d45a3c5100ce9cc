"""Hand-over lists that are full: the entry list (four nodes per unit), where a unit's open nodes do not fit
and its reservation is blanked, and the record list (2^20 units).  The units concerned stay with their lane,
and flags, segment flags and counts equal those of a light pass that hands nothing over."""
import numpy as np
import pytest

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu


def _soup(n, size, seed):
    """Small triangles all through the robot's reach."""
    rng = np.random.default_rng(seed)
    c = rng.uniform([-0.9, -0.9, -0.1], [0.9, 0.9, 1.3], (n, 1, 3))
    return scenes.Mesh((c + rng.normal(0, size, (n, 3, 3))).reshape(-1, 3), np.arange(3 * n).reshape(n, 3), np.array([0, n]))


def _same(a, b, keys):
    for k in keys:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize('kind', ['Linear', 'Quadratic'])
@pytest.mark.parametrize('surface', [False, True])
@pytest.mark.parametrize('steps', [7, 16])
def test_entry_list_full(ctx, panda, kind, surface, steps):
    robot = rtcd.Robot(ctx, panda, spheres=scenes.synth_spheres(panda))
    sc = rtcd.Scene.from_mesh(ctx, _soup(30000, 0.02, 1))
    q = np.repeat(scenes.uniform_poses(panda, 24, seed=3), 12, axis=0)     # every trajectory parked at a pose
    off = np.arange(0, len(q) + 1, 12, dtype=np.uint32)
    never = rtcd.Detector(ctx, kind, robot, sc, light_steps=0xFFFFFFFF)
    det = rtcd.Detector(ctx, kind, robot, sc, light_steps=steps)
    for _ in range(2):      # fresh and used lists
        _same(det.check(q, off, segments=True, counts=True, surface=surface),
              never.check(q, off, segments=True, counts=True, surface=surface), ('flags', 'seg_flags', 'counts'))
        pieces = int(rtcd.segment_offsets(det.kind, off, rtcd.CHECK_SURFACE if surface else 0)[-1])
        assert det.stats()['deferred'] > pieces * 64 / 2       # most units, with more than eight open nodes on average
        _same(det.check(q, off, segments=True, surface=surface), never.check(q, off, segments=True, surface=surface),
              ('flags', 'seg_flags'))


@pytest.mark.parametrize('kind', ['Linear', 'Quadratic'])
@pytest.mark.parametrize('form', [1, 3])
def test_record_list_full(ctx, panda, kind, form):
    robot = rtcd.Robot(ctx, panda, spheres=scenes.synth_spheres(panda))
    sc = rtcd.Scene.from_mesh(ctx, _soup(4000, 0.01, 2))
    n = 500
    q, off = scenes.random_walk_trajectories(panda, n, 90 if kind == 'Quadratic' else 56, seed=4)
    never = rtcd.Detector(ctx, kind, robot, sc, light_steps=0xFFFFFFFF, stage_b_form=form)
    det = rtcd.Detector(ctx, kind, robot, sc, light_steps=1, stage_b_form=form)
    _same(det.check(q, off, segments=True, counts=True), never.check(q, off, segments=True, counts=True),
          ('flags', 'seg_flags', 'counts'))
    assert det.stats()['deferred'] > 1 << 20
