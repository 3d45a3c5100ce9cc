"""The query kernel against the thread-per-item kernel (RTCD_CHECK_FUSED) on the
same scenes: batches on both sides of its grid rules, flags and counts, a share
of the GPU, crowded items that are handed on, and links of one triangle or none."""
import numpy as np
import pytest

from rtcollisiondetection_b200 import rtcd, scenes

pytestmark = pytest.mark.gpu
KINDS = ['RobotToObs', 'ObsToRobot']


@pytest.fixture(scope='module')
def setup(ctx, panda):
    return rtcd.Robot(ctx, panda), {'small': rtcd.Scene.from_mesh(ctx, scenes.discrete_small()),
                                    'shelf': rtcd.Scene.from_mesh(ctx, scenes.reference_scene('medium'))}


# 768 items per SM at 148 SMs and 7 checked links is 16,237 poses
@pytest.mark.parametrize('name', KINDS)
@pytest.mark.parametrize('n,residency', [(1, 0), (9, 0), (677, 0), (4097, 50), (16237, 0), (16239, 0), (20011, 25)])
def test_flags_match_thread_per_item(setup, panda, name, n, residency):
    robot, sc = setup
    q = scenes.uniform_poses(panda, n, seed=n)
    det = rtcd.Detector(robot.ctx, name, robot, sc['small'], residency_percent=residency)
    assert np.array_equal(det.check(q)['flags'], det.check(q, flags=rtcd.CHECK_FUSED)['flags'])


@pytest.mark.parametrize('name', KINDS)
@pytest.mark.parametrize('n', [3, 150, 1100])
def test_counts_match_thread_per_item(setup, panda, name, n):
    """Counting visits every pair, and the shelf's large boards crowd some items far beyond others."""
    robot, sc = setup
    q = scenes.uniform_poses(panda, n, seed=n)
    det = rtcd.Detector(robot.ctx, name, robot, sc['shelf'])
    a, b = det.check(q, counts=True), det.check(q, counts=True, flags=rtcd.CHECK_FUSED)
    assert np.array_equal(a['flags'], b['flags']) and np.array_equal(a['counts'], b['counts'])
    assert np.array_equal(a['flags'], det.check(q)['flags'])


@pytest.mark.parametrize('name', KINDS)
def test_links_of_one_triangle_or_none(ctx, panda, setup, name):
    """Links whose tree is a single leaf, and links without a mesh."""
    _, sc = setup
    m = dict(panda)
    V, T, vo, to = [], [], [0], [0]
    for l in range(len(panda['link_vert_off']) - 1):
        v = panda['link_verts'][panda['link_vert_off'][l]:panda['link_vert_off'][l + 1]]
        t = panda['link_tris'][panda['link_tri_off'][l]:panda['link_tri_off'][l + 1]]
        if l in (3, 6):
            t = t[:1]
        elif l == 4:
            v, t = v[:0], t[:0]
        V.append(v); T.append(t)
        vo.append(vo[-1] + len(v)); to.append(to[-1] + len(t))
    m.update(link_verts=np.concatenate(V), link_tris=np.concatenate(T), link_vert_off=np.asarray(vo, np.uint32),
             link_tri_off=np.asarray(to, np.uint32))
    robot = rtcd.Robot(ctx, m, edges=False)
    det = rtcd.Detector(ctx, name, robot, sc['small'])
    q = scenes.uniform_poses(panda, 500, seed=8)
    a, b = det.check(q, counts=True), det.check(q, counts=True, flags=rtcd.CHECK_FUSED)
    assert np.array_equal(a['flags'], b['flags']) and np.array_equal(a['counts'], b['counts'])
