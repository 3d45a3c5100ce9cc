"""Performance cases of the detectors: the calls that a planner, a controller or a
service makes, each through the public entry points of ``rtcd``.

* ``poses``  - a discrete detector over a batch of configurations: through the
  device-buffer call, through the host-buffer call, through the host-buffer call
  replayed as a CUDA graph (``graph``), and through the upstream call sequence with
  hit counts (``upstream``);
* ``sweeps`` - a continuous detector over a batch of trajectories, with segment
  flags (device), or through the upstream call sequence with counts;
* ``edges``  - a roadmap's straight-line edges checked in one call;
* ``knn``    - the nearest neighbours that make those edges;
* ``served`` - a burst of mixed requests through the continuous-batching server.

A program keeps its context, robot, scenes and detectors, so these are made once
per process; poses, trajectories and requests come from the seed.  Detectors run
with their default settings.
"""
import functools
import math

import numpy as np
import torch

from rtcollisiondetection_b200 import rtcd, scenes

SCENES = {
    'small': scenes.discrete_small,                              # 5,264 triangles
    'shelf_simple': lambda: scenes.reference_scene('simple'),    # 15,008
    'shelf_medium': lambda: scenes.reference_scene('medium'),    # 71,746
    'shelf_dense': lambda: scenes.reference_scene('dense'),      # 202,330
    'dense': scenes.discrete_dense,                              # 428,448
    'sweep': scenes.sweep_scene,                                 # 49,744
    'sparse': scenes.sweep_scene_sparse,                         # 48,784
}


def listed():
    return [
        # a controller asking about its next few configurations
        dict(name='poses_13', path='poses', kind='RobotToObs', scene='shelf_dense', n=13, call='device'),
        # the small batch of an interactive planner
        dict(name='poses_1024_o2r', path='poses', kind='ObsToRobot', scene='small', n=1024, call='device'),
        # the batch the reference quotes its shelves at
        dict(name='poses_4096_r2o', path='poses', kind='RobotToObs', scene='shelf_dense', n=4096, call='device'),
        # a large batch in a dense scene: the headline workload
        dict(name='poses_65536_r2o', path='poses', kind='RobotToObs', scene='dense', n=65536, call='device'),
        # the same end to end: page-locked poses in, flags out, replayed as a graph
        dict(name='poses_65536_o2r_graph', path='poses', kind='ObsToRobot', scene='dense', n=65536, call='graph'),
        # a program written for the reference: prepareUpdateData, check, downloadResult (counts)
        dict(name='poses_1537_counts', path='poses', kind='RobotToObs', scene='shelf_medium', n=1537, call='upstream'),
        # an optimiser's batch of trajectories, linear pieces
        dict(name='linear_4096', path='sweeps', kind='Linear', scene='sweep', n=4096, wp_lo=32, wp_hi=32, call='device'),
        # the same with splines of uneven lengths
        dict(name='quad_4096', path='sweeps', kind='Quadratic', scene='sweep', n=4096, wp_lo=8, wp_hi=64, call='device'),
        # a program written for the reference, curve detector (its semantics, counts)
        dict(name='linear_301_counts', path='sweeps', kind='Linear', scene='shelf_dense', n=301, wp_lo=16, wp_hi=16,
             call='upstream'),
        # a roadmap's edges, 16 configurations each
        dict(name='edges_2000', path='edges', kind='RobotToObs', scene='shelf_dense', n=2000, wp=16),
        # the neighbour lists of that roadmap's construction
        dict(name='knn_20000', path='knn', n=20000, dim=7, k=10),
        # requests of every size arriving at once
        dict(name='served_96', path='served', n=96),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choices(['poses', 'sweeps', 'edges', 'knn', 'served'], [45, 30, 10, 10, 5])[0]
    if path == 'poses':
        call = rng.choice(['device', 'device', 'host', 'graph', 'upstream'])
        return dict(path=path, kind=rng.choice(['RobotToObs', 'ObsToRobot']),
                    scene=rng.choice(['small', 'shelf_simple', 'shelf_medium', 'shelf_dense', 'dense']),
                    n=_log_int(rng, 9, 1536 if call == 'upstream' else 65535), call=call)
    if path == 'sweeps':
        call = rng.choice(['device', 'device', 'device', 'upstream'])
        lo, hi = rng.choice([(8, 16), (16, 16), (32, 32), (8, 64), (8, 128)])
        most = 400 if call == 'upstream' else (1024 if hi == 128 else 4095)
        return dict(path=path, kind=rng.choice(['Linear', 'Quadratic']),
                    scene=rng.choice(['sweep', 'sparse', 'shelf_simple', 'shelf_dense']),
                    n=_log_int(rng, 3, most), wp_lo=lo, wp_hi=hi, call=call)
    if path == 'edges':
        return dict(path=path, kind=rng.choice(['RobotToObs', 'ObsToRobot']),
                    scene=rng.choice(['small', 'shelf_simple', 'shelf_dense']), n=_log_int(rng, 50, 2000),
                    wp=rng.randint(5, 16))
    if path == 'knn':
        return dict(path=path, n=_log_int(rng, 200, 20000), dim=7, k=rng.randint(1, 16))
    return dict(path=path, n=rng.randint(8, 95))


# ------------------------------------------------------------ what a program keeps
@functools.lru_cache(maxsize=None)
def _program():
    """The context, the robot (meshes and spheres) and the stream of its checks."""
    ctx = rtcd.Context(0)
    model = scenes.load_panda()
    return ctx, model, rtcd.Robot(ctx, model, spheres=scenes.synth_spheres(model)), torch.cuda.Stream()


@functools.lru_cache(maxsize=None)
def _scene(name):
    return rtcd.Scene.from_mesh(_program()[0], SCENES[name]())


@functools.lru_cache(maxsize=None)
def _detector(kind, scene):
    ctx, _, robot, _ = _program()
    return rtcd.Detector(ctx, kind, robot, _scene(scene))


@functools.lru_cache(maxsize=None)
def _server():
    """A server over three resident scenes, every slot's workspace sized up front."""
    server = rtcd.Server(_program()[0])
    dets = [_detector(kind, scene) for scene in ('small', 'sweep', 'dense')
            for kind in ('RobotToObs', 'Linear', 'Quadratic')]
    for det in dets:
        server.prepare(det, 1 << 15 if det.sweep else 4096)
    return server, dets


# ------------------------------------------------------------ inputs from the seed
def _limits():
    model = _program()[1]
    return torch.from_numpy(model['lower']).cuda(), torch.from_numpy(model['upper']).cuda()


def _poses(n, gen):
    lo, hi = _limits()
    return (lo + (hi - lo) * torch.rand((n, len(lo)), generator=gen, device='cuda')).contiguous()


def _lengths(case):
    """Waypoints per trajectory: evenly spread over the logarithm of the range."""
    n, lo, hi = case['n'], case['wp_lo'], case['wp_hi']
    at = (np.arange(n) + 0.5) / n
    return np.rint(np.exp(np.log(lo) + at * (np.log(hi) - np.log(lo)))).astype(np.int64)


def _walks(counts, gen):
    """Random walks of N(0, 0.1) rad steps clipped to the joint limits: q on the device, offsets on the host."""
    lo, hi = _limits()
    n, most = len(counts), int(counts.max())
    x = lo + (hi - lo) * torch.rand((n, len(lo)), generator=gen, device='cuda')
    steps = 0.1 * torch.randn((most - 1, n, len(lo)), generator=gen, device='cuda')
    all_q = [x]
    for k in range(most - 1):
        x = torch.minimum(torch.maximum(x + steps[k], lo), hi)
        all_q.append(x)
    keep = torch.arange(most, device='cuda')[None, :] < torch.from_numpy(counts).cuda()[:, None]
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(counts)
    return torch.stack(all_q, 1)[keep].contiguous(), off


def _device_outputs(n, seg):
    return (torch.zeros(n, dtype=torch.uint8, device='cuda'),
            torch.zeros(max(seg, 1), dtype=torch.uint8, device='cuda') if seg is not None else None)


def prepare(case, seed):
    ctx, model, robot, stream = _program()
    gen = torch.Generator(device='cuda')
    gen.manual_seed(seed)
    s = {'case': case, 'ctx': ctx, 'stream': stream}
    path, n = case['path'], case['n']
    if path == 'poses':
        q = _poses(n, gen)
        if case['call'] == 'device':
            s['det'] = _detector(case['kind'], case['scene'])
            s['q'], (s['flags'], _) = q, _device_outputs(n, None)
        elif case['call'] == 'graph':      # a detector of its own: its graph holds this program's buffers
            s['det'] = rtcd.Detector(ctx, case['kind'], robot, _scene(case['scene']))
            s['q'] = q.cpu().pin_memory().numpy()
        elif case['call'] == 'host':
            s['det'] = _detector(case['kind'], case['scene'])
            s['q'] = q.cpu().numpy()
        else:
            s['det'] = rtcd.CollisionDetector(ctx, case['kind'], robot, _scene(case['scene']))
            s['det'].buildSBT()
            s['q'] = q.cpu().numpy()
    elif path == 'sweeps':
        q, off = _walks(np.random.default_rng(seed).permutation(_lengths(case)), gen)
        s['off'] = off
        if case['call'] == 'device':
            s['det'] = _detector(case['kind'], case['scene'])
            s['q'] = q
            s['flags'], s['seg'] = _device_outputs(n, int(rtcd.segment_offsets(s['det'].kind, off)[-1]))
        else:
            s['det'] = rtcd.CollisionDetector(ctx, case['kind'], robot, _scene(case['scene']))
            s['det'].buildSBT()
            s['q'] = q.cpu().numpy()
    elif path == 'edges':
        s['det'] = _detector(case['kind'], case['scene'])
        nodes = max(16, n // 6)
        s['q'] = _poses(nodes, gen)
        s['edges'] = torch.randint(0, nodes, (n, 2), generator=gen, device='cuda', dtype=torch.int32)
        s['flags'], _ = _device_outputs(n, None)
    elif path == 'knn':
        s['q'] = _poses(n, gen)[:, :case['dim']].contiguous()
        s['w'] = np.linspace(1.0, 0.4, case['dim']).astype(np.float32)
        s['idx'] = torch.zeros((n, case['k']), dtype=torch.int32, device='cuda')
        s['dist'] = torch.zeros((n, case['k']), dtype=torch.float32, device='cuda')
    else:
        server, dets = _server()
        rng = np.random.default_rng(seed)
        s['server'], s['requests'] = server, []
        for i in range(n):     # the mix is the case's; poses and trajectories are the seed's
            mix = np.random.default_rng(1000 + i)
            where = 3 * int(mix.integers(0, 3))
            if mix.random() < 0.5:
                m = int(np.rint(np.exp(mix.uniform(0, np.log(4096)))))
                q = rng.uniform(model['lower'], model['upper'], size=(m, len(model['lower']))).astype(np.float32)
                s['requests'].append((dets[where], q, None))
            else:
                kind = 1 + int(mix.integers(0, 2))
                counts = scenes.log_uniform_counts(int(np.rint(np.exp(mix.uniform(0, np.log(1024))))), 8, 128, seed=i)
                q, off = _walks(counts, gen)
                s['requests'].append((dets[where + kind], q.cpu().numpy(), off))
    stream.wait_stream(torch.cuda.current_stream())
    return s


def run(s):
    case = s['case']
    path, n, sp = case['path'], case['n'], s['stream'].cuda_stream
    if path == 'poses':
        if case['call'] == 'device':
            s['det'].check_device(s['q'], n, s['flags'], stream=sp)
            return s['flags']
        if case['call'] == 'upstream':
            s['det'].prepareUpdateData(s['q'], n)
            s['det'].setNCheck(n)
            s['det'].check()
            return s['det'].downloadResult()
        return s['det'].check(s['q'], flags=rtcd.CHECK_GRAPH if case['call'] == 'graph' else 0)['flags']
    if path == 'sweeps':
        if case['call'] == 'device':
            s['det'].check_device(s['q'], n, s['flags'], traj_off=s['off'], seg_dev=s['seg'], stream=sp)
            return s['flags'], s['seg']
        s['det'].prepareUpdateData(s['q'], n, s['off'])
        s['det'].setNCheck(n)
        s['det'].check()
        return s['det'].downloadResult()
    if path == 'edges':
        s['det'].check_edges(s['q'], len(s['q']), s['edges'], n, case['wp'], s['flags'], stream=sp)
        return s['flags']
    if path == 'knn':
        rtcd.knn(s['ctx'], s['q'], n, case['dim'], case['k'], s['idx'], s['dist'], weights=s['w'], stream=sp)
        return s['idx'], s['dist']
    tickets = [s['server'].submit(det, q, off) for det, q, off in s['requests']]
    out = [s['server'].wait(t) for t in tickets]
    return (np.concatenate([o['flags'] for o in out]),
            np.concatenate([o['seg_flags'] for o in out if 'seg_flags' in o] or [np.zeros(0, np.uint8)]))


def exact(case, seed):
    """Collision flags and counts are whole numbers; the neighbour distances in 64 bits."""
    if case['path'] != 'knn':
        return None
    n, k = case['n'], case['k']
    gen = torch.Generator(device='cuda')
    gen.manual_seed(seed)
    w = torch.from_numpy(np.linspace(1.0, 0.4, case['dim']).astype(np.float32)).cuda()
    p = _poses(n, gen)[:, :case['dim']].double() * w.double()
    rows = []
    for a in range(0, n, 1000):
        d2 = torch.zeros((min(1000, n - a), n), dtype=torch.float64, device='cuda')
        for j in range(case['dim']):
            d2 += (p[a:a + 1000, j, None] - p[None, :, j]).square_()
        d2[torch.arange(len(d2), device='cuda'), torch.arange(a, a + len(d2), device='cuda')] = math.inf
        rows.append(d2.topk(k, largest=False).values.sqrt())
    return [None, torch.cat(rows)]


def work(case):
    """Joint values in and flags out, and the chain's arithmetic (28 multiply-adds per joint's product,
    12 for its transform); what the scene costs depends on where the robot is."""
    path, n, fk = case['path'], case['n'], 7 * 2 * (36 + 24)
    if path == 'poses':
        return {'bytes': n * (28 + (4 if case['call'] == 'upstream' else 1)), 'flops': n * fk}
    if path == 'sweeps':
        wp = float(_lengths(case).sum())
        seg = 0.0 if case['call'] == 'upstream' else (wp - n if case['kind'] == 'Linear' else wp / 2)
        return {'bytes': 28 * wp + seg + n * (4 if case['call'] == 'upstream' else 1),
                'flops': wp * (fk + 64 * 18)}
    if path == 'edges':
        return {'bytes': n * (8 + 1) + 28 * max(16, n // 6), 'flops': n * case['wp'] * (fk + 14)}
    if path == 'knn':
        return {'bytes': n * (4 * case['dim'] + 8 * case['k']), 'flops': float(n) * n * 4 * case['dim']}
    return {'bytes': 28.0 * 4000 * n, 'flops': 4000.0 * n * (fk + 32 * 18)}
