"""Neighbour search among few points (k_knn_few): sizes on both sides of its lines, the largest k, masks,
points that are not finite, and exact ties, against the order by distance, then by index."""
import numpy as np
import pytest
import torch

from rtcollisiondetection_b200 import rtcd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [1, 2, 33, 127, 128, 129, 511, 512, 513, 1023, 1024, 1025])
@pytest.mark.parametrize('dim,k', [(1, 1), (7, 10), (16, 32)])
@pytest.mark.parametrize('form', ['plain', 'masked', 'not finite'])
def test_few_points(ctx, n, dim, k, form):
    """Small whole coordinates, weights powers of two: the distances are exact in FP32 and many tie."""
    rng = np.random.default_rng(n * 100 + dim)
    pts = rng.integers(-2, 3, size=(n, dim)).astype(np.float32)
    w = (2.0 ** rng.integers(-1, 2, size=dim)).astype(np.float32)
    mask = (rng.random(n) < 0.4).astype(np.uint8) if form == 'masked' else None
    if form == 'not finite':
        bad = rng.random(n) < 0.2
        pts[bad, rng.integers(0, dim)] = rng.choice([np.nan, np.inf, -np.inf, 1e30], size=bad.sum())
    pd, md = torch.from_numpy(pts).cuda(), torch.from_numpy(mask).cuda() if mask is not None else None
    idx = torch.zeros((n, k), dtype=torch.int32, device='cuda')
    dist = torch.zeros((n, k), dtype=torch.float32, device='cuda')
    rtcd.knn(ctx, pd, n, dim, k, idx, dist, weights=w, mask_dev=md)
    torch.cuda.synchronize()
    with np.errstate(all='ignore'):
        d2 = ((pts[:, None, :] - pts[None, :, :]) ** 2 * (w * w)).sum(-1, dtype=np.float32)
    d2[np.arange(n), np.arange(n)] = np.inf
    if mask is not None:
        d2[mask != 0, :] = np.inf
        d2[:, mask != 0] = np.inf
    d2 = np.where(np.isfinite(d2), d2, np.inf)
    order = np.argsort(d2, axis=1, kind='stable')[:, :k]
    got = np.take_along_axis(d2, order, 1)
    ri = np.full((n, k), 0xFFFFFFFF, np.uint32)
    rd = np.full((n, k), np.finfo(np.float32).max, np.float32)
    ri[:, :order.shape[1]] = np.where(np.isfinite(got), order, 0xFFFFFFFF)
    rd[:, :order.shape[1]] = np.where(np.isfinite(got), np.sqrt(got), np.finfo(np.float32).max)
    assert np.array_equal(idx.cpu().numpy().view(np.uint32), ri)
    assert np.array_equal(dist.cpu().numpy(), rd)
