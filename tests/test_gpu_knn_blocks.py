"""Neighbour search at the edges of its blocks: every number of axes, sizes around the
32-query and 32-point tiles, block shapes of 8 to 32 warps, masks and exact ties."""
import numpy as np
import pytest
import torch

from rtcollisiondetection_b200 import rtcd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,dim,k', [(1, 7, 3), (31, 1, 1), (32, 2, 5), (33, 3, 32), (64, 16, 32), (65, 7, 8),
                                     (257, 4, 9), (1000, 5, 16), (4097, 6, 2), (9001, 7, 10)])
@pytest.mark.parametrize('masked', [False, True])
def test_knn_exact_with_ties(ctx, n, dim, k, masked):
    """Small whole coordinates and weights that are powers of two: every distance is exact in FP32,
    most of them tie, and the lower index has to come first."""
    rng = np.random.default_rng(n + dim + k)
    pts = rng.integers(-3, 4, size=(n, dim)).astype(np.float32)
    w = (2.0 ** rng.integers(-1, 2, size=dim)).astype(np.float32)
    mask = (rng.random(n) < 0.3).astype(np.uint8) if masked else None
    pd = torch.from_numpy(pts).cuda()
    md = torch.from_numpy(mask).cuda() if masked else None
    idx = torch.zeros((n, k), dtype=torch.int32, device='cuda')
    dist = torch.zeros((n, k), dtype=torch.float32, device='cuda')
    rtcd.knn(ctx, pd, n, dim, k, idx, dist, weights=w, mask_dev=md)
    torch.cuda.synchronize()
    gi, gd = idx.cpu().numpy().view(np.uint32), dist.cpu().numpy()
    for a in range(0, n, 500):
        rows = np.arange(a, min(a + 500, n))
        d2 = (((pts[rows, None, :] - pts[None, :, :]) * w) ** 2).sum(-1).astype(np.float64)
        d2[np.arange(len(rows)), rows] = np.inf
        if masked:
            d2[mask[rows] != 0, :] = np.inf
            d2[:, mask != 0] = np.inf
        order = np.argsort(d2, axis=1, kind='stable')[:, :k]
        got = np.take_along_axis(d2, order, 1)
        ri = np.full((len(rows), k), 0xFFFFFFFF, np.uint32)
        rd = np.full((len(rows), k), np.finfo(np.float32).max, np.float32)
        ri[:, :order.shape[1]] = np.where(np.isfinite(got), order, 0xFFFFFFFF)
        rd[:, :order.shape[1]] = np.where(np.isfinite(got), np.sqrt(got), np.finfo(np.float32).max)
        assert np.array_equal(gi[rows], ri)
        assert np.array_equal(gd[rows], rd)
