"""Neighbour searches whose block needs 44 to 48 KB of shared memory, as the first call of their number of
axes in a process (the opt-in for more than 48 KB, lists and static arrays together, outlives a call)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SEARCH = '''
import sys
import torch
from rtcollisiondetection_b200 import rtcd
ctx = rtcd.Context(0)
for n, dim, k in %s:
    g = torch.Generator(device='cuda')
    g.manual_seed(n)
    p = torch.rand((n, dim), device='cuda', generator=g)
    idx = torch.zeros((n, k), dtype=torch.int32, device='cuda')
    dist = torch.zeros((n, k), device='cuda')
    rtcd.knn(ctx, p, n, dim, k, idx, dist)
    torch.cuda.synchronize()
    for a in range(0, n, 1000):
        d2 = (p[a:a + 1000, None, :].double() - p[None, :, :].double()).square().sum(-1)
        d2[torch.arange(len(d2)), torch.arange(a, a + len(d2))] = float('inf')
        want = d2.topk(k, largest=False).values.sqrt()
        mine = d2.gather(1, idx[a:a + 1000].long()).sqrt()
        # (dim + 3) roundings of 2^-24 in the squared distance, half of them after the root
        assert torch.allclose(dist[a:a + 1000].double(), want, rtol=1e-6, atol=0), (n, dim, k)
        assert torch.allclose(mine, want, rtol=1e-6, atol=0), (n, dim, k)
'''


@pytest.mark.parametrize('calls', [[(300, 7, 15), (10000, 6, 16), (10000, 3, 17)],
                                   [(10000, 7, 14), (6000, 6, 4), (6000, 3, 5)], [(6000, 7, 3)]])
def test_first_call_of_a_dimension(calls):
    out = subprocess.run([sys.executable, '-c', SEARCH % calls], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert out.returncode == 0, out.stderr
