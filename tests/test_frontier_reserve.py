"""The rule that keeps a frontier of fixed size from overflowing (frontier_step, csrc/wide.cuh):
a step pops at most (cap - reserve - size) / 3 nodes, but at least one, with reserve = 3 * depth + 4.
Simulated on complete and on ragged 4-wide trees with every child overlapping, the worst case, and
from a start of up to 64 entries, for the frontier's size of 512 and smaller ones."""
import numpy as np
import pytest


def worst(children, start, cap, reserve):
    fr, most, steps = list(start), len(start), 0
    while fr:
        wide = 8 if len(fr) <= 8 else 16 if len(fr) <= 16 else 32
        take = min(len(fr), wide, max(1, (cap - reserve - len(fr)) // 3))
        popped = fr[len(fr) - take:]
        del fr[len(fr) - take:]
        for n in popped:
            fr.extend(children(n))
        most = max(most, len(fr))
        steps += 1
        if steps > 4000:      # a tree of depth 60 is not walked to its end
            break
    return most


@pytest.mark.parametrize('depth', [0, 1, 5, 18, 62])
@pytest.mark.parametrize('cap', [256, 300, 512])
@pytest.mark.parametrize('start', [1, 64])
def test_complete_tree(depth, cap, start):
    """Entries are depths; every node above `depth` has four internal children."""
    assert worst(lambda d: [d + 1] * 4 if d < depth else [], [0] * start, cap, 3 * depth + 4) <= cap


@pytest.mark.parametrize('seed', range(6))
def test_ragged_tree(seed):
    rng = np.random.default_rng(seed)
    depth = int(rng.integers(8, 63))
    p = float(rng.uniform(0.3, 1.0))
    kids = lambda d: [d + 1 + int(rng.integers(0, 3)) for _ in range(4) if rng.random() < p] if d < depth - 3 else []
    assert worst(kids, [0] * 64, 512, 3 * depth + 4) <= 512
