"""What one solve leaves to the next and its CTAs to one another: relabels that start over with a
larger cap while slower CTAs still leave the barrier before."""
import numpy as np
import pytest

from GraphCut import GraphCut

pytestmark = pytest.mark.gpu


def corridors(w, h, nearest, seed):
    """A corridor per row with its sink at x = 0 and excess at distances from `nearest` on, twice
    as far every few rows; every eighth row is joined to the one below."""
    rng = np.random.default_rng(seed)
    up, down, left, right, excess = (np.zeros((h, w), np.int32) for _ in range(5))
    left[:], right[:] = rng.integers(1, 10, (h, w)), rng.integers(0, 10, (h, w))
    down[::8] = rng.integers(0, 3, (len(range(0, h, 8)), w))
    up[1::8] = rng.integers(0, 3, (len(range(1, h, 8)), w))
    excess[:, 0] = -rng.integers(1, 12, h)
    d = nearest
    for y in range(0, h, 3):
        excess[y, min(d, w - 1)] = rng.integers(1, 30)
        d = nearest if d > w else 2 * d + 1
    up[0] = down[-1] = left[:, 0] = right[:, -1] = 0
    return up, down, left, right, excess


@pytest.mark.parametrize("nearest", [10, 40, 300])
def test_relabels_that_start_over(cuda, oracle, nearest):
    """512 tiles, more than a CTA each: no excess within the first caps, again and again."""
    planes = corridors(1024, 512, nearest, nearest)
    f_ref, l_ref = oracle.maxflow_bk(*planes)
    dev = [cuda.from_numpy(p).cuda() for p in planes]
    with GraphCut(1024, 512) as gc:
        for k in range(40):
            gc.upload_capacities(*dev)
            lab = gc.cut_labels()
            assert gc.flow == f_ref, k
            assert np.array_equal(lab.cpu().numpy(), l_ref), k
