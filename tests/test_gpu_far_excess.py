"""Solves whose excess lies far from every sink: the first list of a fresh solve is empty (no
sink in or beside a tile with excess) and the relabel's distance cap (16, then twice as far
whenever no excess lies within it, and each cycle) has to grow, past its last finite value on
the longest grid.  Flow and canonical cut equal the exact oracle's, for the one-launch solve
and the host-driven loop, fresh and after an edit that moves the excess."""
import numpy as np
import pytest

import synth
from GraphCut import GraphCut

pytestmark = pytest.mark.gpu


def far_graph(w, h, seed):
    """Capacities 1..9 everywhere, one block of excess in the first corner, one sink pixel in
    the last (beyond the smallest caps on every grid below)."""
    g = synth.random_graph(w, h, seed, cap_max=9, tlink_max=1)
    for p in (g.up, g.down, g.left, g.right):
        p += 1
    g.excess[:] = 0
    g.excess[0, 0] = 50
    g.excess[h - 1, w - 1] = -40
    return g


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("w,h", [(33, 1), (48, 48), (1, 300), (129, 65), (5000, 1)])
def test_far_excess_matches_oracle(cuda, oracle, w, h, graph):
    g = far_graph(w, h, w + h)
    with GraphCut(w, h, use_graph=graph) as gc:
        gc.upload_capacities(*g.planes())
        f_ref, l_ref = oracle.maxflow_bk(*g.planes())
        lab = gc.cut_labels().cpu().numpy()
        assert gc.flow == f_ref
        assert np.array_equal(lab, l_ref)
        # a warm solve: the excess moves to the other end of the first row (of the column, on
        # the grid one pixel wide: the edited pixels have to be distinct)
        far = w - 1 if w > 1 else h - 1
        t = g.excess.copy()
        t.flat[0], t.flat[far] = -30, 25
        gc.edit_tlinks(np.array([0, far]), np.array([-30, 25]))
        f_ref, l_ref = oracle.maxflow_bk(g.up, g.down, g.left, g.right, t)
        lab = gc.cut_labels().cpu().numpy()
        assert gc.flow == f_ref
        assert np.array_equal(lab, l_ref)


@pytest.mark.parametrize("graph", [True, False])
def test_fresh_and_warm_images_far_apart(cuda, oracle, graph):
    """A pool of three images, one of them solved and edited, the others fresh, of which one
    has no sink near its excess."""
    from session_pool import SessionPool, tiles_of
    graphs = [far_graph(200, 40, 1), synth.make_graph(130, 70, 2), far_graph(64, 90, 3)]
    pool = SessionPool(sum(tiles_of(g.width, g.height) for g in graphs), 3, use_graph=graph)
    for k, g in enumerate(graphs):
        pool.open(k, g.width, g.height, pool.alloc_tiles(g.width, g.height))
        pool.upload_capacities(k, *g.planes())
    pool.solve([1])
    pool.edit_stroke(1, [20, 90], [20, 50], 6, 1000)
    import strokes
    t = strokes.apply(graphs[1].excess, strokes.Stroke(np.array([20, 90], np.int32),
                                                       np.array([20, 50], np.int32), 6, 1000))
    pool.solve([0, 1, 2])
    for k, g in enumerate(graphs):
        f_ref, l_ref = oracle.maxflow_bk(g.up, g.down, g.left, g.right, t if k == 1 else g.excess)
        assert pool.flow(k) == f_ref, k
        assert np.array_equal(pool.labels(k).cpu().numpy(), l_ref), k
    pool.close_pool()
