"""Solves whose excess lies far from every sink: the first list of a fresh solve is empty (no
sink in or beside a tile with excess) and the relabel's distance cap (8, then twice as far
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


@pytest.mark.parametrize("w,h", [(32, 32), (1184, 384), (2848, 160), (1184, 385)])
def test_one_tile_per_cta_and_more(cuda, oracle, w, h):
    """The first pulse without a list (no more tiles than resident CTAs: up to 444 on a B200)
    and with one: 1, 444, 445 and 481 tiles."""
    g = synth.random_graph(w, h, w + h, cap_max=40, tlink_max=60)
    f_ref, l_ref = oracle.maxflow_bk(*g.planes())
    with GraphCut(w, h) as gc:
        gc.upload_capacities(*g.planes())
        lab = gc.cut_labels().cpu().numpy()
        assert gc.flow == f_ref
        assert np.array_equal(lab, l_ref)


def test_solves_of_both_kinds_and_steps_alternate(cuda, oracle):
    """One handle solved by one launch, by the host-driven loop (profiling on) and stepped by
    hand in turn, fresh and warm: each solve starts from what another kind left."""
    g = synth.make_graph(300, 200, 4)
    f_ref, l_ref = oracle.maxflow_bk(*g.planes())
    with GraphCut(g.width, g.height) as gc:
        for k in range(6):
            gc.upload_capacities(*g.planes())
            if k % 3 == 2:
                gc.push()
                gc.push()
            for prof in ((True, False), (False, True))[k % 2]:
                gc.set_profile(prof)
                gc.edit_tlinks(np.array([5, 77]), np.array([1000, -1000]))
                gc.cut()
                gc.edit_tlinks(np.array([5, 77]), g.excess.reshape(-1)[[5, 77]])
                gc.cut()
                assert gc.flow == f_ref, (k, prof)
                assert np.array_equal(gc.labels().cpu().numpy(), l_ref), (k, prof)


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("w,h", [(8, 32), (9, 31), (32, 32), (70, 40)])
def test_snake_distances(cuda, oracle, w, h, graph):
    """Residual edges along one winding path only: distances inside a tile of 255, 256 and more,
    and tiles entered again and again at far distances.  A global relabel gives the distance
    along the path; the solve equals the oracle's."""
    path = [(y, x) for y in range(h) for x in (range(w) if y % 2 == 0 else range(w - 1, -1, -1))]
    planes = [np.zeros((h, w), np.int32) for _ in range(5)]
    up, down, left, right, excess = planes
    for (y0, x0), (y1, x1) in zip(path, path[1:]):
        a, b = {(1, 0): (down, up), (0, 1): (right, left), (0, -1): (left, right)}[y1 - y0, x1 - x0]
        a[y0, x0] = b[y1, x1] = 7
    excess[path[-1]] = 30      # the far end; the sink is the first corner
    excess[0, 0] = -20
    with GraphCut(w, h, use_graph=graph) as gc:
        gc.upload_capacities(*planes)
        gc.startBfs()
        want = np.zeros((h, w), np.int64)
        for d, p in enumerate(path):
            want[p] = d
        assert np.array_equal(gc.dHeight.cpu().numpy(), want)
        gc.upload_capacities(*planes)
        f_ref, l_ref = oracle.maxflow_bk(*planes)
        assert np.array_equal(gc.cut_labels().cpu().numpy(), l_ref)
        assert gc.flow == f_ref
