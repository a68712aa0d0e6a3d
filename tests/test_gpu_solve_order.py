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


def test_solve_after_an_edit_on_another_stream(cuda, oracle):
    """A stroke on slot 0 waits behind other work on its stream; the labels of slot 1 are read on
    a second stream, and slot 0 is solved on a third: the solve has the stroke in it."""
    import strokes
    import synth
    from session_pool import SessionPool, tiles_of
    graphs = [synth.make_graph(300, 200, 1), synth.make_graph(130, 70, 2)]
    stroke = strokes.Stroke(np.array([40, 200], np.int32), np.array([30, 150], np.int32), 9, 900)
    pool = SessionPool(sum(tiles_of(g.width, g.height) for g in graphs), 2)
    a, b, c = (cuda.cuda.Stream() for _ in range(3))
    for k, g in enumerate(graphs):
        pool.open(k, g.width, g.height, pool.alloc_tiles(g.width, g.height))
        pool.upload_capacities(k, *g.planes())
    pool.solve([0, 1])
    with cuda.cuda.stream(a):
        cuda.cuda._sleep(20_000_000)   # about 10 ms
    pool.edit_stroke(0, stroke.xs, stroke.ys, stroke.radius, stroke.value, stream=a)
    with cuda.cuda.stream(b):
        lab1 = pool.labels(1, stream=b)
    b.synchronize()
    assert np.array_equal(lab1.cpu().numpy(), oracle.maxflow_bk(*graphs[1].planes())[1])
    pool.solve([0], stream=c)
    g = graphs[0]
    f_ref, l_ref = oracle.maxflow_bk(g.up, g.down, g.left, g.right, strokes.apply(g.excess, stroke))
    assert pool.flow(0) == f_ref
    assert np.array_equal(pool.labels(0).cpu().numpy(), l_ref)
    cuda.cuda.synchronize()
    pool.close_pool()


@pytest.mark.parametrize("destroy", [False, True])
def test_an_edit_behind_a_refused_call(cuda, oracle, destroy):
    """A stroke waits behind other work on its stream; labels are refused on another stream (the
    edit is not solved yet); then a cut on a third stream, or the end of a handle in caller-owned
    memory, comes after the stroke."""
    import _gcut
    import strokes
    import synth
    g = synth.make_graph(130, 70, 3)
    stroke = strokes.Stroke(np.array([20, 100], np.int32), np.array([10, 60], np.int32), 5, -700)
    arena = cuda.zeros(GraphCut.arena_bytes(g.width, g.height) // 4 + 64, dtype=cuda.int32, device="cuda")
    arena = arena[(-arena.data_ptr() % 256) // 4:]
    a, b, c = (cuda.cuda.Stream() for _ in range(3))
    gc = GraphCut(g.width, g.height, arena=arena)
    gc.upload_capacities(*g.planes())
    gc.cut()
    with cuda.cuda.stream(a):
        cuda.cuda._sleep(20_000_000)
    gc.edit_stroke(stroke.xs, stroke.ys, stroke.radius, stroke.value, stream=a)
    with pytest.raises(_gcut.GCError):
        gc.labels(stream=b)
    if destroy:
        gc.close()
        assert a.query()
        return
    gc.cut(stream=c)
    f_ref, l_ref = oracle.maxflow_bk(g.up, g.down, g.left, g.right, strokes.apply(g.excess, stroke))
    assert gc.flow == f_ref
    assert np.array_equal(gc.labels().cpu().numpy(), l_ref)
    gc.close()


@pytest.mark.parametrize("graph", [True, False])
def test_is_completed_after_a_cut(cuda, oracle, graph):
    """isCompleted once more after startBfs and a cut, fresh and warm: the cut is complete, and the
    next cut's flow is not short of what that call summed.  After a cut that failed there are no
    distances to go by, and isCompleted is refused."""
    import _gcut
    import synth
    g = synth.make_graph(200, 130, 6)
    f_ref, l_ref = oracle.maxflow_bk(*g.planes())
    with GraphCut(g.width, g.height, use_graph=graph) as gc:
        gc.upload_capacities(*g.planes())
        for k in range(3):
            gc.startBfs()
            gc.cut()
            assert gc.isCompleted() and gc.isCompleted(), k
            assert gc.flow == f_ref, k
            gc.cut()
            assert gc.flow == f_ref, k
            assert np.array_equal(gc.labels().cpu().numpy(), l_ref), k
    with GraphCut(200, 32, use_graph=graph, max_cycles=1) as gc:
        gc.upload_capacities(*corridors(200, 32, 150, 1))
        gc.startBfs()
        with pytest.raises(_gcut.GCError):
            gc.cut()      # the excess is too far from the sinks for the first cycle
        with pytest.raises(_gcut.GCError):
            gc.isCompleted()


@pytest.mark.parametrize("graph,first,left_over", [(True, "cut", 13), (False, "cut", 9),
                                                   (True, "startBfs", 16), (False, "startBfs", 16)])
def test_solve_after_one_that_ran_out_of_rounds(cuda, oracle, graph, first, left_over):
    """A row of 24 tiles whose cut or startBfs needs more rounds than allowed fails with a tile
    still queued for the next round (the host-driven rounds run on to the end of their batch).  The
    t-links then change so that excess and sink are in the tiles beside that one: the next cut,
    whose flood has to queue it, is the oracle's."""
    import _gcut
    w, h = 32 * 24, 32
    up, down, left, right, excess = (np.zeros((h, w), np.int32) for _ in range(5))
    left[16, 1:] = 5   # none to the right, where the floods would go on to the end of the row
    far = [32 * 22 + 4, 32 * 3 + 20]
    excess[16, far] = 7, -6
    with GraphCut(w, h, use_graph=graph, max_bfs_rounds=9) as gc:
        gc.upload_capacities(up, down, left, right, excess)
        with pytest.raises(_gcut.GCError):
            getattr(gc, first)()
        idx = 16 * w + np.array([*far, 32 * (left_over + 1) + 4, 32 * (left_over - 1) + 20])
        val = np.array([0, 0, 7, -6])
        gc.edit_tlinks(idx, val)
        excess.flat[idx] = val
        f_ref, l_ref = oracle.maxflow_bk(up, down, left, right, excess)
        lab = gc.cut_labels()
        assert gc.flow == f_ref == 5
        assert np.array_equal(lab.cpu().numpy(), l_ref)


@pytest.mark.parametrize("graph", [True, False])
def test_initial_relabel_is_exact(cuda, oracle, graph):
    """initial_relabel: one global relabel, without a distance cap, before the first pulse, also
    where all excess is further from the sinks than any first cap."""
    planes = corridors(600, 64, 300, 2)
    f_ref, l_ref = oracle.maxflow_bk(*planes)
    with GraphCut(600, 64, use_graph=graph, initial_relabel=True) as gc:
        gc.upload_capacities(*planes)
        gc.set_trace(True)
        lab = gc.cut_labels()
        kinds = [k for k, _ in gc.trace()]
        assert gc.flow == f_ref
        assert np.array_equal(lab.cpu().numpy(), l_ref)
        assert kinds[:kinds.index("discharge")].count("bfs_first") == 1


def test_replay_of_an_upload_after_an_edit(cuda, oracle):
    """An upload captured into a CUDA graph is launched on another stream after a stroke that was
    held back on its own: the upload comes last, and the cut is the uploaded graph's."""
    import synth
    g = synth.make_graph(130, 70, 8)
    planes = [cuda.from_numpy(p).cuda() for p in g.planes()]
    f_ref, l_ref = oracle.maxflow_bk(*g.planes())
    a, b = cuda.cuda.Stream(), cuda.cuda.Stream()
    with GraphCut(g.width, g.height) as gc:
        gc.upload_capacities(*planes)
        gc.cut()
        graph = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(graph):
            gc.upload_capacities(*planes)
        for _ in range(2):
            with cuda.cuda.stream(a):
                cuda.cuda._sleep(20_000_000)
            gc.edit_stroke([3, 100], [5, 60], 4, 500, stream=a)
            with cuda.cuda.stream(b):
                graph.replay()
            cuda.cuda.synchronize()
            assert np.array_equal(gc.cut_labels().cpu().numpy(), l_ref)
            assert gc.flow == f_ref
