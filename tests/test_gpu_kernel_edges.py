"""Kernels at the edges of their tiles and vector widths: scans and compactions around a warp's
step, its run and a chunk, from aligned and unaligned buffers; n-links of the RGBA upload at
widths around a vector and a tile, from aligned and unaligned images; the colour-model fit
around a warp and a cluster's round of samples."""
import numpy as np
import pytest

import synth
from GMM import GMM
from GraphCut import GraphCut
from test_gmm_fit import stroke_samples

pytestmark = pytest.mark.gpu


def _at(torch, a, offset):
    """The int32 array on the device, `offset` elements behind an aligned address."""
    buf = torch.zeros(a.size + offset + 4, dtype=torch.int32, device="cuda")
    v = buf[offset:offset + a.size]
    v.copy_(torch.from_numpy(np.ascontiguousarray(a.reshape(-1), dtype=np.int32)))
    return v


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 511, 513, 4095, 4096, 4097, 12289])
def test_scan_edges(cuda, oracle, n, offset):
    import _gcut
    L, p, s = _gcut.lib(), _gcut.ptr, _gcut.stream_handle()
    rng = np.random.default_rng(n)
    a, b = rng.integers(-3, 4, n).astype(np.int32), rng.integers(-3, 4, n).astype(np.int32)
    st = _gcut.ScanState(0, n)
    dA, dB = _at(cuda, a, offset), _at(cuda, b, offset)
    out, total = _at(cuda, np.zeros(n), offset), cuda.zeros(1, dtype=cuda.int32, device="cuda")
    _gcut.check(L.gc_scan_exclusive(st.handle, p(dA), p(out), p(total), n, s))
    ref, ref_total = oracle.exclusive_scan(a)
    assert np.array_equal(out.cpu().numpy(), ref) and int(total.item()) == ref_total
    for want, call in (
            (a != 0, lambda: L.gc_compact(st.handle, p(dA), p(out), p(total), n, s)),
            (a >= 1, lambda: L.gc_tiles_build(st.handle, p(dA), 3, 1, p(out), p(total), n, s)),
            ((a > 0) | (b < 0), lambda: L.gc_tiles_build_logical(
                st.handle, p(dA), p(dB), 1, 0, 2, 0, 1, p(out), p(total), n, s))):
        _gcut.check(call())
        idx = np.flatnonzero(want)
        assert int(total.item()) == idx.size
        assert np.array_equal(out[:idx.size].cpu().numpy(), idx)
    _gcut.check(L.gc_tiles_incorporate(p(dA), p(dB), 1, 0, 1, 0, 0, 9, n, s))
    assert np.array_equal(dA.cpu().numpy(), np.where((a > 0) & (b > 0), 9, a))
    st.close()


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("lamda", [None, 60])
@pytest.mark.parametrize("w,h", [(1, 1), (4, 33), (5, 3), (31, 64), (32, 32), (36, 65), (64, 31), (67, 40)])
def test_rgba_upload_edges(cuda, oracle, w, h, lamda, offset):
    rng = np.random.default_rng(w * h)
    img = rng.integers(0, 256, (h, w, 3)).astype(np.uint8)
    img[: h // 2] //= 32          # small distances too
    words = (img[..., 0].astype(np.int64) | (img[..., 1].astype(np.int64) << 8)
             | (img[..., 2].astype(np.int64) << 16)).astype(np.int32)
    excess = rng.integers(-50, 51, (h, w)).astype(np.int32)
    f = img.astype(np.int64)
    dv, dh = ((f[1:] - f[:-1]) ** 2).sum(-1), ((f[:, 1:] - f[:, :-1]) ** 2).sum(-1)
    if lamda is None:
        wv, wh = synth.nlinks(img)
    else:
        wv, wh = (np.asarray(oracle.weight_reference(d, lamda)).reshape(d.shape) for d in (dv, dh))
    up, down, left, right = synth.planes_from_weights(wv, wh, excess)
    with GraphCut(w, h) as gc:
        gc.upload_image(_at(cuda, words, offset).view(h, w), _at(cuda, excess, offset).view(h, w),
                        lamda=lamda)
        for name, want in (("dUp", up), ("dDown", down), ("dLeft", left), ("dRight", right),
                           ("dExcess", excess)):
            assert np.array_equal(getattr(gc, name).cpu().numpy(), want), name


@pytest.mark.parametrize("w,h", [(4, 4801), (3, 4763), (1028, 9), (257, 5)])
def test_rgba_table_strips(cuda, w, h):
    """More strips than one wave of CTAs, and columns past a CTA's, in both strip widths; the
    alpha byte takes no part."""
    rng = np.random.default_rng(w)
    img = rng.integers(0, 256, (h, w, 3)).astype(np.uint8)
    alpha = rng.integers(0, 256, (h, w, 1)).astype(np.uint8)
    excess = np.zeros((h, w), np.int32)
    up, down, left, right = synth.planes_from_weights(*synth.nlinks(img), excess)
    with GraphCut(w, h) as gc:
        gc.upload_image(np.concatenate([img, alpha], -1), excess)
        for name, want in (("dUp", up), ("dDown", down), ("dLeft", left), ("dRight", right)):
            assert np.array_equal(getattr(gc, name).cpu().numpy(), want), name


@pytest.mark.parametrize("n,K,full", [(31, 2, False), (33, 5, True), (10240, 4, False),
                                      (10241, 4, True), (20481, 7, False)])
def test_fit_edges(cuda, oracle, n, K, full):
    s = stroke_samples(n, n)
    g = GMM(12, K, tolerance=0.0, full_covariance=full)
    g.fit(s)
    want = oracle.gmm_fit(s, K, 12, tolerance=0.0, full=full)
    assert g.iterations == want["iterations"]
    np.testing.assert_allclose(g.weights, want["weights"], rtol=1e-7, atol=1e-10)
    np.testing.assert_allclose(g.means, want["means"], rtol=1e-7, atol=1e-7)
    np.testing.assert_allclose(g.log_likelihood, want["log_likelihood"], rtol=1e-10)


@pytest.mark.parametrize("npts,radius", [(1, 0), (2, 3), (33, 2), (64, 1), (65, 5), (300, 0)])
def test_stroke_points_in_the_launch_and_copied(cuda, npts, radius):
    """Strokes whose points travel in the launch (up to 64) and longer ones, partly outside the
    image, against the host rasteriser; the state is read on another stream right after."""
    import strokes
    w, h = 150, 90
    rng = np.random.default_rng(npts)
    g = synth.random_graph(w, h, 3, cap_max=5, tlink_max=9)
    xs = rng.integers(-20, w + 20, npts).astype(np.int32)
    ys = rng.integers(-20, h + 20, npts).astype(np.int32)
    want = strokes.apply(g.excess, strokes.Stroke(xs, ys, radius, 77))
    other = cuda.cuda.Stream()
    with GraphCut(w, h) as gc:
        gc.upload_capacities(*g.planes())
        cuda.cuda.synchronize()
        gc.edit_stroke(xs, ys, radius, 77)
        with cuda.cuda.stream(other):
            got = gc.dExcess
            other.synchronize()
        assert np.array_equal(got.cpu().numpy(), want)


def test_upload_captured_after_an_edit(cuda, oracle):
    """A stroke is still on its way when the next upload is captured into a CUDA graph: the
    capture holds the upload alone, and its replay gives the cold solve."""
    torch = cuda
    g = synth.make_graph(130, 70, 5)
    planes = [torch.from_numpy(p).cuda() for p in g.planes()]
    f_ref, l_ref = oracle.maxflow_bk(*g.planes())
    with GraphCut(g.width, g.height) as gc:
        gc.upload_capacities(*planes)
        gc.cut()
        graph = torch.cuda.CUDAGraph()
        gc.edit_stroke([3, 100], [5, 60], 4, 500)
        with torch.cuda.graph(graph):
            gc.upload_capacities(*planes)
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(gc.cut_labels().cpu().numpy(), l_ref)
        assert gc.flow == f_ref
