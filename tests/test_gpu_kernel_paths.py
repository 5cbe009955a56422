"""Device paths at the sizes where they can go wrong, against the CPU oracle bit for bit: windows without a kernel of their
own, the longest image sides, the costs a run keeps (more sources than it keeps, planes without depth), the speckle
tiles' edges and large components, the median's edges, downloads beside running work, sessions that reuse texture arrays."""
import numpy as np
import pytest

from cumulus3d_b200 import fusion, scenes
from cumulus3d_b200.patchstereo import DepthSnapshot, PatchMatchBackend, RunParams, ViewState, _views, c_states
from oracle import oracle

pytestmark = pytest.mark.gpu


def _same(a, b, what):
    for k in ("depth", "normal", "cost"):
        np.testing.assert_array_equal(getattr(a, k), getattr(b, k), err_msg=f"{what} {k}")


def _new(wl):
    return [ViewState.new(c.width, c.height) for c in wl.cams]


@pytest.mark.parametrize("wr,ws", [(1, 1), (2, 2), (4, 1), (6, 2), (7, 1), (7, 2), (10, 1)])
def test_uncompiled_windows_default_tuning(wr, ws):
    """Even and odd row and column counts, four and eight columns unrolled, with and without the weight cache; an image
    side below a tile and one above it."""
    wl = scenes.workload_small(67, 13, views=3, window_radius=wr, window_step=ws, seed=40 + wr)
    gpu, cpu = _new(wl), _new(wl)
    p1, p2 = RunParams(0, False, True, 2, 1), RunParams(0, True, False, 1, 2)
    be = PatchMatchBackend(0)
    with be.begin(wl.input) as s:
        s.run(wl.views, gpu, p1)
        oracle.run(wl.input, wl.views, cpu, p1)
        snap = DepthSnapshot(1, 0, [g.depth.copy() for g in gpu])
        s.run(wl.views, gpu, p2, snap)
        oracle.run(wl.input, wl.views, cpu, p2, snap)
    be.close()
    for a, b in zip(gpu, cpu):
        _same(a, b, f"window {wr},{ws}")


@pytest.mark.parametrize("w,h,f32", [(32768, 12, False), (11, 32768, True), (16385, 9, True)])
def test_largest_image_sides(w, h, f32):
    """The longest sides a session takes: a gather's integer coordinate selects the same footprint at texel 32767 as at 0,
    also where the footprint leaves the image at either end."""
    k, step = (28000.0, 28000.0, w / 2.0, h / 2.0), 0.6
    cams = [scenes.Camera(f"side{i}", k, np.eye(3), np.array([i * step * (w > h), i * step * (h > w), 0.0]), w, h)
            for i in (-1, 0, 1)]
    rng = np.random.default_rng(w)
    img = [rng.random((h, w), np.float32) for _ in cams]
    inp = scenes.kernel_input(cams, img, [[1, 2], [0, 2], [1]], (25.0, 60.0), window_radius=3, gray8=not f32)
    p = RunParams(0, False, True, 1, 1)
    gpu, cpu = [ViewState.new(w, h)], [ViewState.new(w, h)]
    be = PatchMatchBackend(0)
    with be.begin(inp) as s:
        s.run([1], gpu, p)
        costs = s.evaluate(0, [1], gpu)
    be.close()
    oracle.run(inp, [1], cpu, p)
    _same(gpu[0], cpu[0], f"{w} x {h}")
    np.testing.assert_array_equal(costs[0], oracle.evaluate(inp, 0, [1], cpu, False)[0])


@pytest.mark.parametrize("tuning", [0, 42])
@pytest.mark.parametrize("sources", [1, 8, 11])
def test_kept_costs_over_runs(sources, tuning):
    """Three iterations, then a run on other planes (some without depth) of the same session, then a geometric one: the
    costs kept for the first 8 sources never outlive their plane or their run."""
    wl = scenes.workload_small(56, 40, views=12, window_radius=3, seed=61, sources=sources, positions=4)
    rng = np.random.default_rng(5)
    gpu, cpu = _new(wl), _new(wl)
    be = PatchMatchBackend(0, tuning=tuning)
    with be.begin(wl.input) as s:
        p = RunParams(0, False, True, 3, 1)
        s.run(wl.views, gpu, p)
        oracle.run(wl.input, wl.views, cpu, p)
        for a, b in zip(gpu, cpu):
            _same(a, b, "first run")
        for st in gpu:
            st.depth[...] = np.where(rng.random(st.depth.shape) < 0.2, 0.0, st.depth * rng.uniform(0.8, 1.3, st.depth.shape))
        cpu = [g.copy() for g in gpu]
        p = RunParams(0, False, False, 2, 2)
        s.run(wl.views, gpu, p)
        oracle.run(wl.input, wl.views, cpu, p)
        snap = DepthSnapshot(1, 0, [g.depth.copy() for g in gpu])
        p = RunParams(0, True, False, 2, 3)
        s.run(wl.views, gpu, p, snap)
        oracle.run(wl.input, wl.views, cpu, p, snap)
    be.close()
    for a, b in zip(gpu, cpu):
        _same(a, b, f"{sources} sources")


@pytest.mark.parametrize("w,h,frac", [(31, 7, 0.05), (32, 8, 0.1), (33, 9, 0.05), (96, 65, 0.002), (130, 70, 0.03)])
def test_speckles_at_tile_edges(w, h, frac):
    """Components inside, along and across the 32 x 8 tiles of one-iteration maps (many of them), with limits up to more
    than 128 pixels."""
    wl = scenes.workload_small(w, h, views=3, window_radius=3, seed=w + h)
    post = fusion.default_post()
    post.speckle_min_area_frac = frac
    be = PatchMatchBackend(0)
    with be.begin(wl.input) as s:
        s.schedule_resident(wl.views, 1, 0, 0)
        before = s.readout_resident(wl.views)
        removed = s.postprocess_resident(0, wl.views, post)
        after = s.readout_download(0, wl.views)
    be.close()
    n = 0
    for b, a in zip(before, after):
        d, nn = b.depth.copy(), b.normal.copy()
        n += oracle.remove_speckles(d, nn, b.cost, post)
        np.testing.assert_array_equal(a.depth, d)
        np.testing.assert_array_equal(a.normal, nn)
    assert removed == n


@pytest.mark.parametrize("w,sizes", [(64, [2047, 2048, 2049, 2050]), (64, [2049, 300, 5001]), (257, [40000, 2049, 70000])])
def test_speckles_of_large_components(w, sizes):
    """Components on both sides of what one warp takes, in row-major runs of pixels.  Of each, the keys up to the limit are
    just not enough, or just enough, to hold the lower median: an error of one key in either direction shows."""
    total = sum(sizes)
    h = -(-total // w)
    wl = scenes.workload_small(w, h, views=2, window_radius=1, seed=2, sources=1)
    rng = np.random.default_rng(total)
    depth, cost = np.zeros(w * h, np.float32), np.full(w * h, 2.0, np.float32)
    expect, o = np.zeros(w * h, bool), 0
    for i, n in enumerate(sizes):
        depth[o:o + n] = (30.0, 40.0)[i % 2]
        low = n // 2 + i % 2
        cost[o:o + n] = rng.permutation(np.r_[rng.choice([0.125, 0.5, 1.0], low), rng.choice([1.125, 1.5], n - low)])
        expect[o:o + n] = i % 2 == 0
        o += n
    states = []
    for k in range(2):
        st = ViewState.new(w, h)
        st.depth[...], st.cost[...], st.normal[..., 2] = depth.reshape(h, w), cost.reshape(h, w), -1.0
        states.append(st)
    post = fusion.default_post()
    post.speckle_min_area_frac, post.speckle_keep_cost = 1.5, 1.0
    be = PatchMatchBackend(0)
    with be.begin(wl.input) as s:
        s.upload(0, wl.views, states)
        s.median_filter(wl.input, 0, wl.views, states)  # its input stays in the readout planes
        removed = s.postprocess_resident(0, wl.views, post)
        after = s.readout_download(0, wl.views)
    be.close()
    d, nn = states[0].depth.copy(), states[0].normal.copy()
    assert oracle.remove_speckles(d, nn, states[0].cost, post) * 2 == removed == 2 * expect.sum()
    np.testing.assert_array_equal((d == 0).ravel()[:total], expect[:total])
    for a in after:
        np.testing.assert_array_equal(a.depth, d)
        np.testing.assert_array_equal(a.normal, nn)


@pytest.mark.parametrize("repeat,max_batch", [([0, 0], 64), ([1, 0, 1, 1, 2, 0], 64), ([0, 1, 0, 2, 2], 2)])
def test_speckles_of_views_named_more_than_once(repeat, max_batch):
    """Within one launch and across launches: each view is cleaned once, and its erased pixels count once."""
    wl = scenes.workload_small(40, 24, views=3, window_radius=3, seed=11)
    post = fusion.default_post()
    post.speckle_min_area_frac = 0.2
    be = PatchMatchBackend(0, max_batch=max_batch)
    with be.begin(wl.input) as s:
        s.schedule_resident(wl.views, 1, 0, 0)
        before = s.readout_resident(wl.views)
        removed = s.postprocess_resident(0, repeat, post)
        after = s.readout_download(0, wl.views)
    be.close()
    n = 0
    for v, (b, a) in enumerate(zip(before, after)):
        d, nn = b.depth.copy(), b.normal.copy()
        if v in repeat:
            n += oracle.remove_speckles(d, nn, b.cost, post)
        np.testing.assert_array_equal(a.depth, d)
        np.testing.assert_array_equal(a.normal, nn)
    assert removed == n and n > 0


@pytest.mark.parametrize("w,h", [(1, 1), (2, 5), (33, 9)])
def test_median_at_edges_and_ties(w, h):
    wl = scenes.workload_small(w, h, views=2, window_radius=1, seed=3, sources=1)
    rng = np.random.default_rng(w + h)
    states = []
    for c in wl.cams:
        st = ViewState.new(w, h)
        st.depth[...] = np.where(rng.random((h, w)) < 0.2, 0.0, rng.integers(28, 32, (h, w)))
        st.normal[..., 2] = -1.0
        states.append(st)
    be = PatchMatchBackend(0)
    with be.begin(wl.input) as s:
        got = s.median_filter(wl.input, 0, wl.views, states)
    be.close()
    for a, b in zip(got, oracle.median(wl.input, 0, wl.views, states)):
        np.testing.assert_array_equal(a.depth, b.depth)
        np.testing.assert_array_equal(a.normal, b.normal)


@pytest.mark.parametrize("sizes", [[(1, 1)], [(31, 33), (640, 480)], [(801, 603), (67, 13), (801, 603), (1300, 900)]])
def test_downloads_with_and_without_pending_work(sizes):
    """States downloaded while their run is still in flight (pages made present meanwhile, in chunks of 4 MB) hold what an
    idle download holds; arrays of several views in one block, of one view alone, and arrays that had other values."""
    cams = [scenes.formation(w, h, 1, prefix=f"d{i}")[0] for i, (w, h) in enumerate(sizes)]
    cams.append(scenes.formation(64, 48, 1, prefix="src")[1])
    rng = np.random.default_rng(9)
    img = [rng.random((c.height, c.width), np.float32) for c in cams]
    n = len(sizes)
    inp = scenes.kernel_input(cams, img, [[n]] * n + [[0]], (25.0, 60.0), window_radius=3)
    views = list(range(n))
    be = PatchMatchBackend(0)
    with be.begin(inp) as s:
        for p in (RunParams(0, False, True, 3, 1), RunParams(0, False, False, 2, 2)):
            s.run_resident(views, p)
            pending = s.download(0, views)
            idle = s.download(0, views)
            host = [ViewState.new(w, h) for w, h in sizes]
            for st in host:
                st.depth[...], st.normal[...], st.cost[...] = 7.0, 8.0, 9.0
            s._check(s.lib.ps_state_download(s.h, 0, _views(views), n, c_states(host, [])))
            for a, b, c in zip(pending, idle, host):
                _same(a, b, "pending, idle")
                _same(a, c, "pending, filled")
                assert (a.depth > 0).all()
    be.close()


def test_sessions_of_several_sizes_and_formats_in_turn():
    """One backend's sessions reuse the texture arrays of earlier ones by size and format: 8-bit and f32 images of one
    size, another size, and one session with more views than any before."""
    def workload(w, h, views, f32, seed):
        wl = scenes.workload_small(w, h, views=views, window_radius=3, seed=seed, positions=2)
        if f32:
            wl.input = scenes.kernel_input(wl.cams, [np.asarray(i, np.float32) for i in wl.images],
                                           [list(v.sources) for v in wl.input.views], (25.0, 60.0), window_radius=3,
                                           gray8=False)
        return wl
    kinds = [workload(64, 40, 3, False, 5), workload(64, 40, 3, True, 6), workload(48, 40, 3, False, 7),
             workload(64, 40, 5, False, 8)]
    p = RunParams(0, False, True, 1, 1)
    want = []
    for wl in kinds:
        want.append(_new(wl))
        oracle.run(wl.input, wl.views, want[-1], p)
    be = PatchMatchBackend(0)
    for i in (0, 1, 2, 0, 3, 1, 0, 2, 3, 1):
        got = _new(kinds[i])
        with be.begin(kinds[i].input) as s:
            s.run(kinds[i].views, got, p)
        for a, b in zip(got, want[i]):
            _same(a, b, f"session kind {i}")
    be.close()
