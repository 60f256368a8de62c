"""Launch-split and tile-edge checks of the GPU kernels: sizes at the edges of
their tiles, shares and border paths."""
import ctypes

import numpy as np
import pytest

import vlr_b200 as V

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bsdf_queries():
    inp = V.make_bsdf_batch_inputs(914000, seed=41, materials=7)
    inp["material"][::97] = 9          # ids above 6 build UE4
    out, _ = V.bsdf_batch_host(inp)
    return inp, out


@pytest.mark.parametrize("n", [1, 7, 8, 31, 33, 255, 257, 1021, 1024, 1025, 2049, 4096, 4097, 9 * 1024 + 5, 31967, 31968, 31969, 50001,
                               101003, 262147, 524289, 909312, 909313])
def test_bsdf_batch_split_does_not_change_a_query(bsdf_queries, n):
    """A query's outputs do not depend on the batch around it, whatever share,
    group and pass it falls in: each prefix equals the large batch bit for bit."""
    import torch
    inp, want = bsdf_queries
    ins = {k: torch.from_numpy(np.ascontiguousarray(v[:n])).cuda() for k, v in inp.items()}
    outs = {k: torch.full((n, c) if c > 1 else (n,), float("nan"), device="cuda") for k, c in V.BATCH_OUTPUTS.items()}
    V.bsdf_batch_device(ins, outs)
    torch.cuda.synchronize()
    for k, o in outs.items():
        assert np.array_equal(o.cpu().numpy(), want[k][:n], equal_nan=True), k


def test_bsdf_batch_of_middling_size_fills_the_gpu():
    """100,000 queries against 2^20, ten times as many: 0.30 of their time, where
    a split that left warps without passes took 0.44."""
    import torch

    def best(n):
        ins = {k: torch.from_numpy(v).cuda() for k, v in V.make_bsdf_batch_inputs(n, seed=2, materials=7).items()}
        outs = {k: torch.zeros((n, c) if c > 1 else n, device="cuda") for k, c in V.BATCH_OUTPUTS.items()}
        stream = torch.cuda.current_stream()
        t = []
        for _ in range(8):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for _ in range(20):
                V.bsdf_batch_device(ins, outs, stream.cuda_stream)
            e1.record(stream)
            torch.cuda.synchronize()
            t.append(e0.elapsed_time(e1))
        return min(t)

    some, many = best(100000), best(1 << 20)
    assert some < 0.37 * many, (some, many)


def test_bsdf_batch_recorded_vectors_within_the_tables_fit():
    """The recorded outputs with whatever tables the library was built with.
    Fitted tables hold them to the last rounding in all but a few values (1e-6)
    of the BSDFs without a microfacet, and to 1e-5 in 99.9% of all."""
    import os
    g = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "bsdf_batch_2048.npz"))
    out, _ = V.bsdf_batch_host({k[3:]: g[k] for k in g.files if k.startswith("in_")})
    plain = np.isin(g["in_material"], [0, 1, 4])
    for k in ("value", "pdf", "wi", "evalValue", "evalPdf"):
        a, b = out[k].astype(np.float64), g["out_" + k].astype(np.float64)
        rel = np.where((a == b) | (np.isnan(a) & np.isnan(b)), 0.0, np.abs(a - b) / np.maximum(np.abs(b), 1e-30))
        assert np.mean(rel <= 1e-5) >= 0.999 and np.nanmax(rel) <= 2e-3, k
        if k in ("value", "pdf"):
            assert rel[plain].max() <= 1e-6 and np.mean(rel[plain] > 0) <= 0.005, k


def _render_context(W, H, **options):
    from vlr_b200 import vlr as VV, scenes
    ctx = VV.Context()
    ctx.bindOutputBuffer(W, H)
    scene, cam, keep = scenes.cornell_box(ctx, W, H)
    ctx.setScene(scene)
    ctx.setOptions(max_path_length=5, **options)
    return ctx, cam, (scene, keep)


def _colours(film, frames, magnitude=False):
    """XYZ / frames * (W * H) -> Rec.709 (D65) of an FP64 film (magnitude: the
    sum of its terms' absolute values)."""
    L = V.lib()
    L.vlrbCmfStrata.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    cmf = np.zeros(48, np.float32)
    integral = ctypes.c_float()
    assert L.vlrbCmfStrata(cmf.ctypes.data_as(ctypes.c_void_p), ctypes.byref(integral)) == 0
    xyz = film @ cmf.reshape(3, 16).astype(np.float64).T * (film.shape[0] * film.shape[1] / (integral.value * frames))
    m = np.array([[3.2404542, -1.5371385, -0.4985314], [-0.9692660, 1.8760108, 0.0415560],
                  [0.0556434, -0.2040259, 1.0572252]])
    return np.abs(xyz) @ np.abs(m).T if magnitude else xyz @ m.T


@pytest.mark.parametrize("size", [(1, 1), (7, 3), (8, 4), (33, 17), (127, 5), (129, 1), (64, 64)])
@pytest.mark.parametrize("launch_spp", [1, 3])
def test_film_pass_sums_and_converts(size, launch_spp):
    """The output image is the film's conversion after a first call (strata
    stored), a second one (added) and a restart, in one launch or several.  XYZ is
    formed in FP64 and rounded to FP32 (6e-8), the matrix and its three products
    and two sums are FP32: 6 roundings, 4e-7 of the terms' magnitude."""
    W, H = size
    ctx, cam, keep = _render_context(W, H, max_paths_in_flight=W * H * launch_spp)
    totals = []
    for first, spp, frames in ((True, 4, 4), (False, 3, 7), (True, 2, 2)):
        assert ctx.render_samples(cam, first, spp) == frames
        film, image = ctx.read_film(), ctx.read_output()
        want = _colours(film, frames)
        assert np.all(np.abs(image[..., :3] - want) <= 4e-7 * _colours(film, frames, magnitude=True) + 1e-30)
        assert np.all(image[..., 3] == 1)
        totals.append(film.sum())
    if W * H >= 64:
        assert totals[1] > totals[0] > 0 and totals[2] < totals[1]
    ctx.close()


def test_film_pass_of_a_shrunk_preview_leaves_the_rest_empty():
    ctx, cam, keep = _render_context(64, 48)
    ctx.render_samples(cam, True, 2)
    ctx.render(cam, True, shrink=4)
    film = ctx.read_film()
    assert film[:12, :16].sum() > 0
    assert not film[12:].any() and not film[:, 16:].any()
    ctx.close()


def _glowing_box(W, H, spp):
    """A context inside a box that only emits, seen through a field of view so
    narrow that all camera rays weigh the same: every sample adds one value to
    each quarter of its pixel's strata."""
    from vlr_b200 import vlr as VV
    ctx = VV.Context()
    ctx.bindOutputBuffer(W, H)
    mat = ctx.createSurfaceMaterial("DiffuseEmitter")
    mat.set("emittance", VV.rgb(1.0, 1.0, 1.0))
    node = ctx.createTriangleMeshSurfaceNode("wall")
    corners = [(-1, -1), (1, -1), (1, 1), (-1, 1)]
    verts = np.array([[x, y, z, 0, 0, -z, 1, 0, 0, 0, 0] for z in (-1, 1) for x, y in corners], np.float32)
    node.set_vertices(verts)
    node.add_material_group(np.array([0, 1, 2, 0, 2, 3, 4, 6, 5, 4, 7, 6], np.uint32), mat)
    scene = ctx.createScene()
    scene.add_child(node)
    cam = ctx.createCamera("Perspective")
    cam.set_point("position", (0.0, 0.0, 0.0))
    for k, v in (("aspect", 1.0), ("sensitivity", 1.0), ("fovy", 1e-3), ("lens radius", 0.0), ("op distance", 1.0)):
        cam.set(k, v)
    ctx.setScene(scene)
    ctx.setOptions(max_path_length=2, max_paths_in_flight=max(W * H * spp, 1))
    return ctx, cam, (scene, node, mat)


def _quarters(film, frames):
    H, W = film.shape[:2]
    return film.reshape(H, W, 4, 4).sum(axis=3) * (W * H / frames)


@pytest.fixture(scope="module")
def quarter_means():
    ctx, cam, keep = _glowing_box(256, 256, 16)
    ctx.render_samples(cam, True, 16)
    means = _quarters(ctx.read_film(), 16).mean(axis=(0, 1))
    ctx.close()
    return means


@pytest.mark.parametrize("size,spp", [((1, 1), 1), ((1, 1), 64), ((1, 1), 257), ((7, 3), 2), ((7, 3), 3), ((7, 3), 5),
                                      ((7, 3), 9), ((33, 17), 16), ((33, 17), 31), ((64, 64), 33), ((129, 65), 64),
                                      ((320, 200), 12), ((512, 320), 7)])
def test_film_pass_counts_every_sample_once(quarter_means, size, spp):
    """However many threads share a pixel, each sample is in its pixel's sums
    once.  A quarter's sum over n samples is n times a mean over 117.5 nm plus
    noise: the emission varies by less than a half within a quarter, so its
    standard error is below 0.5 / sqrt(12 n); six of them, below half a sample for
    n up to 12, and beyond that over all pixels a loss of one sample in each would
    stand out by far more."""
    (W, H), n = size, spp
    ctx, cam, keep = _glowing_box(W, H, spp)
    for first, frames in ((True, n), (False, 2 * n)):
        ctx.render_samples(cam, first, n)
        rel = _quarters(ctx.read_film(), frames) / quarter_means - 1
        assert np.all(np.abs(rel) < 6 * 0.5 / np.sqrt(12 * frames)), np.abs(rel).max()
        assert np.all(np.abs(rel.mean(axis=(0, 1))) < 6 * 0.5 / np.sqrt(12 * frames * W * H) + 2e-3)
    ctx.close()


def test_film_pass_of_few_pixels_splits_their_samples():
    """64 x 64 pixels of 512 samples are 67 MB of contributions, 10 us of HBM; one
    thread a pixel took 630."""
    ctx, cam, keep = _render_context(64, 64, max_paths_in_flight=64 * 64 * 512)
    ctx.set_profiling(True)
    ms = []
    for _ in range(4):
        ctx.kernel_times(reset=True)
        ctx.render_samples(cam, True, 512)
        ms.append(ctx.kernel_times()[0]["film"]["ms"])
    ctx.close()
    assert min(ms) < 0.2, ms


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 33, 257])
@pytest.mark.parametrize("rounds", [0, 3])
def test_packed_traversal_finds_every_hit(n, rounds):
    """Nodes renumbered in depth-first order: every ray's nearest hit and
    any-hit answer against all triangles in FP64; rays within 1e-4 of an edge
    or of tmax are left out (the FP32 test may decide them either way)."""
    rng = np.random.default_rng(n)
    v = (rng.uniform(0, 1, (n, 1, 3)) + rng.normal(0, 0.3, (n, 3, 3))).astype(np.float32)
    rays = np.zeros((4000, 8), np.float32)
    rays[:, 0:3] = rng.uniform(-0.5, 1.5, (4000, 3))
    rays[:, 3] = 3.0
    d = rng.normal(0, 1, (4000, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    o, dd = rays[:, None, 0:3].astype(float), rays[:, None, 4:7].astype(float)
    p0, e1, e2 = (a[None].astype(float) for a in (v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]))
    pv = np.cross(dd, e2)
    det = (pv * e1).sum(2)
    with np.errstate(divide="ignore", invalid="ignore"):
        u = (pv * (o - p0)).sum(2) / det
        qv = np.cross(o - p0, e1)
        w = (qv * dd).sum(2) / det
        t = (qv * e2).sum(2) / det
    margin = np.minimum(np.minimum(u, w), 1 - u - w)
    hit = (margin > 0) & (t > 0) & (t < 3.0)
    unsure = ((np.abs(margin) < 1e-4) & (t > -1e-3) & (t < 3.001)) | \
             ((margin > -1e-4) & ((np.abs(t) < 1e-4) | (np.abs(t - 3) < 1e-4)))
    ok = ~unsure.any(axis=1)
    near = np.where(hit, t, np.inf).min(axis=1)
    for any_hit in (0, 1):
        hits = np.zeros((4000, 4), np.float32)
        P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
        assert V.lib().vlrbTraceRaysHost(P(v), ctypes.c_uint32(n), ctypes.c_uint32(rounds), P(rays),
                                         ctypes.c_uint32(4000), ctypes.c_uint32(any_hit), P(hits), None) == 0
        found = hits[:, 3].view(np.uint32) != 0xFFFFFFFF
        assert np.array_equal(found[ok], np.isfinite(near)[ok])
        if not any_hit:
            f = ok & found
            assert np.allclose(hits[f, 0], near[f], rtol=1e-4, atol=1e-5)


def _trace(v, rays):
    hits = np.zeros((len(rays), 4), np.float32)
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert V.lib().vlrbTraceRaysHost(P(v), ctypes.c_uint32(len(v)), ctypes.c_uint32(3), P(rays),
                                     ctypes.c_uint32(len(rays)), ctypes.c_uint32(0), P(hits), None) == 0
    return hits


@pytest.fixture(scope="module")
def ray_query():
    rng = np.random.default_rng(9)
    v = (rng.uniform(0, 1, (3000, 1, 3)) + rng.normal(0, 0.05, (3000, 3, 3))).astype(np.float32)
    rays = np.zeros((400000, 8), np.float32)
    rays[:, 0:3] = rng.uniform(-0.5, 1.5, (400000, 3))
    rays[:, 3] = 5.0
    rays[:, 4:7] = rng.normal(0, 1, (400000, 3))
    return v, rays, _trace(v, rays)


@pytest.mark.parametrize("count", [1, 8191, 8192, 32767, 32768, 32769, 65536, 65537, 131073, 300001])
def test_host_copies_at_their_chunk_edges(ray_query, count):
    """Rays up and hits down in one piece, one chunk, two, and several workers'
    chunks: each prefix equals the large call bit for bit."""
    v, rays, want = ray_query
    assert np.array_equal(_trace(v, rays[:count]).view(np.uint32), want[:count].view(np.uint32))


def _memory(kind, a):
    """A copy of array `a` in pinned, registered or device memory, and
    its address."""
    import torch
    rt = torch.cuda.cudart()
    if kind == "pinned":
        t = torch.from_numpy(a.copy()).pin_memory()
        return t, t.data_ptr()
    if kind == "registered":
        b = a.copy()
        assert rt.cudaHostRegister(b.ctypes.data, b.nbytes, 0) in (0, rt.cudaError.success)
        return b, b.ctypes.data
    t = torch.from_numpy(a).cuda()
    return t, t.data_ptr()


@pytest.mark.parametrize("kind", ["pinned", "registered"])
def test_host_copies_of_pinned_arrays(ray_query, kind):
    import torch
    v, rays, want = ray_query
    hits = np.zeros((len(rays), 4), np.float32)
    keep = [_memory(kind, a) for a in (v, rays, hits)]
    assert V.lib().vlrbTraceRaysHost(ctypes.c_void_p(keep[0][1]), ctypes.c_uint32(len(v)), ctypes.c_uint32(3),
                                     ctypes.c_void_p(keep[1][1]), ctypes.c_uint32(len(rays)), ctypes.c_uint32(0),
                                     ctypes.c_void_p(keep[2][1]), None) == 0
    out = np.asarray(keep[2][0])
    assert np.array_equal(out.view(np.uint32), want.view(np.uint32))
    if kind == "registered":
        for k, _ in keep:
            torch.cuda.cudart().cudaHostUnregister(k.ctypes.data)


def test_pinned_arrays_are_not_staged(ray_query):
    """A call's pinned arrays move at the link's rate: faster than pageable ones,
    which a CPU has to copy first."""
    import time
    import torch
    from vlr_b200 import guide
    net = guide.GuideNet(14, seed=1)
    n = 65536
    rng = np.random.default_rng(2)
    arrays = [rng.uniform(0, 1, (n, 3)).astype(np.float32) for _ in range(3)] + [np.zeros((n, 40), np.float32)]
    pinned = [torch.from_numpy(a.copy()).pin_memory().numpy() for a in arrays]
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    best = []
    for s in (arrays, pinned):
        t = []
        for _ in range(20):
            t0 = time.perf_counter()
            assert guide._api().vlrbGuideNetInferHost(net.h, n, *(P(a) for a in s)) == 0
            t.append(time.perf_counter() - t0)
        best.append(min(t))
    net.close()
    assert np.array_equal(arrays[3], pinned[3])
    assert best[1] < best[0], best


def test_device_memory_in_place_of_a_host_array_does_not_crash(ray_query):
    """Whether the driver accepts it or not, the call answers (a CPU copy from a
    device address ends the process)."""
    v, rays, want = ray_query
    keep = _memory("device", rays)
    hits = np.zeros((len(rays), 4), np.float32)
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    r = V.lib().vlrbTraceRaysHost(P(v), ctypes.c_uint32(len(v)), ctypes.c_uint32(3), ctypes.c_void_p(keep[1]),
                                  ctypes.c_uint32(len(rays)), ctypes.c_uint32(0), P(hits), None)
    assert r == V.INTERNAL_ERROR or (r == 0 and np.array_equal(hits.view(np.uint32), want.view(np.uint32)))
    assert np.array_equal(_trace(v, rays[:1000]).view(np.uint32), want[:1000].view(np.uint32))


def test_host_calls_from_several_threads(ray_query):
    """Calls of different sizes at once, more of them than workspaces are kept."""
    from concurrent.futures import ThreadPoolExecutor
    v, rays, want = ray_query
    jobs = [(k * 7919 % 90000, 50000 + 30011 * (k % 5)) for k in range(12)]
    with ThreadPoolExecutor(6) as pool:
        got = list(pool.map(lambda j: _trace(v, rays[j[0]:j[0] + j[1]].copy()), jobs))
    for (a, n), g in zip(jobs, got):
        assert np.array_equal(g.view(np.uint32), want[a:a + n].view(np.uint32))


def test_many_callers_do_not_slow_each_other(ray_query):
    """Small calls of eight threads, per call, against those of one: the work of
    all is on one stream, so a call takes as long as alone (a half for scatter)
    unless the calls beyond the kept workspaces make and undo their own."""
    import time
    from concurrent.futures import ThreadPoolExecutor
    v, rays, _ = ray_query
    v, rays = v[:500].copy(), rays[:1000].copy()

    def per_call(pool, k):
        def calls():
            for _ in range(6):
                _trace(v, rays)
        best = []
        for _ in range(6):
            t0 = time.perf_counter()
            for f in [pool.submit(calls) for _ in range(k)]:
                f.result()
            best.append((time.perf_counter() - t0) / (6 * k))
        return min(best)

    with ThreadPoolExecutor(8) as pool:
        alone, together = per_call(pool, 1), per_call(pool, 8)
    assert together < 1.5 * alone, (together, alone)


def test_kept_memory_gives_way(ray_query):
    """What host calls keep is released when the device has no memory left: with
    it a larger call fits, and so does a renderer; and it goes with the last
    context."""
    import torch
    MB = 1 << 20

    def build(n):
        v = np.random.default_rng(n).uniform(0, 1, (n, 9)).astype(np.float32)
        out = [np.zeros(n, np.uint32), np.zeros(n, np.uint32), np.zeros(2 * n - 2, np.int32),
               np.zeros(6 * n - 6, np.float32)]
        return V.lib().vlrbBvhBuildHost(*(a.ctypes.data_as(ctypes.c_void_p) for a in [v]), ctypes.c_uint32(n),
                                        *(a.ctypes.data_as(ctypes.c_void_p) for a in out), None)

    def free():
        return torch.cuda.mem_get_info()[0]

    def all_but(left):
        torch.cuda.synchronize()
        hog = torch.empty(free() - left, dtype=torch.uint8, device="cuda")
        assert free() < left + 8 * MB
        return hog

    torch.cuda.empty_cache()
    ctx, cam, keep = _render_context(32, 32)
    assert build(600000) == 0                    # about 150 MB are kept
    hog = all_but(100 * MB)
    assert build(800000) == 0                    # needs about 200
    del hog
    torch.cuda.empty_cache()
    hog = all_but(100 * MB)
    ctx.setOptions(max_paths_in_flight=1 << 19)
    ctx.render_samples(cam, True, 512)           # about 120 MB of path state
    del hog
    torch.cuda.empty_cache()
    assert build(600000) == 0
    held = free()
    ctx.close()
    del keep
    assert free() > held + 140 * MB
    before = free()
    assert build(1200000) == 0                   # about 300 MB: above what is kept
    assert free() > before - 8 * MB
    assert build(600000) == 0
    assert np.array_equal(_trace(*ray_query[:2]).view(np.uint32), ray_query[2].view(np.uint32))


@pytest.mark.parametrize("size", [(1, 1), (7, 3), (33, 17), (129, 5)])
def test_guides_accumulate(size):
    """Guides added over three calls against the mean of the same calls' guides
    each on its own (a call's samples follow from its number): the sums are FP64
    and each is rounded once, the colours are three products: 4e-7 of the terms,
    here below 8."""
    W, H = size
    apart = []
    ctx, cam, keep = _render_context(W, H, aux_buffers=True)
    for _ in range(3):
        ctx.render(cam, True)
        apart.append(ctx.read_aux()[0].astype(np.float64))
    ctx.close()
    ctx, cam, keep = _render_context(W, H, aux_buffers=True)
    for k in range(3):
        ctx.render(cam, k == 0)
    together = ctx.read_aux()[0]
    ctx.close()
    assert np.abs(together - sum(apart) / 3).max() < 4e-6 and together[..., :3].max() > 0.01


def test_adding_guides_costs_little_more_than_storing_them():
    """1920 x 1080 guides added to the buffers' (265 MB read, 41 us of HBM) against
    stored: 1.36 times the time; 1.58 with each line's load behind the store of the
    one before."""
    import torch
    stream = torch.cuda.current_stream()

    def best(aux, first):
        ctx, cam, keep = _render_context(1920, 1080, aux_buffers=aux)
        ctx.render(cam, True, stream=stream.cuda_stream)
        t = []
        for _ in range(6):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for _ in range(10):
                ctx.render(cam, first, stream=stream.cuda_stream)
            e1.record(stream)
            torch.cuda.synchronize()
            t.append(e0.elapsed_time(e1) / 10)
        ctx.close()
        return min(t)

    added, stored = (best(True, first) - best(False, first) for first in (False, True))
    assert added < 1.5 * stored, (added, stored)


def _device_bytes(f):
    """Device memory that f() takes and does not give back."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    keep = f()
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0], keep


def test_a_scene_keeps_what_rendering_reads():
    """A grid of a million triangles: 24 B of vertices (two triangles share four of
    them), 20 B of indices and materials, a 128 B record, 112 B of hierarchy and 52 B
    of scratch are 336 B a triangle; a tenth for granularity."""
    from vlr_b200 import vlr as VV
    m = 708
    ctx = VV.Context()
    ctx.bindOutputBuffer(16, 16)
    x, z = np.meshgrid(np.linspace(-1, 1, m + 1), np.linspace(-1, 1, m + 1))
    verts = np.zeros(((m + 1) ** 2, 11), np.float32)
    verts[:, 0], verts[:, 2], verts[:, 4], verts[:, 6] = x.ravel(), z.ravel(), 1, 1
    i = (np.arange(m)[:, None] * (m + 1) + np.arange(m)).ravel().astype(np.uint32)
    idx = np.stack([i, i + m + 1, i + 1, i + 1, i + m + 1, i + m + 2], axis=1).ravel()
    mat = ctx.createSurfaceMaterial("DiffuseEmitter")
    node = ctx.createTriangleMeshSurfaceNode("grid")
    node.set_vertices(verts)
    node.add_material_group(idx, mat)
    scene = ctx.createScene()
    scene.add_child(node)
    cam = ctx.createCamera("Perspective")
    cam.set_point("position", (0.0, 1.0, 2.0))
    ctx.setScene(scene)
    ctx.setOptions(max_path_length=2, max_paths_in_flight=256)
    used, _ = _device_bytes(lambda: ctx.render(cam, True))
    n = ctx.stats()["numTriangles"]
    ctx.close()
    assert n == 2 * m * m
    assert used < 1.1 * 336 * n, used / n


def test_a_path_slot_keeps_what_path_tracing_uses():
    """RNG 8, throughput 16, scalars 16, contribution, ray and hit 64, queues 8,
    nine buckets 36 and a shadow ray 48: 196 B a slot."""
    slots = 1 << 22
    ctx, cam, keep = _render_context(64, 64, max_paths_in_flight=4096)
    ctx.render(cam, True)
    ctx.setOptions(max_paths_in_flight=slots)
    used, _ = _device_bytes(lambda: ctx.render_samples(cam, True, slots // 4096))
    ctx.close()
    assert used < 196 * slots + (8 << 20), used / slots


def _atrous(color, albedo, normal, infinite_variance=False):
    """The denoiser in numpy (float64, guides rounded to halves as stored).
    infinite_variance: what FP32 makes of very bright images."""
    eps = 1e-3
    H, W = color.shape[:2]
    guided = albedo[..., :3].astype(np.float32).sum(axis=2, dtype=np.float32) > eps
    a16 = np.minimum(albedo[..., :3], 65504).astype(np.float16).astype(float)
    n16 = normal[..., :3].astype(np.float16).astype(float)
    filtered = guided & (a16[..., 0] >= 0)   # a negative red marks pixels the passes leave alone
    lum = np.array([0.2126, 0.7152, 0.0722])
    ill = np.where(guided[..., None], color[..., :3] / np.maximum(albedo[..., :3], eps), 0.0).astype(float)
    var = np.zeros((H, W))
    L = ill @ lum
    for y in range(H):
        for x in range(W):
            if guided[y, x]:
                ys, xs = slice(max(y - 1, 0), y + 2), slice(max(x - 1, 0), x + 2)
                l = L[ys, xs][guided[ys, xs]]
                var[y, x] = np.inf if infinite_variance else max((l * l).mean() - l.mean() ** 2, 0.0)
    k = [3 / 8, 1 / 4, 1 / 16]
    for step in (1, 2, 4, 8, 16):
        L = ill @ lum
        num, den, vs = np.zeros_like(ill), np.zeros((H, W)), np.zeros((H, W))
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                y0, y1 = max(0, -dy * step), min(H, H - dy * step)
                x0, x1 = max(0, -dx * step), min(W, W - dx * step)
                if y0 >= y1 or x0 >= x1:
                    continue
                p = (slice(y0, y1), slice(x0, x1))
                q = (slice(y0 + dy * step, y1 + dy * step), slice(x0 + dx * step, x1 + dx * step))
                h = k[abs(dx)] * k[abs(dy)]
                if dx == 0 and dy == 0:
                    w = np.full(L[p].shape, h)
                else:
                    wn = np.maximum((n16[p] * n16[q]).sum(2), 0) ** 128
                    da = ((a16[p] - a16[q]) ** 2).sum(2)
                    w = h * wn * np.exp(-da / 0.02 - np.abs(L[p] - L[q]) / (4 * np.sqrt(var[p]) + 1e-6))
                w = w * filtered[q] * filtered[p]
                num[p] += w[..., None] * ill[q]
                den[p] += w
                vs[p] += w * w * np.where(w > 0, var[q], 0.0)
        g = filtered
        ill[g], var[g] = num[g] / den[g][:, None], vs[g] / den[g] ** 2
    out = color.astype(float).copy()
    out[..., :3] = np.where(guided[..., None], ill * np.maximum(albedo[..., :3], eps), color[..., :3])
    return out


@pytest.mark.parametrize("size", [(5, 3), (37, 21), (70, 66)])
def test_denoiser_matches_numpy(size):
    """The a-trous passes against float64 numpy, on images smaller than the
    widest step (every tap a border test) and with an interior.  The 24 taps
    of a pass and the variance, a difference of squares, are summed in FP32:
    5e-3 of the image's mean at the largest, 1e-4 in the mean."""
    W, H = size
    images = []
    for denoise in (False, True):
        ctx, cam, keep = _render_context(W, H, aux_buffers=True)
        ctx.render(cam, True, denoise=denoise)
        images.append(ctx.read_output())
        aux = ctx.read_aux()
        ctx.close()
    want = _atrous(images[0], *aux)
    off = np.abs(images[1][..., :3] - want[..., :3])
    scale = np.maximum(np.abs(want[..., :3]), np.abs(want[..., :3]).mean())
    assert (off / scale).max() < 5e-3 and (off / scale).mean() < 1e-4


@pytest.mark.parametrize("size", [(2, 2), (6, 4), (45, 40)])
def test_denoiser_of_a_very_bright_image(size):
    """A floor whose illumination is about 1.3e19 everywhere: the sum of four
    squares overflows FP32 and that of the mean does not, so the variance is
    infinite and the luminance term drops out.  That ends in finite colours, at
    the border too.  24 products and a quotient a pass in FP32, five passes:
    1e-4."""
    from vlr_b200 import vlr as VV, scenes
    W, H = size

    def render(emittance, denoise):
        ctx = VV.Context()
        ctx.bindOutputBuffer(W, H)
        desc = scenes.floor_desc(W, H, light_at=(0.0, 0.0))
        desc["camera"]["fovy"] = 0.2
        desc["materials"]["light"] = ("DiffuseEmitter", {"emittance": ("Rec709(D65)",) + (emittance,) * 3})
        for k, mesh in enumerate(desc["meshes"]):
            mesh["name"] = str(k)
        scene, cam, keep = scenes.build(ctx, desc)
        ctx.setScene(scene)
        ctx.setOptions(max_path_length=2, aux_buffers=True)
        for k in range(64):
            ctx.render(cam, k == 0, denoise=denoise and k == 63)
        out = ctx.read_output(), ctx.read_aux()
        ctx.close()
        return out

    lum = np.array([0.2126, 0.7152, 0.0722])
    plain, (albedo, _) = render(1.0, False)
    l = (plain[..., :3] / albedo[..., :3].clip(1e-3)) @ lum
    scale = 1.3e19 / l.mean()
    color, aux = render(scale, False)
    l = (color[..., :3] / albedo[..., :3].clip(1e-3)) @ lum
    assert np.isfinite(color).all() and l.min() > 0.95e19 and l.max() < 1.8e19
    out, _ = render(scale, True)
    want = _atrous(color, *aux, infinite_variance=True)
    assert np.isfinite(out).all()
    assert np.abs(out[..., :3] / want[..., :3] - 1).max() < 1e-4


@pytest.mark.parametrize("n", [1, 127, 128, 129, 256, 257, 18944, 18945, 25000, 37888, 37889, 113664,
                               113665, 113921])
def test_guide_inference_tiles(n):
    """A query's network outputs do not depend on its tile: each prefix equals
    the large batch bit for bit (18,944 rows are one tile per SM, 37,888 two, and
    113,664 fill the resident groups once)."""
    from vlr_b200.guide import GuideNet
    rng = np.random.default_rng(3)
    net = GuideNet(12, seed=1)
    net.set_params(rng.normal(0, 0.2, net.n_weights).astype(np.float32),
                   rng.normal(0, 0.4, net.n_grid).astype(np.float32))
    m = 120000
    pos = rng.uniform(0, 1, (m, 3)).astype(np.float32)
    d = rng.normal(0, 1, (2, m, 3))
    d = (d / np.linalg.norm(d, axis=2, keepdims=True)).astype(np.float32)
    want = net.infer(pos, d[0], d[1])
    assert np.isfinite(want).all() and want.std() > 0
    assert np.array_equal(net.infer(pos[:n], d[0][:n], d[1][:n]), want[:n])
    net.close()
