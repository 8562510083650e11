"""Forms that a call takes by its size against the general form, bit for bit:
batches over four-wide and quad nodes against the child-pair loop, short
queues traced a ray per warp against long ones, the device LBVH at the edges
of its sorts, the Shade stage as three kernels, further samples within a
server step, and the A-Trous row blocks at heights around a block of rows."""
import numpy as np
import pytest

import svgf_cases as S
from renderingengine_b200 import _native as N
from renderingengine_b200 import scenes
from renderingengine_b200.svgf import SvgfReconstruction
from renderingengine_b200.traversal import Scene
from renderingengine_b200.wavefront import FILM_MEAN, FILM_SAMPLE, Renderer, frame_constants
from test_svgf_gpu import _cfg_pair, _compare

pytestmark = pytest.mark.gpu


def _twice(tri, ulps=0):
    """The triangles and a copy of them with IDs of its own, coincident or a
    few ulps away: hits that only ties and rounding tell apart."""
    both = np.concatenate([tri, tri])
    second = both[len(tri):]
    second["metadata"][:, 2] += tri["metadata"][:, 2].max() + 1
    second["identity"][:, 1] += tri["identity"][:, 1].max() + 1
    for _ in range(ulps):
        second["positions"][:, :, 1] = np.nextafter(second["positions"][:, :, 1], np.float32(9))
    return both


def _rays(tri, count, seed):
    """A third random, a third from one point, a third along the axes from
    points on a coarse grid (origins on box planes, zero direction components)."""
    rng = np.random.default_rng(seed)
    p = tri["positions"].reshape(-1, 4)[:, :3].astype(np.float64)
    lo, hi = p.min(0), p.max(0)
    centre, half = (lo + hi) / 2, (hi - lo) / 2 + 1e-3
    o = centre + rng.uniform(-1.2, 1.2, (count, 3)) * half
    d = rng.normal(size=(count, 3))
    a, b = count // 3, 2 * count // 3
    o[a:b] = centre + np.array([0.3, 1.5, 2.1]) * half
    d[a:b] = centre + rng.uniform(-1, 1, (b - a, 3)) * half - o[a:b]
    o[b:] = np.round(o[b:] * 8) / 8
    d[b:] = 0.0
    d[np.arange(b, count), rng.integers(0, 3, count - b)] = rng.choice([-1.0, 1.0], count - b)
    r = np.zeros(count, N.RAY_DTYPE)
    r["origin_tmin"][:, :3], r["origin_tmin"][:, 3] = o, 1e-4
    r["direction_tmax"][:, :3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r["direction_tmax"][:, 3] = np.where(rng.random(count) < 0.2, rng.uniform(0.01, 1, count) * half.max(), 1e30)
    return r


@pytest.mark.parametrize("build", [N.BUILD_FLATTENED_SAH, N.BUILD_LBVH], ids=["sah", "lbvh"])
@pytest.mark.parametrize("triangles,copies,masked", [
    (3, None, False), (9, None, False), (4095, None, False), (4096, None, False), (2048, 0, False), (8192, 0, False),
    (8192, 1, False), (8192, 3, False), (30000, 1, False), (8192, None, True)])
def test_batch_forms_equal_child_pair_loop(native, build, triangles, copies, masked):
    """Counted batches always walk the child pairs.  The quad nodes are there
    from the first any-hit batch of 2^18 rays on."""
    tri = scenes.triangle_soup(triangles, seed=triangles).triangles
    if copies is not None:
        tri = _twice(tri, copies)
    if masked:  # without masks: an error for rays that meet one before a hit
        tri["metadata"][::10, 0] |= 2  # RE_GEOMETRY_FLAG_ALPHA_MASK
    scene = Scene(tri, 5, 1, build)
    for count in (1, 333, (1 << 18) - 1, 1 << 18, 1, 333, 65569):
        rays = _rays(tri, count, seed=count)
        for any_hit in (False, True):
            want, _ = scene.trace(rays, any_hit=any_hit, counters=True)
            got = scene.trace(rays, any_hit=any_hit)
            assert count < 65569 or (want["metadata"][:, 1] == N.HIT_KIND_TRIANGLE).any()
            np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32), err_msg=f"{count} {any_hit}")


@pytest.mark.parametrize("any_hit", [False, True])
def test_captured_batch_equals_child_pair_loop(native, any_hit):
    """The scene's first batch is captured: nothing may be reserved for it.  A
    larger batch outside the capture must leave the graph valid."""
    import torch
    tri = _twice(scenes.triangle_soup(20000, seed=3).triangles, 1)
    scene = Scene(tri, 5, 1, N.BUILD_LBVH)
    rays = _rays(tri, 70_000, 1)
    d_rays = torch.from_numpy(rays.view(np.uint8).reshape(-1)).cuda()
    d_hits = torch.zeros(len(rays) * N.HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        scene.trace_device(d_rays.data_ptr(), d_hits.data_ptr(), len(rays), any_hit,
                           stream=torch.cuda.current_stream().cuda_stream)
    scene.trace(_rays(tri, 300_000, 2), any_hit=any_hit)
    for _ in range(2):
        d_hits.zero_()
        graph.replay()
        torch.cuda.synchronize()
        want, _ = scene.trace(rays, any_hit=any_hit, counters=True)
        np.testing.assert_array_equal(d_hits.cpu().numpy().view(np.uint32), want.view(np.uint32).reshape(-1))


def _morton(tri):
    p = tri["positions"][:, :, :3]
    lo, hi = p.reshape(-1, 3).min(0).astype(np.float64), p.reshape(-1, 3).max(0).astype(np.float64)
    c = ((p.min(1) + p.max(1)) / np.float32(2)).astype(np.float64)
    with np.errstate(divide="ignore", invalid="ignore"):
        q = np.where(hi > lo, (c - lo) / (hi - lo), 0.5)
    q = np.minimum((np.clip(q, 0, 1) * 1024).astype(np.uint64), 1023)
    code = np.zeros(len(tri), np.uint64)
    for bit in range(10):
        for axis in range(3):
            code |= ((q[:, axis] >> np.uint64(bit)) & np.uint64(1)) << np.uint64(3 * bit + 2 - axis)
    return (code << np.uint64(32)) | tri["metadata"][:, 2].astype(np.uint64)


def _check_tree(tri, nodes, order):
    """Leaves in key order, pre-order numbering, every interior node split at
    its keys' highest differing bit, bounds the children's or the triangle's."""
    key = _morton(tri)
    np.testing.assert_array_equal(order, np.argsort(key, kind="stable"))
    key = key[order]
    n = len(tri)
    links = nodes["links"].astype(np.int64)
    leaf = links[:, 1] == 1
    assert len(nodes) == 2 * n - 1 and leaf.sum() == n
    np.testing.assert_array_equal(links[leaf, 0], np.arange(n))
    pos = tri["positions"][order][:, :, :3]
    np.testing.assert_array_equal(nodes["bounds_min"][leaf][:, :3], pos.min(1))
    np.testing.assert_array_equal(nodes["bounds_max"][leaf][:, :3], pos.max(1))
    inner = np.flatnonzero(~leaf)
    if n == 1:
        return
    left, right = links[inner, 0], links[inner, 2]
    np.testing.assert_array_equal(left, inner + 1)
    for b, f in (("bounds_min", np.minimum), ("bounds_max", np.maximum)):
        np.testing.assert_array_equal(nodes[b][inner][:, :3], f(nodes[b][left][:, :3], nodes[b][right][:, :3]))
    first = np.cumsum(leaf) - leaf  # leaves before a node: its first leaf in pre-order
    last = np.empty(len(nodes), np.int64)
    last[leaf] = links[leaf, 0]
    for i in inner[::-1]:
        last[i] = last[links[i, 2]]
    split = first[right]
    diff = key[first[inner]] ^ key[last[inner]]
    bit = np.zeros(len(inner), np.uint64)
    for s in (32, 16, 8, 4, 2, 1):
        over = (diff >> (bit + np.uint64(s))) > 0
        bit[over] += np.uint64(s)
    assert np.all(diff > 0)
    assert np.all((key[split] >> bit) & np.uint64(1) == 1) and np.all((key[split - 1] >> bit) & np.uint64(1) == 0)


@pytest.mark.parametrize("ids", ["ordered", "permuted", "sparse"])
@pytest.mark.parametrize("count", [1, 2, 3, 31, 33, 255, 257, 1023, 1025, 8191, 8193, 65535, 65536, 65537, 70001])
def test_device_lbvh_at_the_edges_of_its_sorts(native, count, ids):
    """65,536 keys are the most that the cluster sort takes.  Triangles on a
    coarse grid share codes, so that IDs decide."""
    import torch
    rng = np.random.default_rng(count)
    tri = scenes.triangle_soup(count, seed=count, max_edge=0.02).triangles
    base = np.round(tri["positions"][:, :1, :3] * 16) / 16
    coarse = rng.random(count) < 0.5
    tri["positions"][coarse, :, :3] += (base - tri["positions"][:, :1, :3])[coarse]
    if ids == "permuted":
        tri = tri[rng.permutation(count)]
    if ids == "sparse":
        tri["metadata"][:, 2] = rng.permutation(count).astype(np.uint32) * 60_013 + 17
    nodes, order = Scene(tri, 5, 1, N.BUILD_LBVH).export_flat()
    _check_tree(tri, nodes, order)
    if ids != "sparse":  # device records number the triangles 0 .. count - 1, at any 4-byte address
        records = torch.from_numpy(np.frombuffer(b"\0" * 4 + tri.tobytes(), np.uint8).copy()).cuda()
        got_nodes, got_order = Scene.from_device(records.data_ptr() + 4, count, 5).export_flat()
        assert got_nodes.tobytes() == nodes.tobytes()
        np.testing.assert_array_equal(got_order, order)


def _film(scene, data, w, h, depth, spp=1, **tuning):
    r = Renderer(w, h, depth)
    r.set_scene(scene, data)
    if tuning:
        r.set_tuning(**tuning)
    for k in range(spp):
        r.render(frame_constants(data.camera, w, h, k, depth, seed=0x5151), accumulate=k > 0)
    tel = r.collect()
    assert tel.fatal_mask == 0 and tel.non_finite == 0
    return r.read(FILM_SAMPLE, w * h).view(np.uint32)


def _coincident():
    data = scenes.add_emissive_triangles(scenes.heightfield_scene(grid=48, spheres=48, seed=2), count=200, seed=5)
    data.triangles = _twice(data.triangles)
    return data


def _unmasked():
    """A tenth of the triangles alpha-masked without masks: rays that meet one
    before a hit end in an error."""
    data = scenes.add_emissive_triangles(scenes.heightfield_scene(grid=48, spheres=48, seed=2), count=200, seed=5)
    data.triangles = data.triangles.copy()
    data.triangles["metadata"][::10, 0] |= 2  # RE_GEOMETRY_FLAG_ALPHA_MASK
    return data


def _loose(data):
    """The scene's flattened tree with every fifth box larger than its
    parent's."""
    nodes, order = Scene(data.triangles, data.fingerprint).export_flat()
    nodes["bounds_min"][5::5, :3] -= 0.05
    nodes["bounds_max"][5::5, :3] += 0.05
    return Scene(np.ascontiguousarray(data.triangles[order]), data.fingerprint, 1, N.BUILD_FLATTENED_SAH, nodes=nodes)


@pytest.mark.parametrize("make,build", [
    (_coincident, lambda d: Scene(d.triangles, d.fingerprint)),
    (_coincident, lambda d: Scene(d.triangles, d.fingerprint, 1, N.BUILD_LBVH)),
    (_coincident, _loose),
    (_unmasked, lambda d: Scene(d.triangles, d.fingerprint)),
], ids=["sah", "lbvh", "loose", "unmasked"])
@pytest.mark.parametrize("w,h", [(1, 1), (33, 7), (97, 61)])
def test_short_queues_equal_long_ones(native, w, h, make, build):
    """A frame alone, its rays traced one per warp, against the same frame
    beside one of a million pixels, traced 32 per warp, where the order of
    visits could show: every surface, the emitter's too, is there twice, or
    masks are missing."""
    data = make()
    scene = build(data)
    for mode in (2, 4):
        films = []
        for others in ([], [((1280, 800), w * h)]):
            r = Renderer(1280, 832, 8)
            r.set_scene(scene, data)
            r.set_tuning(traversal=mode)
            r.render_views([dict(frame=frame_constants(data.camera, *size, 0, 8, seed=0x5151), offset=offset,
                                 key=offset) for size, offset in [((w, h), 0)] + others])
            assert r.collect().fatal_mask == 0
            films.append(r.read_view(FILM_SAMPLE, 0, w * h).view(np.uint32))
        np.testing.assert_array_equal(films[0], films[1], err_msg=str(mode))


@pytest.mark.parametrize("w,h", [(511, 513), (512, 512), (1031, 257)])
def test_default_shade_around_the_three_kernel_line(native, w, h):
    data = scenes.heightfield_scene(grid=48, spheres=48, seed=2)
    scene = Scene(data.triangles, data.fingerprint)
    got = _film(scene, data, w, h, 4)
    for variant in (4, 5):
        np.testing.assert_array_equal(_film(scene, data, w, h, 4, shade_variant=variant), got)


@pytest.mark.parametrize("spp", [1, 2, 5, 9])
def test_server_step_takes_further_samples(native, spp):
    from renderingengine_b200.serving import RenderServer
    data = scenes.cornell_box()
    w, h, depth = 67, 41, 5
    srv = RenderServer(8 << 30, 4 * w * h, max_depth=8, max_batch_views=16)
    srv.register_scene(1, data)
    rid = srv.submit(1, frame_constants(data.camera, w, h, 3, depth, seed=9), spp)
    srv.drain()
    assert srv.stats()["launches"] <= -(-spp // 4)  # the capacity holds four samples
    r = Renderer(w, h, 8)
    r.set_scene(Scene(data.triangles, 77, 1, N.BUILD_LBVH), data)
    for k in range(spp):
        r.render(frame_constants(data.camera, w, h, 3 + k, depth, seed=9), accumulate=k > 0)
    r.collect()
    np.testing.assert_array_equal(srv.result(rid).view(np.uint32), r.read(FILM_MEAN, w * h).view(np.uint32))


@pytest.mark.parametrize("w,h", [(1, 1), (31, 7), (33, 8), (32, 15), (65, 16), (5, 33), (30, 65)])
def test_atrous_row_blocks_match_oracle(native, oracle, w, h):
    """Rows a step apart share a block while eight steps fit the height: the
    five steps 1 to 16 cross that line at each of these heights."""
    native_cfg, py_cfg = _cfg_pair(atrous_iterations=5)
    gpu = SvgfReconstruction(w, h, 2, py_cfg)
    ora = oracle.OracleSvgf(w, h, 2, native_cfg)
    for gb, sig, fi, trig in S.sequence(w, h, 3, 11, hostile=False):
        _compare(gpu.process(gb, sig, fi, trig), ora.process(gb, sig, fi, trig), f"frame {fi}")


@pytest.mark.parametrize("w,h", [(1, 1), (31, 1), (33, 7), (64, 4), (257, 3)])
def test_export_to_any_word_address(native, w, h):
    """Records written a warp at a time to addresses that only words align."""
    import torch
    data = scenes.heightfield_scene(grid=48, spheres=48, seed=2)
    r = Renderer(w, h, 4)
    r.set_scene(Scene(data.triangles, data.fingerprint), data)
    fc = frame_constants(data.camera, w, h, 0, 4, seed=0x5151)
    r.render(fc, accumulate=False)
    r.collect()
    want = r.export_reconstruction(fc, fc)
    sizes = [w * h * N.GBUFFER_DTYPE.itemsize, w * h * N.SIGNAL_DTYPE.itemsize]
    out = [torch.full((s + 32,), 0xA5, dtype=torch.uint8, device="cuda") for s in sizes]
    r.export_reconstruction(fc, fc, gbuffer_ptr=out[0].data_ptr() + 4, signal_ptr=out[1].data_ptr() + 12)
    torch.cuda.synchronize()
    for buf, size, at, records in zip(out, sizes, (4, 12), want):
        got = buf.cpu().numpy()
        assert got[at:at + size].tobytes() == records.tobytes()
        assert np.all(got[:at] == 0xA5) and np.all(got[at + size:] == 0xA5)
