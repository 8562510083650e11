"""Scene memory beside the caller's own work: captures of other streams, work
in flight, and what a scene reports to hold."""
import ctypes
import threading

import numpy as np
import pytest

from renderingengine_b200 import _native as N
from renderingengine_b200 import scenes
from renderingengine_b200.traversal import Scene

pytestmark = pytest.mark.gpu


def _scene(build=N.BUILD_LBVH, triangles=20_000):
    return Scene(scenes.triangle_soup(triangles, seed=9).triangles, 5, 1, build)


def _rays(count, seed=1):
    rng = np.random.default_rng(seed)
    r = np.zeros(count, N.RAY_DTYPE)
    d = rng.normal(size=(count, 3))
    r["origin_tmin"][:, :3], r["origin_tmin"][:, 3] = rng.random((count, 3)), 1e-4
    r["direction_tmax"][:, :3], r["direction_tmax"][:, 3] = d / np.linalg.norm(d, axis=1, keepdims=True), 1e30
    return r


def _beside_capture(mode, call):
    """`call` in another thread (mode thread_local) or this one (relaxed) while
    this thread captures; the capture must end and replay."""
    import torch
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    errors = []

    def run():
        try:
            torch.cuda.set_device(0)
            call()
        except Exception as e:  # reported by the caller's thread
            errors.append(e)

    with torch.cuda.graph(graph, capture_error_mode=mode):
        x.add_(1.0)
        if mode == "thread_local":
            t = threading.Thread(target=run)
            t.start()
            t.join()
        else:
            run()
    assert not errors, errors
    graph.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 1000.0


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
@pytest.mark.parametrize("build", [N.BUILD_LBVH, N.BUILD_FLATTENED_SAH], ids=["lbvh", "sah"])
def test_scene_destroyed_beside_a_capture(native, mode, build):
    scene = _scene(build)
    scene.trace(_rays(300_000), any_hit=True)
    _beside_capture(mode, scene.close)


def test_host_batch_that_grows_its_staging_beside_a_capture(native):
    scene = _scene()
    rays = _rays(5000)
    scene.trace(rays[:100])
    want, _ = scene.trace(rays, counters=True)
    fresh = _scene()
    fresh.trace(rays[:100])
    got = []
    _beside_capture("thread_local", lambda: got.append(fresh.trace(rays)))
    np.testing.assert_array_equal(got[0].view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("build", [N.BUILD_LBVH, N.BUILD_FLATTENED_SAH], ids=["lbvh", "sah"])
def test_scene_destroyed_with_work_in_flight(native, build):
    """Destroying waits for what may still read the scene, on any stream."""
    import torch
    scene = _scene(build)
    rays = _rays(50_000)
    want, _ = scene.trace(rays, counters=True)
    d_rays = torch.from_numpy(rays.view(np.uint8).reshape(-1)).cuda()
    d_hits = torch.zeros(len(rays) * N.HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    stream, done = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(20_000_000)  # about 10 ms
        scene.trace_device(d_rays.data_ptr(), d_hits.data_ptr(), len(rays), stream=stream.cuda_stream)
        done.record()
    scene.close()
    assert done.query()
    other = _scene(build, 30_000)  # takes the memory that was given back
    torch.cuda.synchronize()
    np.testing.assert_array_equal(d_hits.cpu().numpy().view(np.uint32), want.view(np.uint32).reshape(-1))
    other.close()


@pytest.mark.parametrize("any_hit", [False, True])
def test_device_bytes_count_the_quad_nodes(native, any_hit):
    triangles = 20_000
    scene = _scene(N.BUILD_LBVH, triangles)
    before = scene.info().device_bytes
    scene.trace(_rays(1 << 18), any_hit=any_hit)
    assert scene.info().device_bytes == before + 128 * (triangles - 1)  # one for each pair of children


def _device(rays):
    import torch
    return (torch.from_numpy(rays.view(np.uint8).reshape(-1)).cuda(),
            torch.zeros(len(rays) * N.HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda"))


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("busy", ["own", "default"])
def test_device_batches_do_not_wait(native, any_hit, busy):
    """A scene's first large batch, with its stream or the default stream busy,
    returns before either is done; the next one, on another stream, has the same
    hits."""
    import torch
    scene = _scene()
    rays = _rays(1 << 18)
    want, _ = scene.trace(rays, any_hit=any_hit, counters=True)
    scene.close()
    scene = _scene()
    batches = [_device(rays), _device(rays)]
    torch.cuda.synchronize()
    first, second, done = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(first if busy == "own" else torch.cuda.default_stream()):
        torch.cuda._sleep(400_000_000)  # about 200 ms
        done.record()
    for stream, (d_rays, d_hits) in zip((first, second), batches):
        second.wait_stream(first)  # a scene's batches share its work counter
        scene.trace_device(d_rays.data_ptr(), d_hits.data_ptr(), len(rays), any_hit, stream=stream.cuda_stream)
    assert not done.query()
    torch.cuda.synchronize()
    for _, d_hits in batches:
        np.testing.assert_array_equal(d_hits.cpu().numpy().view(np.uint32), want.view(np.uint32).reshape(-1))
    scene.close()


def _blocking_stream():
    """A stream that the legacy default stream waits for, unlike torch's."""
    import torch
    handle = ctypes.c_void_p()
    assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(handle))) == 0
    return torch.cuda.ExternalStream(handle.value)


@pytest.mark.parametrize("any_hit", [False, True])
def test_quad_nodes_made_beside_a_capture_of_a_blocking_stream(native, any_hit):
    """Beside such a capture the legacy default stream is closed.  The batch gets
    its quad nodes all the same, and the capture its end."""
    import torch
    scene = _scene()
    before = scene.info().device_bytes
    rays = _rays(1 << 18)
    want, _ = scene.trace(rays[:1000], any_hit=any_hit, counters=True)
    d_rays, d_hits = _device(rays)
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    own, blocking = torch.cuda.Stream(), _blocking_stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=blocking, capture_error_mode="relaxed"):
        x.add_(1.0)
        scene.trace_device(d_rays.data_ptr(), d_hits.data_ptr(), len(rays), any_hit, stream=own.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 1000.0
    assert scene.info().device_bytes > before
    got = d_hits.cpu().numpy().view(N.HIT_DTYPE)[:1000]
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_export_beside_a_capture(native, mode):
    """The first export of a tree that was built on the device."""
    import torch
    nodes, order = _scene().export_flat()
    scene = _scene()
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    graph, got = torch.cuda.CUDAGraph(), []
    with torch.cuda.graph(graph, stream=_blocking_stream(), capture_error_mode=mode):
        x.add_(1.0)
        t = threading.Thread(target=lambda: got.extend(scene.export_flat()))
        t.start()
        t.join()
    graph.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 1000.0
    assert got[0].tobytes() == nodes.tobytes()
    np.testing.assert_array_equal(got[1], order)


def test_export_keeps_the_current_device(native):
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("needs a second GPU to be current")
    scene = _scene()
    with torch.cuda.device(1):
        scene.export_flat()
        assert torch.cuda.current_device() == 1
