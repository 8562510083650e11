"""The render server's byte budget against what its scenes hold."""
import numpy as np
import pytest

from renderingengine_b200 import _native as N
from renderingengine_b200 import scenes
from renderingengine_b200.serving import RenderServer
from renderingengine_b200.traversal import Scene
from renderingengine_b200.wavefront import frame_constants

pytestmark = pytest.mark.gpu


def _tables(sd):
    return (len(sd.triangles) * 4 + sd.materials.nbytes + len(sd.lights) * (sd.lights.itemsize + 24)
            + sd.fixture_triangles.nbytes)


def _fixed():
    probe = RenderServer(40 << 30, 40000, max_depth=8)
    fixed = probe.stats()["resident_bytes"]
    probe.close()
    return fixed


def _serve(budget, data):
    srv = RenderServer(budget, 40000, max_depth=8)
    ids = []
    for key, sd in enumerate(data):
        srv.register_scene(key, sd)
        ids.append(srv.submit(key, frame_constants(sd.camera, 32, 32, 0, 3), 1))
    srv.drain()
    return srv, [srv.poll(i) for i in ids]


def _lattice(bits):
    """2^sum(bits) small triangles on a lattice of powers of two: a perfectly
    balanced LBVH, whose four-wide nodes are as many as any tree's."""
    n = 1 << sum(bits)
    cells = np.stack(np.unravel_index(np.arange(n), [1 << b for b in bits]), -1)
    at = (cells + 0.25) / np.array([1 << b for b in bits])
    pos = (at[:, None] + np.array([[0, 0, 0], [1, 0, 0], [0, 1, 1]]) * (0.5 / (1 << max(bits)))).astype(np.float32)
    data = scenes.triangle_soup(n, seed=1)
    data.triangles = scenes.canonical_triangles(pos, None, np.zeros(n, np.uint32), np.arange(n, dtype=np.uint32),
                                                np.zeros(n, np.uint32))
    return data


def test_resident_bytes_are_the_scenes_own(native):
    data = [scenes.triangle_soup(40000, seed=4), scenes.heightfield_scene(grid=64, spheres=32, seed=9),
            scenes.cornell_box()]
    fixed = _fixed()
    srv, polls = _serve(40 << 30, data)
    assert all(s.state == N.REQUEST_DONE for s in polls)
    held = sum(Scene(sd.triangles, 77, 1, N.BUILD_LBVH).info().device_bytes + _tables(sd) for sd in data)
    assert srv.stats()["resident_bytes"] == fixed + held


def test_a_scene_above_its_charge_stays_within_the_budget(native):
    """260 bytes a triangle and 1 MiB are asked for before the build; such a
    tree's scene holds 285."""
    big, small = _lattice((6, 6, 5)), scenes.triangle_soup(20000, seed=3)
    n = len(big.triangles)
    held = Scene(big.triangles, 77, 1, N.BUILD_LBVH).info().device_bytes + _tables(big)
    charge = n * 256 + _tables(big) + (1 << 20)
    assert held > charge
    fixed = _fixed()
    srv, polls = _serve(fixed + charge, [big])
    assert polls[0].state == N.REQUEST_FAILED and polls[0].error == N.BUDGET_EXCEEDED
    assert srv.stats()["resident_bytes"] <= srv.stats()["budget_bytes"]
    srv.close()
    srv, polls = _serve(fixed + held + 100, [small, big, small, big])
    assert all(s.state == N.REQUEST_DONE for s in polls)
    st = srv.stats()
    assert st["resident_bytes"] <= st["budget_bytes"] and st["evictions"] > 0
