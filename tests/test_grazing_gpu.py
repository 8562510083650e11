"""Forms of the closest hit where the order of visits decides it
(grazing_cases.py): every form of a call agrees with the loop that it stands
for, bit for bit."""
import numpy as np
import pytest

import grazing_cases as G
from renderingengine_b200 import _native as N
from renderingengine_b200 import scenes
from renderingengine_b200.scenes import Camera
from renderingengine_b200.traversal import Scene
from renderingengine_b200.wavefront import (FILM_PRIMARY_IDENTITY, FILM_PRIMARY_POSITION, FILM_SAMPLE, Renderer,
                                            frame_constants)

pytestmark = pytest.mark.gpu


def _rays(o, d, tmax=1.0):
    r = np.zeros(len(o), N.RAY_DTYPE)
    r["origin_tmin"][:, :3], r["origin_tmin"][:, 3] = o, 1e-4
    r["direction_tmax"][:, :3], r["direction_tmax"][:, 3] = d, tmax
    return r


@pytest.mark.parametrize("build", [N.BUILD_FLATTENED_SAH, N.BUILD_LBVH], ids=["sah", "lbvh"])
@pytest.mark.parametrize("seed,side,clutter", [(1, 4, 70), (2, 6, 30), (3, 10, 6), (4, 10, 14)])
def test_grazing_batches_equal_child_pair_loop(native, build, seed, side, clutter):
    """Counted batches always walk the child pairs; the others take the form of
    their size, before and after a batch of 2^18 rays."""
    data, o, _, d = G.scene(seed, side, clutter)
    scene = Scene(data.triangles, 5, 1, build)
    one = _rays(o, d)
    many = np.resize(one, 1 << 18)
    for rays in (one, many, one):
        for any_hit in (False, True):
            want, _ = scene.trace(rays, any_hit=any_hit, counters=True)
            got = scene.trace(rays, any_hit=any_hit)
            assert (want["metadata"][:, 1] == N.HIT_KIND_TRIANGLE).mean() > 0.9
            differ = (got.view(np.uint32).reshape(len(rays), -1) != want.view(np.uint32).reshape(len(rays), -1)).any(1)
            assert not differ.any(), f"{differ[:len(one)].sum()} of {len(one)} rays, any-hit {any_hit}"


def _views(data, o, forward):
    x = np.array([1.0, 0.0, 0.0], np.float32)
    return [dict(frame=frame_constants(Camera(o[k], forward[k], x, x, 1e-30), 1, 1, 0, 4, seed=0x77 + k), offset=k,
                 key=k) for k in range(len(o))]


def _planes(scene, data, views, n, mode):
    r = Renderer(1280, 832, 4)
    r.set_scene(scene, data)
    r.set_tuning(traversal=mode)
    r.render_views(views)
    assert r.collect().fatal_mask == 0
    return [r.read_view(p, 0, n).view(np.uint32) for p in (FILM_PRIMARY_POSITION, FILM_PRIMARY_IDENTITY, FILM_SAMPLE)]


SCENES = [(1, 4, 70), (2, 6, 30), (5, 6, 6), (6, 6, 150), (7, 6, 2)]


@pytest.mark.parametrize("build", [N.BUILD_FLATTENED_SAH, N.BUILD_LBVH], ids=["sah", "lbvh"])
@pytest.mark.parametrize("seed,side,clutter", SCENES)
def test_grazing_short_queues_equal_long_ones(native, build, seed, side, clutter):
    """Views of one pixel, each looking along a cell's ray, alone (a ray per
    warp) and beside a view of a million pixels (32 rays per warp).  Mode 4 alone:
    with postponed leaves (mode 2) the rays of a warp decide the order of visits
    of one another."""
    data, o, forward, _ = G.scene(seed, side, clutter)
    scene = Scene(data.triangles, data.fingerprint, 1, build)
    n = len(o)
    views = _views(data, o, forward)
    big = dict(frame=frame_constants(data.camera, 1280, 800, 0, 4, seed=0x51), offset=n, key=n)
    alone, beside = _planes(scene, data, views, n, 4), _planes(scene, data, views + [big], n, 4)
    assert len(np.unique(beside[1][:, 1])) > 0.9 * n  # every view sees its own cell
    for a, b in zip(alone, beside):
        assert not (a != b).any(), f"{(a != b).any(1).sum()} of {n} views"


@pytest.mark.parametrize("mode", [2, 4])
@pytest.mark.parametrize("build", [N.BUILD_FLATTENED_SAH, N.BUILD_LBVH], ids=["sah", "lbvh"])
@pytest.mark.parametrize("seed,side,clutter", SCENES)
def test_grazing_warp_per_ray_equals_lane_per_ray(native, build, seed, side, clutter, mode):
    """A short queue gives each ray a warp, or one lane running the mode's loop
    where the scene has alpha-masked triangles: here one that no ray meets."""
    data, o, forward, _ = G.scene(seed, side, clutter)
    far = scenes.canonical_triangles(np.array([[[50, 0, 0], [50, 1, 0], [50, 0, 1]]], np.float32), None, np.zeros(1, np.uint32),
                                     np.full(1, len(data.triangles), np.uint32), np.zeros(1, np.uint32),
                                     first_traversal_id=len(data.triangles))
    data.triangles = np.concatenate([data.triangles, far])
    planes = []
    for masked in (False, True):
        data.triangles["metadata"][-1, 0] |= 2 * masked  # RE_GEOMETRY_FLAG_ALPHA_MASK
        scene = Scene(data.triangles, data.fingerprint, 1, build)
        planes.append(_planes(scene, data, _views(data, o, forward), len(o), mode))
    for a, b in zip(*planes):
        assert not (a != b).any(), f"{(a != b).any(1).sum()} of {len(o)} views"


@pytest.mark.parametrize("mode", [2, 4])
@pytest.mark.parametrize("shrink", [0.5, 0.8, 1.0])
def test_callers_leaf_boxes_smaller_than_their_triangles(native, shrink, mode):
    """A caller's tree whose leaf boxes lie within their parents' but do not hold
    their triangles: hits far before their boxes, warp against lane as above."""
    data = scenes.heightfield_scene(grid=48, spheres=48, seed=2)
    far = scenes.canonical_triangles(np.array([[[50, 0, 0], [50, 1, 0], [50, 0, 1]]], np.float32), None, np.zeros(1, np.uint32),
                                     np.full(1, 1 << 20, np.uint32), data.triangles["identity"][:1, 3],
                                     first_traversal_id=len(data.triangles))
    data.triangles = np.concatenate([data.triangles, far])
    nodes, order = Scene(data.triangles, data.fingerprint).export_flat()
    leaf = nodes["links"][:, 1] > 0
    centre = (nodes["bounds_min"][leaf] + nodes["bounds_max"][leaf]) / 2
    for b in ("bounds_min", "bounds_max"):
        nodes[b][leaf] = centre + (nodes[b][leaf] - centre) * np.float32(shrink)
    data.triangles = np.ascontiguousarray(data.triangles[order])
    at = int(np.argmax(data.triangles["positions"][:, 0, 0]))
    view = dict(frame=frame_constants(data.camera, 118, 80, 0, 4, seed=0x51), offset=0, key=0)
    planes = []
    for masked in (False, True):
        data.triangles["metadata"][at, 0] |= 2 * masked  # RE_GEOMETRY_FLAG_ALPHA_MASK
        scene = Scene(data.triangles, data.fingerprint, 1, N.BUILD_FLATTENED_SAH, nodes=nodes)
        planes.append(_planes(scene, data, [view], 118 * 80, mode))
    for a, b in zip(*planes):
        assert not (a != b).any(), f"{(a != b).any(1).sum()} of {118 * 80} pixels"
