"""Performance cases of the wavefront path tracer's public entry points.

Each case is one call, or one short sequence of calls, that a program using
this package makes: tracing ray batches, rendering frames (single views, ReSTIR
sequences, batches of views), rebuilding acceleration structures for moving
geometry, and reconstructing a noisy frame.  Sizes and options are those of the
package's benchmark workloads and tests (workloads.py, bench.py) together with
the small, odd and ragged ones that interactive tools and probes use.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs and handles a program holds before the call
    run(state)          one pass through the public entry points
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   the outputs in 64 bits, where they are plain arithmetic
"""
from __future__ import annotations

import math

import numpy as np
import torch

from renderingengine_b200 import _native as N
from renderingengine_b200 import autotune, scenes, workloads
from renderingengine_b200.svgf import (PLANE_ACCEPTED, PLANE_ATROUS, PLANE_HISTORY_LENGTH, PLANE_MOMENTS, PLANE_SVGF,
                                       PLANE_TEMPORAL, PLANE_VARIANCE, SvgfConfig, SvgfReconstruction)
from renderingengine_b200.traversal import Scene
from renderingengine_b200.wavefront import (ESTIMATOR_MIS, ESTIMATOR_RESTIR, FILM_DIRECT_DIFFUSE,
                                            FILM_INDIRECT_DIFFUSE, FILM_MEAN, FILM_PRIMARY_IDENTITY,
                                            FILM_PRIMARY_NORMAL, FILM_PRIMARY_POSITION, FILM_SAMPLE, Renderer,
                                            frame_constants)

TMAX = 16.0  # every scene fits the unit cube or the Cornell box; a finite tMax keeps miss records small


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # A tool's probe: a few hundred rays against a tiny scene (picking,
        # light-probe visibility).  Launch latency is all there is.
        dict(name="trace_probe", kind="trace", scene="cornell", size=0, build="sah", rays=500, camera=True, any=False,
             host=False),
        # The benchmark's trace workload: one 1080p frame of camera rays over
        # the 2,424,832-triangle heightfield, GPU LBVH.
        dict(name="trace_camera_1080p", kind="trace", scene="heightfield", size=1024, build="lbvh", rays=2_073_600,
             camera=True, any=False, host=False),
        # Occlusion queries of a baker: incoherent any-hit rays, an odd count,
        # over a flattened-SAH soup.
        dict(name="trace_any_soup", kind="trace", scene="soup", size=60_000, build="sah", rays=400_009, camera=False,
             any=True, host=False),
        # The convenience call on host arrays (Scene.trace): rays up, hits down.
        dict(name="trace_host", kind="trace", scene="heightfield", size=192, build="sah", rays=300_001, camera=False,
             any=False, host=True),
        # A thumbnail: small frame, small scene, four samples, default tuning.
        dict(name="frame_cornell_256", kind="frame", scene="cornell", size=0, build="sah", width=256, height=256,
             depth=8, spp=4, tuned=False, env=False),
        # The headline frame: 1920x1080, 1 spp, depth 8, GPU LBVH, the shipped
        # B200 tuning.
        dict(name="frame_heightfield_1080p", kind="frame", scene="heightfield", size=1024, build="lbvh", width=1920,
             height=1080, depth=8, spp=1, tuned=True, env=False),
        # A window of odd size, lit by an environment map, default tuning.
        dict(name="frame_env_odd", kind="frame", scene="heightfield", size=256, build="sah", width=801, height=449,
             depth=6, spp=1, tuned=False, env=True),
        # Interactive many-light frames: two ReSTIR DI frames of a sequence
        # (the second with temporal reuse) and the export to reconstruction.
        dict(name="restir_720p", kind="restir", size=512, lights=10_000, width=1280, height=720, depth=8),
        # Reconstruction of that sequence: two SVGF frames, five A-Trous
        # iterations, sigma_n 128 (the many-light configuration).
        dict(name="svgf_720p", kind="svgf", width=1280, height=720, iterations=5, phi_normal=128.0),
        # A service's launch: one sample of many views over four scenes.
        dict(name="views_batch", kind="views", views=16, size=256, lights=2_000, depth=6),
        # Moving geometry: a 600k-triangle scene rebuilt from device records,
        # then one 720p batch of camera rays traced against it.
        dict(name="scene_rebuild", kind="build", scene="heightfield", size=512, rays=921_600),
        # The allocation-free rebuild of a skinned mesh between a frame's
        # launches.
        dict(name="lbvh_static_50k", kind="lbvh", triangles=50_003),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "frame", "frame", "restir", "svgf", "views", "build", "lbvh"])
    if kind == "trace":
        scene = rng.choice(["cornell", "heightfield", "soup", "soup"])
        size = {"cornell": 0, "heightfield": _log(rng, 48, 512), "soup": _log(rng, 5_000, 300_000)}[scene]
        host = rng.random() < 0.2
        return dict(kind=kind, scene=scene, size=size, build=rng.choice(["sah", "lbvh"]),
                    rays=_log(rng, 200, 400_000 if host else 1_500_000), camera=rng.random() < 0.5,
                    any=rng.random() < 0.35, host=host)
    if kind == "frame":
        scene = rng.choice(["cornell", "heightfield", "heightfield", "soup"])
        size = {"cornell": 0, "heightfield": _log(rng, 48, 512), "soup": _log(rng, 5_000, 200_000)}[scene]
        w = _log(rng, 96, 1600)
        return dict(kind=kind, scene=scene, size=size, build=rng.choice(["sah", "lbvh"]), width=w,
                    height=max(64, int(w * rng.uniform(0.5, 0.8))), depth=rng.randint(3, 8),
                    spp=rng.choice([1, 1, 4]) if w < 600 else 1, tuned=rng.random() < 0.5,
                    env=scene == "heightfield" and rng.random() < 0.3)
    if kind == "restir":
        w = _log(rng, 160, 1280)
        return dict(kind=kind, size=_log(rng, 64, 384), lights=_log(rng, 100, 10_000), width=w,
                    height=max(90, int(w * rng.uniform(0.5, 0.65))), depth=rng.randint(3, 8))
    if kind == "svgf":
        w = _log(rng, 96, 1920)
        return dict(kind=kind, width=w, height=max(60, int(w * rng.uniform(0.5, 0.6))), iterations=rng.randint(3, 5),
                    phi_normal=rng.choice([64.0, 128.0]))
    if kind == "views":
        return dict(kind=kind, views=rng.randint(2, 20), size=_log(rng, 64, 384), lights=_log(rng, 100, 4_000),
                    depth=rng.randint(3, 6))
    if kind == "build":
        scene = rng.choice(["heightfield", "soup"])
        return dict(kind=kind, scene=scene,
                    size=_log(rng, 64, 512) if scene == "heightfield" else _log(rng, 10_000, 400_000),
                    rays=_log(rng, 5_000, 900_000))
    return dict(kind="lbvh", triangles=_log(rng, 300, 65_536))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _scene_data(kind: str, size: int, seed: int) -> scenes.SceneData:
    if kind == "cornell":
        return scenes.cornell_box()
    if kind == "soup":
        # Random triangles in the unit cube; edges shrink with the count.
        return scenes.triangle_soup(size, seed=seed, max_edge=min(0.2, 0.8 / size ** (1.0 / 3.0)))
    return scenes.heightfield_scene(grid=size, spheres=min(4096, max(8, size * size // 256)), seed=seed)


def _triangles(case) -> int:
    if case.get("scene", "heightfield") == "cornell":
        return 36
    if case.get("scene") == "soup":
        return case["size"]
    return 2 * case["size"] ** 2 + 80 * min(4096, max(8, case["size"] ** 2 // 256))


def _camera(data: scenes.SceneData, seed: int) -> scenes.Camera:
    scale = 0.05 if data.name.startswith("cornell") else 0.02
    return workloads.jittered_camera(data.camera, np.random.default_rng(seed), scale)


def _ray_records(case, data, seed: int) -> np.ndarray:
    n = case["rays"]
    if case.get("camera", True):
        w = max(1, int(round(math.sqrt(n * 16.0 / 9.0))))
        h = -(-n // w)
        rays = scenes.pinhole_rays(_camera(data, seed), w, h, seed=seed)[:n]
    elif data.name.startswith("cornell"):
        rays = scenes.random_rays((-0.9, -0.9, -2.9), (0.9, 0.9, -1.1), n, seed=seed)
    else:
        rays = scenes.random_rays((0, 0, 0), (1, 0.6, 1), n, seed=seed)
    rays[:, 7] = TMAX
    return scenes.to_ray_records(rays)


def _upload(records: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(records).view(np.uint8).reshape(-1)).cuda()


class _Buffer:
    """Device memory of a library object as an array a torch tensor can view;
    the tensor keeps the object alive."""

    def __init__(self, owner, ptr: int, shape: tuple, typestr: str):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 2}


def _view(owner, ptr: int, shape: tuple, typestr: str = "<f4") -> torch.Tensor:
    return torch.as_tensor(_Buffer(owner, ptr, shape, typestr), device="cuda")


def _film(r: Renderer, pixels: int, planes) -> list:
    """Film planes as (pixels, 4) tensors over the renderer's own memory:
    values of the float planes, words of the identity plane."""
    out = []
    for p in planes:
        if p == FILM_PRIMARY_IDENTITY:
            out.append(_view(r, r.film_pointer(p), (pixels, 4), "<i4"))
        elif p == FILM_PRIMARY_NORMAL:  # .w holds the material index as bits
            full = _view(r, r.film_pointer(p), (pixels, 4))
            out += [full[:, :3], full.view(torch.int32)[:, 3]]
        else:
            out.append(_view(r, r.film_pointer(p), (pixels, 4)))
    return out


FRAME_PLANES = (FILM_MEAN, FILM_SAMPLE, FILM_DIRECT_DIFFUSE, FILM_INDIRECT_DIFFUSE, FILM_PRIMARY_POSITION,
                FILM_PRIMARY_NORMAL, FILM_PRIMARY_IDENTITY)


def _hit_views(hits: torch.Tensor, n: int) -> list:
    words = hits.view(torch.int32).view(n, 24)
    return [words.view(torch.float32)[:, :12], words[:, 12:20]]


def prepare(case, seed):
    return {"trace": _prepare_trace, "frame": _prepare_frame, "restir": _prepare_restir, "svgf": _prepare_svgf,
            "views": _prepare_views, "build": _prepare_build, "lbvh": _prepare_lbvh}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _build_kind(case) -> int:
    return N.BUILD_LBVH if case["build"] == "lbvh" else N.BUILD_FLATTENED_SAH


# -- ray batches ------------------------------------------------------------
def _prepare_trace(case, seed):
    data = _scene_data(case["scene"], case["size"], seed)
    scene = Scene(data.triangles, data.fingerprint, build_kind=_build_kind(case))
    records = _ray_records(case, data, seed + 1)
    n = len(records)
    if case["host"]:
        return dict(run=_run_trace_host, scene=scene, rays=records, any=case["any"])
    rays = _upload(records)
    hits = torch.zeros(n * 96, dtype=torch.uint8, device="cuda")
    return dict(run=_run_trace, scene=scene, rays=rays, hits=hits, n=n, any=case["any"], out=_hit_views(hits, n))


def _run_trace(s):
    s["scene"].trace_device(s["rays"].data_ptr(), s["hits"].data_ptr(), s["n"], any_hit=s["any"])
    return s["out"]


def _run_trace_host(s):
    hits = s["scene"].trace(s["rays"], any_hit=s["any"])
    words = hits.view(np.int32).reshape(len(hits), 24)
    return [words.view(np.float32)[:, :12], words[:, 12:20]]


# -- frames -------------------------------------------------------------------
def _prepare_frame(case, seed):
    data = _scene_data(case["scene"], case["size"], seed)
    if case["env"]:
        data.lights = np.concatenate([data.lights, scenes.environment_light(light_id=1)])
        data.extra["environment"] = scenes.sky_environment(256, 128, seed=seed)
    scene = Scene(data.triangles, data.fingerprint, build_kind=_build_kind(case))
    w, h = case["width"], case["height"]
    r = Renderer(w, h, case["depth"])
    if case["tuned"]:
        autotune.apply(r, autotune.load("b200_frame_lbvh"))
    r.set_scene(scene, data)
    cam = _camera(data, seed + 1)
    frames = [frame_constants(cam, w, h, k, case["depth"], seed=seed, estimator=ESTIMATOR_MIS)
              for k in range(case["spp"])]
    return dict(run=_run_frame, scene=scene, renderer=r, frames=frames, out=_film(r, w * h, FRAME_PLANES))


def _run_frame(s):
    for k, f in enumerate(s["frames"]):
        s["renderer"].render(f, accumulate=k > 0)
    return s["out"]


# -- ReSTIR sequences -----------------------------------------------------------
def _prepare_restir(case, seed):
    data = scenes.add_emissive_triangles(_scene_data("heightfield", case["size"], seed), count=case["lights"],
                                         seed=seed + 7)
    scene = Scene(data.triangles, data.fingerprint, build_kind=N.BUILD_LBVH)
    w, h = case["width"], case["height"]
    r = Renderer(w, h, case["depth"])
    r.set_restir(**workloads.RESTIR_MANY_LIGHTS)
    r.set_scene(scene, data, light_selection=1)
    path = workloads.camera_path(_camera(data, seed + 1), 60, seed=seed)
    frames = [frame_constants(path[k], w, h, k, case["depth"], seed=seed, estimator=ESTIMATOR_RESTIR)
              for k in range(2)]
    gbuffer = torch.zeros(w * h, 16, dtype=torch.int32, device="cuda")
    signal = torch.zeros(w * h, 6, dtype=torch.float32, device="cuda")
    out = _film(r, w * h, (FILM_SAMPLE, FILM_INDIRECT_DIFFUSE, FILM_PRIMARY_POSITION, FILM_PRIMARY_IDENTITY))
    out += [gbuffer.view(torch.float32)[:, :13], gbuffer[:, 13:], signal]
    return dict(run=_run_restir, scene=scene, renderer=r, frames=frames, gbuffer=gbuffer, signal=signal, out=out)


def _run_restir(s):
    r = s["renderer"]
    r.restir_reset()
    previous = None
    for f in s["frames"]:
        r.render(f, accumulate=False)
        r.export_reconstruction(f, previous, gbuffer_ptr=s["gbuffer"].data_ptr(), signal_ptr=s["signal"].data_ptr())
        previous = f
    return s["out"]


# -- batches of views -------------------------------------------------------------
def _prepare_views(case, seed):
    field = _scene_data("heightfield", case["size"], seed)
    datas = [(scenes.cornell_box(), 0, False), (field, 0, False),
             (scenes.add_emissive_triangles(field, count=case["lights"], seed=seed + 7), 1, True),
             (_scene_data("soup", 4 * case["size"] ** 2 // 3, seed + 3), 0, False)]
    rng = np.random.default_rng(1000 + case["views"])  # resolutions belong to the case, cameras to the seed
    sizes = [((256, 256), (512, 512), (640, 360), (333, 217))[int(rng.integers(0, 4))] for _ in range(case["views"])]
    offsets = np.concatenate([[0], np.cumsum([w * h for w, h in sizes])])
    total = int(offsets[-1])
    # The path pool is sized as a width x height; any factors that cover it do.
    r = Renderer(1024, -(-total // 1024), case["depth"])
    r.set_restir(**workloads.RESTIR_MANY_LIGHTS)
    keep = []
    for k, (data, selection, _) in enumerate(datas):
        scene = Scene(data.triangles, data.fingerprint, build_kind=N.BUILD_LBVH)
        r.bind_scene(k, scene, data, light_selection=selection)
        keep.append(scene)
    views = []
    for v, (w, h) in enumerate(sizes):
        data, _, restir = datas[v % 4]
        f = frame_constants(_camera(data, seed + 10 + v), w, h, 0, case["depth"], seed=seed + v,
                            estimator=ESTIMATOR_RESTIR if restir else ESTIMATOR_MIS)
        views.append(dict(frame=f, slot=v % 4, offset=int(offsets[v]), accumulate=False, key=100 + v))
    return dict(run=_run_views, renderer=r, scenes=keep, views=views,
                out=_film(r, total, (FILM_SAMPLE, FILM_INDIRECT_DIFFUSE, FILM_PRIMARY_IDENTITY)))


def _run_views(s):
    s["renderer"].restir_reset()
    s["renderer"].render_views(s["views"])
    return s["out"]


# -- acceleration structures --------------------------------------------------------
def _prepare_build(case, seed):
    data = _scene_data(case["scene"], case["size"], seed)
    records = _upload(data.triangles)
    rays = _upload(_ray_records(case, data, seed + 1))
    n = case["rays"]
    hits = torch.zeros(n * 96, dtype=torch.uint8, device="cuda")
    return dict(run=_run_build, records=records, count=len(data.triangles), fingerprint=data.fingerprint, rays=rays,
                hits=hits, n=n, out=_hit_views(hits, n))


def _run_build(s):
    scene = Scene.from_device(s["records"].data_ptr(), s["count"], s["fingerprint"])
    scene.trace_device(s["rays"].data_ptr(), s["hits"].data_ptr(), s["n"])
    scene.close()
    return s["out"]


def _prepare_lbvh(case, seed):
    # A deforming sheet: triangle strips over a smooth displaced grid, IDs in
    # index order.
    n = case["triangles"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    side = int(math.ceil(math.sqrt(n / 2.0)))
    phase = torch.rand(6, generator=g, device="cuda") * 6.28

    def vertex(i, j):
        x, z = i / side, j / side
        y = 0.1 * torch.sin(9 * x + phase[0]) * torch.cos(7 * z + phase[1]) + 0.03 * torch.sin(31 * x + 23 * z + phase[2])
        x = x + 0.01 * torch.sin(40 * z + phase[3])
        return torch.stack([x, y, z, torch.ones_like(x)], -1)

    t = torch.arange(n, device="cuda")
    cell, odd = t // 2, (t % 2).float()
    i, j = (cell // side).float(), (cell % side).float()
    positions = torch.stack([vertex(i, j), vertex(i + odd, j + 1), vertex(i + 1, j + 1 - odd)], 1)
    positions = (positions.view(n, 12) + 1e-4 * torch.rand(n, 12, generator=g, device="cuda")).contiguous()
    ids = torch.arange(n, dtype=torch.int32, device="cuda")
    order = torch.zeros(n, dtype=torch.int32, device="cuda")
    nodes = torch.zeros(n - 1, 8, dtype=torch.int32, device="cuda")
    bounds = nodes.view(torch.float32)
    out = [order, bounds[:, 0:3], bounds[:, 4:7], nodes[:, 3], nodes[:, 7]]
    return dict(run=_run_lbvh, lib=N.load(), positions=positions, ids=ids, n=n, order=order, nodes=nodes, out=out)


def _run_lbvh(s):
    N.check(s["lib"].re_lbvh_build_static(s["positions"].data_ptr(), s["ids"].data_ptr(), s["n"],
                                          s["order"].data_ptr(), s["nodes"].data_ptr(), None))
    return s["out"]


# -- reconstruction ---------------------------------------------------------------
PAN = (1.37, -0.61)  # pixels the camera pans between the two frames


def _svgf_inputs(case, seed, frame: int):
    """A panning camera over a field of curved objects under an empty sky:
    guide planes and a one-sample noisy signal, as (pixels, 16) and (pixels,
    6) words."""
    w, h = case["width"], case["height"]
    rng = np.random.default_rng([seed, 77])
    centers = rng.random((40, 2)) * (w * 1.1, h) - (w * 0.05, -h * 0.1)
    dev = torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")
    y, x = torch.meshgrid(torch.arange(h, device=dev, dtype=torch.float64),
                          torch.arange(w, device=dev, dtype=torch.float64), indexing="ij")
    wx, wy = x + PAN[0] * frame, y + PAN[1] * frame
    c = torch.from_numpy(centers).to(dev)
    obj = torch.stack([(wx - cx) ** 2 + 2.0 * (wy - cy) ** 2 for cx, cy in c]).argmin(0)
    cx, cy = c[obj, 0], c[obj, 1]
    u, v = (wx - cx) / (0.3 * w), (wy - cy) / (0.3 * h)
    depth = 2.0 + 0.15 * obj + 0.4 * u * u + 0.3 * v * v + 0.2 * torch.sin(3 * u + 2 * v)
    normal = torch.stack([-0.8 * u, -0.6 * v, torch.ones_like(u)], -1)
    normal = normal / normal.norm(dim=-1, keepdim=True)
    tex = 0.5 + 0.5 * torch.sin(wx * 0.21) * torch.sin(wy * 0.17)
    tint = torch.from_numpy(rng.uniform(0.2, 0.9, (40, 3))).to(dev)[obj]
    dalb = tint * (0.3 + 0.6 * tex[..., None])
    salb = 0.04 + 0.5 * tint * (obj % 3 == 0)[..., None]
    surface = wy > 0.08 * h
    gb = torch.zeros(h, w, 16, dtype=torch.float32, device=dev)
    gb[..., 0] = depth
    gb[..., 1:4] = normal
    gb[..., 4:7] = dalb
    gb[..., 7:10] = salb
    gb[..., 10] = depth
    gb[..., 11] = PAN[0] / w
    gb[..., 12] = PAN[1] / h
    words = gb.view(torch.int32)
    words[..., 13] = (obj % 7).int()
    words[..., 14] = obj.int()
    words[..., 15] = torch.where(surface, N.GBUFFER_VALID | N.GBUFFER_MOTION_VALID, 0).int()
    gb[~surface] = 0.0
    g = torch.Generator(device=dev).manual_seed(seed * 2 + frame)
    light = (0.6 + 0.4 * torch.sin(2.1 * u) * torch.cos(1.7 * v))[..., None]
    noise = torch.rand(h, w, 6, generator=g, device=dev)
    fire = torch.where(torch.rand(h, w, 1, generator=g, device=dev) < 0.01, 12.0, 1.0)
    sig = torch.empty(h, w, 6, dtype=torch.float32, device=dev)
    sig[..., :3] = dalb * light * (2.0 * noise[..., :3]) * fire
    sig[..., 3:] = salb * light * (noise[..., 3:] ** 4 * 5.0) * fire
    sig[~surface] = 0.0
    return gb.view(h * w, 16), sig.view(h * w, 6)


def _svgf_config(case) -> SvgfConfig:
    return SvgfConfig(atrous_iterations=case["iterations"], phi_normal=case["phi_normal"])


def _prepare_svgf(case, seed):
    w, h = case["width"], case["height"]
    inputs = [_svgf_inputs(case, seed, f) for f in range(2)]
    svgf = SvgfReconstruction(w, h, 2, _svgf_config(case))
    out = [_view(svgf, svgf.plane_pointer(p), (w * h, 6)) for p in (PLANE_SVGF, PLANE_ATROUS, PLANE_TEMPORAL)]
    out += [_view(svgf, svgf.plane_pointer(PLANE_VARIANCE), (w * h,)), _view(svgf, svgf.plane_pointer(PLANE_MOMENTS), (w * h, 2)),
            _view(svgf, svgf.plane_pointer(PLANE_HISTORY_LENGTH), (w * h,), "<i4"),
            _view(svgf, svgf.plane_pointer(PLANE_ACCEPTED), (w * h,), "<i4")]
    return dict(run=_run_svgf, svgf=svgf, inputs=inputs, width=w, height=h, out=out)


def _run_svgf(s):
    for f, (gb, sig) in enumerate(s["inputs"]):
        s["svgf"].process_device(gb.data_ptr(), sig.data_ptr(), s["width"], s["height"], f, reset_trigger=f == 0)
    return s["out"]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "trace":
        n, t = case["rays"], _triangles(case)
        # Per ray: its record and hit record, and one root-to-leaf path of
        # box tests (two children a level, ~20 operations each) and a
        # triangle test; the scene's triangles once.
        return {"bytes": n * (64 + 96) + t * 64, "flops": n * (math.log2(t) * 40 + 60)}
    if kind == "frame":
        px = case["width"] * case["height"] * case["spp"]
        t = _triangles(case)
        # Film and primary-surface planes written, scene read; about three
        # path segments and two shadow rays a pixel, each a root-to-leaf path
        # and ~400 operations of shading.
        return {"bytes": px * 11 * 16 + t * 128, "flops": px * (5 * (math.log2(t) * 40 + 60) + 3 * 400)}
    if kind == "restir":
        px = 2 * case["width"] * case["height"]
        t = _triangles(case) + case["lights"]
        # As a frame, plus reservoirs and surfaces read and written, 32
        # candidates a pixel at ~300 operations, and the exported records.
        return {"bytes": px * (11 * 16 + 2 * 256 + 2 * 96 + 88) + t * 128,
                "flops": px * (5 * (math.log2(t) * 40 + 60) + 3 * 400 + 32 * 300)}
    if kind == "views":
        rng = np.random.default_rng(1000 + case["views"])
        sizes = [((256, 256), (512, 512), (640, 360), (333, 217))[int(rng.integers(0, 4))] for _ in range(case["views"])]
        px = sum(w * h for w, h in sizes)
        t = 2 * case["size"] ** 2
        return {"bytes": px * 11 * 16 + 4 * t * 128, "flops": px * (5 * (math.log2(t) * 40 + 60) + 3 * 400 + 8 * 300)}
    if kind == "svgf":
        px = 2 * case["width"] * case["height"]
        # Guide, signal and history records in; history, planes out; 25 taps
        # of two signals an iteration at ~40 operations, 49 in the bootstrap.
        return {"bytes": px * (88 + 64 + 64 + 4 * 24 + 24), "flops": px * (case["iterations"] * 25 * 40 + 49 * 20)}
    if kind == "build":
        t, n = _triangles(case), case["rays"]
        return {"bytes": t * (176 + 64 + 64 + 2 * 48 + 64) + n * 160, "flops": t * 200 + n * (math.log2(t) * 40 + 60)}
    return {"bytes": case["triangles"] * (48 + 4 + 4 + 32), "flops": case["triangles"] * 150}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "trace" and case["scene"] == "cornell" and not case["any"]:
        return _exact_trace(case, seed)
    if case["kind"] == "svgf":
        return _exact_svgf(case, seed)
    return None


def _exact_trace(case, seed):
    """Every ray against every triangle (Moller-Trumbore), nearest hit."""
    data = _scene_data(case["scene"], case["size"], seed)
    rays = _ray_records(case, data, seed + 1)
    tri = data.triangles["positions"][:, :, :3]
    p0 = tri[:, 0].astype(np.float64)
    e1, e2 = tri[:, 1].astype(np.float64) - p0, tri[:, 2].astype(np.float64) - p0
    out = np.zeros((len(rays), 12))
    for a in range(0, len(rays), 100_000):
        o = rays["origin_tmin"][a:a + 100_000, :3].astype(np.float64)
        d = rays["direction_tmax"][a:a + 100_000, :3].astype(np.float64)
        tmin = rays["origin_tmin"][a:a + 100_000, 3].astype(np.float64)
        best, which = np.full(len(o), TMAX), np.full(len(o), -1)
        bu, bv, front = np.zeros(len(o)), np.zeros(len(o)), np.zeros(len(o), bool)
        for k in range(len(p0)):
            p = np.cross(d, e2[k])
            det = p @ e1[k]
            with np.errstate(divide="ignore", invalid="ignore"):
                inv = 1.0 / det
                tv = o - p0[k]
                u = (tv * p).sum(1) * inv
                q = np.cross(tv, e1[k])
                v = (d * q).sum(1) * inv
                t = (q @ e2[k]) * inv
                ok = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > tmin) & (t < best)
            best, which = np.where(ok, t, best), np.where(ok, k, which)
            bu, bv, front = np.where(ok, u, bu), np.where(ok, v, bv), np.where(ok, det > 0, front)
        hit = which >= 0
        sign = np.where(front, 1.0, -1.0)[:, None]
        gn = np.cross(e1, e2)
        gn = (gn / np.linalg.norm(gn, axis=1, keepdims=True))[which] * sign
        nn = data.triangles["normals"][which][:, :, :3].astype(np.float64)
        sn = (1 - bu - bv)[:, None] * nn[:, 0] + bu[:, None] * nn[:, 1] + bv[:, None] * nn[:, 2]
        sn = sn / np.linalg.norm(sn, axis=1, keepdims=True) * sign
        rec = np.concatenate([o + d * best[:, None], best[:, None], gn, bu[:, None], sn, bv[:, None]], 1)
        rec[~hit] = 0.0
        rec[~hit, 3] = TMAX
        out[a:a + 100_000] = rec
    return [out, None]


def _shifted(t: torch.Tensor, dy: int, dx: int) -> torch.Tensor:
    """t at (y + dy, x + dx), zero outside the image."""
    h, w = t.shape[:2]
    out = torch.zeros_like(t)
    y0, y1 = max(0, -dy), min(h, h - dy)
    x0, x1 = max(0, -dx), min(w, w - dx)
    if y0 < y1 and x0 < x1:
        out[y0:y1, x0:x1] = t[y0 + dy:y1 + dy, x0 + dx:x1 + dx]
    return out


def _luma(sig: torch.Tensor) -> torch.Tensor:
    return ((sig[..., :3] + sig[..., 3:]) * torch.tensor([0.2126, 0.7152, 0.0722], dtype=sig.dtype,
                                                         device=sig.device)).sum(-1)


def _exact_svgf(case, seed):
    """The two frames in 64 bits: demodulation, temporal accumulation,
    variance bootstrap and the edge-avoiding A-Trous iterations."""
    w, h = case["width"], case["height"]
    c = _svgf_config(case)
    f32 = lambda v: float(np.float32(v))  # noqa: E731 -- the configuration is held in 32 bits
    hist = None
    for f in range(2):
        gb32, sig32 = _svgf_inputs(case, seed, f)
        ints = gb32.view(torch.int32).view(h, w, 16)
        gb, raw = gb32.double().view(h, w, 16), sig32.double().view(h, w, 6)
        ok = (ints[..., 15] & N.GBUFFER_VALID) != 0
        moving = (ints[..., 15] & N.GBUFFER_MOTION_VALID) != 0
        albedo = gb[..., 4:10].clamp(min=f32(c.minimum_albedo))
        demod = raw / albedo
        lum = _luma(demod)
        normal = gb[..., 1:4]
        norm = normal.norm(dim=-1, keepdim=True)
        filterable = ok & (norm[..., 0] > 1e-10)
        normal = torch.where(norm > 1e-20, normal / norm.clamp(min=1e-20),
                             torch.tensor([0.0, 0.0, 1.0], dtype=normal.dtype, device=normal.device))
        depth, epd = gb[..., 0], gb[..., 10]
        acc, m1, m2 = demod, lum, lum * lum
        hlen = torch.ones_like(lum)
        if hist is not None:
            hsig, hm1, hm2, hdepth, hnormal, hobj, hmat, hvalid, hhlen = hist
            y, x = torch.meshgrid(torch.arange(h, device=gb.device, dtype=torch.float64),
                                  torch.arange(w, device=gb.device, dtype=torch.float64), indexing="ij")
            u, v = (x + 0.5) / w + gb[..., 11], (y + 0.5) / h + gb[..., 12]
            live = filterable & moving & (epd >= 0) & (u >= 0) & (v >= 0) & (u < 1) & (v < 1)
            sx, sy = u * w - 0.5, v * h - 0.5
            bx, by = sx.floor(), sy.floor()
            fx, fy = sx - bx, sy - by

            def tap(px, py):
                inside = (px >= 0) & (py >= 0) & (px < w) & (py < h)
                ix, iy = px.clamp(0, w - 1).long(), py.clamp(0, h - 1).long()
                tol = f32(c.absolute_depth_threshold) + f32(c.relative_depth_threshold) * torch.maximum(
                    epd.abs(), hdepth[iy, ix].abs())
                good = (inside & hvalid[iy, ix] & ((epd - hdepth[iy, ix]).abs() <= tol)
                        & ((normal * hnormal[iy, ix]).sum(-1) >= f32(c.normal_cosine_threshold))
                        & (ints[..., 13] == hmat[iy, ix]) & (ints[..., 14] == hobj[iy, ix]))
                return good, ix, iy

            ws = torch.zeros_like(lum)
            s_sig, s1, s2, sl = torch.zeros_like(demod), ws.clone(), ws.clone(), ws.clone()
            for ty in range(2):
                for tx in range(2):
                    wt = (fx if tx else 1 - fx) * (fy if ty else 1 - fy)
                    good, ix, iy = tap(bx + tx, by + ty)
                    wt = torch.where(good & (wt > 0), wt, 0.0)
                    s_sig += hsig[iy, ix] * wt[..., None]
                    s1 += hm1[iy, ix] * wt
                    s2 += hm2[iy, ix] * wt
                    sl += hhlen[iy, ix] * wt
                    ws += wt
            bilinear = ws > 0
            d = ws.clamp(min=1e-30)
            s_sig, s1, s2, sl = s_sig / d[..., None], s1 / d, s2 / d, (sl / d + 0.5).floor()
            # The nearest valid tap of the 3 x 3 neighbourhood otherwise.
            nx, ny = (u * w).floor(), (v * h).floor()
            best = torch.full_like(lum, math.inf)
            for oy in (-1, 0, 1):
                for ox in (-1, 0, 1):
                    good, ix, iy = tap(nx + ox, ny + oy)
                    d2 = (nx + ox + 0.5 - u * w) ** 2 + (ny + oy + 0.5 - v * h) ** 2
                    take = good & ~bilinear & (d2 < best)
                    best = torch.where(take, d2, best)
                    s_sig = torch.where(take[..., None], hsig[iy, ix], s_sig)
                    s1, s2 = torch.where(take, hm1[iy, ix], s1), torch.where(take, hm2[iy, ix], s2)
                    sl = torch.where(take, hhlen[iy, ix], sl)
            accepted = live & (bilinear | torch.isfinite(best))
            hlen = torch.where(accepted, sl.clamp(max=c.max_history_length - 1) + 1, 1.0)
            ca = (1.0 / hlen).clamp(min=f32(c.minimum_color_alpha))
            ma = (1.0 / hlen).clamp(min=f32(c.minimum_moments_alpha))
            acc = torch.where(accepted[..., None], s_sig * (1 - ca[..., None]) + demod * ca[..., None], demod)
            m1 = torch.where(accepted, s1 * (1 - ma) + lum * ma, lum)
            m2 = torch.where(accepted, s2 * (1 - ma) + lum * lum * ma, lum * lum)
        tvar = (m2 - m1 * m1).clamp(min=0)
        hist = (acc, m1, m2, depth, normal, ints[..., 14], ints[..., 13], filterable, hlen)

    mat, obj = ints[..., 13] + 1, ints[..., 14] + 1  # zero marks a tap outside the image

    def guide(dy, dx, depth_den, phi):
        same = ((_shifted(mat, dy, dx) == mat) & (_shifted(obj, dy, dx) == obj)
                & _shifted(filterable, dy, dx) & filterable)
        dw = torch.exp(-(_shifted(depth, dy, dx) - depth).abs() / depth_den)
        nw = (normal * _shifted(normal, dy, dx)).sum(-1).clamp(0, 1) ** phi
        return torch.where(same, dw * nw, 0.0)

    def bootstrap(sig, length, variance):
        l = _luma(sig)
        ws, s1, s2 = torch.zeros_like(l), torch.zeros_like(l), torch.zeros_like(l)
        scale = (depth.abs() * f32(0.02)).clamp(min=f32(0.01))
        r = c.spatial_radius
        for dy in range(-r, r + 1):
            for dx in range(-r, r + 1):
                wt = guide(dy, dx, scale, 32.0)
                lt = _shifted(l, dy, dx)
                ws += wt
                s1 += lt * wt
                s2 += lt * lt * wt
        d = ws.clamp(min=1e-300)
        spatial = torch.where(ws > 0, (s2 / d - (s1 / d) ** 2).clamp(min=0), 0.0)
        blend = (length / c.short_history_length).clamp(0, 1)
        out = (spatial * (1 - blend) + variance * blend).clamp(min=f32(c.minimum_variance))
        return torch.where(filterable, out, f32(c.minimum_variance))

    kernel = (1.0, 4.0, 6.0, 4.0, 1.0)

    def atrous(sig, var):
        for it in range(c.atrous_iterations):
            step = 1 << it
            l = _luma(sig)
            den = (f32(c.phi_luminance) * var.sqrt()).clamp(min=f32(1e-4))
            scale = (f32(c.phi_depth) * (depth.abs() * f32(0.01)).clamp(min=f32(0.01)) * step).clamp(min=f32(1e-6))
            ws, wv, ss = torch.zeros_like(l), torch.zeros_like(l), torch.zeros_like(sig)
            for ky in range(-2, 3):
                for kx in range(-2, 3):
                    dy, dx = ky * step, kx * step
                    wt = guide(dy, dx, scale, f32(c.phi_normal)) * torch.exp(-(_shifted(l, dy, dx) - l).abs() / den)
                    wt = wt * (kernel[kx + 2] * kernel[ky + 2])
                    ss += _shifted(sig, dy, dx) * wt[..., None]
                    wv += _shifted(var, dy, dx) * wt * wt
                    ws += wt
            d = ws.clamp(min=1e-300)
            sig = torch.where((ws > 0)[..., None], ss / d[..., None], sig)
            var = torch.where(ws > 0, (wv / (d * d)).clamp(min=f32(c.minimum_variance)), var)
        return sig

    variance = bootstrap(acc, hlen, tvar)
    svgf = atrous(acc, variance) * albedo
    plain = atrous(demod, bootstrap(demod, torch.ones_like(lum), torch.zeros_like(lum))) * albedo
    flat = lambda t: t.reshape(h * w, -1).squeeze(-1)  # noqa: E731
    return [flat(svgf), flat(plain), flat(acc * albedo), flat(variance), torch.stack([flat(m1), flat(m2)], -1), None,
            None]
