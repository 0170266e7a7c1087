"""The library's performance cases: what its users have it do, at the sizes they do it.

Eight kinds of work, each through the public Python entry points:

* query        closest hits of a batch of rays (GB300Scene.trace_closest): picking and visibility
               queries, from a thousand rays to millions
* progressive  an interactive viewer's step: one sample per pixel with the default (plain) renderer,
               then the RGBA8 image on the host
* plain        a few samples per pixel of a still frame on the plain renderer
* wave         a still frame on the wavefront renderer, the command line's default
* views        many views of one scene in one batch, each resolved to an image
* adjoint      one step of a material optimisation: forward frame, image loss, gradients
* tile         a 64K-path preview on the allocation-free entry point
* build        a new frame of an animated mesh: scene from host arrays with the GPU builder, then a
               batch of queries on it

Scenes and sizes are those of cudart_gb300.scenes and of bench.py.  A seed changes the rays, the
random numbers of a render, the optimisation target and, for `build`, the geometry's pose.
"""
import ctypes
import dataclasses
import functools
import math

import numpy as np
import torch

from cudart_gb300 import GB300Batch, GB300Renderer, GB300Scene, camera_from_json, load, make_options, scenes

FLT_MAX = float(np.finfo(np.float32).max)
TILE_PATHS = 65536          # CRT_NOALLOC_MAX_PATHS
VIEW_SIZES = [(256, 256), (512, 512), (768, 432), (1024, 1024)]


def listed():
    return [
        # the smallest call: a thousand rays into the 36-triangle box, launch and latency
        {"name": "query_small", "do": "query", "scene": "cornell", "detail": 0, "nodes": "q8", "rays": 1000},
        # a million scattered visibility queries, an odd count, default node encoding
        {"name": "query_mixed", "do": "query", "scene": "mixed", "detail": 5, "nodes": "q8", "rays": 1000003},
        # a large batch into the 2.17M-triangle scene, FP32 nodes
        {"name": "query_large", "do": "query", "scene": "large", "detail": 1024, "nodes": "f32", "rays": 8388608},
        # the viewer loop with every default: 512x512, one sample, image to the host
        {"name": "progressive_512", "do": "progressive", "scene": "cornell", "detail": 0, "nodes": "q8",
         "width": 512, "height": 512, "spp": 1, "depth": 6},
        # the drop-in renderer on the mixed scene at its own size
        {"name": "plain_mixed_720p", "do": "plain", "scene": "mixed", "detail": 5, "nodes": "f32",
         "width": 1280, "height": 720, "spp": 16, "depth": 8},
        # the Cornell box at its own size and samples: a short wavefront pass
        {"name": "wave_cornell_512", "do": "wave", "scene": "cornell", "detail": 0, "nodes": "f32",
         "width": 512, "height": 512, "spp": 16, "depth": 5},
        # an image whose sides divide by nothing, on the quantised nodes
        {"name": "wave_mixed_ragged", "do": "wave", "scene": "mixed", "detail": 5, "nodes": "q8",
         "width": 1001, "height": 563, "spp": 32, "depth": 8},
        # the headline frame: 1080p, 256 samples, 2.17M triangles
        {"name": "wave_large_1080p", "do": "wave", "scene": "large", "detail": 1024, "nodes": "f32",
         "width": 1920, "height": 1080, "spp": 256, "depth": 8},
        # sixteen of the batched-views workload's views at its lowest sample count
        {"name": "views_16", "do": "views", "scene": "mixed", "detail": 5, "nodes": "f32", "views": 16, "spp": 16,
         "depth": 8},
        # an iteration of the material inversion at its own size
        {"name": "adjoint_512", "do": "adjoint", "scene": "inversion", "detail": 32, "nodes": "q8",
         "width": 512, "height": 512, "spp": 64, "depth": 6},
        # the largest preview the allocation-free entry point takes
        {"name": "tile_64k", "do": "tile", "scene": "mixed", "detail": 5, "nodes": "f32",
         "width": 256, "height": 64, "spp": 4, "depth": 8},
        # a new 2.17M-triangle frame: upload, build, 100,000 queries
        {"name": "build_large", "do": "build", "scene": "large", "detail": 1024, "nodes": "f32", "rays": 100000},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["query", "progressive", "plain", "wave", "views", "adjoint", "tile", "build"])
    scene = rng.choice({"query": ["cornell", "mixed", "large"], "progressive": ["cornell", "mixed", "large"],
                        "plain": ["cornell", "mixed", "large"], "wave": ["cornell", "mixed", "large"],
                        "views": ["mixed"], "adjoint": ["inversion"], "tile": ["cornell", "mixed", "large"],
                        "build": ["mixed", "large"]}[kind])
    detail = {"cornell": 0, "mixed": rng.randint(2, 5), "large": _log_int(rng, 128, 1024),
              "inversion": rng.randint(8, 48)}[scene]
    case = {"do": kind, "scene": scene, "detail": detail, "nodes": rng.choice(["q8", "f32"])}
    if kind == "query":
        return {**case, "rays": _log_int(rng, 1000, 8000000)}
    if kind == "build":
        return {**case, "rays": _log_int(rng, 1000, 100000)}
    if kind == "views":
        return {**case, "views": rng.randint(2, 16), "spp": rng.choice([4, 8, 16]), "depth": rng.randint(4, 8)}
    if kind == "tile":
        width = _log_int(rng, 16, 256)
        height = _log_int(rng, 16, 64)
        return {**case, "width": width, "height": height, "spp": rng.randint(1, TILE_PATHS // (width * height)),
                "depth": rng.randint(2, 8)}
    limit = {"progressive": 1, "plain": 16, "wave": 64, "adjoint": 64}[kind]
    wide = {"progressive": 1280, "plain": 1280, "wave": 1920, "adjoint": 512}[kind]
    width = _log_int(rng, wide // 8, wide)
    height = max(48, int(width * rng.uniform(0.5, 1.0)))
    return {**case, "width": width, "height": height, "spp": _log_int(rng, 1, limit), "depth": rng.randint(3, 8)}


# ---------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=6)
def _arrays(scene, detail):
    """The scene's host arrays, as a loader hands them over."""
    if scene == "cornell":
        return scenes.cornell_box()
    if scene == "mixed":
        return scenes.mixed_mid(subdiv=detail)
    if scene == "large":
        return scenes.large_textured(grid=detail, tex_size=detail)
    return scenes.material_inversion(n_boxes=detail)


def _posed(sc, seed):
    """The mesh turned about the vertical axis by an angle of the seed's."""
    a = 2.0 * math.pi * np.random.default_rng(seed).random()
    rot = np.array([[math.cos(a), 0.0, math.sin(a)], [0.0, 1.0, 0.0], [-math.sin(a), 0.0, math.cos(a)]], np.float32)
    return dataclasses.replace(sc, positions=sc.positions @ rot.T, normals=sc.normals @ rot.T)


def _rays(sc, n, seed):
    """Half from the eye to points spread over the surface, half from such points into the hemisphere
    above them, shuffled: [n, 8] float32 on the GPU (origin, tmin, direction, tmax)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    p = torch.from_numpy(np.ascontiguousarray(sc.positions, np.float32)).cuda()
    face = torch.randint(0, sc.n_tris, (n,), generator=gen, device="cuda")
    if sc.n_tris > 1000:     # spread over space rather than over the many small faces of dense meshes
        some = torch.randint(0, sc.n_tris, (n,), generator=gen, device="cuda")
        area = lambda f: torch.linalg.norm(torch.linalg.cross(p[f, 1] - p[f, 0], p[f, 2] - p[f, 0]), dim=1)
        face = torch.where(area(some) > area(face), some, face)
    s, r = torch.rand(n, generator=gen, device="cuda").sqrt(), torch.rand(n, generator=gen, device="cuda")
    w = torch.stack([1 - s, s * (1 - r), s * r], 1)
    point = (w[:, :, None] * p[face]).sum(1)
    normal = torch.nn.functional.normalize(torch.linalg.cross(p[face, 1] - p[face, 0], p[face, 2] - p[face, 0]), dim=1)
    eye = torch.tensor(np.asarray(sc.camera.eye, np.float32), device="cuda")
    out = torch.randn(n, 3, generator=gen, device="cuda")
    out = torch.where((out * normal).sum(1, keepdim=True) < 0, -out, out)
    from_eye = torch.rand(n, 1, generator=gen, device="cuda") < 0.5
    rays = torch.empty(n, 8, device="cuda")
    rays[:, 0:3] = torch.where(from_eye, eye.expand(n, 3), point)
    rays[:, 3] = 1e-4
    rays[:, 4:7] = torch.nn.functional.normalize(torch.where(from_eye, point - eye, out), dim=1)
    rays[:, 7] = FLT_MAX
    return rays


def _views(sc, case, seed):
    """Views of the batched-views workload's hemisphere, in its four sizes."""
    rng = np.random.default_rng(seed)
    got = []
    for k in range(case["views"]):
        theta, phi = rng.uniform(0.05, 0.45 * math.pi), 2 * math.pi * k / case["views"] + rng.uniform(-0.05, 0.05)
        eye = 12 * np.array([math.cos(theta) * math.sin(phi), math.sin(theta), math.cos(theta) * math.cos(phi)])
        target = rng.uniform(-0.2, 0.2, 3)
        w, h = VIEW_SIZES[k % len(VIEW_SIZES)]
        got.append(scenes.View(scenes.CameraSpec(fov_deg=14.0, eye=tuple(eye), view_dir=tuple(target - eye)), w, h,
                               case["spp"]))
    return got


def prepare(case, seed):
    sc = _arrays(case["scene"], case["detail"])
    st = {"case": case, "do": case["do"]}
    if case["do"] == "build":
        st["arrays"] = _posed(sc, seed)
        st["rays"] = _rays(st["arrays"], case["rays"], seed)
        return st
    # trees of the large scene come from the GPU builder (a user with new geometry waits 20 times longer
    # for the host's), the others from the default one
    st["scene"] = GB300Scene(sc, node_format=case["nodes"], builder="gpu" if case["scene"] == "large" else "host")
    if case["do"] == "query":
        st["rays"] = _rays(sc, case["rays"], seed)
        return st
    if case["do"] == "views":
        st["batch"] = GB300Batch(st["scene"], _views(sc, case, seed), mode="wavefront", seed=seed,
                                 max_depth=case["depth"])
        return st
    w, h, spp = case["width"], case["height"], case["spp"]
    if case["do"] == "tile":
        st["camera"] = camera_from_json(sc.camera, w, h)
        st["options"] = make_options(max_depth=case["depth"], seed=seed, mode="wavefront")
        st["accum"] = torch.zeros(w * h, 4, device="cuda")
        return st
    mode = "megakernel" if case["do"] in ("progressive", "plain") else "wavefront"
    st["render"] = GB300Renderer(st["scene"], w, h, spp, max_depth=case["depth"], seed=seed, mode=mode)
    if case["do"] == "progressive":
        st["image"] = np.zeros((h, w, 4), np.uint8)
    if case["do"] == "adjoint":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        st["stream"] = torch.cuda.Stream()
        st["render"].set_stream(st["stream"].cuda_stream)
        st["target"] = torch.rand(w * h, 3, generator=gen, device="cuda")
        st["weights"] = torch.zeros(w * h, 4, device="cuda")
        n = len(sc.materials)
        st["kd"], st["ka"] = torch.zeros(n, 3, device="cuda"), torch.zeros(n, 3, device="cuda")
    return st


# ---------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------
def _accum(r):
    """The renderer's accumulator as a tensor, with the renderer kept for as long as its memory is looked at."""
    image = r.accum_tensor()
    image.renderer = r
    return image


def _run_adjoint(st):
    """Forward frame, gradient of the squared image error, adjoint on the samples after the frame's."""
    r, spp = st["render"], st["case"]["spp"]
    with torch.cuda.stream(st["stream"]):
        r.restart(0)
        r.render(spp)
        image = _accum(r)
        st["weights"][:, :3] = (image[:, :3] / spp - st["target"]) * (2.0 / (spp * image.shape[0]))
        st["kd"].zero_()
        st["ka"].zero_()
        r.adjoint(spp, spp, st["weights"].data_ptr(), st["kd"].data_ptr(), st["ka"].data_ptr())
    return {"image": image, "kd": st["kd"], "ka": st["ka"]}


def _run_tile(st):
    c = st["case"]
    st["accum"].zero_()
    status = load().crt_render_tile_noalloc(
        st["scene"].handle, ctypes.byref(st["camera"]), c["width"], c["height"], ctypes.byref(st["options"]), 0,
        c["width"] * c["height"], 0, c["spp"], st["accum"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if status:
        raise RuntimeError(load().crt_last_error().decode())
    return {"accum": st["accum"]}


def run(state):
    do = state["do"]
    if do in ("query", "build"):
        if do == "build":
            state["scene"] = GB300Scene(state["arrays"], node_format=state["case"]["nodes"], builder="gpu")
        face, t, uv = state["scene"].trace_closest(state["rays"])
        return {"face": face, "t": t, "uv": uv}
    if do == "views":
        batch = state["batch"]
        load().crt_render_restart(batch.handle, 0)
        batch.render()
        return [batch.resolve(k) for k in range(len(batch))]
    if do == "adjoint":
        return _run_adjoint(state)
    if do == "tile":
        return _run_tile(state)
    r = state["render"]
    r.restart(0)
    if do == "progressive":
        r.render_one_sample_per_pixel()
        return {"accum": _accum(r), "image": r.copy_image_bytes(state["image"])}
    r.render()
    return {"accum": _accum(r)}


# ---------------------------------------------------------------------------------------------------
# what a pass cannot do without, and what it should return
# ---------------------------------------------------------------------------------------------------
def _ray_flops(n_tris):
    """One path down a tree of eight-wide nodes (12 operations per child box) and one triangle test."""
    return 96.0 * max(1, math.ceil(math.log(n_tris, 8))) + 50.0


def work(case):
    n = {"cornell": 36, "mixed": 12 + 5 * 20 * 4 ** case["detail"], "inversion": 12 + 12 * case["detail"],
         "large": 2 * (case["detail"] - 1) ** 2 + 64 * 20 * 4 ** 3 + 8}[case["scene"]]
    depth = max(1, math.ceil(math.log(n, 8)))
    touched = lambda rays: min(48.0 * n, rays * (80.0 * depth + 48.0))     # of the scene, each record once
    if case["do"] in ("query", "build"):
        rays = case["rays"]
        bytes_, flops = rays * 48.0 + touched(rays), rays * _ray_flops(n)
        if case["do"] == "build":      # 25 floats in per triangle; its records and its share of the nodes out
            bytes_, flops = bytes_ + n * (100.0 + 128.0 + 25.0), flops + n * 200.0
        return {"bytes": bytes_, "flops": flops}
    if case["do"] == "views":
        pixels = sum(w * h for w, h in (VIEW_SIZES[k % len(VIEW_SIZES)] for k in range(case["views"])))
    else:
        pixels = case["width"] * case["height"]
    rays = 2.0 * pixels * case["spp"]           # a camera ray and a shadow ray of every sample, no bounce counted
    bytes_ = 16.0 * pixels + touched(rays)
    if case["do"] in ("progressive", "views"):
        bytes_ += 4.0 * pixels
    if case["do"] == "adjoint":                 # forward, and the adjoint's two traces
        rays, bytes_ = 3.0 * rays, bytes_ + 16.0 * pixels * 2
    return {"bytes": bytes_, "flops": rays * _ray_flops(n)}


def exact(case, seed):
    """Closest hits against every triangle in 64 bits, for the batches where that is quick.  The distance
    alone: coplanar faces of the boxes and the floor tie, and the tie decides the face and its barycentrics.
    A path's radiance has no such value (its random decisions follow from rounded numbers)."""
    sc = _arrays(case["scene"], case["detail"])
    if case["do"] != "query" or sc.n_tris * case["rays"] > 5e8 or sc.n_tris > 1000:
        return None
    rays = _rays(sc, case["rays"], seed).double()
    p = torch.from_numpy(np.ascontiguousarray(sc.positions, np.float32)).cuda().float()
    v, e1, e2 = p[:, 0].double(), (p[:, 1] - p[:, 0]).double(), (p[:, 2] - p[:, 0]).double()
    eps = float(np.float32(1e-5))
    got = []
    for part in rays.split(max(1, 2000000 // sc.n_tris)):
        o, tmin, d, tmax = part[:, None, 0:3], part[:, 3:4], part[:, None, 4:7], part[:, 7:8]
        pv = torch.linalg.cross(d.expand(-1, len(v), -1), e2.expand(len(part), -1, -1))
        det = (e1 * pv).sum(2)
        tv = o - v
        u = (tv * pv).sum(2) / det
        qv = torch.linalg.cross(tv, e1.expand(len(part), -1, -1))
        w = (d * qv).sum(2) / det
        t = (e2 * qv).sum(2) / det
        hit = (det.abs() >= eps) & (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (t > eps) & (t > tmin) & (t < tmax)
        got.append(torch.where(hit, t, torch.full_like(t, FLT_MAX)).min(1).values)
    return {"face": None, "t": torch.cat(got), "uv": None}
