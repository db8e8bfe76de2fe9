"""The render path's performance cases: what a program that uses polyred_gb300 has it do.

A case is a dict of plain values. `kind` names the entry point:

  render    render.NewRenderer(...).Render(): one frame into host arrays, the whole Python call
  frame     pr_render of a resident scene into device outputs (a frame loop with a fixed scene)
  stream    pr_frame_submit: the scene uploaded anew from page-locked memory, the frame read back
  batch     Batch.render: several scenes and views as one job
  grad      diff.shade and its backward: radiance of a view and the gradients of all eight parameters
  depthmap  pr_depth_map_noalloc: triangles into a caller's depth map

`scene` names the content: `field` (a field of UV spheres, four materials, a point and a directional
light), `soup` (small random triangles), `ground` and `textured` (spheres on a plane that crosses the
near plane). Sizes are those of the repository's own workloads and tests, and odd ones between them.
"""
import ctypes as C
import math

import numpy as np
import torch

from polyred_gb300 import _abi, batch as pb, diff, native, procedural, render, scene as sc

F32 = np.float32
IMAGE = ("rgba", "tri_id", "depth")
GBUFFER = IMAGE + ("nor", "face_nor", "world_pos", "uvd", "vcol", "mat_id")
WORDS = {"rgba": 1, "tri_id": 1, "depth": 1, "nor": 4, "face_nor": 4, "world_pos": 4, "uvd": 4, "vcol": 1, "mat_id": 1}


def listed():
    frame = {"kind": "frame", "scene": "field", "spheres": 256, "lon": 63, "lat": 32, "width": 1920, "height": 1080,
             "msaa": 1, "shadow": 2048, "ao": True, "gbuffer": False}
    return [
        # the first program anyone writes: one sphere on a ground, Render() into host arrays
        {"name": "render_small", "kind": "render", "scene": "ground", "width": 800, "height": 500, "msaa": 1, "shadow": 0},
        # the same scene kept on the GPU: an interactive viewer's frame, where launches and latency count
        {"name": "frame_small", **frame, "scene": "ground", "spheres": 1, "lon": 64, "lat": 32, "width": 800,
         "height": 500, "shadow": 0, "ao": False},
        # a thumbnail of a small field with everything on, at a size no tile divides
        {"name": "frame_ragged", **frame, "spheres": 24, "lon": 37, "lat": 19, "width": 641, "height": 479, "shadow": 700},
        # image textures with and without mipmaps at full HD, shadow map of the frame's size
        {"name": "frame_textured", **frame, "scene": "textured", "spheres": 2, "lon": 64, "lat": 32, "shadow": -1,
         "ao": False},
        # the repository's headline workload
        {"name": "frame_field", **frame},
        # the same frame with the whole G-buffer kept, for a deferred pass of the caller's own
        {"name": "gbuffer_field", **frame, "gbuffer": True},
        # offline quality: MSAA 2, a 3840 x 2160 framebuffer
        {"name": "frame_msaa2", **frame, "msaa": 2},
        # the stress scene: ten million pixel-sized triangles at 4K, no shadows
        {"name": "frame_soup_4k", **frame, "scene": "soup", "spheres": 0, "lon": 0, "lat": 0, "tris": 10_000_000,
         "width": 3840, "height": 2160, "shadow": 0, "ao": False},
        # a host whose scene changes every frame: upload, frame and readback through page-locked memory
        {"name": "stream_field", **frame, "kind": "stream"},
        # dataset rendering: five scenes of 1k to 500k triangles, four views each, sixteen shadowed lights
        {"name": "batch_views", "kind": "batch", "scenes": 5, "views": 4, "lights": 16, "lo": 1_000, "hi": 500_000,
         "width": 1280, "height": 720, "shadow": 1024, "ao": True},
        # one view's step of an inverse-rendering loop
        {"name": "grad_field", "kind": "grad", "spheres": 256, "lon": 63, "lat": 32, "width": 1920, "height": 1080,
         "shadow": 2048},
        # a depth map for a caller that allocates nothing, at the entry point's largest sizes
        {"name": "depthmap_1k", "kind": "depthmap", "spheres": 16, "lon": 63, "lat": 33, "width": 1024, "height": 1024},
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    def size(lo, hi):
        w = log(lo, hi)
        return w, max(32, int(w * rng.uniform(0.45, 0.8)))

    kind = rng.choice(["frame", "frame", "frame", "frame", "render", "stream", "batch", "grad", "depthmap"])
    field = {"spheres": log(2, 256), "lon": log(8, 63), "lat": log(6, 32)}
    if kind == "render":
        w, h = size(160, 1280)
        return {"kind": kind, "scene": rng.choice(["ground", "textured"]), "width": w, "height": h,
                "msaa": rng.choice([1, 1, 2]), "shadow": rng.choice([0, -1])}
    if kind == "batch":
        w, h = size(160, 1280)
        lo = log(1_000, 20_000)
        return {"kind": kind, "scenes": rng.randint(1, 5), "views": rng.randint(1, 4), "lights": rng.randint(1, 16),
                "lo": lo, "hi": log(lo, 400_000), "width": w, "height": h, "shadow": log(200, 1024),
                "ao": rng.random() < 0.75}
    if kind == "grad":
        w, h = size(160, 1920)
        return {"kind": kind, **field, "width": w, "height": h, "shadow": log(256, 2048)}
    if kind == "depthmap":
        w, h = size(100, 1000)
        return {"kind": kind, "spheres": log(1, 16), "lon": log(6, 62), "lat": log(6, 32), "width": w, "height": h}
    w, h = size(96, 1920)
    scene = rng.choice(["field", "field", "field", "soup", "ground", "textured"]) if kind == "frame" else "field"
    c = {"kind": kind, "scene": scene, **field, "width": w, "height": h,
         "msaa": rng.choice([1, 1, 1, 2, 3]) if w <= 1000 else 1,
         "shadow": rng.choice([0, -1, log(256, 2048)]), "ao": rng.random() < 0.6,
         "gbuffer": kind == "frame" and rng.random() < 0.3}
    if scene == "soup":
        c.update(tris=log(2_000, 5_000_000), shadow=0, ao=False)
    return c


# ------------------------------------------------------------------ scenes

def _sphere(lon, lat):
    """A UV sphere's triangles: unit positions (n, 3, 3) wound outward, uv (n, 3, 2)."""
    th, ph = np.pi * np.arange(lat + 1) / lat, 2 * np.pi * np.arange(lon + 1) / lon
    P = np.stack([np.sin(th)[:, None] * np.cos(ph), np.cos(th)[:, None] * np.ones_like(ph),
                  -np.sin(th)[:, None] * np.sin(ph)], -1)
    P[0], P[lat] = (0, 1, 0), (0, -1, 0)
    uv = np.stack(np.broadcast_arrays(np.arange(lon + 1) / lon, (np.arange(lat + 1) / lat)[:, None]), -1)
    j, i = (v.reshape(-1) for v in np.meshgrid(np.arange(lat), np.arange(lon), indexing="ij"))
    a, b, c, d = (j * (lon + 1) + i + k for k in (0, 1, lon + 1, lon + 2))
    t = np.concatenate([np.stack([a, c, d], -1)[j < lat - 1], np.stack([a, d, b], -1)[(j > 0) & (j < lat - 1)],
                        np.stack([a, c, b], -1)[j == lat - 1]])
    P, uv = P.reshape(-1, 3), uv.reshape(-1, 2)
    p = P[t]
    flip = (np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]) * p.mean(1)).sum(-1) < 0
    t[flip] = t[flip][:, [0, 2, 1]]
    return P[t], uv[t]


def _field_numbers(case, seed):
    """Centres, radii, materials and the camera of a sphere field, as float32 values."""
    g = np.random.default_rng(seed)
    n = case["spheres"]
    return {"centre": g.uniform(-10, 10, (n, 3)).astype(F32), "radius": g.uniform(0.2, 1.5, n).astype(F32),
            "material": g.integers(0, 4, n), "eye": (np.array([0, 4, 24]) + g.uniform(-0.5, 0.5, 3)).astype(F32),
            "light": (np.array([14, 18, 12]) + g.uniform(-1, 1, 3)).astype(F32)}


def _mesh(case, mat_id=0, seed=0):
    p, uv = _sphere(case["lon"], case["lat"])
    n = len(p)
    pos, nor = np.ones((n, 3, 4), F32), np.zeros((n, 3, 4), F32)
    pos[..., :3], nor[..., :3] = p, p
    col = np.random.default_rng(seed).integers(40, 216, (n, 3, 4)).astype(np.uint8)
    col[..., 3] = 255
    return sc.Mesh(pos, nor, uv, col, np.full(n, mat_id, np.int32))


MATERIALS = [(0.8, 0.3, 0.2, 32, False), (0.2, 0.5, 0.8, 16, False), (0.3, 0.8, 0.3, 64, True), (0.9, 0.9, 0.9, 8, False)]


def _field(case, seed, ao, painted=0):
    """The sphere field; every painted-th sphere without a material (its vertex colours show)."""
    f = _field_numbers(case, seed)
    mats = [sc.BlinnPhong(diffuse=sc.color_from_value(r, g, b), specular=sc.color_from_value(0.5, 0.5, 0.5), shininess=s,
                          ambient_occlusion=ao, receive_shadow=True, flat_shading=flat) for r, g, b, s, flat in MATERIALS]
    mesh, paint = _mesh(case, 0, seed), _mesh(case, -1, seed)
    s = sc.Scene()
    for k in range(case["spheres"]):
        bare = painted and k % painted == 0
        o = sc.Geometry(paint) if bare else sc.Geometry(mesh, mats[f["material"][k]])
        r = f["radius"][k]
        s.add(o.scale(r, r, r).translate(*f["centre"][k]))
    s.add(sc.Point(position=f["light"], intensity=1.0, cast_shadow=True),
          sc.Directional(direction=(-1, -1, -0.5), intensity=0.6, cast_shadow=True), sc.Ambient(intensity=0.1))
    cam = sc.Perspective(position=f["eye"], target=(0, 0, 0), up=(0, 1, 0), fov=60, aspect=case["width"] / case["height"],
                         near=0.1, far=100)
    return s, cam


def _plane_scene(case, seed):
    """The repository's small or textured scene, seen from a seeded place."""
    make = procedural.small_scene if case["scene"] == "ground" else procedural.textured_scene
    s, cam = make(case["width"], case["height"])
    cam.position = (cam.position + np.random.default_rng(seed).uniform(-0.2, 0.2, 3)).astype(F32)
    return s, cam


def _soup_tensors(case, seed):
    """A soup of pixel-sized triangles on the GPU: centroids uniform on screen, view depth U[0.1, 100], areas
    log-normal about 1 px, 30% wound backwards, unprojected through a camera at the origin."""
    n, W, H = case["tris"], case["width"] * case["msaa"], case["height"] * case["msaa"]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def u(lo, hi, *shape):
        return torch.rand(*shape, generator=g, device="cuda") * (hi - lo) + lo

    depth, side = u(0.1, 100.0, n), torch.exp(torch.randn(n, generator=g, device="cuda") * 0.5) * (4 / math.sqrt(3)) ** 0.5
    ang = u(0, 2 * math.pi, n)[:, None] + torch.tensor([0, 2, 4], device="cuda") * (math.pi / 3)
    reach = u(0.6, 1.4, n, 3) * side[:, None] / math.sqrt(3)
    sx, sy = u(0, W, n)[:, None] + torch.cos(ang) * reach, u(0, H, n)[:, None] + torch.sin(ang) * reach
    flip = u(0, 1, n) < 0.3
    sx[flip], sy[flip] = sx[flip].flip(1), sy[flip].flip(1)
    t = math.tan(math.radians(60) / 2)
    pos = torch.ones(n, 3, 4, device="cuda")
    pos[..., 0] = (sx / W * 2 - 1) * (t * W / H) * depth[:, None]
    pos[..., 1] = (sy / H * 2 - 1) * t * depth[:, None]
    pos[..., 2] = -depth[:, None]
    nrm = torch.linalg.cross(pos[:, 1, :3] - pos[:, 0, :3], pos[:, 2, :3] - pos[:, 0, :3])
    nor = torch.zeros(n, 3, 4, device="cuda")
    nor[..., :3] = (nrm / (nrm.norm(dim=-1, keepdim=True) + 1e-30))[:, None]
    col = torch.randint(0, 256, (n, 3, 4), generator=g, device="cuda", dtype=torch.uint8)
    col[..., 3] = 255
    return pos, nor, torch.zeros(n, 3, 2, device="cuda"), col, torch.zeros(n, dtype=torch.int32, device="cuda")


def _shadow_size(case):
    if case["shadow"] < 0:
        return case["width"] * case["msaa"], case["height"] * case["msaa"]
    return (case["shadow"], case["shadow"]) if case["shadow"] else None


def _opts(case, scene, cam):
    return dict(width=case["width"], height=case["height"], camera=cam, scene=scene, perspective=True,
                shadow_map=case["shadow"] != 0, gamma=True, background=(0, 0, 0, 0), shadow_size=_shadow_size(case),
                directional_shadows=True, msaa=case["msaa"])


# ------------------------------------------------------------------ prepare and run

def _device_outputs(case, names):
    W, H, m = case["width"], case["height"], case["msaa"]
    od = _abi.pr_outputs()
    od.size, od.flags = C.sizeof(_abi.pr_outputs), _abi.PR_OUT_DEVICE_PTRS
    types = {np.uint8: torch.uint8, np.uint32: torch.int32, np.int32: torch.int32, np.float32: torch.float32}
    outs = {}
    for k in names:
        ch, dt = render.Outputs.FIELDS[k]
        h, w = (H, W) if k == "rgba" else (H * m, W * m)
        outs[k] = torch.empty((h, w, ch) if ch > 1 else (h, w), dtype=types[dt], device="cuda")
        setattr(od, k, outs[k].data_ptr())
    return outs, od


def _prepare_frame(case, seed):
    lib, dev = native.load(), render.Device(0)
    if case["scene"] == "soup":
        tensors = _soup_tensors(case, seed)
        s = sc.Scene(sc.Point(position=(0, 5, 5)), sc.Ambient(intensity=0.1))
        cam = sc.Perspective(position=(0, 0, 0), target=(0, 0, -1), up=(0, 1, 0), fov=60,
                             aspect=case["width"] / case["height"], near=0.1, far=120)
        mat = sc.BlinnPhong(diffuse=sc.color_from_value(0.8, 0.3, 0.2), specular=sc.color_from_value(0.5, 0.5, 0.5),
                            shininess=32)
        flat = render.FlatScene(sc.Scene(sc.Geometry(_mesh({"lon": 3, "lat": 2}), mat)))
        desc = flat.desc()
        desc.flags, desc.n_tris, flat.objects[0].n_tris = _abi.PR_SCENE_DEVICE_PTRS, case["tris"], case["tris"]
        desc.pos, desc.nor, desc.uv, desc.col, desc.mat_id = (t.data_ptr() for t in tensors)
    else:
        s, cam = _field(case, seed, case["ao"]) if case["scene"] == "field" else _plane_scene(case, seed)
        tensors, flat = None, render.FlatScene(s)
        desc = flat.desc()
    torch.cuda.synchronize()
    native.check(lib.pr_scene_upload(dev.handle, C.byref(desc)))
    opts = _opts(case, s, cam)
    fd = render.FrameDesc(opts, pb.shadow_cams(opts))
    outs, od = _device_outputs(case, GBUFFER if case["gbuffer"] else IMAGE)
    return {"kind": "frame", "lib": lib, "dev": dev, "fd": fd, "od": od, "outs": outs, "keep": (flat, tensors)}


def _prepare_stream(case, seed):
    lib, dev = native.load(), render.Device(0)
    s, cam = _field(case, seed, case["ao"])
    flat = render.FlatScene(s)
    for name in ("pos", "nor", "uv", "col", "mat_id"):
        a = getattr(flat, name)
        pinned = render.host_array(a.shape, a.dtype)
        pinned[...] = a
        setattr(flat, name, pinned)
    desc = flat.desc()
    opts = _opts(case, s, cam)
    fd = render.FrameDesc(opts, pb.shadow_cams(opts))
    out = render.Outputs(case["width"], case["height"], IMAGE, pinned=True, msaa=case["msaa"])
    # a synchronous frame sizes the context's buffers, as pr_frame_submit asks for
    native.check(lib.pr_scene_upload(dev.handle, C.byref(desc)))
    native.check(lib.pr_render(dev.handle, C.byref(fd.desc), C.byref(out.desc)))
    return {"kind": "stream", "lib": lib, "dev": dev, "fd": fd, "desc": desc, "out": out, "keep": flat}


def _prepare_render(case, seed):
    s, cam = _plane_scene(case, seed)
    opts = [render.Size(case["width"], case["height"]), render.Camera(cam), render.Scene(s), render.MSAA(case["msaa"]),
            render.GammaCorrection(True), render.ShadowMap(case["shadow"] != 0), render.CUDA(render.Device(0))]
    return {"kind": "render", "renderer": render.NewRenderer(*opts)}


def _prepare_batch(case, seed):
    b = pb.Batch(0)
    n, specs = case["scenes"], []
    for k in range(n):
        tris = case["lo"] * (case["hi"] / case["lo"]) ** (k / max(n - 1, 1))
        s = pb.sphere_scene(int(tris), seed * 64 + k, case["lights"], case["ao"])
        i = b.add_scene(s)
        for cam in pb.ring_cameras(case["views"], case["width"], case["height"]):
            o = pb.view_opts(s, cam, case["width"], case["height"], case["shadow"])
            specs.append((i, o, pb.shadow_cams(o)))
    arr, outs, keep = b.views(specs, IMAGE)
    return {"kind": "batch", "batch": b, "arr": arr, "outs": outs, "keep": keep}


def _prepare_grad(case, seed):
    s, cam = _field(case, seed, False, painted=8)
    r = diff.DiffRenderer(s, [diff.View(cam, case["width"], case["height"])], shadow_size=(case["shadow"],) * 2)
    p = {k: v.requires_grad_(True) for k, v in r.initial_params().items()}
    return {"kind": "grad", "renderer": r, "params": p, "g": _grad_image(case, seed)}


def _grad_image(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    return torch.randn(case["height"], case["width"], 4, generator=g, device="cuda") * 1e-3


def _ortho(case):
    """The depth map's camera as the descriptor takes it: looking down -z from (0, 0, 20), a box of +-12."""
    view, proj = np.eye(4), np.diag([1 / 12, 1 / 12, 0, 1.0])
    view[2, 3] = -20.0
    n, f = 0.0, -40.0
    proj[2, 2], proj[2, 3] = 2 / (n - f), (f + n) / (f - n)
    return view.astype(F32), proj.astype(F32)


def _prepare_depthmap(case, seed):
    f, mesh, n = _field_numbers(case, seed), _mesh(case), case["spheres"]
    objects = (_abi.pr_object * n)()
    for k in range(n):
        r, c = f["radius"][k], f["centre"][k]
        objects[k].first_tri, objects[k].n_tris = k * mesh.n_tris, mesh.n_tris
        objects[k].model[:] = [r, 0, 0, c[0], 0, r, 0, c[1], 0, 0, r, c[2], 0, 0, 0, 1]
    pos = torch.from_numpy(mesh.pos).cuda().repeat(n, 1, 1).contiguous()
    depth = torch.zeros(case["height"], case["width"], device="cuda")
    view, proj = _ortho(case)
    d = _abi.pr_depth_map_desc()
    d.size, d.n_tris, d.n_objects, d.width, d.height = C.sizeof(d), n * mesh.n_tris, n, case["width"], case["height"]
    d.pos, d.objects, d.depth = pos.data_ptr(), objects, depth.data_ptr()
    d.view[:], d.proj[:] = view.reshape(-1).tolist(), proj.reshape(-1).tolist()
    return {"kind": "depthmap", "lib": native.load(), "desc": d, "depth": depth, "keep": (pos, objects)}


def prepare(case, seed):
    return {"render": _prepare_render, "frame": _prepare_frame, "stream": _prepare_stream, "batch": _prepare_batch,
            "grad": _prepare_grad, "depthmap": _prepare_depthmap}[case["kind"]](case, seed)


def run(state):
    kind = state["kind"]
    if kind == "frame":
        native.check(state["lib"].pr_render(state["dev"].handle, C.byref(state["fd"].desc), C.byref(state["od"])))
        return state["outs"]
    if kind == "render":
        state["renderer"].Render()
        return state["renderer"].outputs()
    if kind == "stream":
        native.check(state["lib"].pr_frame_submit(state["dev"].handle, C.byref(state["desc"]), C.byref(state["fd"].desc),
                                                  C.byref(state["out"].desc)))
        return state["out"].arrays
    if kind == "batch":
        state["batch"].render(state["arr"])
        return state["outs"]
    if kind == "depthmap":
        native.check(state["lib"].pr_depth_map_noalloc(C.byref(state["desc"])))
        return state["depth"]
    p = state["params"]
    radiance = diff.shade(p, state["renderer"], 0)
    grads = torch.autograd.grad(radiance, [p[k] for k in diff.PARAM_NAMES], state["g"])
    return {"radiance": radiance, **dict(zip(diff.PARAM_NAMES, grads))}


# ------------------------------------------------------------------ work

def _tris(case):
    if case.get("scene") == "soup":
        return case["tris"]
    if case["kind"] == "render" or case.get("scene") in ("ground", "textured"):
        return 3970 if case["scene"] == "ground" else 4932
    return case["spheres"] * 2 * case["lon"] * (case["lat"] - 1)


def work(case):
    """Bytes: the scene's 136 B a triangle, each output and each shadow map once. Flops: about 200 a triangle and
    pass (transform, culls, edges), 100 a pixel and light (Blinn-Phong, shadow lookup), 4 an occlusion tap."""
    if case["kind"] == "batch":
        n = case["scenes"]
        tris = sum(case["lo"] * (case["hi"] / case["lo"]) ** (k / max(n - 1, 1)) for k in range(n))
        views, px = n * case["views"], case["width"] * case["height"]
        maps = views * case["lights"] * case["shadow"] ** 2
        return {"bytes": 136 * tris + 12 * px * views + 4 * maps,
                "flops": 200 * tris * case["views"] * (1 + case["lights"]) + px * views * 100 * case["lights"]
                + (0.3 * px * views * 8 * 98 * 4 if case["ao"] else 0)}
    tris, px = _tris(case), case["width"] * case["height"] * case.get("msaa", 1) ** 2
    if case["kind"] == "depthmap":
        return {"bytes": 48 * tris + 8 * px, "flops": 200 * tris}
    lights = 1 if case.get("scene") in ("ground", "soup", "textured") else 2
    maps = lights * case["shadow"] ** 2 if case["shadow"] > 0 else lights * px if case["shadow"] < 0 else 0
    if case["kind"] == "grad":
        return {"bytes": 136 * tris + 96 * 2 * tris + 4 * maps + 32 * px, "flops": 600 * tris + 400 * px * lights}
    words = sum(WORDS[k] for k in (GBUFFER if case.get("gbuffer") else IMAGE))
    return {"bytes": 136 * tris + 4 * words * px + 4 * maps,
            "flops": 200 * tris * (1 + (lights if case["shadow"] else 0)) + 100 * px * lights
            + (0.3 * px * 8 * 98 * 4 if case.get("ao") else 0)}


# ------------------------------------------------------------------ in 64 bits

def _t(a):
    return torch.as_tensor(np.asarray(a, np.float64), device="cuda")


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _look(eye, target):
    eye, target = _t(eye), _t(target)
    f = _unit(target - eye)
    x = _unit(torch.linalg.cross(f, _t([0, 1, 0])))
    y = _unit(torch.linalg.cross(x, f))
    m = torch.eye(4, dtype=torch.float64, device="cuda")
    m[:3, :3] = torch.stack([x, y, -f])
    m[:3, 3] = -(m[:3, :3] @ eye)
    return m


def _perspective(fov, aspect, n, f):
    t = math.tan(math.radians(fov) / 2)
    return _t([[-1 / (float(F32(aspect)) * t), 0, 0, 0], [0, -1 / t, 0, 0],
               [0, 0, (n + f) / (n - f), 2 * n * f / (n - f)], [0, 0, 1, 0]])


def _viewport(W, H):
    return _t([[W / 2, 0, 0, W / 2], [0, H / 2, 0, H / 2], [0, 0, 1, 0], [0, 0, 0, 1]])


def _bary(px, py, s):
    """Barycentric weights of points against screen triangles s (n, 3, >=2)."""
    x, y = s[..., 0], s[..., 1]
    area = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (y[:, 1] - y[:, 0]) * (x[:, 2] - x[:, 0])
    b0 = (x[:, 2] - x[:, 1]) * (py - y[:, 1]) - (y[:, 2] - y[:, 1]) * (px - x[:, 1])
    b1 = (px - x[:, 0]) * (y[:, 2] - y[:, 0]) - (py - y[:, 0]) * (x[:, 2] - x[:, 0])
    return torch.stack([b0 / area, b1 / area, 1 - b0 / area - b1 / area], -1)


def _raster(world, pv, W, H):
    """Depth (greatest wins) and winning triangle (-1: none) per pixel, rows bottom-up, and every triangle's screen
    vertices (x, y, z, clip w)."""
    dev = world.device
    scr = torch.empty(len(world), 3, 4, dtype=torch.float64, device=dev)
    vp = _viewport(W, H)
    for at in range(0, len(world), 1 << 21):
        clip = world[at: at + (1 << 21)] @ (vp @ pv).T
        scr[at: at + (1 << 21)] = torch.cat([clip[..., :3] / clip[..., 3:], clip[..., 3:]], -1)
    e1, e2 = scr[:, 1, :2] - scr[:, 0, :2], scr[:, 2, :2] - scr[:, 0, :2]
    lo, hi = scr[..., :2].amin(1), scr[..., :2].amax(1)
    x0, y0 = torch.ceil(lo[:, 0] - 0.5).clamp(min=0), torch.ceil(lo[:, 1] - 0.5).clamp(min=0)
    x1, y1 = torch.floor(hi[:, 0] - 0.5).clamp(max=W - 1), torch.floor(hi[:, 1] - 0.5).clamp(max=H - 1)
    front = (e1[:, 0] * e2[:, 1] - e1[:, 1] * e2[:, 0] > 0) & (x0 <= x1) & (y0 <= y1)
    del e1, e2, lo, hi
    ids = front.nonzero()[:, 0]
    x0, y0, bw = x0[ids].long(), y0[ids].long(), (x1 - x0 + 1)[ids].long()
    count = bw * (y1[ids].long() - y0 + 1)
    depth = torch.full((W * H,), -math.inf, dtype=torch.float64, device=dev)
    win = torch.full((W * H,), len(world), dtype=torch.int64, device=dev)
    ends = torch.cumsum(count, 0)
    total, start = int(ends[-1]) if len(ends) else 0, 0
    kept = []
    for upto in range(1 << 24, total + (1 << 24), 1 << 24):
        stop = int(torch.searchsorted(ends, min(upto, total), right=True))
        part = torch.arange(start, stop, device=dev)
        start = stop
        rep = torch.repeat_interleave(part, count[part])
        if not len(rep):
            continue
        k = torch.arange(len(rep), device=dev) - (ends[rep] - count[rep] - (ends[part[0]] - count[part[0]]))
        px, py = x0[rep] + k % bw[rep], y0[rep] + k // bw[rep]
        s = scr[ids[rep]]
        b = _bary(px + 0.5, py + 0.5, s)
        inside = (b >= -1e-7).all(-1)
        z, i, t = (b * s[..., 2]).sum(-1)[inside], (px + py * W)[inside], ids[rep][inside]
        depth.scatter_reduce_(0, i, z, "amax")
        kept.append((i, z, t))
    for i, z, t in kept:
        first = z == depth[i]
        win.scatter_reduce_(0, i[first], t[first], "amin")
    win[win == len(world)] = -1
    return depth.reshape(H, W), win.reshape(H, W), scr


def _field_world(case, seed):
    f = _field_numbers(case, seed)
    p, uv = _sphere(case["lon"], case["lat"])
    p, n = _t(p.astype(F32)), case["spheres"]
    world = torch.ones(n, len(p), 3, 4, dtype=torch.float64, device="cuda")
    world[..., :3] = p * _t(f["radius"])[:, None, None, None] + _t(f["centre"])[:, None, None]
    nor = p / _t(f["radius"])[:, None, None, None]
    return f, world.reshape(-1, 3, 4), nor.reshape(-1, 3, 3), _t(uv.astype(F32)).repeat(n, 1, 1)


def _camera(case, seed):
    if case.get("scene") == "soup":
        return _look((0, 0, 0), (0, 0, -1)), _perspective(60, case["width"] / case["height"], 0.1, 120)
    return (_look(_field_numbers(case, seed)["eye"], (0, 0, 0)),
            _perspective(60, case["width"] / case["height"], 0.1, 100))


def _up(a):
    """Rows bottom-up to the images' top-down."""
    return a.flip(0).contiguous()


def _winners(case, seed, world, W, H):
    view, proj = _camera(case, seed)
    depth, win, scr = _raster(world, proj @ view, W, H)
    y, x = (win >= 0).nonzero(as_tuple=True)
    t = win[y, x]
    back = torch.linalg.inv(view) @ torch.linalg.inv(proj) @ torch.linalg.inv(_viewport(W, H))
    b = _bary(x + 0.5, y + 0.5, scr[t])
    flat = scr[t].clone()
    flat[..., 3] = 1.0
    m = (flat @ back.T)[..., :3]  # the vertices' screen positions unprojected, not divided by w
    return {"depth": depth, "win": win, "x": x, "y": y, "t": t, "b": b, "scr": scr[t], "m": m, "back": back,
            "z": depth[y, x]}


def _exact_frame(case, seed):
    if case["scene"] not in ("field", "soup"):
        return None  # the ground crosses the near plane: what the clipper makes of it is the reference's own rule
    W, H = case["width"] * case["msaa"], case["height"] * case["msaa"]
    if case["scene"] == "soup":
        pos, nor, uv, _, _ = _soup_tensors(case, seed)
        world, nor, uv = pos.double(), nor[..., :3].double(), uv.double()
        del pos
    else:
        _, world, nor, uv = _field_world(case, seed)
    w = _winners(case, seed, world, W, H)
    out = dict.fromkeys(GBUFFER if case.get("gbuffer") else IMAGE)
    out["depth"] = _up(torch.where(w["win"] >= 0, w["depth"], 0.0))
    if not case.get("gbuffer"):
        return out
    t, b, x, y = w["t"], w["b"], w["x"], w["y"]

    def put(v, last):
        a = torch.zeros(H, W, 4, dtype=torch.float64, device="cuda")
        a[y, x] = torch.cat([v, torch.full((len(v), 1), last, dtype=torch.float64, device="cuda")], -1) if last is not None else v
        return _up(a)

    out["nor"] = put(_unit((b[..., None] * nor[t]).sum(1)), 0.0)
    out["face_nor"] = put(_unit(torch.linalg.cross(w["m"][:, 1] - w["m"][:, 0], w["m"][:, 2] - w["m"][:, 0])), 0.0)
    out["world_pos"] = put((b[..., None] * w["m"]).sum(1), 1.0)

    def at(dx, dy):
        q = _bary(x + 0.5 + dx, y + 0.5 + dy, w["scr"]) / -w["scr"][..., 3]
        return (q[..., None] * uv[t]).sum(1) / q.sum(-1, keepdim=True)

    c = at(0, 0)
    out["uvd"] = put(torch.cat([c, ((at(1, 0) - c) ** 2).sum(-1, keepdim=True), ((at(0, 1) - c) ** 2).sum(-1, keepdim=True)], -1), None)
    return out


def _shadow_camera(eye, centre, view, proj):
    """The orthographic light camera fitted about the main camera's frustum."""
    lv = _look(eye, centre)
    corner = _t([[a, b, c, 1] for a in (1, -1) for b in (1, -1) for c in (1, -1)])
    v = corner @ (lv @ torch.linalg.inv(view) @ torch.linalg.inv(proj)).T
    v = v[:, :3] / v[:, 3:]
    (l, b, n0), (r, t, f0) = v.amin(0).tolist(), v.amax(0).tolist()
    n, f = f0, n0 - 2
    return lv, _t([[2 / (r - l), 0, 0, (l + r) / (l - r)], [0, 2 / (t - b), 0, (b + t) / (b - t)],
                   [0, 0, 2 / (n - f), (f + n) / (f - n)], [0, 0, 0, 1]])


def _exact_grad(case, seed):
    W, H, S = case["width"], case["height"], case["shadow"]
    f, world, nor, _ = _field_world(case, seed)
    w = _winners(case, seed, world, W, H)
    per = len(world) // case["spheres"]
    t, b = w["t"], w["b"]
    ball = t // per
    painted, kind = ball % 8 == 0, torch.as_tensor(f["material"], device="cuda")[ball]
    # shadows: each light's map, then 0.5 for every light that does not reach the pixel
    view, proj = _camera(case, seed)
    way = np.array([-1, -1, -0.5]) / np.linalg.norm([-1, -1, -0.5])
    centre = (np.minimum(-1, f["light"].astype(np.float64)) + np.maximum(1, f["light"].astype(np.float64))) / 2
    screen = torch.stack([w["x"].double(), w["y"].double(), w["z"], torch.ones_like(w["z"])], -1) @ w["back"].T
    hidden = torch.zeros(len(t), dtype=torch.float64, device="cuda")
    for eye in (f["light"], centre - way):
        lv, lp = _shadow_camera(eye, centre, view, proj)
        shadow = _raster(world, lp @ lv, S, S)[0].clamp(min=0).reshape(-1)
        q = screen @ (_viewport(S, S) @ lp @ lv).T
        q = q[:, :3] / q[:, 3:]
        i = q[:, 0].trunc().long() + q[:, 1].trunc().long() * S
        ok = (i > 0) & (i < S * S)
        hidden += (ok & (q[:, 2] < shadow[i.clamp(0, S * S - 1)] - 0.03)).double()
    fac = 0.5 ** hidden
    # the radiance as a function of the parameters
    mats = [MATERIALS[m] for k, m in enumerate(f["material"]) if k % 8]  # one entry a sphere that has a material
    slot = torch.as_tensor(np.cumsum(np.arange(case["spheres"]) % 8 != 0) - 1, device="cuda")[ball]
    half = math.floor(0.5 * 255 + 0.5) / 255
    col = np.random.default_rng(seed).integers(40, 216, (per, 3, 4)).astype(np.uint8)
    col[..., 3] = 255
    n_m = max(len(mats), 0)
    kd = _t([[math.floor(v * 255 + 0.5) / 255 for v in m[:3]] for m in mats]).reshape(-1, 3)
    p = {"vertex_color": _t(col / 255.0).repeat(case["spheres"], 1, 1), "vertex_normal": None, "kd": kd,
         "ks": torch.full((n_m, 3), half, dtype=torch.float64, device="cuda"), "shininess": _t([m[3] for m in mats]),
         "light_pos": _t(np.stack([f["light"], np.zeros(3)])), "light_intensity": _t([1.0, float(F32(0.6))]),
         "ambient": _t([float(F32(0.1))])}
    p["vertex_normal"] = torch.zeros_like(p["vertex_color"])
    p["vertex_normal"][..., :3] = _t(_sphere(case["lon"], case["lat"])[0].astype(F32)).repeat(case["spheres"], 1, 1)
    p = {k: v.requires_grad_(True) for k, v in p.items()}
    radiance = torch.zeros(H, W, 4, dtype=torch.float64, device="cuda")
    radiance[..., 3] = 255.0
    g = _up(_grad_image(case, seed).double())[w["y"], w["x"], :3]
    loss = torch.zeros((), dtype=torch.float64, device="cuda")
    bare, lit = painted.nonzero()[:, 0], (~painted).nonzero()[:, 0]
    if len(bare):
        q = b[bare] / -w["scr"][bare][..., 3]
        R = 255 * ((q / q.sum(-1, keepdim=True))[..., None] * p["vertex_color"][t[bare]][..., :3]).sum(1)
        radiance[w["y"][bare], w["x"][bare], :3] = R.detach()
        loss = loss + (R * g[bare]).sum()
    if len(lit):
        x = (b[lit][..., None] * w["m"][lit]).sum(1)
        k = slot[lit]
        scale = _t(f["radius"])[ball[lit]][:, None, None]
        n = _unit((b[lit][..., None] * (p["vertex_normal"][t[lit]][..., :3] / scale)).sum(1))
        fn = _unit(torch.linalg.cross(w["m"][lit][:, 1] - w["m"][lit][:, 0], w["m"][lit][:, 2] - w["m"][lit][:, 0]))
        n = torch.where((kind[lit] == 2)[:, None], fn, n)
        V = _unit(_t(f["eye"]) - x)
        diffuse, specular = 0.0, 0.0
        for i in range(2):
            if i == 0:
                D = p["light_pos"][0] - x
                far = D.norm(dim=-1, keepdim=True)
                L, I = D / far, p["light_intensity"][0] / far
            else:
                L, I = -_t(way).expand_as(x), p["light_intensity"][1].expand(len(x), 1)
            Hv = _unit(L + V)
            nh = (n * Hv).sum(-1, keepdim=True).clamp(0, 1)
            power = torch.where(nh > 0, nh.clamp(min=1e-300) ** p["shininess"][k][:, None], 0.0)
            diffuse = diffuse + (n * L).sum(-1, keepdim=True).clamp(0, 1) * 255.0 * I
            specular = specular + power * 255.0 * I
        R = fac[lit][:, None] * (p["ambient"][0] * 255.0 + p["kd"][k] * diffuse + p["ks"][k] * specular).clamp(0, 255)
        radiance[w["y"][lit], w["x"][lit], :3] = R.detach()
        loss = loss + (R * g[lit]).sum()
    grads = torch.autograd.grad(loss, list(p.values()), allow_unused=True, materialize_grads=True) if loss.requires_grad \
        else [torch.zeros_like(v) for v in p.values()]
    return {"radiance": _up(radiance), **dict(zip(p, grads))}


def _exact_depthmap(case, seed):
    _, world, _, _ = _field_world(case, seed)
    view, proj = (_t(m) for m in _ortho(case))
    return _raster(world, proj @ view, case["width"], case["height"])[0].clamp(min=0)


def exact(case, seed):
    if case["kind"] in ("frame", "stream") and case["scene"] in ("field", "soup"):
        return _exact_frame(case, seed)
    if case["kind"] == "grad":
        return _exact_grad(case, seed)
    if case["kind"] == "depthmap":
        return _exact_depthmap(case, seed)
    return None  # cameras inside the scene, or a ground through the near plane
