"""The work this renderer is asked to do, as cases that can be timed and compared.

A case is one pass through the public entry points:

  frame   Renderer.SetTransform + RenderMesh of a mesh that is resident on the
          GPU, colour, depth and triangle id left there: what an application
          does once per displayed image;
  viewer  the same on a mesh in page-locked host memory, and GetBackBuffer:
          what the reference's viewer does (RealtimeViewer/Main.cpp:71-95);
  batch   RenderBatched of many meshes and cameras prepared once
          (PrepareBatch): image generation for learning systems;
  step    one gradient step of the differentiable form: RenderBatched for the
          visibility, edxr_shade_visible for the colour, edxr_backward for the
          gradients of an L2 image loss.

Every renderer runs with its default launch tunables: an application that
never calls the autotuner.  Scenes come from edxraster_gb300/scenes.py, sizes
from the benchmark's workloads and the tests.
"""
import ctypes
import math

import numpy as np
import torch

from edxraster_gb300 import _lib, scenes
from edxraster_gb300 import renderer as R

NO_TRIANGLE = 0xFFFFFFFF


def listed():
    def frame(name, scene, size, width, height, shader=R.PS_BLINN_PHONG, depth=R.DEPTH_LESS, msaa=0):
        return {"name": name, "kind": "frame", "scene": scene, "size": size, "width": width, "height": height,
                "shader": shader, "depth": depth, "msaa": msaa}

    return [
        # a thumbnail or a preview pane: launch and host latency
        frame("sphere_320x180", "sphere", 32, 320, 180),
        # the smallest of the benchmark's workloads: one object, mostly background
        frame("sphere_720p", "sphere", 32, 1280, 720),
        # a mid-sized scene in a window of no round size, the reference's depth function
        frame("terrain_1366x769", "terrain", 301, 1366, 769, R.PS_LAMBERTIAN_ALBEDO, R.DEPTH_LEQUAL),
        # the headline workload: 2,097,152 triangles at 1920x1080
        frame("terrain_1080p", "terrain", 1024, 1920, 1080),
        # binning stress: a million independent triangles of very uneven size at 3840x2160, deep overdraw
        frame("stress_4k", "stress", 1_000_000, 3840, 2160),
        # the reference's default pixel shader: textured albedo, trilinear, three texture slots
        frame("textured_720p", "terrain", 256, 1280, 720, R.PS_LAMBERTIAN_TEXTURED, R.DEPTH_LEQUAL),
        # the reference's Blinn-Phong shader as written (ks 3, exponent 200), shaded in FP64
        frame("reference_shader_720p", "terrain", 256, 1280, 720, R.PS_BLINN_PHONG_REFERENCE, R.DEPTH_LEQUAL),
        # anti-aliased frames: the headline workload with 4 samples, one object with 8
        frame("terrain_1080p_4x", "terrain", 1024, 1920, 1080, msaa=2),
        frame("sphere_720p_8x", "sphere", 32, 1280, 720, msaa=3),
        # the viewer's loop on the headline mesh: positions and indices uploaded, RGBA8 read back, every frame
        {"name": "viewer_terrain_1080p", "kind": "viewer", "scene": "terrain", "size": 1024, "width": 1920,
         "height": 1080, "shader": R.PS_BLINN_PHONG, "depth": R.DEPTH_LESS, "msaa": 0},
        # many meshes of uneven size (500 to 200,000 triangles), four cameras each, in one pass
        {"name": "batch_256_views", "kind": "batch", "meshes": 64, "views": 4, "most": 200_000, "width": 512,
         "height": 512},
        # the differentiable configuration: a torus of 50,000 triangles in 64 views
        {"name": "step_64_views", "kind": "step", "size": 250, "views": 64, "width": 256, "height": 256},
    ]


def draw(rng):
    def log_uniform(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame"] * 5 + ["viewer", "batch", "batch", "step", "step"])
    if kind == "batch":
        side = log_uniform(64, 512)
        return {"kind": kind, "meshes": log_uniform(2, 64), "views": rng.randint(1, 4),
                "most": log_uniform(5_000, 200_000), "width": side, "height": rng.randint(max(48, side // 2), side)}
    if kind == "step":
        side = log_uniform(64, 256)
        return {"kind": kind, "size": log_uniform(40, 250), "views": log_uniform(2, 64), "width": side,
                "height": rng.randint(max(48, side // 2), side)}
    # window sizes: any width, the heights of wide and of tall windows
    width = log_uniform(160, 3840)
    height = min(2160, max(90, int(width * rng.uniform(0.5, 1.0))))
    scene = rng.choice(["sphere", "terrain", "terrain", "stress"])
    size = {"sphere": lambda: log_uniform(12, 128), "terrain": lambda: log_uniform(96, 1024),
            "stress": lambda: log_uniform(2_000, 1_000_000)}[scene]()
    msaa = rng.choice([0, 0, 0, 1, 2, 3]) if kind == "frame" and width <= 1920 else 0
    shaders = [R.PS_BLINN_PHONG] * 3 + [R.PS_LAMBERTIAN_ALBEDO, R.PS_LAMBERTIAN]
    if scene == "terrain" and not msaa:
        shaders += [R.PS_LAMBERTIAN_TEXTURED, R.PS_BLINN_PHONG_REFERENCE]
    return {"kind": kind, "scene": scene, "size": size, "width": width, "height": height,
            "shader": rng.choice(shaders), "depth": rng.choice([R.DEPTH_LESS, R.DEPTH_LEQUAL]), "msaa": msaa}


# --------------------------------------------------------------------------
# inputs

def _scene(case, seed):
    """(mesh, view, textures) of a frame or viewer case."""
    w, h, size = case["width"], case["height"], case["size"]
    textures = []
    if case["scene"] == "sphere":
        sc = scenes.sphere_scene(w, h, seed=seed, slices=size, stacks=2 * size)
    elif case["scene"] == "terrain":
        sc = scenes.terrain_scene(size, w, h, seed=seed)
    else:
        sc = scenes.stress_scene(size, w, h, seed=seed)
    sc.view.shader, sc.view.depth_func = case["shader"], case["depth"]
    if case["shader"] == R.PS_BLINN_PHONG_REFERENCE:
        sc.view.ks, sc.view.shininess = 3.0, 200.0
    if case["shader"] == R.PS_LAMBERTIAN_TEXTURED:
        # an 8-bit image, a float image of no round size and a constant colour; 24 repeats across the ground
        rng = np.random.default_rng(seed + 1)
        textures = [rng.integers(0, 256, (512, 512, 4)).astype(np.uint8),
                    rng.uniform(0.0, 1.0, (120, 300, 4)).astype(np.float32),
                    np.array([[[0.9, 0.6, 0.3, 1.0]]], np.float32)]
        sc.mesh.uvs = (sc.mesh.uvs * np.float32(24.0)).astype(np.float32)
        sc.mesh.texture_ids = rng.choice(3, sc.mesh.nt, p=[0.6, 0.3, 0.1]).astype(np.uint32)
    return sc.mesh, sc.view, textures


def _batch(case, seed):
    """(meshes, views) of a batch case."""
    meshes = scenes.batched_meshes(case["meshes"], 500, case["most"], seed=seed)
    views = []
    for m in range(len(meshes)):
        for v in scenes.orbit_views(case["views"], case["width"], case["height"], seed=seed + 1000 + m):
            v.mesh = m
            views.append(v)
    return meshes, views


def _step(case, seed):
    """(mesh, views, target images) of a step case."""
    rng = np.random.default_rng(seed)
    mesh = scenes.torus(case["size"], max(16, case["size"] * 2 // 5), 1.0, 0.35)
    mesh.albedo = rng.uniform(0.1, 0.9, size=(mesh.nv, 3)).astype(np.float32)
    views = scenes.orbit_views(case["views"], case["width"], case["height"], seed=seed + 1)
    target = rng.uniform(0.0, 1.0, (case["views"], case["height"], case["width"], 4)).astype(np.float32)
    return mesh, views, target


def prepare(case, seed):
    dev = torch.device("cuda")
    r = R.Renderer()
    r.Initialize(case["width"], case["height"])
    state = {"case": case, "renderer": r, "wrapped": {}}
    if case["kind"] in ("frame", "viewer"):
        mesh, view, textures = _scene(case, seed)
        R.configure(r, view)
        if textures:
            r.SetTextures(textures)
        if case["msaa"]:
            r.SetMSAAMode(case["msaa"])
        state["view"] = view
        state["mesh"] = R.DeviceMesh.from_mesh(mesh, dev) if case["kind"] == "frame" else R.HostMesh(mesh, pinned=True)
    elif case["kind"] == "batch":
        meshes, views = _batch(case, seed)
        state["batch"] = r.PrepareBatch([R.DeviceMesh.from_mesh(m, dev) for m in meshes], views)
    else:
        mesh, views, target = _step(case, seed)
        state["mesh"] = R.DeviceMesh.from_mesh(mesh, dev)
        state["batch"] = r.PrepareBatch([state["mesh"]], views)
        state["target"] = torch.from_numpy(target).to(dev)
    torch.cuda.synchronize()
    return state


# --------------------------------------------------------------------------
# one pass

class _DeviceArray:
    """A renderer-owned device buffer, for torch.as_tensor."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (int(ptr), False),
                                         "version": 3, "strides": None}


class _Outputs(dict):
    """Outputs in the renderer's own buffers: they live as long as the renderer."""

    renderer = None


def _images(state, o, lead, depth_lead):
    """Colour, depth and triangle id of the last pass as tensors (made once per buffer)."""
    key = (o.color, o.depth, o.triangle_id)
    if key not in state["wrapped"]:
        hw = (o.height, o.width)
        out = _Outputs(color=torch.as_tensor(_DeviceArray(o.color, lead + hw + (4,), "<f4"), device="cuda"),
                       depth=torch.as_tensor(_DeviceArray(o.depth, depth_lead + hw, "<f4"), device="cuda"),
                       triangle_id=torch.as_tensor(_DeviceArray(o.triangle_id, depth_lead + hw, "<i4"), device="cuda"))
        out.renderer = state["renderer"]
        state["wrapped"] = {key: out}
    return state["wrapped"][key]


def _run_step(state):
    r, mesh, target = state["renderer"], state["mesh"], state["target"]
    with torch.cuda.stream(r.stream):
        r.RenderBatched(state["batch"], None, state["case"]["width"], state["case"]["height"], synchronize=False)
        color = torch.empty_like(target)
        abi = mesh.abi()
        _lib.check(r._lib.edxr_shade_visible(r._h, ctypes.byref(abi), None, color.data_ptr()))
        # loss = sum((colour - target)^2 over RGB); the adjoint ignores alpha
        grad = 2.0 * (color - target)
        g = {k: torch.zeros_like(getattr(mesh, k)) for k in ("albedo", "normals", "positions")}
        g["light"], g["ks"], g["shininess"] = (torch.zeros(n, device="cuda") for n in (3, 1, 1))
        grads = _lib.Grads(*[g[k].data_ptr() for k in ("albedo", "normals", "positions", "light", "ks", "shininess")])
        _lib.check(r._lib.edxr_backward(r._h, ctypes.byref(abi), None, grad.data_ptr(), ctypes.byref(grads)))
    torch.cuda.current_stream().wait_stream(r.stream)
    return dict(g, color=color)


def run(state):
    case, r = state["case"], state["renderer"]
    if case["kind"] == "step":
        return _run_step(state)
    if case["kind"] == "batch":
        r.RenderBatched(state["batch"], None, case["width"], case["height"])
        o = r.BatchOutputs()
        return _images(state, o, (o.num_views,), (o.num_views,))
    view = state["view"]
    r.SetTransform(view.mv, view.proj, view.raster)
    if case["kind"] == "viewer":
        r.RenderMesh(state["mesh"], synchronize=False)
        out = _Outputs(image=r.GetBackBuffer(copy=False))
        out.renderer = r
        return out
    r.RenderMesh(state["mesh"])
    o = r.DeviceOutputs()
    return _images(state, o, (), (o.samples,) if o.samples > 1 else ())


def work(case):
    """Bytes: 36 per vertex (position, normal, albedo), 12 per triangle, 24 per
    pixel (RGBA32F, depth, id; 16 + 8 per sample with several).  A step reads
    its mesh once per view for the visibility, and writes colour, reads the
    ids and the targets and reads colour again, and touches the gradients."""
    pixels = case["width"] * case["height"]
    if case["kind"] == "batch":
        # triangle counts are log-uniform from 500 to `most`, twice as many triangles as vertices
        tris = case["meshes"] * (case["most"] - 500) / math.log(case["most"] / 500)
        return {"bytes": tris * (18 + 12) + case["meshes"] * case["views"] * pixels * 24, "flops": 0}
    if case["kind"] == "step":
        n = case["size"] * max(16, case["size"] * 2 // 5)
        return {"bytes": n * (36 + 24) + n * 36 + case["views"] * pixels * (24 + 4 + 16 + 16 + 16 + 4 + 16),
                "flops": 0}
    size = case["size"]
    nv, nt = {"sphere": lambda: (size * (2 * size - 1) + 2, 2 * size * (2 * size - 1)),
              "terrain": lambda: ((size + 1) ** 2, 2 * size * size),
              "stress": lambda: (3 * size, size)}[case["scene"]]()
    per_pixel = 4 if case["kind"] == "viewer" else 16 + 8 * (1 << case["msaa"])
    return {"bytes": nv * 36 + nt * 12 + pixels * per_pixel, "flops": 0}


# --------------------------------------------------------------------------
# the same outputs in 64 bits
#
# Which triangle wins a pixel is decided on the 1/16-pixel grid that the
# vertices are snapped to, with float32 depths (the reference's arithmetic),
# so the visibility is restated in that arithmetic, with numpy and torch; what
# is computed at the winner (depth, colour, gradients) is then 64 bits.

def _transform(m, p):
    """Rows of m times (p, 1) in float32, summed left to right."""
    m = np.asarray(m, np.float32)
    return np.stack([((m[i, 0] * p[:, 0] + m[i, 1] * p[:, 1]) + m[i, 2] * p[:, 2]) + m[i, 3] for i in range(4)], 1)


def _product(a, b):
    a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
    return ((a[:, [0]] * b[0] + a[:, [1]] * b[1]) + a[:, [2]] * b[2]) + a[:, [3]] * b[3]


def _distance(plane, c):
    """Signed distance (as the clipper forms it) and whether c is inside plane L, R, B, T, F, N."""
    x, y, z, w = c[..., 0], c[..., 1], c[..., 2], c[..., 3]
    return [(w + x, x >= -w), (-w + x, x <= w), (w + y, y >= -w), (-w + y, y <= w), (-w + z, z <= w), (z, z >= 0)][plane]


def _clip(clip, tri):
    """Triangles that straddle a plane (three clip-space vertices each): the
    fan pieces' vertices (n,3,4), the weights of the source vertices (n,3,3),
    the source triangles and the pieces' numbers in their fans."""
    n = len(clip)
    poly = np.zeros((n, 17, 7), np.float32)
    poly[:, :3, :4] = clip
    poly[:, :3, 4:] = np.eye(3, dtype=np.float32)
    count = np.full(n, 3)
    outside = np.stack([~_distance(k, clip)[1] for k in range(6)], -1)  # (n,3,6)
    cut = outside.any(1) & ~outside.all(1)
    for k in range(6):
        rows = np.nonzero(cut[:, k])[0]
        new, m = np.zeros_like(poly[rows]), np.zeros(len(rows), int)
        for i in range(int(count[rows].max(initial=0))):
            live = np.nonzero(i < count[rows])[0]
            a = poly[rows[live], i]
            b = poly[rows[live], np.where(i + 1 == count[rows[live]], 0, i + 1)]
            (da, ina), (db, inb) = _distance(k, a), _distance(k, b)
            with np.errstate(divide="ignore", invalid="ignore"):  # edges that do not cross are not used
                t = (da / (da - db))[:, None]
                mid = a * (np.float32(1) - t) + b * t
            w = mid[:, 3]
            mid[:, [0, 0, 1, 1, 2, 2][k]] = [-w, w, -w, w, w, 0 * w][k]
            put = live[ina != inb]
            new[put, m[put]] = mid[ina != inb]
            m[put] += 1
            put = live[inb]
            new[put, m[put]] = b[inb]
            m[put] += 1
        poly[rows], count[rows] = new, m
    used = np.arange(17)[None] < count[:, None]
    count[(used & (poly[..., 3] <= 0)).any(1)] = 0
    for s in (2, 1, 0):  # a vertex of weight one is that source vertex itself
        at = used & (poly[..., 4 + s] == 1)
        poly[at, :4] = np.broadcast_to(clip[:, None, s], poly[..., :4].shape)[at]
        poly[at, 4:] = np.eye(3, dtype=np.float32)[s]
    pieces = [(np.nonzero(count > f + 1)[0], f) for f in range(1, 15)]
    pick = np.concatenate([r for r, _ in pieces])
    fan = np.concatenate([np.full(len(r), f) for r, f in pieces])
    v = np.stack([poly[pick, 0], poly[pick, fan], poly[pick, fan + 1]], 1)
    return v[..., :4], v[..., 4:], tri[pick], fan


def _set_up(mesh, view):
    """Raster triangles of a frame: snapped vertices, depths, 1/w, weights of the source vertices, order."""
    clip = _transform(_product(view.proj, view.mv), mesh.positions)[mesh.indices.astype(np.int64)]
    out = np.stack([~_distance(k, clip)[1] for k in range(6)], -1)
    whole = np.nonzero(~out.any((1, 2)))[0]
    part = np.nonzero(out.any((1, 2)) & ~out.all(1).any(1))[0]
    pc, pw, ptri, fan = _clip(clip[part], part)
    c = np.concatenate([clip[whole], pc])
    weight = np.concatenate([np.broadcast_to(np.eye(3, dtype=np.float32), (len(whole), 3, 3)), pw])
    tri = np.concatenate([whole, ptri])
    order = np.concatenate([whole * 16, ptri * 16 + fan])
    inv_w = np.float32(1) / c[..., 3]
    ndc = (c[..., :3] * inv_w[..., None]).reshape(-1, 3)
    at = _transform(view.raster, ndc)[:, :2].reshape(-1, 3, 2) * np.float32(16)
    snapped = np.trunc(at).astype(np.int64)
    x, y = snapped[..., 0], snapped[..., 1]
    det = (x[:, 0] - x[:, 2]) * (y[:, 1] - y[:, 2]) - (x[:, 2] - x[:, 1]) * (y[:, 2] - y[:, 0])
    keep = np.nonzero(det > 0)[0]
    ext = [np.ptp(a[keep], 1) + 1024 for a in (x, y)]
    if len(keep) and (2.0 * ext[0] * ext[1]).max() >= 2 ** 30:
        return None  # 32-bit edge values may wrap: not restated here
    return {"x": x[keep], "y": y[keep], "det": det[keep], "z": ndc[:, 2].reshape(-1, 3)[keep], "inv_w": inv_w[keep],
            "weight": weight[keep], "tri": tri[keep], "order": order[keep]}


def _winners(s, view, offset, dev):
    """Per pixel the winning raster triangle (-1: none) at `offset` sixteenths from the pixel centres."""
    W, H = view.width, view.height
    less = view.depth_func == R.DEPTH_LESS
    best = torch.full((H * W,), (0x3F800000 << 32) | (0 if less else NO_TRIANGLE), dtype=torch.int64, device=dev)
    x, y = torch.from_numpy(s["x"]).to(dev), torch.from_numpy(s["y"]).to(dev)
    z = torch.from_numpy(s["z"]).to(dev)
    inv_det = torch.from_numpy(np.float32(1) / s["det"].astype(np.float32)).to(dev)
    rank = torch.from_numpy(s["order"]).to(dev) + 1
    x0 = torch.clamp((x.amin(1) - 8 - offset + 15) >> 4, min=0)
    x1 = torch.clamp((x.amax(1) - 8 - offset) >> 4, max=W - 1)
    y0 = torch.clamp((y.amin(1) - 8 - offset + 15) >> 4, min=0)
    y1 = torch.clamp((y.amax(1) - 8 - offset) >> 4, max=H - 1)
    wide = torch.clamp(x1 - x0 + 1, min=0)
    area = wide * torch.clamp(y1 - y0 + 1, min=0)
    some = torch.nonzero(area).flatten()
    ends = torch.cumsum(area[some], 0).cpu()
    at = 0
    while at < len(some):
        # up to 16 Mi (triangle, pixel) pairs at a time
        before = int(ends[at - 1]) if at else 0
        to = max(at + 1, int(torch.searchsorted(ends, before + (1 << 24), right=True)))
        t = torch.repeat_interleave(some[at:to], area[some[at:to]])
        first = torch.cumsum(area[some[at:to]], 0) - area[some[at:to]]
        local = torch.arange(len(t), device=dev) - torch.repeat_interleave(first, area[some[at:to]])
        px, py = x0[t] + local % wide[t], y0[t] + local // wide[t]
        cx, cy = px * 16 + 8 + offset, py * 16 + 8 + offset
        inside, edge = torch.ones_like(t, dtype=torch.bool), []
        for k in range(3):
            xa, ya, xb, yb = x[t, k], y[t, k], x[t, (k + 1) % 3], y[t, (k + 1) % 3]
            e = (ya - yb) * (cx - xa) + (xb - xa) * (cy - ya)
            edge.append(e)
            inside &= e >= ((yb > ya) | ((ya == yb) & (xa > xb))).long()
        t, px, py, e1, e2 = t[inside], px[inside], py[inside], edge[1][inside], edge[2][inside]
        l0, l1 = e1.float() * inv_det[t], e2.float() * inv_det[t]
        l2 = (torch.ones_like(l0) - l0) - l1
        d = (l0 * z[t, 0] + l1 * z[t, 1]) + l2 * z[t, 2] + 0.0
        bits = d.view(torch.int32).long()
        bits = torch.where(bits >= 0, bits, bits ^ 0x7FFFFFFF)
        key = (bits << 32) | (rank[t] if less else NO_TRIANGLE - rank[t])
        best.scatter_reduce_(0, (py * W + px)[~torch.isnan(d)], key[~torch.isnan(d)], "amin")
        at = to
    low = best & NO_TRIANGLE
    won = low if less else NO_TRIANGLE - low
    order, slot = torch.sort(torch.from_numpy(s["order"]).to(dev))
    if not len(order):
        return torch.full((H * W,), -1, dtype=torch.int64, device=dev)
    return torch.where(won > 0, slot[torch.searchsorted(order, won - 1).clamp(max=len(order) - 1)], -1)


def _eye(view):
    inv = np.linalg.inv(np.asarray(view.mv, np.float64))
    return torch.from_numpy(inv[:3, 3] / inv[3, 3])


def _shade(P, N, A, light, eye, ks, shininess, shader):
    """The pixel shaders on interpolated position, normal and albedo."""
    N = N / N.norm(dim=-1, keepdim=True)
    L = light / light.norm()
    diffuse = ((N * L).sum(-1).clamp(min=0) + 0.2)[:, None] * (3.0 / math.pi)
    color = diffuse * A if shader in (R.PS_BLINN_PHONG, R.PS_LAMBERTIAN_ALBEDO, R.PS_LAMBERTIAN_TEXTURED) \
        else diffuse.expand(-1, 3)
    if shader in (R.PS_BLINN_PHONG, R.PS_BLINN_PHONG_REFERENCE):
        E = eye - P
        H = L + E / E.norm(dim=-1, keepdim=True)
        nh = (N * (H / H.norm(dim=-1, keepdim=True))).sum(-1)
        if shader == R.PS_BLINN_PHONG:
            nh = nh.clamp(min=0)
        color = color + (ks * nh ** shininess)[:, None]
    return color


def _mips(textures, dev):
    """Every level of every texture in one pool, and [slot][level] -> (first texel, width, height)."""
    pool, table, at = [], [], 0
    for t in textures:
        img = t.astype(np.float64) / 255.0 if t.dtype == np.uint8 else t.astype(np.float64)
        levels = []
        while True:
            h, w = img.shape[:2]
            levels.append((at, w, h))
            pool.append(img.reshape(-1, 4))
            at += w * h
            if w == 1 and h == 1:
                break
            ys = [np.minimum(2 * np.arange(max(1, h // 2)) + q, h - 1) for q in (0, 1)]
            xs = [np.minimum(2 * np.arange(max(1, w // 2)) + q, w - 1) for q in (0, 1)]
            img = sum(img[a][:, b] for a in ys for b in xs) / 4.0
        table.append(levels)
    deep = max(len(t) for t in table)
    flat = torch.tensor([[t[min(k, len(t) - 1)] for k in range(deep)] for t in table], device=dev)
    return torch.from_numpy(np.concatenate(pool)).to(dev), flat, torch.tensor([len(t) - 1 for t in table], device=dev)


def _trilinear(mips, slot, uv, d0, d1):
    pool, table, last = mips
    size = table[slot, 0][:, 1:].double()
    r = torch.maximum(((d0 * size) ** 2).sum(-1), ((d1 * size) ** 2).sum(-1))
    lod = torch.minimum(0.5 * torch.log2(r.clamp(min=1.0)), last[slot].double())
    out = 0
    for q in (0, 1):
        level = torch.minimum(lod.floor().long() + q, last[slot])
        first, w, h = table[slot, level].unbind(-1)
        f = (uv - uv.floor()) * torch.stack([w, h], -1) - 0.5
        lo, part = f.floor(), f - f.floor()
        texel = lambda i, j: pool[first + (lo[:, 1].long() + j) % h * w + (lo[:, 0].long() + i) % w]  # noqa: E731
        tx, ty = part[:, :1], part[:, 1:]
        level_color = (texel(0, 0) * (1 - tx) + texel(1, 0) * tx) * (1 - ty) + \
            (texel(0, 1) * (1 - tx) + texel(1, 1) * tx) * ty
        share = (lod - lod.floor())[:, None]
        out = out + level_color * (share if q else 1 - share)
    return out[:, :3]


def _exact_frame(mesh, view, textures, offsets, dev):
    """(colour (H,W,4), depth per sample) of one frame in 64 bits, or None."""
    s = _set_up(mesh, view)
    if s is None:
        return None
    W, H = view.width, view.height
    t64 = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev).double()  # noqa: E731
    x, y, det, z, inv_w, weight = (t64(s[k]) for k in ("x", "y", "det", "z", "inv_w", "weight"))
    source = torch.from_numpy(mesh.indices.astype(np.int64)[s["tri"]]).to(dev)
    light, eye = t64(view.light), _eye(view).to(dev)
    mips = _mips(textures, dev) if textures else None

    def flat_weights(t, px, py, offset=0):
        cx, cy = px * 16.0 + 8 + offset, py * 16.0 + 8 + offset
        e1 = (y[t, 1] - y[t, 2]) * (cx - x[t, 2]) + (x[t, 2] - x[t, 1]) * (cy - y[t, 2])
        e2 = (y[t, 2] - y[t, 0]) * (cx - x[t, 2]) + (x[t, 0] - x[t, 2]) * (cy - y[t, 2])
        return torch.stack([e1 / det[t], e2 / det[t], 1 - e1 / det[t] - e2 / det[t]], -1)

    def source_weights(t, px, py):
        """Perspective-correct weights of the input triangle's vertices at the pixel centre."""
        b = flat_weights(t, px, py) * inv_w[t]
        b = b / b.sum(-1, keepdim=True)
        return (b[:, :, None] * weight[t]).sum(1)

    total = torch.zeros((H * W, 4), dtype=torch.float64, device=dev)
    depths = []
    for o in offsets:
        won = _winners(s, view, o, dev)
        at = torch.nonzero(won >= 0).flatten()
        t, px, py = won[at], at % W, at // W
        depth = torch.ones(H * W, dtype=torch.float64, device=dev)
        depth[at] = (flat_weights(t, px, py, o) * z[t]).sum(-1)
        depths.append(depth.reshape(H, W))
        b, v = source_weights(t, px, py), source[t]
        mix = lambda a: (b[:, :, None] * t64(a)[v]).sum(1)  # noqa: E731
        if textures:
            uvs = t64(mesh.uvs)[v]
            uv = lambda i, j: (source_weights(t, i, j)[:, :, None] * uvs).sum(1)  # noqa: E731
            qx, qy = px & ~1, py & ~1
            slot = torch.from_numpy(mesh.texture_ids.astype(np.int64)[s["tri"]]).to(dev)[t]
            albedo = _trilinear(mips, slot, uv(px, py), uv(qx + 1, qy) - uv(qx, qy), uv(qx, qy + 1) - uv(qx, qy))
        else:
            albedo = mix(mesh.albedo)
        c = _shade(mix(mesh.positions), mix(mesh.normals), albedo, light, eye, view.ks, view.shininess, view.shader)
        if len(offsets) > 1:  # the resolve averages 8-bit sample colours
            c = torch.floor(c.clamp(0, 1) * 255 + 0.5) / 255
        total[at] += torch.cat([c, torch.ones_like(c[:, :1])], -1)
    color = (total / len(offsets)).reshape(H, W, 4)
    return color, (torch.stack(depths) if len(offsets) > 1 else depths[0])


def _exact_step(case, seed, dev):
    mesh, views, target = _step(case, seed)
    t64 = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev).double()  # noqa: E731
    pos, nrm, alb = (t64(a).requires_grad_() for a in (mesh.positions, mesh.normals, mesh.albedo))
    ks, shin = (t64(np.array([a])).requires_grad_() for a in (views[0].ks, views[0].shininess))
    lights, colors = [], []
    index = torch.from_numpy(mesh.indices.astype(np.int64)).to(dev)
    target = t64(target)
    for i, view in enumerate(views):
        s = _set_up(mesh, view)
        if s is None or view.ks != views[0].ks or view.shininess != views[0].shininess:
            return None
        won = _winners(s, view, 0, dev)
        at = torch.nonzero(won >= 0).flatten()
        v = index[torch.from_numpy(s["tri"]).to(dev)[won[at]]]
        p, n, a = pos[v], nrm[v], alb[v]
        mvp = t64(_product(view.proj, view.mv))
        clip = p @ mvp[:, :3].T + mvp[:, 3]
        # NDC of the pixel centres: the raster matrix maps each axis by itself
        u = ((at % view.width) + 0.5 - float(view.raster[0, 3])) / float(view.raster[0, 0])
        w = ((at // view.width) + 0.5 - float(view.raster[1, 3])) / float(view.raster[1, 1])
        b = torch.linalg.cross((clip[..., 0] - u[:, None] * clip[..., 3]), (clip[..., 1] - w[:, None] * clip[..., 3]))
        b = (b / b.sum(-1, keepdim=True))[:, :, None]
        light = t64(view.light).requires_grad_()
        c = _shade((b * p).sum(1), (b * n).sum(1), (b * a).sum(1), light, _eye(view).to(dev), ks, shin, view.shader)
        img = torch.zeros((view.height * view.width, 4), dtype=torch.float64, device=dev)
        img[at] = torch.cat([c.detach(), torch.ones_like(c[:, :1])], -1)
        ((c - target[i].reshape(-1, 4)[at, :3]) ** 2).sum().backward()
        colors.append(img.reshape(view.height, view.width, 4))
        lights.append(light.grad)
    return {"albedo": alb.grad, "normals": nrm.grad, "positions": pos.grad, "light": torch.stack(lights).sum(0),
            "ks": ks.grad, "shininess": shin.grad, "color": torch.stack(colors)}


# 1/16-pixel sample offsets per log2 of the sample count, the same in x and y (FrameBuffer.cpp:107-191 as
# Rasterizer.h:247 reads it)
_SAMPLES = [[0], [4, -4], [-2, 6, -6, 2], [1, -1, 5, -3, -5, -7, 3, 7]]


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if case["kind"] == "viewer":
        return None  # bytes
    if case["kind"] == "step":
        return _exact_step(case, seed, dev)
    if case["kind"] == "batch":
        meshes, views = _batch(case, seed)
        frames = [_exact_frame(meshes[v.mesh], v, [], [0], dev) for v in views]
        if any(f is None for f in frames):
            return None
        return {"color": torch.stack([f[0] for f in frames]), "depth": torch.stack([f[1] for f in frames]),
                "triangle_id": None}
    mesh, view, textures = _scene(case, seed)
    f = _exact_frame(mesh, view, textures, _SAMPLES[case["msaa"]], dev)
    return None if f is None else {"color": f[0], "depth": f[1], "triangle_id": None}
