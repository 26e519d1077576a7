"""Workloads of the rasteriser, each one pass through its public entry points.

``listed()`` gives the standing cases and ``draw(rng)`` more of the same
ranges; ``prepare`` builds what a program holds before the call (resident
meshes and textures, page-locked buffers), ``run`` makes the call and returns
its whole outputs, ``work`` says what a pass cannot do without, and ``exact``
gives the depth image in 64 bits by plain torch.

Kinds of case:
  frame    Context.render on resident meshes, outputs left on the device
  view     Renderer.render() and its getters: images in host memory
  update   a mesh and texture sent anew with every frame, RGB8 and depth read
           back, three contexts in turn on one upload stream
  noalloc  mr_render_noalloc on the caller's device arrays
  batch    Context.render_batch, outputs left on the device
Scenes: "sphere" (UV sphere under a point light), "icosphere" (displaced,
textured, shared vertices), "soup" (unshared 1-4 pixel triangles, exact ties),
"prims" (a hierarchy of primitives, one mesh each).
"""
import ctypes as C
import math

import numpy as np
import torch

from minirender_gb300 import abi, capi
from minirender_gb300 import projection as pj
from minirender_gb300 import scene as S
from minirender_gb300 import workloads as W
from minirender_gb300.batch import BatchRenderer
from minirender_gb300.frame import FrameState
from minirender_gb300.renderer import Renderer


def _case(name, kind, scene, size, width, height, **more):
    c = {"name": name, "kind": kind, "scene": scene, "size": size, "width": width, "height": height}
    c.update(more)
    return c


def listed():
    return [
        # the smallest request of a serving stream: a thumbnail of a small soup, bound by launches
        _case("soup_thumbnail", "frame", "soup", 1000, 128, 128),
        # one simple object in a preview window
        _case("sphere_480p", "frame", "sphere", 32, 640, 480),
        # a scene of many meshes with triangles from one pixel to much of the screen, one frame per call
        _case("prims_720p", "frame", "prims", 64, 1280, 720),
        # an odd-sized sensor image: orthographic, float texture, float colour and normals besides the rest
        _case("ortho_normals_odd", "frame", "icosphere", 6, 1001, 563, ortho=True, float_texture=True, everything=True),
        # one large scanned mesh, textured and near-clipped, at full HD
        _case("mesh_1080p", "frame", "icosphere", 8, 1920, 1080),
        # heavy overdraw and ties: a ten-million-triangle soup at 4K
        _case("soup_4k", "frame", "soup", 10_000_000, 3840, 2160),
        # the Renderer mirror as an application uses it: render, then image and depth in host memory
        _case("view_480p", "view", "prims", 64, 640, 480),
        # an animated mesh: all vertices and texels re-sent with every frame, results read back
        _case("update_1080p", "update", "icosphere", 8, 1920, 1080),
        # a caller that may not allocate: device arrays in, device images out, synchronous
        _case("noalloc_1080p", "noalloc", "icosphere", 7, 1920, 1080),
        # a few small views of small scenes in one launch, default tiling
        _case("batch_views", "batch", "prims", 16, 256, 256, scenes=24),
        # what a render server batches: soups of mixed sizes
        _case("batch_soups", "batch", "soup", 300_000, 1280, 720, scenes=16, tile_w=16, tile_h=16, threads=64),
        # dataset generation: 256 scenes of 64 primitives, mixed resolutions
        _case("batch_256", "batch", "prims", 64, 0, 0, scenes=256, tile_w=64, tile_h=32, threads=256),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def frame_size(lo=128, hi=3840):
        w = log(lo, hi)
        return w, max(96, min(2160, int(round(w * rng.uniform(0.5, 1.0)))))

    what = rng.choice(["soup", "soup", "sphere", "prims", "icosphere", "icosphere", "view", "noalloc", "batch", "batch"])
    if what == "soup":
        w, h = frame_size()
        return _unnamed("frame", "soup", log(1000, 4_000_000), w, h)
    if what == "sphere":
        w, h = frame_size(128, 1920)
        return _unnamed("frame", "sphere", rng.randint(8, 128), w, h)
    if what == "prims":
        w, h = frame_size(256, 1920)
        return _unnamed("frame", "prims", rng.randint(1, 96), w, h)
    if what == "icosphere":
        w, h = frame_size(320, 2560)
        return _unnamed("frame", "icosphere", rng.randint(3, 8), w, h, ortho=rng.random() < 0.25,
                        float_texture=rng.random() < 0.25, everything=rng.random() < 0.25)
    if what == "view":
        w, h = frame_size(128, 1280)
        return _unnamed("view", "prims", rng.randint(4, 64), w, h)
    if what == "noalloc":
        w, h = frame_size(128, 1920)
        return _unnamed("noalloc", "icosphere", rng.randint(3, 7), w, min(h, (1 << 21) // w))
    tile_w, tile_h, threads = rng.choice([(0, 0, 0), (16, 16, 64), (32, 32, 256), (64, 32, 256)])
    if rng.random() < 0.4:
        w, h = frame_size(128, 1920)
        return _unnamed("batch", "soup", log(1000, 400_000), w, h, scenes=rng.randint(2, 16),
                        tile_w=tile_w, tile_h=tile_h, threads=threads)
    w, h = frame_size(128, 1280)
    return _unnamed("batch", "prims", rng.randint(2, 64), w, h, scenes=rng.randint(2, 64),
                    tile_w=tile_w, tile_h=tile_h, threads=threads)


def _unnamed(*a, **more):
    c = _case("", *a, **more)
    del c["name"]
    return c


# ------------------------------------------------------------------ scenes
def _soup(n, width, height, seed, palette=64, dup_frac=0.05):
    """workloads.config3's soup, made on the GPU: 95 % unique triangles of 1-4
    square pixels parallel to the image plane at uniform depth, then exact
    copies of some in another colour."""
    g = torch.Generator("cuda").manual_seed(seed)
    rnd = lambda k: torch.rand(k, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    n_dup = int(round(n * dup_frac))
    n_u = n - n_dup
    P = pj.projection_frustum(pj.deg2rad(60), np.float32(width) / np.float32(height), 0.1, 100)
    cx, cy, d = rnd(n_u) * width, rnd(n_u) * height, 0.2 + rnd(n_u) * 49.8
    rad = torch.sqrt(4 * (1 + 3 * rnd(n_u)) / math.sqrt(3)) / math.sqrt(3)
    rot = rnd(n_u) * (2 * math.pi)
    ang = rot[:, None] - torch.tensor([0, 2 * math.pi / 3, 4 * math.pi / 3], dtype=torch.float64, device="cuda")
    xn = 2 * (cx[:, None] + rad[:, None] * torch.cos(ang)) / width - 1
    yn = 1 - 2 * (cy[:, None] + rad[:, None] * torch.sin(ang)) / height
    z = d[:, None].expand(n_u, 3)
    verts = torch.stack([xn * z / float(P[0, 0]), yn * z / float(P[1, 1]), -z], -1).reshape(-1, 3).float()
    nrm = torch.stack([rnd(n_u) * 0.9 - 0.45, rnd(n_u) * 0.9 - 0.45, torch.ones_like(d)], 1)
    nrm = (nrm / nrm.norm(dim=1, keepdim=True)).float()
    pal = palette * palette
    col = torch.randint(0, pal, (n_u,), device="cuda", generator=g)
    src = torch.sort(torch.randint(0, n_u, (n_dup,), device="cuda", generator=g)).values
    col = torch.cat([col, (col[src] + 1 + torch.randint(0, pal - 1, (n_dup,), device="cuda", generator=g)) % pal])
    face = torch.cat([torch.arange(n_u, device="cuda"), src])
    corner = (3 * face[:, None] + torch.arange(3, device="cuda")).reshape(-1)
    host = lambda t, dt: t.to(dt).cpu().numpy()  # noqa: E731
    k = np.arange(pal)
    uvs = np.stack([(k % palette + 0.5) / palette, (k // palette + 0.5) / palette], 1).astype(np.float32)
    tex = np.random.default_rng(seed + 1).integers(0, 256, (palette, palette, 3)).astype(np.uint8)
    mesh = S.TriMesh(host(verts, torch.float32), host(nrm, torch.float32), host(corner, torch.int32),
                     normalsI=host(face.repeat_interleave(3), torch.int32), texcoords=uvs,
                     texcoordsI=host(col.repeat_interleave(3), torch.int32),
                     material=S.Material(specular=(0.3, 0.3, 0.3), shininess=8, texture=tex))
    scene = S.Scene()
    scene.add(mesh)
    st = FrameState(width=width, height=height, projection=P, light=np.array([0.2, 0.4, 1.0], np.float32),
                    ambient=scene.ambientLight)
    return st, scene


def _sphere(segments, width, height, seed):
    rng = np.random.default_rng(seed)
    st, scene = W.config1(width, height)
    mesh = W.create_sphere(1.0, segments, 2 * segments)
    mesh.material = S.Material(diffuse=rng.uniform(0.2, 1, 3), specular=(1, 1, 1), shininess=32)
    scene.children = [mesh]
    st.view = pj.mat_mul(st.view, pj.rotate_x(float(rng.uniform(-1, 1))))
    return st, scene


def _icosphere(level, width, height, seed, ortho=False, float_texture=False, everything=False):
    st, scene = W.config2(level=level, width=width, height=height, tex_size=1024, seed=seed)
    if float_texture:
        m = scene.children[0].material
        m.texture = m.texture.astype(np.float32) / np.float32(255)
    if ortho:
        a = width / height
        st.projection = pj.projection_ortho(-1.1 * a, 1.1 * a, -1.1, 1.1, 0.5, 10)
    st.save_normals = everything
    return st, scene


def _one(case, seed):
    w, h, n = case["width"], case["height"], case["size"]
    if case["scene"] == "soup":
        return _soup(n, w, h, seed)
    if case["scene"] == "sphere":
        return _sphere(n, w, h, seed)
    if case["scene"] == "prims":
        return W.config4_scene(seed, n, (w, h))
    return _icosphere(n, w, h, seed, case.get("ortho", False), case.get("float_texture", False),
                      case.get("everything", False))


def _scenes(case, seed):
    """The frames of a batch; a soup batch holds sizes and resolutions from a
    tenth of the case's to all of it, a batch without a size of its own the
    four resolutions of workloads.RESOLUTIONS in turn."""
    out = []
    for k in range(case["scenes"]):
        c = dict(case)
        if not case["width"]:
            c["width"], c["height"] = W.RESOLUTIONS[k % len(W.RESOLUTIONS)]
        if case["scene"] == "soup":
            f = 0.1 ** (k / max(1, case["scenes"] - 1))
            c.update(size=max(100, int(case["size"] * f)), width=max(64, int(case["width"] * math.sqrt(f))),
                     height=max(64, int(case["height"] * math.sqrt(f))))
        out.append(_one(c, 1000 * seed + k))
    return out


# ------------------------------------------------------------------ passes
class _Array:
    """Device memory of a context as torch sees it; the tensor made of it
    holds this object, and so the context that owns the memory."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


class _Outputs(dict):
    """Outputs that live in a context's memory: the context stays as long as they do."""

    owner = None


def _pin(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


def prepare(case, seed):
    s = {"case": case, "views": {}}
    if case["kind"] == "batch":
        br = BatchRenderer(0)
        if case.get("tile_w"):
            br.ctx.set_batch_tiling(case["tile_w"], case["tile_h"], case["threads"], 64)
        s["keep"] = br
        s["ctx"], s["args"], s["outputs"] = br.ctx, br.prepare(_scenes(case, seed)), br.outputs
        return s
    st, scene = _one(case, seed)
    if case["kind"] == "noalloc":
        return _prepare_noalloc(s, st, scene)
    s["outputs"] = abi.MR_OUT_DEFAULT | (abi.MR_OUT_RGB_F32 if case.get("everything") else 0)
    lanes = []
    for _ in range(3 if case["kind"] == "update" else 1):
        r = Renderer(0)
        r.state = st
        r.setScene(scene)
        lanes.append((r, r.prepare()))
    s["keep"] = r = lanes[0][0]
    s["ctx"], s["args"] = r.ctx, lanes[0][1]
    if case["kind"] == "update":
        s["outputs"] = abi.MR_OUT_RGB8 | abi.MR_OUT_DEPTH
        mesh = scene.children[0]
        idx = _pin(mesh.indices).numpy()
        pinned = S.TriMesh(_pin(mesh.vertices).numpy(), _pin(mesh.normals).numpy(), idx, normalsI=idx,
                           texcoords=_pin(mesh.texcoords).numpy(), texcoordsI=idx, material=mesh.material)
        s["mesh"], s["desc"], s["tex"] = pinned, pinned.desc(), _pin(mesh.material.texture).numpy()
        s["upload"] = torch.cuda.Stream()
        s["lanes"], s["next"] = [], 0
        for r, (frame, rs, n) in lanes:
            r.ctx.set_upload_stream(s["upload"].cuda_stream)
            rgb8 = torch.empty((st.height, st.width, 3), dtype=torch.uint8).pin_memory()
            depth = torch.empty((st.height, st.width), dtype=torch.float32).pin_memory()
            s["lanes"].append({"r": r, "ctx": r.ctx, "frame": frame, "rs": rs, "n": n, "mesh": rs[0].mesh,
                               "tex": rs[0].material.texture, "rgb8": rgb8, "depth": depth})
    return s


def _prepare_noalloc(s, st, scene):
    flat = S.flatten(scene)
    rs, _ = capi.collect_shapes(flat.nodes)
    mesh, tex = flat.meshes[0], flat.textures[0]
    dev = [torch.from_numpy(a).cuda() for a in (mesh.vertices, mesh.normals, mesh.texcoords, mesh.indices, tex)]
    v, n, uv, idx, t = dev
    desc = abi.mr_mesh_desc(v.data_ptr(), len(v), n.data_ptr(), len(n), uv.data_ptr(), len(uv),
                            idx.data_ptr(), len(idx), idx.data_ptr(), len(idx), idx.data_ptr(), len(idx))
    H, Wd = st.height, st.width
    out = [torch.empty((H, Wd, 3), dtype=torch.uint8, device="cuda"),
           torch.empty((H, Wd), dtype=torch.float32, device="cuda"),
           torch.empty((H, Wd), dtype=torch.int32, device="cuda")]
    frame, xf, mat = st.to_c(), (C.c_float * 16)(*rs[0].transform), rs[0].material
    s.update(keep=(dev, rs, frame, desc, xf, mat), out=out,
             call=(C.byref(frame), C.byref(desc), C.addressof(xf), C.byref(mat), t.data_ptr(), tex.shape[0],
                   tex.shape[1], 1, out[0].data_ptr(), out[1].data_ptr(), out[2].data_ptr()))
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "frame":
        s["ctx"].render(*s["args"], s["outputs"])
        return _frame_outputs(s)
    if kind == "batch":
        s["ctx"].render_batch(*s["args"], s["outputs"])
        return _batch_outputs(s)
    if kind == "view":
        r = s["keep"]
        r.render()
        return {"rgb8": r.getImageRGB8(), "depth": r.getDepth()}
    if kind == "update":
        L = s["lanes"][s["next"]]
        s["next"] = (s["next"] + 1) % len(s["lanes"])
        L["ctx"].update_mesh(L["mesh"], s["desc"])
        L["ctx"].update_texture(L["tex"], s["tex"])
        L["ctx"].render(L["frame"], L["rs"], L["n"], s["outputs"])
        L["ctx"].read_async(L["rgb8"].numpy(), L["depth"].numpy())
        return {"rgb8": L["rgb8"], "depth": L["depth"]}
    rc = capi.lib().mr_render_noalloc(*s["call"], torch.cuda.current_stream().cuda_stream)
    if rc != abi.MR_OK:
        raise RuntimeError(capi.lib().mr_status_string(rc).decode())
    return {"rgb8": s["out"][0], "depth": s["out"][1], "ids": s["out"][2]}


def _view(s, name, ptr, shape, typestr):
    got = s["views"].get(name)
    if got is None or got[0] != ptr:
        got = s["views"][name] = (ptr, torch.as_tensor(_Array(s["ctx"], ptr, shape, typestr), device="cuda"))
    return got[1]


def _frame_outputs(s):
    o = s["ctx"].outputs()
    H, Wd = o.height, o.width
    out = _Outputs(rgb8=_view(s, "rgb8", o.rgb8, (H, Wd, 3), "|u1"), depth=_view(s, "depth", o.depth, (H, Wd), "<f4"),
                   ids=_view(s, "ids", o.tri_id, (H, Wd), "<i4"))
    out.owner = s["ctx"]
    if s["case"].get("everything"):
        out["image"] = _view(s, "image", o.rgb_f32, (H, Wd, 3), "<f4")
        out["normals"] = _view(s, "normals", o.normals, (H, Wd, 3), "<f4")
    return out


def _batch_outputs(s):
    """Every scene's outputs; those of one batch lie back to back, so one
    tensor per kind of output covers them all."""
    first, last, L = abi.mr_outputs(), abi.mr_outputs(), capi.lib()
    scenes, n = s["args"][0], s["args"][1]
    L.mr_get_batch_outputs(s["ctx"].h, 0, C.byref(first))
    L.mr_get_batch_outputs(s["ctx"].h, n - 1, C.byref(last))
    if "pixels" not in s:
        s["pixels"] = sum(scenes[i].frame.width * scenes[i].frame.height for i in range(n))
    px = s["pixels"]
    if last.depth + 4 * last.width * last.height != first.depth + 4 * px:
        raise RuntimeError("the outputs of a batch no longer lie back to back")
    out = _Outputs(rgb8=_view(s, "rgb8", first.rgb8, (px, 3), "|u1"), depth=_view(s, "depth", first.depth, (px,), "<f4"),
                   ids=_view(s, "ids", first.tri_id, (px,), "<i4"))
    out.owner = s["ctx"]
    return out


# ------------------------------------------------------------------ work
def _counts(case):
    """Triangles, vertices, normals and texel bytes of one frame (a frame of
    primitives: the mean of the generator)."""
    n = case["size"]
    if case["scene"] == "sphere":
        return 4 * n * (n - 1), 2 * n * (n - 1) + 2, 2 * n * (n - 1) + 2, 0
    if case["scene"] == "icosphere":
        return 20 * 4 ** n, 10 * 4 ** n + 2, 10 * 4 ** n + 2, 3 * 1024 * 1024 * (4 if case.get("float_texture") else 1)
    if case["scene"] == "soup":
        u = n - int(round(0.05 * n))
        return n, 3 * u, u, 3 * 64 * 64
    return 540 * n, 330 * n, 330 * n, 0


def work(case):
    frames = case.get("scenes", 1)
    px = (case["width"] * case["height"] or sum(w * h for w, h in W.RESOLUTIONS) / len(W.RESOLUTIONS))
    T, V, N, tex = _counts(case)
    if case["kind"] == "batch" and case["scene"] == "soup":  # sizes fall off to a tenth
        f = sum(0.1 ** (k / max(1, frames - 1)) for k in range(frames)) / frames
        T, V, N, px = T * f, V * f, N * f, px * f
    indices = 36 if case["scene"] == "soup" else 12
    per_px = 3 + 4 + (0 if case["kind"] in ("update", "view") else 4) + (24 if case.get("everything") else 0)
    textured = case["scene"] in ("icosphere", "soup")
    mesh = 12 * V + 12 * N + indices * T + (8 * (V if case["scene"] == "icosphere" else 4096) if textured else 0)
    # an update's mesh and texels cross the host link; the rest is read where it lies
    return {"bytes": frames * (mesh + tex + per_px * px), "flops": frames * (70 * V + 20 * N + 60 * T + 120 * px)}


# ------------------------------------------------------------------ 64 bits
def exact(case, seed):
    """The depth image in 64 bits: every triangle's covered pixel centres
    (homogeneous edge functions, so triangles through the near plane need no
    clipping), nearest first.  Bytes, ids and shaded images have no value of
    their own there: which triangle a pixel on an edge shows is a rounding."""
    none = {"rgb8": None, "depth": None, "ids": None}
    if case.get("everything"):
        none.update(image=None, normals=None)
    if case["kind"] == "batch" and case["scenes"] > 32:
        return None
    if case["kind"] in ("view", "update"):
        del none["ids"]
    frames = _scenes(case, seed) if case["kind"] == "batch" else [_one(case, seed)]
    depths = [_exact_depth(st, scene) for st, scene in frames]
    none["depth"] = torch.cat([d.reshape(-1) for d in depths]) if case["kind"] == "batch" else depths[0]
    return none


def _world(node, parent):
    m = parent @ np.asarray(node.transform, np.float64).reshape(4, 4)
    if isinstance(node, S.TriMesh):
        yield node, m
    for c in node.children:
        yield from _world(c, m)


def _exact_depth(st, scene):
    Wd, H = st.width, st.height
    P = torch.as_tensor(np.asarray(st.projection, np.float64).reshape(4, 4), device="cuda")
    view = np.asarray(st.view, np.float64).reshape(4, 4)
    persp = float(P[3, 3]) == 0
    near = float(P[2, 3] / (P[2, 2] - 1)) if persp else float((P[2, 3] + 1) / P[2, 2])  # distance
    tri = []
    for mesh, m in _world(scene, np.eye(4)):
        mv = torch.as_tensor(view @ m, device="cuda")
        v = torch.as_tensor(mesh.vertices, device="cuda").double() @ mv[:3, :3].T + mv[:3, 3]
        tri.append(v[torch.as_tensor(mesh.indices.reshape(-1, 3), device="cuda").long()])
    tri = torch.cat(tri)
    out = torch.full((H * Wd,), 1e11, dtype=torch.float64, device="cuda")

    def screen(v):
        w = v @ P[3, :3] + P[3, 3]
        x, y = (v @ P[0, :3] + P[0, 3]) / w, (v @ P[1, :3] + P[1, 3]) / w
        return (1 + x) * (Wd / 2), (1 - y) * (H / 2)

    front = tri[..., 2] <= -near
    tri, front = tri[front.any(1)], front[front.any(1)]
    # bounding box over the corners in front and the points where edges meet the near plane
    a, b = tri, tri.roll(-1, 1)
    dz = b[..., 2] - a[..., 2]
    t = torch.where(dz.abs() > 1e-12, (-near - a[..., 2]) / dz, torch.zeros_like(dz))
    crossing = a + t[..., None] * (b - a)
    use = torch.cat([front, front != front.roll(-1, 1)], 1)
    px, py = screen(torch.cat([a, crossing], 1))
    big = 1e30

    def box(p, n):
        lo = torch.where(use, p, torch.full_like(p, big)).amin(1)
        hi = torch.where(use, p, torch.full_like(p, -big)).amax(1)
        on = (hi >= 0) & (lo <= n)
        return lo.clamp(0, n - 1).floor().long(), hi.clamp(0, n - 1).floor().long(), on

    x0, x1, onx = box(px, Wd)
    y0, y1, ony = box(py, H)
    keep = onx & ony
    tri, x0, x1, y0, y1 = tri[keep], x0[keep], x1[keep], y0[keep], y1[keep]
    bw = x1 - x0 + 1
    area = bw * (y1 - y0 + 1)
    if area.numel() == 0:
        return out.reshape(H, Wd)
    ends = torch.cumsum(area, 0)
    start, k = 0, 0
    while k < len(area):  # some millions of (triangle, pixel) pairs at a time
        stop = int(torch.searchsorted(ends, start + 16_000_000, right=True))
        stop = max(stop, k + 1)
        i = torch.repeat_interleave(torch.arange(k, stop, device="cuda"), area[k:stop])
        j = torch.arange(i.numel(), device="cuda") - (ends[i] - area[i] - start)
        x, y = x0[i] + j % bw[i], y0[i] + j // bw[i]
        T = tri[i]
        xn, yn = (x + 0.5) / (Wd / 2) - 1, 1 - (y + 0.5) / (H / 2)
        if persp:
            ray = torch.stack([(xn + P[0, 2]) / P[0, 0], (yn + P[1, 2]) / P[1, 1], -torch.ones_like(xn)], 1)
            e = [(ray * torch.linalg.cross(T[:, q], T[:, p])).sum(1) for p, q in ((1, 2), (2, 0), (0, 1))]
            det = (T[:, 0] * torch.linalg.cross(T[:, 2], T[:, 1])).sum(1)
            total = e[0] + e[1] + e[2]
            z = det / total  # ray parameter: the distance along -z
            hit = (e[0] >= 0) & (e[1] >= 0) & (e[2] >= 0) & (total > 0) & (z >= near)
        else:
            X, Y = [(T[:, c, 0] * P[0, 0] + P[0, 3]) for c in range(3)], [(T[:, c, 1] * P[1, 1] + P[1, 3]) for c in range(3)]
            e = [(X[p] - xn) * (Y[q] - yn) - (X[q] - xn) * (Y[p] - yn) for p, q in ((1, 2), (2, 0), (0, 1))]
            total = e[0] + e[1] + e[2]
            z = sum(e[c] * (T[:, c, 2] * P[2, 2] + P[2, 3]) for c in range(3)) / total
            hit = (e[0] >= 0) & (e[1] >= 0) & (e[2] >= 0) & (total > 0) & (T[..., 2].amax(1) <= -near)
        at = (y * Wd + x)[hit]
        out.scatter_reduce_(0, at, z[hit], "amin")
        start, k = int(ends[stop - 1]), stop
    return out.reshape(H, Wd)
