"""Sizes at which the kernels' splits and dispatch rules change, against the
oracle: visible ids and depth bit for bit, RGB8 within 1."""
import numpy as np
import pytest

from minirender_gb300 import projection as pj
from minirender_gb300 import scene as S
from minirender_gb300.frame import FrameState
from minirender_gb300.renderer import Renderer
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _same(got, want, what):
    assert np.array_equal(got["ids"], want["ids"]), f"{what}: visible ids differ"
    assert np.array_equal(got["depth"].view(np.uint32), want["depth"].view(np.uint32)), f"{what}: depth"
    d = np.abs(got["rgb8"].astype(np.int16) - want["rgb8"].astype(np.int16))
    assert d.max(initial=0) <= 1, f"{what}: rgb8"


def _render(st, sc):
    r = Renderer(0)
    try:
        r.state = st
        r.setScene(sc)
        r.render()
        return {"rgb8": r.getImageRGB8(), "depth": r.getDepth(), "ids": r.getTriangleIds()}
    finally:
        r.close()


def _boxes(widths, heights, w, h, meshes=1):
    """Front-facing triangles whose bounding boxes are the given widths and
    heights, overlapping at random depths, one unit per pixel; spread over
    `meshes` renderables."""
    rng = np.random.default_rng(len(widths) * 100 + meshes)
    v = []
    for bw in widths:
        for bh in heights:
            x = rng.uniform(-w / 2, w / 2 - bw + 1)
            y = rng.uniform(-h / 2, h / 2 - bh + 1)
            z = -rng.uniform(2, 50, 3)
            m = rng.uniform(0, bw - 1)
            v.append([[x, y, z[0]], [x + bw - 1, y + 0.3, z[1]], [x + m, y + bh - 1, z[2]]])
    v = np.array(v, np.float32)
    sc = S.Scene()
    for part in np.array_split(v, meshes):
        idx = np.arange(3 * len(part), dtype=np.int32)
        nrm = np.tile(np.array([[0.2, 0.3, 1]], np.float32), (3 * len(part), 1))
        sc.add(S.TriMesh(part.reshape(-1, 3), nrm, idx, normalsI=idx,
                         material=S.Material(diffuse=rng.uniform(0.2, 1, 3), shininess=12)))
    st = FrameState(width=w, height=h, projection=pj.projection_ortho(-w / 2, w / 2, -h / 2, h / 2, 1, 60),
                    light=np.array([0.3, 0.4, 1], np.float32))
    return st, sc


@pytest.mark.parametrize("meshes", [1, 3])
def test_large_triangle_column_segments(product_lib, meshes):
    """Widths and heights on either side of the column segments (16 columns up
    to a width of 256, then 32, 48, ...) and row blocks of large triangles."""
    st, sc = _boxes((9, 15, 16, 17, 31, 33, 65, 255, 256, 257, 511, 513, 769, 1025, 1300), (8, 31, 32, 33, 65, 90), 1400,
                    100, meshes)
    _same(_render(st, sc), O.render(st, sc), "boxes")


def _skewed():
    m = np.array(pj.projection_perspective(-0.5, 0.5, -0.4, 0.4, 1, 50), np.float32).reshape(4, 4)
    m[0, 1] = 0.2
    return m


_PROJECTIONS = {
    "symmetric": lambda: pj.projection_perspective(-0.5, 0.5, -0.4, 0.4, 1, 50),
    "off_axis": lambda: pj.projection_perspective(-0.3, 0.6, -0.5, 0.2, 1, 50),
    "skewed": _skewed,
    "ortho": lambda: pj.projection_ortho(-4, 5, -3, 4, 1, 50),
}


def _awkward(shared: bool):
    """Triangles of 1 to 30 pixels, some through the near plane, some with a
    corner at z = 0, infinite, NaN or near the largest float."""
    rng = np.random.default_rng(12 + shared)
    n = 400
    c = np.stack([rng.uniform(-6, 6, n), rng.uniform(-5, 5, n), -rng.uniform(0.5, 40, n)], 1)
    v = (c[:, None] + rng.normal(0, 0.4, (n, 3, 3)) * [1, 1, 0.6]).astype(np.float32)
    for k, bad in enumerate((0.0, -0.0, np.inf, -np.inf, np.nan, 3e38, -3e38, 1e-40)):
        for axis in range(3):
            v[3 * k + axis + 40, rng.integers(0, 3), axis] = bad
    v[100, :, 2] = 0.0
    v = v.reshape(-1, 3)
    idx = np.arange(3 * n, dtype=np.int32)
    if shared:  # neighbouring triangles use each other's corners
        idx = np.concatenate([idx, np.roll(idx, 1), np.roll(idx, 2)]).astype(np.int32)
    nrm = rng.normal(size=(3 * n, 3)).astype(np.float32)
    sc = S.Scene()
    sc.add(S.TriMesh(v, nrm, idx, normalsI=idx, material=S.Material(shininess=8)))
    return sc


@pytest.mark.parametrize("shared", [False, True], ids=["soup", "shared"])
@pytest.mark.parametrize("projection", sorted(_PROJECTIONS))
def test_projection_forms(product_lib, projection, shared):
    """The short projection of perspective matrices without skew, its general
    form, and the corners that must take the general form."""
    st = FrameState(width=120, height=90, projection=_PROJECTIONS[projection](),
                    light=np.array([0.2, 0.4, 1], np.float32))
    sc = _awkward(shared)
    ref = O.render(st, sc)
    assert (ref["ids"] != 0xFFFFFFFF).sum() > 500
    got = _render(st, sc)
    assert np.array_equal(got["ids"], ref["ids"])
    assert np.array_equal(got["depth"].view(np.uint32), ref["depth"].view(np.uint32))


@pytest.mark.parametrize("small_max", [0, 64])
@pytest.mark.parametrize("tiling", [(4, 16, 64), (8, 8, 128), (16, 16, 256), (32, 2, 64), (64, 32, 256), (128, 8, 128),
                                    (256, 16, 256), (64, 64, 64)])
def test_batch_strips(product_lib, tiling, small_max):
    """The strips a tile is cut into (at most 256 pixels, rows of 4 to 256
    columns), at frame edges that cut tiles, strips and rows, for records
    narrower and wider than a strip."""
    from minirender_gb300 import workloads as W
    from minirender_gb300.batch import BatchRenderer
    items = [_boxes((9, 33, 257, 700), (8, 33, 90), 771, 101), W.config4_scene(3, 16, (131, 77)),
             _boxes((3, 12), (5, 17), 33, 31, 2), W.config1(64, 47)]
    br = BatchRenderer(0)
    try:
        br.ctx.set_batch_tiling(tiling[0], tiling[1], tiling[2], 64)
        br.ctx.set_batch_small_max(small_max)
        br.render(items)
        for k, (st, sc) in enumerate(items):
            _same(br.read(k), O.render(st, sc), f"scene {k}")
    finally:
        br.close()


@pytest.mark.parametrize("meshes", [1, 3])
def test_shared_indices_with_unused_tail(product_lib, meshes):
    """One index per corner for all attributes, with more vertices than
    normals and texcoords (the rest unused), under every set of attributes
    that the fragments read."""
    from minirender_gb300 import workloads as W
    st, sc = W.config2(level=3, width=150, height=110, tex_size=32)
    m = sc.children[0]
    extra = np.full((7, 3), np.nan, np.float32)
    verts = np.concatenate([m.vertices, extra])
    sc.children = []
    for k in range(meshes):
        xf = np.eye(4, dtype=np.float32)
        xf[0, 3] = 0.8 * (k - (meshes - 1) / 2)
        mat = S.Material(diffuse=(0.2 + 0.2 * k, 0.6, 0.5), shininess=0 if k == 1 else 9,
                         texture=m.material.texture if k != 2 else None)
        sc.add(S.TriMesh(verts, m.normals, m.indices, normalsI=m.indices, texcoords=m.texcoords,
                         texcoordsI=m.indices, material=mat, transform=xf))
    for lighting, texturing, point in ((True, True, False), (True, False, True), (False, True, False), (False, False, False)):
        st.lighting, st.texturing, st.light_is_point = lighting, texturing, point
        _same(_render(st, sc), O.render(st, sc), f"lighting {lighting}, texturing {texturing}, point {point}")


@pytest.mark.parametrize("noalloc", [False, True])
def test_record_shares(product_lib, noalloc):
    """More large triangles in one part of the triangle list than a share of
    the fixed record store holds (the rest is rasterised by the setup), beside
    parts with none; in the growing store every one finds room."""
    import test_zz_no_alloc as N
    st, sc = N._strips(5000, 640, 480, 9)
    m = sc.children[0]
    v = m.vertices.reshape(-1, 3, 3).copy()
    t = np.arange(len(v))
    v[(t // 32) % 16 > 2] *= np.float32([0.02, 0.02, 1])  # small ones outside three shares of sixteen
    v = np.concatenate([v, np.tile(v[:96], (120, 1, 1))])  # and the large ones of those, again and again
    idx = np.arange(3 * len(v), dtype=np.int32)
    nrm = np.tile(np.array([[0.2, 0.3, 1]], np.float32), (3 * len(v), 1))
    sc.children = [S.TriMesh(v.reshape(-1, 3), nrm, idx, normalsI=idx, material=m.material)]
    ref = O.render(st, sc)
    got = N._noalloc(st, sc, calls=1)[0] if noalloc else _render(st, sc)
    _same(got, ref, "strips")


def test_batches_of_growing_and_shrinking_frames(product_lib):
    """A batch leaves the visibility words empty for the next one; the words a
    larger batch adds (its buffer grown, maybe in place) are cleared first."""
    from minirender_gb300 import workloads as W
    from minirender_gb300.batch import BatchRenderer
    br = BatchRenderer(0)
    try:
        for w, h in ((64, 48), (65, 49), (400, 301), (31, 17), (801, 602), (801, 602)):
            item = W.config4_scene(w, 8, (w, h))
            br.render([item, item])
            ref = O.render(*item)
            for k in range(2):
                _same(br.read(k), ref, f"{w}x{h} scene {k}")
    finally:
        br.close()


def _share_of_warp(w):
    """layout.h's share_of_warp."""
    h = (w // 16 * 0x9E3779B1) & 0xFFFFFFFF
    h = ((h ^ (h >> 15)) * 0x2C1B3C6D) & 0xFFFFFFFF
    return (w ^ (h >> 28)) % 16


@pytest.mark.parametrize("noalloc", [False, True])
def test_overfull_record_shares(product_lib, noalloc):
    """Warps of 32 triangles, 29 of them large, in three shares of sixteen: each
    of these holds more than the fixed store has room for in a share, the last
    warp that finds room not for all of its own; the others hold one each.  In
    the growing store every large triangle has a record."""
    import test_zz_no_alloc as N
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    warps = max(16 * sms, 16 * 150)
    t = np.arange(32 * warps)
    share = np.array([_share_of_warp(w) for w in range(warps)])[t // 32]
    large = np.where(share < 3, t % 32 < 29, t % (32 * 97) == 5)
    per_share = np.bincount(share[large], minlength=16)
    cap = 32768 // 16  # of the fixed store
    assert per_share[:3].min() > cap and 0 < per_share[3:].max() < cap and cap % 29
    rng = np.random.default_rng(5)
    w, h = 320, 240
    size = np.where(large, 12.0, 1.6)[:, None]  # boxes of 13x13 and 2x2 or 3x3 pixels
    c = np.stack([rng.uniform(-w / 2, w / 2 - 13, t.size), rng.uniform(-h / 2, h / 2 - 13, t.size)], 1)
    z = -rng.uniform(2, 50, (t.size, 3, 1))
    v = np.concatenate([np.stack([c, c + size * [1, 0], c + size * [0.5, 1]], 1), z], 2).astype(np.float32)
    idx = np.arange(3 * t.size, dtype=np.int32)
    nrm = np.tile(np.array([[0.2, 0.3, 1]], np.float32), (3 * t.size, 1))
    sc = S.Scene()
    sc.add(S.TriMesh(v.reshape(-1, 3), nrm, idx, normalsI=idx, material=S.Material()))
    st = FrameState(width=w, height=h, projection=pj.projection_ortho(-w / 2, w / 2, -h / 2, h / 2, 1, 60),
                    light=np.array([0.3, 0.4, 1], np.float32))
    ref = O.render(st, sc)
    if noalloc:
        _same(N._noalloc(st, sc, calls=2)[1], ref, "fixed store")
        return
    r = Renderer(0)
    try:
        r.state = st
        r.setScene(sc)
        r.render()
        _same({"rgb8": r.getImageRGB8(), "depth": r.getDepth(), "ids": r.getTriangleIds()}, ref, "growing store")
        assert r.stats().binned == large.sum()
    finally:
        r.close()


@pytest.mark.parametrize("n,box,frame", [(600, 900, 1000), (900, 500, 600), (2500, 250, 300), (30000, 100, 400)])
def test_spilled_blocks(product_lib, n, box, frame):
    """Large triangles whose blocks pass the fixed store's list, from a few
    hundred spilled records (many warps on each) to more than there are warps,
    and with records whose first blocks found room."""
    import test_zz_no_alloc as N
    rng = np.random.default_rng(n)
    side = box * rng.uniform(0.6, 1, (n, 1))
    at = np.stack([rng.uniform(-frame / 2, frame / 2 - 0.6 * box, n), rng.uniform(-frame / 2, frame / 2 - 0.6 * box, n)], 1)
    third = rng.uniform(0, 1, (n, 1))
    z = -rng.uniform(2, 50, (n, 3, 1))
    v = np.concatenate([np.stack([at, at + side * [1, 0.02], at + side * np.concatenate([third, np.ones((n, 1))], 1)], 1), z], 2)
    idx = np.arange(3 * n, dtype=np.int32)
    nrm = np.tile(np.array([[0.2, 0.3, 1]], np.float32), (3 * n, 1))
    sc = S.Scene()
    sc.add(S.TriMesh(v.astype(np.float32).reshape(-1, 3), nrm, idx, normalsI=idx, material=S.Material()))
    st = FrameState(width=frame, height=frame, projection=pj.projection_ortho(-frame / 2, frame / 2, -frame / 2, frame / 2, 1, 60),
                    light=np.array([0.3, 0.4, 1], np.float32))
    ref = O.render(st, sc)
    _same(N._noalloc(st, sc, calls=2)[1], ref, "fixed store")
    r = Renderer(0)
    try:
        r.state = st
        r.setScene(sc)
        r.render()
        assert r.stats().bin_entries > 1 << 17  # blocks the fixed store lists
        _same({"rgb8": r.getImageRGB8(), "depth": r.getDepth(), "ids": r.getTriangleIds()}, ref, "growing store")
    finally:
        r.close()


@pytest.mark.parametrize("meshes", [1, 3])
@pytest.mark.parametrize("shared", [False, True], ids=["soup", "shared"])
@pytest.mark.parametrize("w,h", [(65536, 20), (20, 65536), (40000, 33)])
def test_frames_of_the_largest_sides(product_lib, w, h, shared, meshes):
    """Coordinates past 32767 (the small raster packs two into 32 bits) and
    triangles as long as the frame (column segments of thousands of columns)."""
    rng = np.random.default_rng(w + shared)
    n = 600
    small = np.arange(n) % 20 > 0
    size = np.stack([np.where(small, rng.uniform(1, 11, n), rng.uniform(0.1, 1, n) * w),
                     np.where(small, rng.uniform(1, 11, n), rng.uniform(0.1, 1, n) * h)], 1)
    at = np.stack([rng.uniform(-w / 2, w / 2, n), rng.uniform(-h / 2, h / 2, n)], 1)
    at[::3] = [w / 2, h / 2] - at[::3] % 12  # many in the last columns and rows
    at = np.where(small[:, None], at, np.minimum(at, [w / 2, h / 2] - size))
    z = -rng.uniform(2, 50, (n, 3, 1))
    v = np.concatenate([np.stack([at, at + size * [1, 0.1], at + size * [0.4, 1]], 1), z], 2).astype(np.float32)
    sc = S.Scene()
    for part in np.array_split(v, meshes):
        k = 3 * len(part)
        idx = np.arange(k, dtype=np.int32)
        if shared:
            idx = np.concatenate([idx, idx])
        nrm = np.tile(np.array([[0.2, 0.3, 1]], np.float32), (k, 1))
        sc.add(S.TriMesh(part.reshape(-1, 3), nrm, idx, normalsI=idx, material=S.Material()))
    st = FrameState(width=w, height=h, projection=pj.projection_ortho(-w / 2, w / 2, -h / 2, h / 2, 1, 60),
                    light=np.array([0.3, 0.4, 1], np.float32))
    ref = O.render(st, sc)
    drawn = np.nonzero(ref["ids"] != 0xFFFFFFFF)
    assert drawn[1 if w > h else 0].max() > 0.99 * max(w, h)
    _same(_render(st, sc), ref, "frame")
    from minirender_gb300.batch import BatchRenderer
    br = BatchRenderer(0)
    try:
        br.render([(st, sc), (st, sc)])
        for k in range(2):
            _same(br.read(k), ref, f"batch scene {k}")
    finally:
        br.close()


@pytest.mark.parametrize("shared", [False, True], ids=["soup", "shared"])
@pytest.mark.parametrize("hollow", [False, True], ids=["empty", "vertices_only"])
def test_runs_of_empty_renderables(product_lib, shared, hollow):
    """Renderables without triangles (with and without vertices) between others
    of 1 to 40: the search for a triangle's or vertex's renderable steps over
    32 of them and searches past more."""
    rng = np.random.default_rng(9 + shared)
    nothing = np.zeros((5 if hollow else 0, 3), np.float32)
    sc = S.Scene()
    for run in (0, 1, 30, 31, 32, 33, 64, 500, 0, 0, 2):
        for _ in range(run):
            sc.add(S.TriMesh(nothing, nothing, np.zeros(0, np.int32), material=S.Material()))
        for n in (1, 2, 40, 1):
            c = np.concatenate([rng.uniform(-70, 60, (n, 1, 2)), -rng.uniform(2, 50, (n, 1, 1))], 2)
            v = (c + [[0, 0, 0], [9, 1, 0], [3, 8, 0]]).astype(np.float32).reshape(-1, 3)
            idx = np.arange(3 * n, dtype=np.int32)
            idx = np.concatenate([idx] * (3 if shared else 1))
            nrm = rng.normal(size=(3 * n, 3)).astype(np.float32)
            sc.add(S.TriMesh(v, nrm, idx, normalsI=idx, material=S.Material(diffuse=rng.uniform(0.2, 1, 3))))
    st = FrameState(width=160, height=120, projection=pj.projection_ortho(-80, 80, -60, 60, 1, 60),
                    light=np.array([0.3, 0.4, 1], np.float32))
    ref = O.render(st, sc)
    _same(_render(st, sc), ref, "frame")
    from minirender_gb300.batch import BatchRenderer
    br = BatchRenderer(0)
    try:
        br.render([(st, sc), (st, sc)])
        for k in range(2):
            _same(br.read(k), ref, f"batch scene {k}")
    finally:
        br.close()
