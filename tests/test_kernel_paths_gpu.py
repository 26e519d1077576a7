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
    """Widths and heights on either side of the column segments (32 columns up
    to a width of 512, then 64, 96, ...) and row blocks of large triangles."""
    st, sc = _boxes((9, 31, 32, 33, 64, 65, 511, 512, 513, 545, 1025, 1300), (8, 31, 32, 33, 65, 90), 1400, 100, meshes)
    _same(_render(st, sc), O.render(st, sc), "boxes")
