"""The render server's budget covers what a batch holds for the vertex pass:
meshes with shared vertices are charged for its buffers, and a batch that also
holds soups runs it only where the budget makes up for them."""
import numpy as np
import pytest

from minirender_gb300 import abi, capi
from minirender_gb300 import workloads as W
from minirender_gb300.scene import Material, Scene, TriMesh
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FRAME = 64 * 48


@pytest.fixture(scope="module")
def ctx(product_lib):
    c = capi.Context(0)
    yield c
    c.close()


def _shared(level, own_normals=False):
    """An icosphere: two triangles a vertex, one index a corner for every
    attribute or (own_normals) an index array of its own for the normals."""
    st, sc = W.config2(level=level, width=64, height=48, tex_size=8)
    m = sc.children[0]
    return st, TriMesh(m.vertices, m.normals, m.indices, normalsI=m.indices.copy() if own_normals else m.indices,
                       material=Material())


def _soup(n):
    st, sc = W.config3(n_tris=n, width=64, height=48, seed=3)
    m = sc.children[0]
    return st, TriMesh(m.vertices, m.normals, m.indices, normalsI=m.normalsI, material=Material())


def _charges(m):
    """(resident mesh, request without the vertex pass, the pass) in bytes, as
    the server counts them; the last bytes (tables of one renderable, scene
    and tiles) are left to _SLACK."""
    T, V, N = m.n_triangles, len(m.vertices), len(m.normals)
    records = 128 * T if 3 * T < 2 * V else 0
    mesh = 12 * V + 12 * N + 36 * T + T // 8 + 4096 + records
    unified = m.normalsI.ctypes.data == m.indices.ctypes.data
    run = 48 * V + 16 * T + (0 if unified else 16 * N) if 3 * T >= 2 * V else 24 * V + 16 * N
    return mesh, (8 + 3 + 4 + 4) * FRAME + 144 * T, run


_SLACK = 4096


def _oracle(st, mesh):
    sc = Scene()
    sc.add(mesh)
    return O.render(st, sc)


def _buffers():
    return {"rgb8": np.zeros((48, 64, 3), np.uint8), "depth": np.zeros((48, 64), np.float32),
            "ids": np.zeros((48, 64), np.uint32)}


def _same(a, b):
    return (np.array_equal(a["ids"], b["ids"]) and
            np.array_equal(a["depth"].view(np.uint32), b["depth"].view(np.uint32)) and
            np.abs(a["rgb8"].astype(int) - b["rgb8"].astype(int)).max() <= 1)


@pytest.mark.parametrize("own_normals", [False, True], ids=["one_index", "own_normals"])
def test_shared_vertices_are_charged_for_the_pass(ctx, own_normals):
    """48 bytes a vertex, 16 a triangle, and 16 a normal where normals have
    indices of their own: a budget short of that is refused, one that holds it
    renders, and soups are charged as without the pass."""
    from minirender_gb300.server import RenderServer
    st, m = _shared(6, own_normals)
    own = sum(_charges(m))
    for budget, fits in ((own - 1, False), (own + _SLACK, True)):
        srv = RenderServer(ctx, budget_bytes=budget, slots=1, max_batch=4)
        try:
            out = _buffers()
            if fits:
                assert srv.wait(srv.submit(st, m, mesh_key=1, out=out)).status == 0
                assert _same(out, _oracle(st, m))
            else:
                with pytest.raises(capi.MRError) as e:
                    srv.submit(st, m, mesh_key=1, out=out)
                assert e.value.code == abi.MR_E_BUDGET
        finally:
            srv.close()
    st, m = _soup(30_000)
    srv = RenderServer(ctx, budget_bytes=sum(_charges(m)) + _SLACK, slots=1, max_batch=4)
    try:
        out = _buffers()
        assert srv.wait(srv.submit(st, m, mesh_key=2, out=out)).status == 0
        assert _same(out, _oracle(st, m))
    finally:
        srv.close()


@pytest.mark.parametrize("room", [1 << 16, 64 << 20], ids=["no_room", "room"])
def test_soups_among_shared_vertices(ctx, room):
    """A batch of both kinds, in a budget with and without room for the soups'
    share of the vertex pass: the same pixels, and the budget holds."""
    from minirender_gb300.server import RenderServer
    reqs = [_shared(6), _soup(60_000)]
    refs = [_oracle(st, m) for st, m in reqs]
    budget = sum(sum(_charges(m)) for _, m in reqs) + room
    srv = RenderServer(ctx, budget_bytes=budget, slots=1, max_batch=2)
    try:
        sizes = []
        for rep in range(4):
            tickets = []
            for k in (0, 1, 0, 1, 0, 1):
                out = _buffers()
                st, m = reqs[k]
                tickets.append((k, out, srv.submit(st, m, mesh_key=10 + k, out=out)))
                assert srv.stats()["committed_bytes"] <= budget
            for k, out, t in tickets:
                info = srv.wait(t)
                sizes.append(info.batch_size)
                assert info.status == 0 and _same(out, refs[k])
        assert max(sizes) == 2
        s = srv.stats()
        assert s["committed_bytes"] == s["resident_bytes"] <= budget
    finally:
        srv.close()
