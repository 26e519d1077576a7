"""Which frame the Renderer mirror's outputs belong to, with a fake library
that numbers its frames: the first getter decides, whatever the context
renders afterwards; and contexts are released whatever a read answers."""
import numpy as np
import pytest

from minirender_gb300 import abi, capi
from minirender_gb300 import workloads as W
from minirender_gb300.renderer import Renderer


class FakeLib:
    """mr_render counts frames; mr_read fills every array with the frame's
    number; `fail` is the status of the named calls."""

    def __init__(self):
        self.frames, self.hw, self.reads, self.destroyed, self.fail = 0, None, [], 0, {}

    def __getattr__(self, name):  # uploads, updates, frees
        return lambda *a: self.fail.get(name, 0)

    def mr_create(self, device, out):
        out._obj.value = 1
        return 0

    def mr_destroy(self, h):
        self.destroyed += 1
        return 0

    def mr_last_error(self, h):
        return b"fake"

    def mr_render(self, h, frame, rs, n, outputs):
        rc = self.fail.get("mr_render", 0)
        if rc == 0:
            self.frames += 1
            self.hw = (frame._obj.height, frame._obj.width)
        return rc

    def mr_get_outputs(self, h, o):
        if self.hw is None:
            return abi.MR_E_INVALID
        o._obj.height, o._obj.width = self.hw
        o._obj.rgb8 = o._obj.depth = o._obj.rgb_f32 = o._obj.tri_id = 1
        return 0

    def mr_read(self, h, rgb8, depth, image, ids, normals):
        rc = self.fail.get("mr_read", 0)
        self.reads.append([n for n, p in zip(("rgb8", "depth", "image", "ids", "normals"),
                                             (rgb8, depth, image, ids, normals)) if p])
        if rc == 0:
            H, W_ = self.hw
            import ctypes as C
            for p, t, k in ((rgb8, C.c_uint8, 3), (depth, C.c_float, 1), (image, C.c_float, 3), (ids, C.c_uint32, 1)):
                if p:
                    np.ctypeslib.as_array((t * (H * W_ * k)).from_address(p))[:] = self.frames
        return rc


@pytest.fixture
def fake(monkeypatch, product_lib):
    f = FakeLib()
    f.mr_collect_shapes = product_lib.mr_collect_shapes
    made, init = [], capi.Context.__init__

    def keep(self, device=0):
        init(self, device)
        made.append(self)

    monkeypatch.setattr(capi.Context, "__init__", keep)
    monkeypatch.setattr(capi, "lib", lambda: f)
    yield f
    for c in made:  # nothing of the fake's reaches the library
        c.h = None


def _renderer():
    r = Renderer(0)
    r.state, sc = W.config1(8, 6)
    r.setScene(sc)
    return r


GETTERS = {"rgb8": "getImageRGB8", "depth": "getDepth", "image": "getImage", "ids": "getTriangleIds"}


def _frames(r):
    return {k: int(np.unique(getattr(r, g)()).item()) for k, g in GETTERS.items()}


@pytest.mark.parametrize("first", list(GETTERS.values()))
def test_outputs_of_one_frame_after_another_render_on_the_context(fake, first):
    r = _renderer()
    r.render()
    getattr(r, first)()
    r.ctx.render(*r.prepare(), abi.MR_OUT_DEFAULT)
    r.ctx.render(*r.prepare(), abi.MR_OUT_DEFAULT)
    assert _frames(r) == dict.fromkeys(GETTERS, 1)
    r.render()
    assert _frames(r) == dict.fromkeys(GETTERS, 4)


def test_outputs_are_the_contexts_frame_when_first_asked_for(fake):
    r = _renderer()
    r.render()
    r.ctx.render(*r.prepare(), abi.MR_OUT_DEFAULT)
    assert _frames(r) == dict.fromkeys(GETTERS, 2)


def test_what_could_not_be_read_is_of_no_other_frame(fake):
    """After a read of the rest that fails, the outputs not read are gone, not
    the next frame's."""
    r = _renderer()
    r.render()
    r.getDepth()
    fake.fail["mr_read"] = abi.MR_E_CUDA
    r.ctx.render(*r.prepare(), abi.MR_OUT_DEFAULT)
    del fake.fail["mr_read"]
    assert int(np.unique(r.getDepth()).item()) == 1
    with pytest.raises(KeyError):
        r.getImage()
    r.render()
    assert _frames(r) == dict.fromkeys(GETTERS, 3)


def test_a_render_reads_nothing_of_the_frame_it_replaces(fake):
    r = _renderer()
    for _ in range(3):
        r.render()
        r.getDepth()
    assert fake.reads == [["depth"]] * 3


def test_outputs_stay_after_a_render_that_fails(fake):
    r = _renderer()
    r.render()
    r.getDepth()
    r.state.width = 99
    fake.fail["mr_render"] = abi.MR_E_INVALID
    with pytest.raises(capi.MRError):
        r.render()
    # arrays of the frame that was rendered, not of the one that was refused
    assert r.getImageRGB8().shape == (6, 8, 3)
    assert _frames(r) == dict.fromkeys(GETTERS, 1)
    del fake.fail["mr_render"]
    with pytest.raises(capi.MRError):
        fake.fail["mr_render"] = abi.MR_E_INVALID
        r.ctx.render(*r.prepare(), abi.MR_OUT_DEFAULT)
    assert _frames(r) == dict.fromkeys(GETTERS, 1)


@pytest.mark.parametrize("closer", ["renderer", "context"])
def test_outputs_after_close(fake, closer):
    r = _renderer()
    r.render()
    r.getDepth()
    (r if closer == "renderer" else r.ctx).close()
    assert fake.destroyed == 1
    assert _frames(r) == dict.fromkeys(GETTERS, 1)


def test_close_releases_the_context_when_a_read_fails(fake):
    r = _renderer()
    r.render()
    r.getDepth()
    fake.fail["mr_read"] = abi.MR_E_CUDA
    r.close()
    assert fake.destroyed == 1 and r.ctx.h is None
    assert int(np.unique(r.getDepth()).item()) == 1
    c = capi.Context(0)

    class Reader:
        def rest(self):
            raise MemoryError

    reader = Reader()
    c.hold(reader.rest)
    with pytest.raises(MemoryError):
        c.close()
    assert fake.destroyed == 2 and c.h is None


def test_a_first_read_that_fails_keeps_nothing(fake):
    r = _renderer()
    r.render()
    fake.fail["mr_read"] = abi.MR_E_BAD_INDEX
    for _ in range(2):
        with pytest.raises(capi.MRError):
            r.getDepth()
    r.ctx.render(*r.prepare(), abi.MR_OUT_DEFAULT)
    del fake.fail["mr_read"]
    assert _frames(r) == dict.fromkeys(GETTERS, 2)
