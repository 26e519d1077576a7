"""The Renderer mirror's outputs are those of the frame its first getter read,
also when its context renders another frame before the other getters, or is
closed."""
import numpy as np
import pytest

from minirender_gb300 import abi
from minirender_gb300 import workloads as W
from minirender_gb300.renderer import Renderer
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("then", ["render", "close"])
def test_outputs_of_one_frame(product_lib, then):
    (st, sc), (st2, sc2) = W.config1(96, 64), W.config4_scene(5, 8, (130, 70))
    ref = O.render(st, sc)
    r, other = Renderer(0), Renderer(0)
    try:
        r.state = st
        r.setScene(sc)
        r.render()
        rgb8 = r.getImageRGB8()
        if then == "render":
            other.ctx.close()
            other.ctx, other.state = r.ctx, st2
            other.setScene(sc2)
            other.render()
            assert np.array_equal(other.getTriangleIds(), O.render(st2, sc2)["ids"])
        else:
            r.ctx.close()
        assert np.array_equal(r.getTriangleIds(), ref["ids"])
        assert np.array_equal(r.getDepth().view(np.uint32), ref["depth"].view(np.uint32))
        assert np.abs(rgb8.astype(int) - ref["rgb8"].astype(int)).max() <= 1
        assert r.getImage().shape == (64, 96, 3) and r.getImageRGB8() is rgb8
    finally:
        other.close()
        r.close()
