"""What a batch slot keeps from one batch to the next -- its visibility words,
which a batch leaves empty -- when a batch was only recorded into the caller's
graph, when small triangles are switched off and on again, and when a recorded
batch is replayed between others; against the oracle."""
import ctypes as C

import numpy as np
import pytest

from minirender_gb300 import abi, capi
from minirender_gb300 import workloads as W
from minirender_gb300.batch import BatchRenderer
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _same(got, want, what):
    assert np.array_equal(got["ids"], want["ids"]), f"{what}: visible ids differ"
    assert np.array_equal(got["depth"].view(np.uint32), want["depth"].view(np.uint32)), f"{what}: depth"
    d = np.abs(got["rgb8"].astype(np.int16) - want["rgb8"].astype(np.int16))
    assert d.max(initial=0) <= 1, f"{what}: rgb8"


class _Device:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (ptr, False), "version": 3}


def _wipe(ctx, scene, value):
    """Overwrites a scene's outputs of the last batch on the device."""
    import torch
    o = abi.mr_outputs()
    assert capi.lib().mr_get_batch_outputs(ctx.h, scene, C.byref(o)) == 0
    px = o.width * o.height
    for ptr, n in ((o.rgb8, 3 * px), (o.depth, 4 * px), (o.tri_id, 4 * px)):
        torch.as_tensor(_Device(ptr, n), device="cuda").fill_(value)
    torch.cuda.synchronize()


def test_words_after_a_batch_that_was_only_recorded(product_lib):
    """A batch recorded into the caller's graph and not run leaves the words of
    its new buffer undefined; a batch without words (small_max 0) in between
    says nothing about them, so the next one with words clears them.  The
    recorded batch replays to the same pixels."""
    import torch
    items = [W.config4_scene(1, 12, (150, 110)), W.config1(97, 64)]
    refs = [O.render(*i) for i in items]
    br = BatchRenderer(0)
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()

    def check(what):
        for k, ref in enumerate(refs):
            _same(br.read(k), ref, f"{what}, scene {k}")

    try:
        br.ctx.set_stream(stream.cuda_stream)
        br.ctx.set_batch_graphs(False)  # the caller's graph instead of the library's
        args = br.prepare(items)
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            br.ctx.render_batch(*args)
        br.ctx.set_batch_small_max(0)
        br.render(items)
        check("small_max 0")
        br.ctx.set_batch_small_max(64)
        br.render(items)
        check("small_max 64")
        for k in range(2):
            for s in range(len(items)):
                _wipe(br.ctx, s, 0x55)
            with torch.cuda.stream(stream):
                graph.replay()
            check(f"replay {k}")
        br.render(items)
        check("after the replays")
    finally:
        torch.cuda.synchronize()
        br.close()


def test_small_max_set_between_a_batch_and_its_read(product_lib):
    """The words belong to the batch as it was staged: a small_max set before
    the batch is read (and, its record list too short, run again) changes the
    next batch only."""
    from test_kernel_paths_gpu import _boxes
    # 1200 triangles over nearly all of 1200 tiles: more pairs than the list
    # first holds (2^20); the others are small
    st, sc = _boxes([3, 5, 7] * 10 + [312] * 30, [3, 6] * 10 + [235] * 40, 320, 240)
    ref = O.render(st, sc)
    br = BatchRenderer(0)
    try:
        br.ctx.set_batch_tiling(4, 16, 64, 64)
        for first, then in ((64, 0), (0, 64), (64, 64)):
            br.ctx.set_batch_small_max(first)
            br.render([(st, sc)])
            br.ctx.set_batch_small_max(then)
            _same(br.read(0), ref, f"{first} then {then}")
        assert br.ctx.batch_stats().bin_entries > 1 << 20
    finally:
        br.close()
