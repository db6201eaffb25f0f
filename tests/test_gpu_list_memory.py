"""The per-draw bin lists: what a draw of many small triangles holds of the
device's memory, the fallback of a draw whose pairs do not fit (asserted to
have run), and their growth for the submissions after it. Images against the
oracle, bit for bit."""
import ctypes

import numpy as np
import pytest

import cpvulkan_gb300 as c
from tests.test_gpu_binning import SIZES

pytestmark = pytest.mark.gpu


def _lists(ctx):
    out = (ctypes.c_uint64 * 2)()
    lib = ctypes.CDLL(c.ICD_PATH)
    lib.cpv_queue_list_stats.argtypes = [ctypes.c_void_p, ctypes.c_uint64 * 2]
    lib.cpv_queue_list_stats(ctx.queue, out)
    return out[0], out[1]


def _frames(ctx, scene, n):
    r = c.Renderer(ctx, scene)
    out = []
    for _ in range(n):
        r.render(1)
        out.append(r.readback())
    r.close()
    return out


def _equal(frames, oracle, scene):
    colour, depth, _ = oracle.render(scene)
    return all(np.array_equal(a, colour) and np.array_equal(b, depth) for a, b in frames)


@pytest.mark.parametrize("tris,width,height,tile", SIZES)
def test_lists_that_hold_nothing(native, oracle, monkeypatch, tris, width, height, tile):
    for k, v in {"CPV_DIRECT_PRIMS": "0", "CPV_FILTER_PRIMS": "0", "CPV_LIST_CAPACITY": "0", "CPV_TILE": tile}.items():
        monkeypatch.setenv(k, v)
    ctx = c.Context()
    try:
        scene = c.Scene(c.PROGRAM, 4, [c.PROGRAM_CUBE, 0x10 | 0x20 | 0x1000, width, height, tris])
        frames = _frames(ctx, scene, 3)
        assert _lists(ctx)[1] > 0  # no pair fitted, so every frame filtered
    finally:
        ctx.close()
    assert _equal(frames, oracle, scene)


@pytest.mark.parametrize("tris,width,height,tile", [(700, 1041, 1030, "8"), (1100, 640, 360, "16")])
def test_lists_grow_after_a_draw_that_needs_more(native, oracle, monkeypatch, tris, width, height, tile):
    for k, v in {"CPV_DIRECT_PRIMS": "0", "CPV_FILTER_PRIMS": "0", "CPV_LIST_START": "1", "CPV_TILE": tile}.items():
        monkeypatch.setenv(k, v)
    ctx = c.Context()
    try:
        scene = c.Scene(c.PROGRAM, 4, [c.PROGRAM_CUBE, 0x10 | 0x20 | 0x1000, width, height, tris])
        frames = _frames(ctx, scene, 1)
        held, need = _lists(ctx)  # after the read-back's submission, which grows the lists
        assert held >= need > 1024  # (the smallest allocation: the frame did not fit)
        r = c.Renderer(ctx, scene)  # eager, captured, replayed
        for _ in range(3):
            r.render(1)
            frames.append(r.readback())
        r.close()
        assert _lists(ctx) == (held, need)
    finally:
        ctx.close()
    assert _equal(frames, oracle, scene)


def test_a_graph_is_captured_again_when_lists_grow(native, oracle, monkeypatch):
    """A replayed command buffer that does not fit leaves its need too."""
    for k, v in {"CPV_DIRECT_PRIMS": "0", "CPV_FILTER_PRIMS": "0", "CPV_LIST_START": "1"}.items():
        monkeypatch.setenv(k, v)
    ctx = c.Context()
    try:
        scene = c.Scene(c.PROGRAM, 4, [c.PROGRAM_CUBE, 0x10 | 0x20 | 0x1000, 640, 360, 1100])
        monkeypatch.setenv("CPV_LIST_CAPACITY", "1")
        r = c.Renderer(ctx, scene)
        frames = []
        for step in range(8):
            if step == 4:
                monkeypatch.delenv("CPV_LIST_CAPACITY")
            r.render(1)
            frames.append(r.readback())
        r.close()
        held, need = _lists(ctx)
        assert 0 < need <= held
    finally:
        ctx.close()
    assert _equal(frames, oracle, scene)


def test_memory_of_many_small_triangles(native):
    """70000 triangles over 1024 bins: lists of at most 2^23 pairs, 64 MiB.
    (Room for every primitive in every bin took 512 MiB.)"""
    ctx = c.Context()
    try:
        scene = c.Scene(c.PROGRAM, 3, [c.PROGRAM_CUBE, 0x10, 2048, 2048, 70000])
        h = c.SceneHeader.from_address(scene.ptr)
        v = np.ctypeslib.as_array(ctypes.cast(h.vertex_data, ctypes.POINTER(ctypes.c_float)), (h.vertex_bytes // 32, 8))
        v[:, :2] *= 0.01
        _frames(ctx, scene, 2)
        held, need = _lists(ctx)
        assert 70000 < held <= 1 << 23 and need == 0
    finally:
        ctx.close()
