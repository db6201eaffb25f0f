"""The sparse schedule's choice between per-pixel lists and the immediate
walk: batches of small and large primitives and slivers whose areas lie below
and above the limit, pixels whose lists overflow on either side of it, with
depth, stencil and blending, per draw (filtered and by lists) and batched,
tiles of 8 to 32 pixels — against the oracle, byte for byte."""
import ctypes

import numpy as np
import pytest

import cpvulkan_gb300 as c

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["filter", "lists", "batched"])
@pytest.mark.parametrize("tile", ["8", "16", "32"])
@pytest.mark.parametrize("variant", [0x20, 0x10 | 0x20, 0x18])
@pytest.mark.parametrize("tris,big,size", [(40, 0.5, 2.0), (300, 0.1, 0.3), (300, 0.7, 0.3), (700, 0.4, 1.0), (700, 1.0, 0.2)])
def test_dense(gpu_ctx, oracle, monkeypatch, mode, tile, variant, tris, big, size):
    monkeypatch.setenv("CPV_TILE", tile)
    monkeypatch.setenv("CPV_DIRECT_PRIMS", "0")
    monkeypatch.setenv("CPV_FILTER_PRIMS", "0" if mode == "lists" else "1000000")
    if mode == "batched":
        monkeypatch.setenv("CPV_BATCH_MIN_DRAWS", "1")
    width, height = 53, 37
    scene = c.Scene(c.PROGRAM, 8, [c.PROGRAM_CUBE, variant, width, height, tris])
    h = c.SceneHeader.from_address(scene.ptr)
    v = np.ctypeslib.as_array(ctypes.cast(h.vertex_data, ctypes.POINTER(ctypes.c_float)), (h.vertex_bytes // 32, 8))
    t = v[: tris * 3].reshape(tris, 3, 8)
    rng = np.random.default_rng(5)
    scale = np.where(rng.random((tris, 1, 1)) < big, size, 0.06) * np.where(rng.random((tris, 1, 1)) < 0.2, [[[1.0, 0.02]]], [[[1.0, 1.0]]])
    xy = rng.uniform(-0.9, 0.9, (tris, 1, 2)) + rng.uniform(-1.0, 1.0, (tris, 3, 2)) * scale
    t[:, :, :2] = (xy * t[:, :, 3:4]).astype(np.float32)
    r = c.Renderer(gpu_ctx, scene)
    r.render(1)
    colour, depth = r.readback()
    r.close()
    want, want_depth, _ = oracle.render(scene)
    assert np.array_equal(colour, want)
    if want_depth is not None:
        keep = 5 if scene.depth_format == c.VK_FORMAT_D32_SFLOAT_S8_UINT else want_depth.shape[2]  # the texel's padding is not compared
        assert np.array_equal(depth[..., :keep], want_depth[..., :keep])
