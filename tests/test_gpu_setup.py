"""Triangle set-up where its coverage pretest and its index fetch decide:
boxes of 1 to 6 pixels a side, on the target's edges and across tiles,
coordinates far outside, infinite and NaN, index buffers that end inside a
triangle, 16- and 32-bit indices — batched and per draw, against the oracle,
byte for byte."""
import ctypes

import numpy as np
import pytest

import cpvulkan_gb300 as c

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batched", [0, 1])
@pytest.mark.parametrize("odd", ["none", "far", "inf", "nan"])
@pytest.mark.parametrize("size", [0.5, 1.5, 3.0, 4.5])
@pytest.mark.parametrize("index,cut", [(None, 0), (np.uint16, 0), (np.uint16, 9), (np.uint32, 18)])
def test_setup(gpu_ctx, oracle, monkeypatch, batched, odd, size, index, cut):
    monkeypatch.setenv("CPV_BATCH", str(batched))
    monkeypatch.setenv("CPV_BATCH_MIN_DRAWS", "1")
    monkeypatch.setenv("CPV_DIRECT_PRIMS", "0")
    width, height, tris = 61, 45, 2000
    indices = None  # kept alive while the scene points at it
    scene = c.Scene(c.PROGRAM, 5, [c.PROGRAM_CUBE, 0x10 | 0x20 | (0x1000 if index else 0), width, height, tris])
    h = c.SceneHeader.from_address(scene.ptr)
    v = np.ctypeslib.as_array(ctypes.cast(h.vertex_data, ctypes.POINTER(ctypes.c_float)), (h.vertex_bytes // 32, 8))
    rng = np.random.default_rng(11)
    t = v[: tris * 3].reshape(tris, 3, 8)
    centre = rng.uniform(-1.1, 1.1, (tris, 1, 2))
    xy = centre + rng.uniform(-size, size, (tris, 3, 2)) / [width, height]
    if odd != "none":
        value = {"far": 1e12, "inf": np.inf, "nan": np.nan}[odd]
        which = rng.random((tris, 3, 2))
        xy = np.where(which < 0.01, value, np.where(which > 0.99, -value, xy))
    t[:, :, :2] = (xy * t[:, :, 3:4]).astype(np.float32)
    if index is not None:
        old = np.ctypeslib.as_array(ctypes.cast(h.index_data, ctypes.POINTER(ctypes.c_uint16)), (h.index_bytes // 2,))
        indices = old.astype(index)
        h.index_data, h.index_type, h.index_bytes = indices.ctypes.data, 1 if index is np.uint32 else 0, indices.nbytes - cut
    r = c.Renderer(gpu_ctx, scene)
    r.render(1)
    colour, depth = r.readback()
    r.close()
    want, want_depth, _ = oracle.render(scene)
    del indices
    assert np.array_equal(colour, want)
    nan = np.isnan(depth.view(np.float32)) & np.isnan(want_depth.view(np.float32))
    assert ((depth.view(np.uint32) == want_depth.view(np.uint32)) | nan).all()
