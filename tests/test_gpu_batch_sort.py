"""The batched binning (pair emission, radix sort by tile) where its shape
changes: one tile, the most tiles one digit sorts and one row more, ragged
targets; few pairs, primitives on more tiles than one lane writes, whole
chunks and their remainders, several chunks of set-up blocks, blocks without
pairs, no pair at all and more pairs than the buffers hold — against the
oracle, byte for byte."""
import ctypes

import numpy as np
import pytest

import cpvulkan_gb300 as c

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(16, 16), (512, 512), (528, 512), (1000, 700)])
@pytest.mark.parametrize("tris,scale,shift", [(1, 1.0, 0.0), (40, 1.0, 0.0), (257, 0.3, 0.0), (30000, 0.05, 0.3), (600000, 0.004, 0.5), (300, 1.0, 50.0)])
@pytest.mark.parametrize("capacity", [0, 100])
def test_batch_sort(gpu_ctx, oracle, monkeypatch, width, height, tris, scale, shift, capacity):
    monkeypatch.setenv("CPV_BATCH_MIN_DRAWS", "1")
    monkeypatch.setenv("CPV_TILE", "16")
    if capacity:
        if tris > 30000:
            pytest.skip("every tile scans every primitive")
        monkeypatch.setenv("CPV_BATCH_PAIR_CAPACITY", str(capacity))
    scene = c.Scene(c.PROGRAM, 9, [c.PROGRAM_CUBE, 0x10 | 0x20, width, height, tris])
    h = c.SceneHeader.from_address(scene.ptr)
    v = np.ctypeslib.as_array(ctypes.cast(h.vertex_data, ctypes.POINTER(ctypes.c_float)), (h.vertex_bytes // 32, 8))
    v[:, :2] = v[:, :2] * scale + shift * v[:, 3:4]
    v[: len(v) // 4, 0] += 40 * v[: len(v) // 4, 3] * (tris > 1000)  # whole set-up blocks off screen
    r = c.Renderer(gpu_ctx, scene)
    got = []
    for _ in range(2):
        r.render(1)
        got.append(r.readback())
    r.close()
    colour, depth, _ = oracle.render(scene)
    for g_colour, g_depth in got:
        assert np.array_equal(g_colour, colour)
        assert np.array_equal(g_depth, depth)
