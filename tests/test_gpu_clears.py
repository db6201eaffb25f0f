"""Load-op clears made by the first draw's raster: targets of one tile, ragged
tiles and many tiles that geometry covers wholly, in a corner or not at all,
in texels of 1 to 16 bytes and every depth format, per draw (walked whole,
filtered, binned), batched, and with blending that reads the cleared colour
— against the oracle, byte for byte, over three frames."""
import ctypes

import numpy as np
import pytest

import cpvulkan_gb300 as c

pytestmark = pytest.mark.gpu
MODES = {"direct": {"CPV_DIRECT_PRIMS": "1000000", "CPV_DIRECT_LIMIT": "4000000000"}, "filter": {"CPV_DIRECT_PRIMS": "0", "CPV_FILTER_PRIMS": "1000000"},
         "lists": {"CPV_DIRECT_PRIMS": "0", "CPV_FILTER_PRIMS": "0"}, "batched": {"CPV_BATCH_MIN_DRAWS": "1"}}


def place(scene, where):
    h = c.SceneHeader.from_address(scene.ptr)
    v = np.ctypeslib.as_array(ctypes.cast(h.vertex_data, ctypes.POINTER(ctypes.c_float)), (h.vertex_bytes // 32, 8))
    if where == "corner":
        v[:, :2] = (v[:, :2] / v[:, 3:4] * 0.1 - 0.85) * v[:, 3:4]
    elif where == "nowhere":
        v[:, 0] += 40 * v[:, 3]


@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("where", ["everywhere", "corner", "nowhere"])
@pytest.mark.parametrize("fmt,depth,blend,width,height", [(9, 0x8, 0, 16, 16), (0, 0x18, 0x20, 17, 33), (97, 0x10, 0x20, 100, 70), (109, 0x18, 0, 65, 15),
                                                          (77, 0, 0x20, 48, 64), (0, 0x40000010, 0, 50, 50)])
def test_clears(gpu_ctx, oracle, monkeypatch, mode, where, fmt, depth, blend, width, height):
    for k, v in MODES[mode].items():
        monkeypatch.setenv(k, v)
    scene = c.Scene(c.PROGRAM, 4, [c.PROGRAM_CUBE, depth | blend | 0x1000, width, height, 70, 0, fmt])
    place(scene, where)
    r = c.Renderer(gpu_ctx, scene)
    got = []
    for _ in range(3):  # eager, captured, replayed: each starts from the last one's image
        r.render(1)
        got.append(r.readback())
    r.close()
    colour, dep, _ = oracle.render(scene)
    for g_colour, g_depth in got:
        if scene.color_format:
            assert np.array_equal(g_colour, colour)
        if dep is not None:
            keep = 5 if scene.depth_format == c.VK_FORMAT_D32_SFLOAT_S8_UINT else dep.shape[2]  # the texel's padding is not compared
            assert np.array_equal(g_depth[..., :keep], dep[..., :keep])
