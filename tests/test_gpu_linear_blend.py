"""Blending of flat colours through every path a pipeline can take (linear
constants in registers, blend tables, the general blend) against the oracle,
byte for byte: blend operations and factors, write masks, colours outside
[0, 1], infinite and NaN, byte orders, lines and points, and targets of one
block, ragged blocks and several tiles."""
import ctypes

import numpy as np
import pytest

import cpvulkan_gb300 as c

pytestmark = pytest.mark.gpu
# (src colour, dst colour, op, src alpha, dst alpha, op), 0: no blending
EQUATIONS = {
    "none": None, "src over": (6, 7, 0, 1, 7, 0), "additive": (1, 1, 0, 1, 1, 0), "subtract": (6, 1, 1, 1, 7, 2), "reverse subtract": (2, 12, 2, 6, 3, 1),
    "constants": (10, 13, 0, 12, 11, 0), "zero": (0, 3, 0, 0, 0, 0), "one minus source": (3, 2, 0, 7, 6, 0), "max": (1, 1, 4, 1, 1, 4),
    "destination colour": (4, 5, 0, 8, 9, 0), "destination alpha": (8, 9, 0, 1, 1, 0)}
PATHS = {"linear": {}, "tables": {"CPV_LINEAR_BLEND": "0"}, "general": {"CPV_BLEND_TABLES": "0"}}


def set_state(scene, equation, mask):
    """Blend state and write mask of the scene's pipelines (cpv_scene_pipeline)."""
    h = c.SceneHeader.from_address(scene.ptr)
    assert h.num_pipelines == 1
    words = (ctypes.c_uint32 * 81).from_address(h.pipelines)
    words[22] = 0 if equation is None else 1
    for i, v in enumerate(equation or (1, 0, 0, 1, 0, 0)):
        words[23 + i] = v
    constants = (ctypes.c_float * 4).from_address(h.pipelines + 29 * 4)
    constants[:] = [0.3, 0.6, -0.2, 1.5]
    assert words[80] == 0xF
    words[80] = mask


def wild(scene):
    h = c.SceneHeader.from_address(scene.ptr)
    v = np.ctypeslib.as_array(ctypes.cast(h.vertex_data, ctypes.POINTER(ctypes.c_float)), (h.vertex_bytes // 24, 6))
    v[0::9, 2:] *= -1
    v[3::9, 2:] *= 3
    v[6::18, 2] = np.nan
    v[12::27, 3] = np.inf
    v[15::27, 5] = 0.0


@pytest.mark.parametrize("path", list(PATHS))
@pytest.mark.parametrize("equation", list(EQUATIONS))
@pytest.mark.parametrize("variant,width,height,mask", [(0, 8, 4, 0xF), (0x200, 37, 21, 0xF), (0, 70, 50, 0x5), (0x10400, 33, 40, 0xF), (0x30800, 40, 33, 0xB),
                                                       (0x10000, 20, 20, 0xF)])
def test_flat_blend(gpu_ctx, oracle, monkeypatch, path, equation, variant, width, height, mask):
    for k, v in PATHS[path].items():
        monkeypatch.setenv(k, v)
    scene = c.Scene(c.PROGRAM, 4, [c.PROGRAM_FLATQUAD, variant | 0x1000, width, height, 150])
    set_state(scene, EQUATIONS[equation], mask)
    wild(scene)
    r = c.Renderer(gpu_ctx, scene)
    r.render(2)
    colour, _ = r.readback()
    r.close()
    ref, _, _ = oracle.render(scene)
    assert np.array_equal(colour, ref)
