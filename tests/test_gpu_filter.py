"""Linear filtering against the oracle's binary64 lerps, bit for bit: sizes
whose coordinates lie on both sides of the binary32 path's lower bound of 2,
texels that are zero, small or arbitrary (their lerps on both sides of its
bound of 2^-8), up- and downscaling, and repeat / mirror addressing of
power-of-two and other sizes through the textured program."""
import numpy as np
import pytest

import cpvulkan_gb300 as c

pytestmark = pytest.mark.gpu
RGBA8 = 37


def texels(rng, kind, w, h):
    if kind == "random":
        return rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    if kind == "sparse":  # mostly zeros among small values
        return (rng.integers(0, 4, (h, w, 4)) * (rng.random((h, w, 4)) < 0.3)).astype(np.uint8)
    return rng.choice(np.array([0, 1, 255], np.uint8), (h, w, 4))


@pytest.mark.parametrize("kind", ["random", "sparse", "extremes"])
@pytest.mark.parametrize("src_size,dst_size", [((1, 1), (7, 5)), ((2, 3), (61, 47)), ((5, 4), (333, 77)), ((64, 33), (97, 201)), ((257, 130), (64, 31)),
                                               ((40, 40), (1021, 9))])
def test_linear_blit(gpu_ctx, oracle, kind, src_size, dst_size):
    rng = np.random.default_rng(11)
    src = texels(rng, kind, *src_size)
    dst = np.zeros((dst_size[1], dst_size[0], 4), np.uint8)
    ref = dst.copy()
    gpu_ctx.blit(src.reshape(-1), src_size, 1, RGBA8, [(0, 0, 0, *src_size, 0, 0, 0, *dst_size)], 1, dst=dst.reshape(-1), dst_size=dst_size)
    oracle.blit(src, RGBA8, ref, RGBA8, (0, 0, *src_size, 0, 0, *dst_size), 1)
    assert np.array_equal(dst, ref)


@pytest.mark.parametrize("side", [64, 300])
@pytest.mark.parametrize("variant", [0x10, 0x10 | 0x8000])
def test_textured_program(gpu_ctx, oracle, side, variant):
    # texture coordinates in [-2, 3]: repeat (and, with the LOD bias, clamp
    # to edge and lerps between levels of 64 down to 1 texels)
    scene = c.Scene(c.PROGRAM, 6, [c.PROGRAM_TEXLIT, variant | 0x1000, side, side, 40])
    r = c.Renderer(gpu_ctx, scene)
    r.render(1)
    colour, depth = r.readback()
    r.close()
    ref_colour, ref_depth, _ = oracle.render(scene)
    assert np.array_equal(colour, ref_colour) and np.array_equal(depth, ref_depth)
