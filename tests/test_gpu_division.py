"""Interpolation by prepared reciprocals against the oracle's IEEE divisions,
bit for bit in 32-bit float colours and depth: varyings, clip w, areas and
weights inside, at and far outside the ranges in which the reciprocals are
used, zeros, infinities and pixel centres exactly on edges; per draw and, by
the override, batched."""
import ctypes

import numpy as np
import pytest

import cpvulkan_gb300 as c

pytestmark = pytest.mark.gpu
RGBA32F = 109


def vertices(scene):
    """The scene's vertices (position, colour) as a writable array."""
    h = c.SceneHeader.from_address(scene.ptr)
    n = h.vertex_bytes // 32
    return np.ctypeslib.as_array(ctypes.cast(h.vertex_data, ctypes.POINTER(ctypes.c_float)), (n, 8))


def colours(scale):
    def change(v):
        v[:, 4:] *= np.float32(scale)
    return change


def clip(scale):
    def change(v):
        v[:, :4] *= np.float32(scale)
    return change


def mixed_colours(v):
    v[0::5, 4] = 0.0
    v[1::5, 5] = -0.0
    v[2::7, 6] = np.float32(2.0 ** -41)
    v[3::7, 7] = np.float32(2.0 ** 21)
    v[4::11, 4] = np.float32(1e-42)
    v[5::11, 5] = np.float32("inf")
    v[6::3, 6] *= -1


def mixed_w(v):
    for i, e in enumerate((0, 19, 21, -19, -21, 40, -60)):
        v[i::7, :4] *= np.float32(2.0 ** e)


def on_edges(v):
    # triangle vertices on pixel centres of a 16 x 16 target: weights of exactly zero
    rng = np.random.default_rng(3)
    v[:, :2] = (rng.integers(0, 16, (len(v), 2)) + 0.5) / 8.0 - 1.0
    v[:, 2] = np.where(rng.random(len(v)) < 0.5, -0.0, 0.0)
    v[:, 3] = 1.0


def tiny(v):
    v[:, :2] = v[:, :2] * np.float32(2.0 ** -27)


CHANGES = {"as they are": lambda v: None, "colours 2^-42": colours(2.0 ** -42), "colours 2^22": colours(2.0 ** 22), "colours 2^100": colours(2.0 ** 100),
           "colours 0": colours(0.0), "clip 2^21": clip(2.0 ** 21), "clip 2^-22": clip(2.0 ** -22), "clip 2^-70": clip(2.0 ** -70),
           "mixed colours": mixed_colours, "mixed w": mixed_w, "on edges": on_edges, "tiny": tiny}


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("change", list(CHANGES))
def test_interpolation(gpu_ctx, oracle, monkeypatch, change, batched):
    monkeypatch.setenv("CPV_QUICK_DIV", "1")
    if batched:
        monkeypatch.setenv("CPV_BATCH_MIN_DRAWS", "1")
    # D32, compare ALWAYS: every fragment's depth and colour is written
    scene = c.Scene(c.PROGRAM, 2, [c.PROGRAM_CUBE, 0x10 | 0xC0 | 0x1000, 16, 16, 40, 0, RGBA32F])
    CHANGES[change](vertices(scene))
    r = c.Renderer(gpu_ctx, scene)
    r.render(1)
    colour, depth = r.readback()
    r.close()
    ref_colour, ref_depth, _ = oracle.render(scene)
    for got, ref in ((colour, ref_colour), (depth, ref_depth)):
        # the sign and payload of a NaN (zero-area triangles, infinite
        # varyings) are not defined by the operations
        nan = np.isnan(got.view(np.float32)) & np.isnan(ref.view(np.float32))
        assert np.array_equal(got.view(np.uint32)[~nan], ref.view(np.uint32)[~nan])
