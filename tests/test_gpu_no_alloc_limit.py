"""cpv_queue_submit_no_alloc with a raised CPV_DIRECT_LIMIT: a draw whose tile
rectangles do not fit the fixed 32 MiB array is walked whole by every tile
(nothing of it is written to the array) and gives vkQueueSubmit's image; one
above the limit is refused before any launch; one that fits still bins."""
import numpy as np
import pytest

import cpvulkan_gb300 as c

pytestmark = pytest.mark.gpu

# 2 x 1499^2 triangles: 36 MB of rectangles; 6 x 4 tiles
LARGE = (c.HEIGHTFIELD, [1500, 96, 64])


def _image(ctx, scene):
    r = c.Renderer(ctx, scene)
    try:
        r.render(1)
        return r.readback()
    finally:
        r.close()


@pytest.mark.parametrize("config,params", [LARGE, (c.HEIGHTFIELD, [256, 640, 360]), (c.BLEND, [3000, 640, 360])])
def test_raised_limit_renders(native, gpu_ctx, monkeypatch, config, params):
    scene = c.Scene(config, 5, params)
    want = _image(gpu_ctx, scene)
    monkeypatch.setenv("CPVH_SUBMIT", "no_alloc")
    monkeypatch.setenv("CPV_DIRECT_LIMIT", "4000000000")
    ctx = c.Context()
    try:
        got = _image(ctx, scene)
    finally:
        ctx.close()
    for g, w in zip(got, want):
        assert (g is None and w is None) or np.array_equal(g, w)


@pytest.mark.parametrize("limit", [None, str(2 * 1499 * 1499 * 24 - 1)])
def test_above_the_limit_is_refused(native, monkeypatch, limit):
    monkeypatch.setenv("CPVH_SUBMIT", "no_alloc")
    if limit:
        monkeypatch.setenv("CPV_DIRECT_LIMIT", limit)
    ctx = c.Context()
    r = c.Renderer(ctx, c.Scene(LARGE[0], 5, LARGE[1]))
    try:
        before = c.kernel_launches()
        with pytest.raises(RuntimeError):
            r.render(1)
        assert "fixed scratch holds 33554432" in c.icd_last_error() and c.kernel_launches() == before
    finally:
        r.close()
        ctx.close()
