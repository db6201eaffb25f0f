"""Per-draw binning: the ways a tile finds its primitives (walked whole,
filtered from all rectangles, from its bin's list, from all rectangles when
the list overflows) give the oracle's image bit for bit, at primitive counts
and target sizes around the rows, bins and filter steps of the kernels. The
scenes blend and depth-test overlapping triangles, so a primitive lost,
doubled or out of order changes pixels."""
import numpy as np
import pytest

import cpvulkan_gb300 as c

pytestmark = pytest.mark.gpu

MODES = {
    "direct": {"CPV_DIRECT_PRIMS": "1000000", "CPV_DIRECT_LIMIT": "4000000000"},
    "filter": {"CPV_DIRECT_PRIMS": "0", "CPV_FILTER_PRIMS": "1000000"},
    "lists": {"CPV_DIRECT_PRIMS": "0", "CPV_FILTER_PRIMS": "0"},
    "long rows": {"CPV_DIRECT_PRIMS": "0", "CPV_FILTER_PRIMS": "0", "CPV_BIN_ROW_PRIMS": "512"},
    "overflow": {"CPV_DIRECT_PRIMS": "0", "CPV_FILTER_PRIMS": "0", "CPV_LIST_CAPACITY": "1"},
}
# triangles, width, height, tile: one tile; a bin's edge; ragged rows; more
# than 1024 bins of 4 x 4 tiles
SIZES = [(1, 9, 7, "16"), (255, 64, 64, "16"), (256, 65, 63, "16"), (257, 130, 33, "8"), (700, 1041, 1030, "8"), (1100, 200, 150, "32")]


@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("tris,width,height,tile", SIZES)
def test_every_mode_equals_the_oracle(native, oracle, monkeypatch, mode, tris, width, height, tile):
    for k, v in MODES[mode].items():
        monkeypatch.setenv(k, v)
    monkeypatch.setenv("CPV_TILE", tile)
    ctx = c.Context()  # scratch of its own: the list's capacity is this test's
    try:
        scene = c.Scene(c.PROGRAM, 4, [c.PROGRAM_CUBE, 0x10 | 0x20 | 0x1000, width, height, tris])
        r = c.Renderer(ctx, scene)
        got = []
        for _ in range(3):  # eager, captured, replayed
            r.render(1)
            got.append(r.readback())
        r.close()
    finally:
        ctx.close()
    colour, depth, _ = oracle.render(scene)
    for g_colour, g_depth in got:
        assert np.array_equal(g_colour, colour) and np.array_equal(g_depth, depth)
