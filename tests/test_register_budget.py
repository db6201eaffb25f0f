"""The register budget of the per-draw raster of flat pipelines with depth or
stencil operations, in resident CTAs of 256 threads (compile-only device)."""
import pytest

import cpvulkan_gb300 as c
from tests.test_pipeline_compile import _module_source, compile_ctx  # noqa: F401


@pytest.mark.parametrize("variant", [0x10, 0x10 | 0x20, 0x18 | 0x100 | 0x20, 0x10 | (2 << 28)])
def test_flat_pipelines_with_depth(compile_ctx, variant):  # noqa: F811
    text = _module_source(compile_ctx, c.PROGRAM_FLATQUAD, variant)
    assert "#define CPV_LINEAR_BLEND 0\n" in text and "#define CPV_SCHEDULE 0\n" in text
    assert "#define CPV_PLAIN_MIN_BLOCKS 5\n" in text
