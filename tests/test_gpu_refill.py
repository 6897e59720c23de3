"""Traversal kernels that refill idle lanes (deep trees) against the plain ones,
which a render with traversal counters runs.

Every ray meets the same nodes and triangles in the same order in both. The one
freedom is the order in which a path's shadow rays add into its radiance (float
atomics): a few roundings of 2^-24 of the sum per sample, so rtol 1e-6 holds
every pixel."""
import numpy as np
import pytest

from renderer_gb300 import GpuScene, PerPixelRenderer, _abi, workloads

pytestmark = pytest.mark.gpu


def scene(levels):
    return workloads.icosphere_scene(levels=levels, width=64, height=48, env_size=(16, 8))


# one ray, a warp and one more, a block's edge, ragged, several rays per lane;
# trees on both sides of the rule
@pytest.mark.parametrize("width,height,xs", [(1, 1, 1), (33, 1, 1), (129, 1, 1), (61, 47, 2), (640, 451, 4)])
@pytest.mark.parametrize("levels", [3, 4, 6])
@pytest.mark.parametrize("sem", [_abi.SEM_REFERENCE, _abi.SEM_PHYSICAL])
def test_refilled_render(ctx, width, height, xs, levels, sem):
    s = scene(levels)
    g = GpuScene(ctx, s)
    out = []
    for flags in (_abi.RENDER_TIME_KERNELS, _abi.RENDER_COUNT_TRAVERSAL):
        r = PerPixelRenderer(g, s.camera_struct(width, height), {"pt-x-samples": xs, "pt-y-samples": 1}, seed=11,
                             max_depth=5)
        r.params.semantics = sem
        r.params.flags = flags
        out.append((r.render(), r.stats))
    (a, sa), (b, sb) = out
    np.testing.assert_allclose(a, b, rtol=1e-6, atol=1e-9)
    for k in ("paths", "extension_rays", "shadow_rays", "nonfinite"):
        assert getattr(sa, k) == getattr(sb, k), k
