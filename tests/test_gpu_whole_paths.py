"""Renders by whole paths (k_path for small wavefronts, k_finish for the last
paths of large ones) against the same renders by one launch per bounce and
kernel, which GBRT_RENDER_TIME_KERNELS asks for.

Both run the same arithmetic on the same random numbers. The one freedom is the
order in which a path's shadow rays add into its radiance (float atomics in the
kernels per bounce): a few roundings of 2^-24 of the sum per sample, so rtol
1e-6 holds every pixel."""
import numpy as np
import pytest

from renderer_gb300 import GpuScene, PerPixelRenderer, _abi, workloads
from tests.test_csg import csg_scene
from tests.test_instances import instanced_cornell
from tests.test_texture import textured_room

pytestmark = pytest.mark.gpu


def render(g, s, width, height, xs, depth, sem, flags, batch=0):
    cam = s.camera_struct(width, height)
    r = PerPixelRenderer(g, cam, {"pt-x-samples": xs, "pt-y-samples": 1}, seed=7, max_depth=depth, batch_paths=batch)
    r.params.semantics = sem
    r.params.flags = flags
    return r.render(), r.stats


def compare(ctx, s, width, height, xs, depth, sem, batch=0):
    g = GpuScene(ctx, s)
    a, sa = render(g, s, width, height, xs, depth, sem, 0, batch)
    b, sb = render(g, s, width, height, xs, depth, sem, _abi.RENDER_TIME_KERNELS, batch)
    np.testing.assert_allclose(a, b, rtol=1e-6, atol=1e-9)
    for k in ("paths", "extension_rays", "shadow_rays", "nonfinite"):
        assert getattr(sa, k) == getattr(sb, k), k
    return sa, sb


# one path, a warp and one more, a block's edge, a ragged image
@pytest.mark.parametrize("width,height", [(1, 1), (33, 1), (127, 1), (43, 3), (67, 45)])
@pytest.mark.parametrize("sem", [_abi.SEM_REFERENCE, _abi.SEM_PHYSICAL])
def test_small_wavefronts(ctx, width, height, sem):
    sa, sb = compare(ctx, workloads.cornell_box(), width, height, 1, 8, sem)
    assert sa.kernel_launches < sb.kernel_launches


@pytest.mark.parametrize("make", [csg_scene, lambda: instanced_cornell(40)[0], textured_room])
@pytest.mark.parametrize("sem", [_abi.SEM_REFERENCE, _abi.SEM_PHYSICAL])
def test_extended_scenes(ctx, make, sem):
    compare(ctx, make(), 61, 47, 2, 6, sem)


# above the one-warp blocks; several wavefronts, the last one ragged
@pytest.mark.parametrize("batch", [0, 10007])
def test_several_wavefronts(ctx, batch):
    compare(ctx, workloads.cornell_box(), 160, 127, 1, 5, _abi.SEM_REFERENCE, batch)


# more paths than k_path takes: bounces, then k_finish
@pytest.mark.parametrize("sem", [_abi.SEM_REFERENCE, _abi.SEM_PHYSICAL])
def test_large_wavefronts_end_in_one_launch(ctx, sem):
    compare(ctx, workloads.icosphere_scene(levels=4, env_size=(64, 32)), 1021, 701, 1, 12, sem)
