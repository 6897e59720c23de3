"""Which launches a render takes: whole paths (k_path) for small wavefronts, one
set of launches per bounce for larger ones, whose last paths k_finish may end.
Either schedule gives the image of
the kernels per bounce (GBRT_RENDER_TIME_KERNELS) up to the order in which a
path's shadow rays add into its radiance: rtol 1e-6."""
import numpy as np
import pytest

from renderer_gb300 import GpuScene, PerPixelRenderer, _abi, workloads
from tests.test_instances import instanced_cornell

pytestmark = pytest.mark.gpu


def lanes():
    """Threads of a whole-path kernel resident at once."""
    import torch
    return 512 * torch.cuda.get_device_properties(0).multi_processor_count


def render(gs, paths, depth, sem, flags=0):
    r = PerPixelRenderer(gs, gs.data.camera_struct(paths, 1), {"pt-x-samples": 1, "pt-y-samples": 1}, seed=3,
                         max_depth=depth)
    r.params.semantics = sem
    r.params.flags = flags
    return r.render(), r.stats


# four instances in a room, nine levels: at most one path a lane
@pytest.mark.parametrize("sem", [_abi.SEM_REFERENCE, _abi.SEM_PHYSICAL])
def test_instances_take_whole_paths_up_to_one_a_lane(ctx, sem):
    gs = GpuScene(ctx, instanced_cornell(40)[0])
    n, depth = lanes(), 5
    for paths, whole in ((n // 2 + 1, True), (n, True), (n + 1, False), (2 * n - 3, False), (3 * n, False)):
        film, st = render(gs, paths, depth, sem)
        assert (st.kernel_launches < 3 * depth) == whole, paths
        want, sw = render(gs, paths, depth, sem, _abi.RENDER_TIME_KERNELS)
        np.testing.assert_allclose(film, want, rtol=1e-6, atol=1e-9)
        assert st.extension_rays == sw.extension_rays and st.shadow_rays == sw.shadow_rays


# Launches of a wavefront of more paths than k_path takes: camera rays, three a
# bounce, accumulation, film, and one of k_finish before bounces 2, 3, 4, 6, 8,
# 12 ... with four bounces left, or with any in a deep tree.
@pytest.mark.parametrize("deep,depth,finishes", [(False, 1, 0), (False, 3, 0), (False, 5, 0), (False, 6, 1), (False, 8, 3),
                                                 (False, 12, 5), (False, 64, 10), (True, 2, 0), (True, 3, 1), (True, 5, 3)])
def test_launches_that_look_for_the_last_paths(ctx, deep, depth, finishes):
    s = workloads.icosphere_scene(levels=6, env_size=(16, 8)) if deep else workloads.cornell_box()
    _, st = render(GpuScene(ctx, s), 6 * lanes(), depth, _abi.SEM_REFERENCE)
    assert st.kernel_launches == 3 + 3 * depth + finishes
