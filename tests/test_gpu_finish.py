"""k_finish, the kernel that ends a wavefront's last paths, in every variant:
renders and chains whose bounces from the third on are launched as usual
against the same ones with those launches left out (GBRT_FAULT_LATE_LAUNCHES), so
that every path still alive there is run by k_finish or lost.

Both run the same arithmetic on the same random numbers; a path's shadow rays
may add into its radiance in another order (a few roundings of 2^-24 of the
sum): rtol 1e-6 for every pixel."""
import numpy as np
import pytest

from renderer_gb300 import Context, GpuScene, PerPixelRenderer, _abi, lib, workloads
from renderer_gb300.chains import EnergyRedistributionRenderer, MetropolisRenderer
from renderer_gb300.guiding import guide_params, render_guided
from tests.test_csg import csg_scene
from tests.test_instances import instanced_cornell
from tests.test_texture import textured_room

pytestmark = pytest.mark.gpu

SCENES = {"plain": workloads.cornell_box, "csg": csg_scene, "instanced": lambda: instanced_cornell(40)[0],
          "textured": textured_room, "deep": lambda: workloads.icosphere_scene(levels=5, env_size=(64, 32))}


@pytest.fixture(scope="module")
def fctx(gbrt_built):
    c = Context(0)
    yield c
    c.close()


def late_launches(ctx, left_out):
    assert lib().gbrt_debug_fault(ctx.handle, _abi.FAULT_LATE_LAUNCHES, int(left_out)) == _abi.OK


def both(ctx, run):
    out = []
    for left_out in (False, True):
        late_launches(ctx, left_out)
        try:
            out.append(run())
        finally:
            late_launches(ctx, False)
    return out


@pytest.mark.parametrize("scene", SCENES)
@pytest.mark.parametrize("sem", [_abi.SEM_REFERENCE, _abi.SEM_PHYSICAL])
@pytest.mark.parametrize("width,height,xs,depth", [(1, 1, 1, 8), (33, 1, 1, 3), (61, 47, 2, 6), (353, 331, 1, 12)])
def test_renders(fctx, scene, sem, width, height, xs, depth):
    gs = GpuScene(fctx, SCENES[scene]())

    def run():
        r = PerPixelRenderer(gs, gs.data.camera_struct(width, height), {"pt-x-samples": xs, "pt-y-samples": 1}, seed=7,
                             max_depth=depth)
        r.params.semantics = sem
        return r.render(), r.stats

    (a, sa), (b, sb) = both(fctx, run)
    np.testing.assert_allclose(a, b, rtol=1e-6, atol=1e-9)
    for k in ("paths", "extension_rays", "shadow_rays", "nonfinite"):
        assert getattr(sa, k) == getattr(sb, k), k
    assert sb.kernel_launches == 1 + 2 * 3 + 1 + 2  # camera rays, two bounces, k_finish, accumulation, film


@pytest.mark.parametrize("scene", ["plain", "instanced"])
def test_passes_of_a_guided_render(fctx, scene):
    gs = GpuScene(fctx, SCENES[scene]())
    cam = gs.data.camera_struct(61, 47)
    r = PerPixelRenderer(gs, cam, {"pt-x-samples": 1, "pt-y-samples": 1}, seed=7, max_depth=8)
    r.params.semantics = _abi.SEM_PHYSICAL
    (a, sa), (b, sb) = both(fctx, lambda: render_guided(gs, cam, r.params, None, guide_params(passes=3)))
    np.testing.assert_allclose(a, b, rtol=1e-6, atol=1e-9)
    assert sa.extension_rays == sb.extension_rays and sa.shadow_rays == sb.shadow_rays


# The chains move by their radiance: a last bit of it turns an acceptance over
# with a probability of about 2^-23 a mutation, so of these 40,000 mutations none
# is expected to, and one would show in at most a few pixels.
@pytest.mark.parametrize("scene", SCENES)
@pytest.mark.parametrize("chains", [1, 127, 2500])
def test_metropolis(fctx, scene, chains):
    gs = GpuScene(fctx, SCENES[scene]())

    def run():
        m = MetropolisRenderer(gs, gs.data.camera_struct(50, 50), {"met-mutations": 16, "met-bootstrap": 3000}, seed=2,
                               max_depth=6, chains=chains)
        return m.render(), m.stats

    (a, sa), (b, sb) = both(fctx, run)
    assert (~np.isclose(a, b, rtol=1e-4, atol=1e-7).all(-1)).sum() <= 20
    assert abs(int(sa.accepted) - int(sb.accepted)) <= 20
    assert sb.normaliser == pytest.approx(sa.normaliser, rel=1e-6)


@pytest.mark.parametrize("scene", ["plain", "csg", "textured"])
def test_energy_redistribution(fctx, scene):
    gs = GpuScene(fctx, SCENES[scene]())

    def run():
        m = EnergyRedistributionRenderer(gs, gs.data.camera_struct(40, 30), {"erpt-mutations": 10}, seed=2, max_depth=6)
        return m.render(), m.stats

    (a, sa), (b, sb) = both(fctx, run)
    assert sa.chains == sb.chains
    assert (~np.isclose(a, b, rtol=1e-4, atol=1e-7).all(-1)).sum() <= 20
    assert abs(int(sa.accepted) - int(sb.accepted)) <= 20
