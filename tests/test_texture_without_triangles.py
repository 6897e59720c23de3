"""Textured scenes without a triangle list: a textured sphere, quad and plane
(default and spherical texture coordinates), alone and beside a CSG object,
against the oracle path by path for both estimators.

The tolerance is that of the textured room's parity test (tests/test_texture.py):
the same shading in the same precision."""
import numpy as np
import pytest

from oracle.binding import OracleScene
from renderer_gb300 import _abi, workloads
from renderer_gb300.scene import render_params
from tests.test_texture import checker

pytestmark = pytest.mark.gpu


def textured_shapes(csg):
    s = workloads.cornell_box(64, 64)
    m = s.add_material(_abi.MAT_TEXTURE, kd=(0.9, 0.8, 0.7), exponent=1.5, texture=s.add_texture(checker(16)))
    c, r, _ = s.spheres[0]
    s.spheres[0] = (c, r, m)
    s.quads[2] = (*s.quads[2][:4], m)  # the back wall
    s.planes = [((0, 1, 0, 0.5), m)]
    if csg:
        s.add_csg(s.csg_leaf(_abi.CSG_SPHERE, (0.0, 1.2, 0.0), (0.25, 0, 0), m))
    assert s.tri_pos is None
    return s


@pytest.mark.parametrize("csg", [False, True])
@pytest.mark.parametrize("semantics", [_abi.SEM_REFERENCE, _abi.SEM_PHYSICAL])
def test_textured_shapes_path_level_parity(ctx, semantics, csg):
    from tests.test_gpu_render import gpu_render
    s = textured_shapes(csg)
    prm = render_params(2, 2, 0.5, 6, 9, semantics=semantics)
    (film, _, _), _ = gpu_render(ctx, s, prm)
    orc = OracleScene(s).render(s.camera_struct(), prm, rng_mode=1)["film"]
    close = np.isclose(film, orc, rtol=2e-3, atol=1e-5).all(-1)
    assert close.mean() > 0.97, close.mean()
    assert film.mean() == pytest.approx(orc.mean(), rel=5e-3)
