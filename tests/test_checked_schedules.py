"""The checked build (tests/test_checked_build.py) on the schedules that its small
images do not take by themselves: the wavefront kernels per bounce (queue slots
of every scene), refilled traversal (trees of eight levels and more), k_finish, and
the no-allocation render by the kernels per bounce on its stale state. Every call
has to succeed in the checked build (a bad index would be its status), and the
schedules have to agree: rtol 1e-6 for the order of a path's shadow additions
(as in tests/test_gpu_whole_paths.py), 1e-5 between the two builds."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r'''
import ctypes as C, os, sys
sys.path.insert(0, os.environ["GBRT_ROOT"])
import numpy as np
import torch
import renderer_gb300
renderer_gb300.LIB_PATH = sys.argv[1]
from renderer_gb300 import GpuScene, PerPixelRenderer, _abi, check, lib, workloads
from renderer_gb300.chains import MetropolisRenderer
from renderer_gb300.runtime import Context
from tests.test_csg import csg_scene
from tests.test_instances import instanced_cornell
from tests.test_texture import textured_room
out = {}
with Context(0) as ctx:
    late = lambda on: check(lib().gbrt_debug_fault(ctx.handle, _abi.FAULT_LATE_LAUNCHES, on), ctx.handle)
    scenes = {"cornell": workloads.cornell_box(48, 48), "csg": csg_scene(), "instanced": instanced_cornell(40)[0],
              "textured": textured_room(), "deep": workloads.icosphere_scene(levels=5, width=64, height=48, env_size=(16, 8))}
    for name, s in scenes.items():
        g = GpuScene(ctx, s)
        cam = s.camera_struct()
        for sem in (_abi.SEM_REFERENCE, _abi.SEM_PHYSICAL):
            # 1009 paths a wavefront: ragged queues, several wavefronts
            for batch in (0, 1009):
                r = PerPixelRenderer(g, cam, {"pt-x-samples": 2, "pt-y-samples": 1}, seed=3, max_depth=8, batch_paths=batch)
                r.params.semantics = sem
                for how, flags in (("whole", 0), ("bounces", _abi.RENDER_TIME_KERNELS), ("finish", 0)):
                    late(how == "finish")
                    r.params.flags = flags
                    out["%s_%d_%d_%s" % (name, sem, batch, how)] = r.render()
                    late(0)
            d = [torch.zeros(cam.width * cam.height * 3, dtype=t, device="cuda") for t in (torch.float32, torch.float64)]
            late(1)  # no whole paths: the kernels per bounce
            r.params.batch_paths, r.params.flags = 0, 0
            for call in range(2):
                check(lib().gbrt_render_device_noalloc(g.handle, C.byref(cam), C.byref(r.params), C.c_void_p(d[0].data_ptr()),
                                                       C.c_void_p(d[1].data_ptr()), None, None), ctx.handle)
            late(0)
            out["%s_%d_0_noalloc" % (name, sem)] = d[0].cpu().numpy().reshape(cam.height, cam.width, 3)
        late(1)
        m = MetropolisRenderer(g, cam, {"met-mutations": 2, "met-bootstrap": 500}, seed=2, chains=300)
        out[name + "_mlt"] = m.render()
        late(0)
np.savez(sys.argv[2], **out)
'''


def _run(lib_path, out_path):
    env = dict(os.environ, GBRT_ROOT=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD, lib_path, str(out_path)], capture_output=True, text=True, env=env,
                       cwd=ROOT, timeout=900)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return np.load(out_path)


def _checked_lib():
    """The checked library, built unless it is newer than every source."""
    from renderer_gb300 import build
    srcs = [os.path.join(d, f) for d in (build.CSRC, os.path.join(ROOT, "include")) for f in os.listdir(d)]
    newest = max(os.path.getmtime(f) for f in srcs)
    if os.path.exists(build.LIB_CHECKED) and os.path.getmtime(build.LIB_CHECKED) > newest:
        return build.LIB_CHECKED
    return build.build(checked=True)


def test_checked_schedules(tmp_path):
    from renderer_gb300 import LIB_PATH
    a = _run(_checked_lib(), tmp_path / "checked.npz")
    b = _run(LIB_PATH, tmp_path / "normal.npz")
    assert set(a.files) == set(b.files) and len(a.files) == 5 * (2 * (2 * 3 + 1) + 1)
    for k in a.files:
        assert np.isfinite(a[k]).all() and a[k].max() > 0, k
        if k.endswith("_mlt"):
            # as in tests/test_gpu_finish.py: a last bit may turn an acceptance over
            assert (~np.isclose(a[k], b[k], rtol=1e-4, atol=1e-6).all(-1)).sum() <= 20, k
            continue
        np.testing.assert_allclose(a[k], b[k], rtol=1e-5, atol=1e-6, err_msg=k)
        name, sem, batch, how = k.split("_")
        np.testing.assert_allclose(a[k], a["%s_%s_0_whole" % (name, sem)], rtol=1e-6, atol=1e-9, err_msg=k)
