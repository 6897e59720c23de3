"""pathtrace.cu refuses to compile without the flags that keep its sums of
products as they are written (build.py FLAGS)."""
import os
import subprocess

import pytest

from renderer_gb300.build import ARCH, COMMON, CSRC, FLAGS, nvcc


@pytest.mark.parametrize("flags", [True, False])
def test_contraction_is_off(flags):
    extra = FLAGS["pathtrace.cu"] if flags else []
    r = subprocess.run([nvcc(), *ARCH, *COMMON, *extra, "-E", os.path.join(CSRC, "pathtrace.cu")], capture_output=True,
                       text=True)
    assert (r.returncode == 0) == flags
    if flags:
        assert "-fmad=false" in extra
    else:
        assert "-fmad=false" in r.stderr
