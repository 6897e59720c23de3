"""gbrt_guide_eval lays small evaluations out on the host and larger ones on the
device: a row's mixture does not depend on which (equal bit for bit), on both
sides of the line and for a call that writes over its inputs."""
import numpy as np
import pytest

from renderer_gb300 import check, lib
from renderer_gb300.guiding import Guide
from tests.test_guide import BOUNDS, init_weights, random_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 127, 129, 511, 512, 513, 1024])
def test_small_and_large_agree(ctx, n):
    g = Guide(ctx, BOUNDS, seed=3)
    g.set_weights(init_weights(8) * 2)
    x = random_inputs(4099, BOUNDS, np.random.default_rng(5))
    want = g.eval(x)
    np.testing.assert_array_equal(g.eval(x[:n]), want[:n])
    np.testing.assert_array_equal(g.eval(x[-n:]), want[-n:])
    buf = np.zeros(n * 40, np.float32)
    buf[:n * 9] = x[:n].ravel()
    check(lib().gbrt_guide_eval(g.handle, buf.ctypes.data, n, buf.ctypes.data), ctx.handle)
    np.testing.assert_array_equal(buf.reshape(n, 40), want[:n])
    g.close()
