"""gbrt_guide_eval with the mixtures written over the inputs: every input is read
before the first mixture is written, also when the rows are evaluated in more
than one piece (2^20 rows)."""
import numpy as np
import pytest

from renderer_gb300 import check, lib
from renderer_gb300.guiding import Guide
from tests.test_guide import BOUNDS, init_weights, random_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 257, (1 << 20) + 5])
def test_mixtures_over_inputs(ctx, n):
    g = Guide(ctx, BOUNDS, seed=3)
    g.set_weights(init_weights(8) * 2)
    x = random_inputs(n, BOUNDS, np.random.default_rng(n))
    want = g.eval(x)
    buf = np.zeros(n * 40, np.float32)
    buf[:n * 9] = x.ravel()
    check(lib().gbrt_guide_eval(g.handle, buf.ctypes.data, n, buf.ctypes.data), ctx.handle)
    np.testing.assert_array_equal(buf.reshape(n, 40), want)
    g.close()
