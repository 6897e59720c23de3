"""The rows of gbrt_guide_eval / gbrt_guide_gradient around the edges of the
kernels that lay them out: one row, a block's and a tile's edges, and more rows
than one piece of an evaluation."""
import numpy as np
import pytest

from oracle import guide_ref as gr
from tests.test_guide import BOUNDS, init_weights, random_inputs, random_samples

pytestmark = pytest.mark.gpu


@pytest.fixture
def guide(ctx):
    from renderer_gb300.guiding import Guide
    g = Guide(ctx, BOUNDS, seed=3)
    g.set_weights(init_weights(8) * 2)
    yield g
    g.close()


# A row's mixture does not depend on the rows around it: equal bit for bit.
@pytest.mark.parametrize("n", [1, 85, 86, 128, 257, 4099, (1 << 20) + 5])
def test_eval_rows(guide, n):
    x = random_inputs(n, BOUNDS, np.random.default_rng(n))
    got = guide.eval(x)
    assert got.shape == (n, 40)
    k = max(1, n - 131)
    np.testing.assert_array_equal(got[k - 1:], guide.eval(x[k - 1:]))
    np.testing.assert_array_equal(got[:min(n, 7)], guide.eval(x[:min(n, 7)]))


# Both sides round the same tensors to bfloat16 (one ulp is 2^-8) and differ by
# the roundings that fall to the other side: below a few times 2^-8 of the
# gradient even for one row, far below what a misplaced column would change.
@pytest.mark.parametrize("n", [1, 63, 64, 65, 257, 2049])
def test_sample_rows(guide, n):
    s = random_samples(n, BOUNDS, np.random.default_rng(n))
    g, loss = guide.gradient(s)
    want, gref = gr.loss_and_grad(guide.weights(), s, BOUNDS, bf16=True)
    assert loss == pytest.approx(want, rel=2e-2, abs=2e-2)
    x = g[:gref.size].astype(np.float64)
    assert np.linalg.norm(x - gref) < 0.1 * np.linalg.norm(gref)
