"""The small-batch backward kernel at its edges (four samples per block, up to
one block per SM, any input width) against the numpy oracle: FP32 against
float64, 1e-4 of the largest component as for the other K7 kernels."""
import numpy as np
import pytest

from hisvsim_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 43, 64])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 64, 589, 592, 593])
def test_small_batches_match_oracle(d, n):
    from oracle import mlp

    rng = np.random.default_rng(100 * d + n)
    x = rng.normal(0, 1, (n, d)).astype(np.float32)
    y = np.sin(x.sum(axis=1)).astype(np.float32)
    m = abi.Mlp(d, seed=d)
    loss, g = m.gradients(x, y)
    wl, wg = mlp.loss_and_grad(m.params().astype(np.float64), x, y)
    assert loss == pytest.approx(wl, rel=1e-4)
    assert np.abs(g - wg).max() <= 1e-4 * np.abs(wg).max()
    m.close()
