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


def test_calls_share_the_models_buffers():
    """Calls of growing and shrinking sizes, beyond the kept size and from several
    threads, on one model give what fresh models give, bit for bit."""
    from concurrent.futures import ThreadPoolExecutor

    rng = np.random.default_rng(7)
    d = 43
    sets = [rng.normal(0, 1, (n, d)).astype(np.float32) for n in (3, 5000, 17, 120000, 1, 5000)]
    want = []
    for x in sets:
        m = abi.Mlp(d, seed=1)
        want.append((m.predict(x), m.gradients(x, x[:, 0].copy())))
        m.close()
    m = abi.Mlp(d, seed=1)
    for x, (p, (loss, g)) in zip(sets, want):
        assert np.array_equal(m.predict(x), p)
        got = m.gradients(x, x[:, 0].copy())
        assert got[0] == loss and np.array_equal(got[1], g)
    with ThreadPoolExecutor(4) as ex:
        for x, p in zip(sets * 4, ex.map(m.predict, sets * 4)):
            assert np.array_equal(p, want[[id(s) for s in sets].index(id(x))][0])
    # training, with other calls in between, equals training without them
    a, b = abi.Mlp(d, seed=2), abi.Mlp(d, seed=2)
    x = sets[1]
    la = a.train(x, x[:, 0].copy(), 2, 256, 1e-3, 5)
    lb = [b.train(x, x[:, 0].copy(), 2, 256, 1e-3, 5)]
    b.predict(sets[3])
    assert np.array_equal(np.asarray(la), np.asarray(lb[0])) and np.array_equal(a.params(), b.params())
    for k in (a, b, m):
        k.close()
