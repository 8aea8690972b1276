"""Readout kernels against numpy in FP64: <ZZ> of many pairs in one pass (pairs
within and across the thread, register and chunk bits of the kernel, more pairs
than one pass holds), marginals of every slot, and samples found on the device.
Sums of up to 2^17 probabilities in FP64 differ by their order: 1e-13."""
import numpy as np
import pytest

from hisvsim_b200 import abi

pytestmark = pytest.mark.gpu


def _state(n, dtype, seed, zeros=False):
    rng = np.random.default_rng(seed)
    a = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    if zeros:  # long runs without mass, the last amplitudes among them
        a[rng.uniform(size=1 << n) < 0.7] = 0
        a[: 1 << (n - 2)] = 0
        a[-(1 << (n - 2)):] = 0
        a[1 << (n - 1)] = 1.0
    a /= np.linalg.norm(a)
    st = abi.State(n, dtype)
    st.load(a.astype(st.np_dtype))
    p = np.abs(st.raw().astype(complex)) ** 2
    return st, p


@pytest.mark.parametrize("dtype", [abi.C128, abi.C64])
@pytest.mark.parametrize("n", [1, 2, 5, 8, 9, 12, 13, 16, 17])
def test_zz_and_marginals(n, dtype):
    st, p = _state(n, dtype, n)
    x = np.arange(1 << n)
    z = 1.0 - 2.0 * ((x[:, None] >> np.arange(n)) & 1)
    pairs = [(i, j) for i in range(n) for j in range(i, n)][:70]
    got = st.expect_zz(pairs)
    want = np.array([np.sum(p * z[:, i] * z[:, j]) for i, j in pairs])
    assert np.abs(got - want).max() <= 1e-13
    for q in range(n):
        assert abs(st.probability(q) - p[((x >> q) & 1) == 0].sum()) <= 1e-13


@pytest.mark.parametrize("dtype", [abi.C128, abi.C64])
@pytest.mark.parametrize("n,samples,zeros", [(1, 7, False), (4, 50, False), (6, 50, True),
                                             (12, 300, True), (16, 300, False), (17, 1000, True)])
def test_samples_follow_the_distribution(n, samples, zeros, dtype):
    """The seeded sample points walked against numpy's cumulative sum; a point
    within 1e-12 of a step may fall on either side."""
    st, p = _state(n, dtype, 50 + n, zeros and n > 2)
    seed = 1234567 + n
    got = st.measure(list(range(n)), samples, seed)
    idx = (got.astype(np.int64) << np.arange(n)).sum(axis=1)
    raw = np.random.RandomState(seed)._bit_generator.random_raw(2 * samples).astype(np.float64)
    u = np.sort((raw[0::2] + raw[1::2] * 2.0 ** 32) / 2.0 ** 64)
    cum = np.cumsum(p)
    assert np.all(p[idx] > 0)
    assert np.all(cum[idx] >= u - 1e-12)
    assert np.all(cum[idx] - p[idx] <= u + 1e-12)


@pytest.mark.parametrize("n,samples", [(1, 300), (10, 5000), (16, 5000), (17, 3001)])
def test_many_samples_of_a_small_state(n, samples):
    """More samples than one block searches: the points of the seed, as in
    test_samples_follow_the_distribution."""
    st, p = _state(n, abi.C128, 90 + n, n > 2)
    seed = 77 + n
    got = st.measure(list(range(n)), samples, seed)
    idx = (got.astype(np.int64) << np.arange(n)).sum(axis=1)
    raw = np.random.RandomState(seed)._bit_generator.random_raw(2 * samples).astype(np.float64)
    u = np.sort((raw[0::2] + raw[1::2] * 2.0 ** 32) / 2.0 ** 64)
    cum = np.cumsum(p)
    assert np.all(p[idx] > 0)
    assert np.all(cum[idx] >= u - 1e-12)
    assert np.all(cum[idx] - p[idx] <= u + 1e-12)
