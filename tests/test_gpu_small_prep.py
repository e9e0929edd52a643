"""Preparation of small matrices: gene statistics at the 4,096 cells where a warp per
row gives way to spans of the array, for short, long and empty rows; size factors at
the 16,384 cells where one block gives way to three kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(rng, n, lens):
    cols = [np.sort(rng.choice(n, k, replace=False)).astype(np.int32) for k in lens]
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    return ptr, np.concatenate(cols), rng.integers(1, 60000, int(ptr[-1])).astype(np.uint16)


# mean and variance come from exact integer sums: theta_0 is rounded a few times
# after them, and its numerator cancels by less than 1e3 on these counts
@pytest.mark.parametrize("n", [40, 4095, 4096, 4097, 16385])
@pytest.mark.parametrize("rows", ["short", "long"])
def test_statistics(dv, orc, n, rows):
    rng = np.random.default_rng(n)
    lens = rng.integers(1, 16, 700) if rows == "short" else np.r_[n, n - 1, rng.integers(n // 2, n, 30)]
    lens = np.minimum(np.r_[lens, 0, 1, n // 2], n)
    ptr, col, val = _csr(rng, n, lens)
    off = rng.normal(0, 0.3, n)
    got = dv.estimate_dispersion((ptr, col, val, n), off)
    np.testing.assert_array_equal(got, dv.estimate_dispersion((ptr, col, val.astype(np.float32), n), off))
    some = np.r_[:10, len(lens) - 3:len(lens)]
    Y = np.zeros((len(some), n))
    for i, g in enumerate(some):
        Y[i, col[ptr[g]:ptr[g + 1]]] = val[ptr[g]:ptr[g + 1]]
    np.testing.assert_allclose(got[some], orc.estimate_dispersion(Y, off), rtol=1e-12)


@pytest.mark.parametrize("n", [2, 16383, 16384, 16385])
@pytest.mark.parametrize("method", ["normed_sum", "psinorm"])
def test_size_factors(dv, orc, n, method):
    rng = np.random.default_rng(n)
    Y = rng.poisson(3.0, (12, n)) + 1.0
    # psinorm keeps the columns' minima in FP32 (1 ulp of 6e-8 of a logarithm's size)
    np.testing.assert_allclose(dv.calculate_sf(Y, method), orc.calculate_sf(Y, method),
                               rtol=1e-12 if method == "normed_sum" else 1e-6)
    if n > 2:
        Y[:, 5] = 0.0
        with pytest.raises(Exception, match="all zeros"):
            dv.calculate_sf(Y, "normed_sum")
