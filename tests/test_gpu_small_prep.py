"""Preparation of small matrices: gene statistics at the 4,096 cells where a warp per
row gives way to spans of the array, for short, long and empty rows, and the CSR check
at the same line; beta_0 at the 3,072 cells where one entry a lane gives way to several;
size factors at the 16,384 cells where one block gives way to three kernels."""
import ctypes as C

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


# X'X of normal columns with n >= 4 p has a condition of about 9, and its sums and
# the right-hand side's are rounded n times at most: 9 * 3,100 * 1e-16 of the largest
@pytest.mark.parametrize("n", [150, 3071, 3072, 3073])
@pytest.mark.parametrize("p", [1, 4, 5, 8, 9, 16, 17, 32])
def test_initial_coefficients(dv, orc, n, p):
    rng = np.random.default_rng(n + p)
    lens = np.minimum(np.r_[n, n - 1, 0, 1, 31, 32, 33, rng.integers(1, n // 2, 40)], n)
    ptr, col, val = _csr(rng, n, lens)
    X = np.c_[np.ones(n), rng.normal(size=(n, p - 1))]
    off = rng.normal(0, 0.3, n)
    Y = np.zeros((len(lens), n))
    for g in range(len(lens)):
        Y[g, col[ptr[g]:ptr[g + 1]]] = val[ptr[g]:ptr[g + 1]]
    want = orc.init_beta(Y, X, off)
    for v in (val, val.astype(np.float32)):
        got = dv.init_beta((ptr, col, v, n), X, off)
        np.testing.assert_allclose(got, want, rtol=0, atol=1e-11 * np.abs(want).max())


@pytest.mark.parametrize("n", [4096, 4097])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_check_of_short_rows_and_long(dv, n, shift):
    import torch
    from devil_b200 import _lib as L

    rng = np.random.default_rng(n + shift)
    lens = np.r_[0, 1, 0, 31, 32, 33, n, 2, rng.integers(0, 9, 2000), n - 1, 0]
    ptr, col, val = _csr(rng, n, lens)
    G, d = len(lens), torch.device("cuda")
    rp, X = torch.tensor(ptr, device=d), torch.ones(n, dtype=torch.float64, device=d)
    vi = torch.tensor(val.view(np.int16), device=d)
    buf = torch.zeros(len(col) + shift, dtype=torch.int32, device=d)[shift:]
    out = torch.zeros(3 * G, dtype=torch.float64, device=d)
    at = [C.c_void_p(out.data_ptr() + 8 * G * i) for i in range(3)]
    res = L.FitResult(at[0], at[1], at[2], None, None, None, None, None, None, None, None)
    counts = L.Counts(L.COUNTS_CSR_U16, 0, G, n, len(col), vi.data_ptr(), rp.data_ptr(), buf.data_ptr())
    opts = L.FitOpts()
    L.load().devil_fit_opts_default(C.byref(opts))
    opts.max_iter, opts.init_beta_rough = 0, 1
    ctx = dv.context()

    def run(c, r=ptr):
        buf.copy_(torch.tensor(c))
        rp.copy_(torch.tensor(r))
        torch.cuda.synchronize()
        rc = L.load().devil_fit_device(ctx.h, C.byref(counts), C.c_void_p(X.data_ptr()), 1, None, 0,
                                       C.byref(opts), C.byref(res))
        ctx.synchronize()
        return rc

    assert run(col) == L.OK
    inside = np.setdiff1d(np.arange(len(col)), ptr)  # entries with one before them in their row
    for e in np.r_[inside[:3], inside[-3:], rng.choice(inside, 12)]:
        bad = col.copy()
        bad[e] = bad[e - 1]
        assert run(bad) == L.ERR_ARG, e
    for e in (0, 1, len(col) - 1):
        for v in (-1, n):
            bad = col.copy()
            bad[e] = v
            assert run(bad) == L.ERR_ARG, (e, v)
    for g, v in ((3, -1), (7, ptr[6]), (G - 1, len(col) + 1), (G, len(col) - 1)):
        r = ptr.copy()
        r[g] = v
        assert run(col, r) == L.ERR_ARG, (g, v)
