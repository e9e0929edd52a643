"""Column sums, gene statistics and the CSR check on matrices whose rows cut
the scans' spans, pieces and column tiles anywhere: few long rows, many short
and empty ones, columns beyond one tile of 49,152, any nnz mod 8, and arrays
that start off a 16-byte boundary.  Integer results, so bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(rng, n, lens):
    rows = [np.sort(rng.choice(n, k, replace=False)).astype(np.int32) for k in lens]
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = np.concatenate(rows)
    return ptr, col, rng.integers(1, 65536, len(col)).astype(np.uint16)


CASES = {
    "one_tile_dense": (2001, [2001] * 30 + [0, 1, 7]),
    "two_tiles": (49153, [49153] * 17 + [3, 0, 0, 49152]),
    "three_tiles_ragged": (120000, [120000] * 16 + list(range(0, 3000, 11))),
    "sparse_columns": (60000, [500] * 40 + [0] * 9 + [60000]),
    "short_rows": (300, [k % 5 for k in range(4000)] + [300]),
}


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_scans_are_exact(dv, name, shift):
    import torch
    from devil_b200 import _lib as L

    n, lens = CASES[name]
    rng = np.random.default_rng(len(lens))
    ptr, col, val = _matrix(rng, n, lens)
    G = len(lens)
    want = np.zeros(n)
    np.add.at(want, col, val.astype(np.float64))
    d = torch.device("cuda")
    rp = torch.tensor(ptr, device=d)
    # shift 1: both arrays start one element off their allocation
    ci = torch.zeros(len(col) + shift, dtype=torch.int32, device=d)[shift:]
    vi = torch.zeros(len(col) + shift, dtype=torch.int16, device=d)[shift:]
    ci.copy_(torch.tensor(col))
    vi.copy_(torch.tensor(val.view(np.int16)))
    X = torch.ones(n, dtype=torch.float64, device=d)
    out = {k: torch.zeros(s, dtype=t, device=d) for k, s, t in
           [("beta", G, torch.float64), ("theta", G, torch.float64), ("it", G, torch.int32), ("sf", n, torch.float64)]}
    at = {k: C.c_void_p(v.data_ptr()) for k, v in out.items()}
    counts = L.Counts(L.COUNTS_CSR_U16, 0, G, n, len(col), vi.data_ptr(), rp.data_ptr(), ci.data_ptr())
    opts = L.FitOpts()
    L.load().devil_fit_opts_default(C.byref(opts))
    opts.max_iter, opts.size_factors, opts.init_beta_rough = 0, L.SF_NORMED_SUM, 1
    res = L.FitResult(at["beta"], at["theta"], at["it"], None, None, None, None, None, at["sf"], None, None)
    ctx = dv.context()
    torch.cuda.synchronize()
    ctx.check(L.load().devil_fit_device(ctx.h, C.byref(counts), C.c_void_p(X.data_ptr()), 1, None, 0,
                                        C.byref(opts), C.byref(res)))
    ctx.synchronize()
    # size factors: the column sums over their geometric mean
    sf = out["sf"].cpu().numpy()
    np.testing.assert_allclose(sf / sf[0], want / want[0], rtol=4e-16 * 4)
    # rough beta_0 = log1p(row mean): the exact row sums
    sums = np.add.reduceat(np.append(val.astype(np.float64), 0), np.minimum(ptr[:-1], len(val)))
    sums[np.diff(ptr) == 0] = 0
    np.testing.assert_allclose(out["beta"].cpu().numpy(), np.log1p(sums / n), rtol=1e-15)


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_check_finds_a_fault_at_any_place(dv, shift):
    import torch
    from devil_b200 import _lib as L

    rng = np.random.default_rng(shift)
    n = 1000
    ptr, col, val = _matrix(rng, n, [40, 0, 333, 1, 2, 1000, 0, 5])
    d = torch.device("cuda")
    rp, X = torch.tensor(ptr, device=d), torch.ones(n, dtype=torch.float64, device=d)
    vi = torch.tensor(val.view(np.int16), device=d)
    buf = torch.zeros(len(col) + shift, dtype=torch.int32, device=d)[shift:]
    out = torch.zeros(3 * 8, dtype=torch.float64, device=d)
    at = [C.c_void_p(out.data_ptr() + 64 * i) for i in range(3)]
    res = L.FitResult(at[0], at[1], at[2], None, None, None, None, None, None, None, None)
    counts = L.Counts(L.COUNTS_CSR_U16, 0, 8, n, len(col), vi.data_ptr(), rp.data_ptr(), buf.data_ptr())
    opts = L.FitOpts()
    L.load().devil_fit_opts_default(C.byref(opts))
    opts.max_iter, opts.init_beta_rough = 0, 1
    ctx = dv.context()
    inside = np.setdiff1d(np.arange(len(col)), ptr)  # entries with one before them in their row

    def run(c):
        buf.copy_(torch.tensor(c))
        torch.cuda.synchronize()
        rc = L.load().devil_fit_device(ctx.h, C.byref(counts), C.c_void_p(X.data_ptr()), 1, None, 0,
                                       C.byref(opts), C.byref(res))
        ctx.synchronize()
        return rc

    assert run(col) == L.OK
    for e in np.unique(np.concatenate([inside[:6], inside[-6:], rng.choice(inside, 20)])):
        bad = col.copy()
        bad[e] = bad[e - 1]  # not above the index before it
        assert run(bad) == L.ERR_ARG, e
    for e in (0, 1, len(col) - 1):
        for v in (-1, n):
            bad = col.copy()
            bad[e] = v
            assert run(bad) == L.ERR_ARG, (e, v)
