"""The slice-ordered copy of the counts: rows shorter and longer than the
2,048-entry tiles, designs on both sides of the 24 rows and of the 1,024 keys
where the copy changes kernels."""
import numpy as np
import pytest

from test_gpu_parity import check_mats

pytestmark = pytest.mark.gpu


# sums of FP64 terms per cluster with the Gauss rules' bound (1e-11 of the sum of
# the terms' sizes); the residual sums cancel by less than 1e4 and the meat
# squares them: 1e-6 of the diagonal scale
@pytest.mark.parametrize("counts", ["u16", "float"])
@pytest.mark.parametrize("rows,n", [(23, 9000), (24, 9000), (61, 20000), (256, 20000)])
def test_meat_at_tile_edges_matches_oracle(dv, orc, counts, rows, n):
    rng = np.random.default_rng(rows)
    x = rng.integers(0, rows, n)
    x[:rows] = np.arange(rows)
    X = np.stack([np.ones(n), x / rows], 1)
    lens = [1, 31, 2047, 2048, 2049, 4096, 6200, n]
    cols, vals = [], []
    for m in lens:
        cols.append(np.sort(rng.choice(n, m, replace=False)).astype(np.int32))
        vals.append(rng.integers(1, 40000, m) if m < 40 else rng.poisson(2.0, m) + 1)
    rowptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = np.concatenate(cols)
    val = np.concatenate(vals).astype(np.uint16 if counts == "u16" else np.float32)
    G = len(lens)
    Y = np.zeros((G, n))
    for g in range(G):
        Y[g, cols[g]] = vals[g]
    sf = np.exp(rng.normal(0, 0.3, n))
    b = np.stack([np.log(Y.sum(1) / sf.sum()), np.full(G, 0.1)], 1)
    th = np.linspace(0.2, 1.5, G)
    ends = np.asarray([n // 3, n // 2, n], np.int32)
    meat = dv.compute_clustered_meat(X, (rowptr, col, val, n), b, th, sf, ends)
    assert dv.context().engine(3) == "groups"
    ref = np.stack([orc.clustered_meat_fast(X, Y[g], b[g], th[g], sf, ends) for g in range(G)])
    check_mats(meat, ref, np.ones(G, bool), 1e-6, "meat")


# the same bounds on a converged step: see the tolerances of the design-group tests (1e-8)
@pytest.mark.parametrize("clusters", [32, 33])
def test_fit_at_key_line_matches_oracle(dv, orc, clusters):
    """32 design rows in 32 and 33 clusters: MLE fits cut the slices by cluster (1,024 and 1,056 keys)."""
    rng = np.random.default_rng(clusters)
    n, G = 9000, 5
    x = rng.integers(0, 32, n)
    X = np.stack([np.ones(n), x / 32], 1)
    Y = rng.poisson(rng.gamma(2.0, 0.5, (G, n)) * 4.0 * np.exp(0.5 * X[:, 1])).astype(np.float64)
    sf = np.exp(rng.normal(0, 0.2, n))
    cl = np.sort(np.concatenate([np.arange(clusters), rng.integers(0, clusters, n - clusters)]))
    off = orc.offset_vector(0.0, n, sf)
    th0, b0 = orc.estimate_dispersion(Y, off), orc.init_beta(Y, X, off)
    ref = orc.cpu_fit(Y, X, off, th0, b0, orc.OD_MLE, 200, 1e-3)
    fit = dv.fit_devil(Y, X, overdispersion="MLE", size_factors=sf, clusters=cl)
    assert dv.context().engine(0) == "groups"
    np.testing.assert_array_equal(fit["iterations"]["beta_iters"], ref["iters"])
    assert np.abs(fit["beta"] - ref["beta"]).max() <= 1e-8
