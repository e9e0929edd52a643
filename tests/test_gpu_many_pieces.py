"""A clustered meat whose slices, cut by design row alone, would give more pieces
(slice x cluster) than a block's shared memory holds: two design rows in 2,048
clusters and 18 M cells."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_meat_of_many_clusters(dv):
    n, C, G = 18_000_000, 2048, 2
    rng = np.random.default_rng(1)
    cond = np.arange(n) % 2
    X = np.column_stack([np.ones(n), cond])
    lens = [40000, 300000]
    cols = [np.unique(rng.integers(0, n, k)).astype(np.int32) for k in lens]
    vals = [rng.integers(1, 9, len(c)).astype(np.uint16) for c in cols]
    rowptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int64)
    b = np.array([[-4.0, 0.3], [-2.5, -0.2]])
    th = np.array([0.4, 1.5])
    ends = ((np.arange(1, C + 1) * n) // C).astype(np.int32)
    meat = dv.compute_clustered_meat(X, (rowptr, np.concatenate(cols), np.concatenate(vals), n), b, th, np.ones(n), ends)
    assert dv.context().kernel(3) == "grp_pass"
    starts = np.concatenate([[0], ends[:-1]])
    for g in range(G):
        mu = np.exp(b[g, 0] + b[g, 1] * cond)
        r = -mu
        r[cols[g]] += vals[g]
        r /= 1 + th[g] * mu
        s = np.column_stack([np.add.reduceat(r, starts), np.add.reduceat(r * cond, starts)])
        ref = s.T @ s * (C / (C - 1) / n)
        # the cluster sums carry the rules' 1e-11 of the sum of the terms' sizes and
        # are not small beside it (counts well off the coefficients): 1e-9
        np.testing.assert_allclose(meat[g], ref, rtol=1e-9)


# the same terms summed in another order; the residual sums cancel by at most 1e4
# and the meat squares them: 1e-10 of the diagonal scale
def test_meat_of_a_fit_cut_at_the_clusters(dv):
    """A fit with MLE cuts its slices at the clusters (every piece is a slice), the
    single step by design row (three pieces a slice)."""
    from devil_b200 import synthetic
    P = synthetic.make("binary", seed=3, G=20, n=30000)
    clusters = np.repeat([1, 2, 3], [8000, 2000, 20000])
    f = dv.fit_devil((P.rowptr, P.col, P.val, P.n), P.X, clusters=clusters, overdispersion="MLE", size_factors=P.sf_true)
    meat = dv.compute_clustered_meat(P.X, (P.rowptr, P.col, P.val, P.n), f["beta"], f["overdispersion"], P.sf_true,
                                     np.array([8000, 10000, 30000], np.int32))
    d = np.sqrt(np.einsum("gii->gi", meat))
    assert np.nanmax(np.abs(f["meat"] - meat) / (d[:, :, None] * d[:, None, :])) <= 1e-10
