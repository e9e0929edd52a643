"""Bread and meat of continuous designs of three to eight columns: the sizes
where they move from the register engine to the FP64 matrix tiles, genes and
cells off the tiles' multiples of 32, cluster ends inside a chunk of 32 cells."""
import numpy as np
import pytest

from devil_b200 import synthetic
from test_gpu_parity import check_mats

pytestmark = pytest.mark.gpu


def _ends(n, k):
    return np.unique(np.r_[(np.arange(1, k) * n) // k + 5, n]).astype(np.int32)


# FP64 sums of at most 16,400 positive terms (1e-13 relative), inverted at a
# condition below 1e3 on these designs; the meat's residual sums cancel by at most
# 1e3: 1e-10 of the diagonal scale
@pytest.mark.parametrize("p,G,n,clusters,kernel", [
    (3, 1, 65, 0, "reg_pass"), (4, 33, 1000, 0, "reg_pass"), (5, 31, 3001, 0, "reg_pass"), (8, 300, 1500, 0, "reg_pass"),
    (5, 300, 16400, 0, "cell64"), (8, 1001, 5000, 0, "cell64"),
    (3, 1, 97, 3, "reg_pass"), (3, 33, 3000, 75, "cell64"), (4, 65, 1025, 50, "cell64"), (4, 33, 3000, 40, "reg_pass"),
    (5, 31, 1000, 7, "reg_pass"), (5, 33, 1001, 40, "cell64"), (8, 31, 2500, 75, "cell64"), (8, 64, 3000, 7, "reg_pass"),
])
@pytest.mark.parametrize("counts", ["u16", "float"])
def test_routes_match_oracle(dv, orc, p, G, n, clusters, kernel, counts):
    P = synthetic.make("continuous", seed=p + n, G=G, n=n, p=p)
    val = P.val if counts == "u16" else P.val.astype(np.float32)
    csr, b, th, sf = (P.rowptr, P.col, val, n), P.beta_true, P.theta_true, P.sf_true
    some = np.unique(np.r_[0, G // 2, G - 1])  # (the oracle takes a while)
    Y = P.subset_genes(some).dense()
    if clusters:
        ends = _ends(n, clusters)
        got = dv.compute_clustered_meat(P.X, csr, b, th, sf, ends)
        ref = [orc.clustered_meat_fast(P.X, y, b[g], th[g], sf, ends) for g, y in zip(some, Y)]
    else:
        got = dv.compute_hessian(b, th, csr, P.X, sf)
        ref = [orc.compute_hessian(b[g], th[g], y, P.X, sf) for g, y in zip(some, Y)]
    assert dv.context().kernel(3) == kernel
    check_mats(got[some], np.stack(ref), np.ones(len(some), bool), 1e-10, "matrix")


def test_line_of_four_columns(dv):
    # eight blocks an SM of 32 genes x 2,048 cells: 1,184 blocks
    rng = np.random.default_rng(4)
    for n, kernel in ((36 * 2048, "reg_pass"), (38 * 2048, "cell64")):
        X = np.column_stack([np.ones(n), rng.normal(size=(n, 3))])
        cols = np.sort(rng.choice(n, 100, replace=False)).astype(np.int32)
        x = (np.array([0] * 1000 + [100]), cols, np.ones(100, np.uint16), n)
        dv.compute_hessian(np.tile([0.5, 0.1, 0.0, -0.1], (1000, 1)), np.ones(1000), x, X, np.ones(n))
        assert dv.context().kernel(3) == kernel
