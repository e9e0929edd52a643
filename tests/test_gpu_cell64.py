"""The FP64 per-cell passes (MOM moments, bread, clustered meat) at designs of
p = 9..32 continuous columns: tiles of 32 genes and 32 cells with remainders,
every register class of the contraction (p = 9, 13, 14, 17, 18, 23, 24, 28,
32), cluster ends inside a chunk, counts of both types."""
import numpy as np
import pytest

from devil_b200 import synthetic
from test_gpu_parity import check_mats

pytestmark = pytest.mark.gpu


# FP64 sums of at most 3,000 positive terms (1e-13 relative), inverted at a
# condition below 1e3 on these designs: 1e-10 of the diagonal scale; the MOM
# numerator cancels by at most 1e3 at the true coefficients: 1e-10 relative
@pytest.mark.parametrize("p,G,n", [(9, 1, 65), (13, 31, 1000), (14, 33, 1023), (17, 32, 97), (18, 64, 1025),
                                   (23, 5, 2049), (24, 40, 700), (28, 33, 1500), (32, 70, 1025), (32, 3, 3001)])
@pytest.mark.parametrize("counts", ["u16", "float"])
def test_steps_match_oracle(dv, orc, p, G, n, counts):
    P = synthetic.make("continuous", seed=100 * p + G, G=G, n=n, p=p)
    val = P.val if counts == "u16" else P.val.astype(np.float32)
    csr, Y = (P.rowptr, P.col, val, n), P.dense()
    b, th, sf = P.beta_true, P.theta_true, P.sf_true
    ones = np.ones(G, bool)
    bread = dv.compute_hessian(b, th, csr, P.X, sf)
    assert dv.context().engine(3) == "shared"
    check_mats(bread, np.stack([orc.compute_hessian(bb, t, y, P.X, sf) for bb, t, y in zip(b, th, Y)]), ones, 1e-10,
               "bread")
    mom = dv.estimate_mom_dispersion(csr, P.X, b, sf)
    np.testing.assert_allclose(mom, [orc.mom_dispersion(y, P.X, bb, sf) for y, bb in zip(Y, b)], rtol=1e-10, atol=1e-12)
    ends = np.unique(np.r_[1, 2, 33, n // 3, n // 3 + 31, n - 1, n]).astype(np.int32)
    meat = dv.compute_clustered_meat(P.X, csr, b, th, sf, ends)
    check_mats(meat, np.stack([orc.clustered_meat_fast(P.X, y, bb, t, sf, ends) for y, bb, t in zip(Y, b, th)]), ones,
               1e-10, "meat")
