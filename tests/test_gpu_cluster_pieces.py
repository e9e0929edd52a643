"""The clustered meat of a grouped design at cluster ends that cut a design
row's slices (at most 16,384 cells each) in the middle, leave single cells,
and span several slices."""
import numpy as np
import pytest

from devil_b200 import synthetic
from test_gpu_parity import check_mats

pytestmark = pytest.mark.gpu


# the per-cluster sums carry the Gauss rules' bound (1e-11 of the sum of the
# terms' sizes); at the true coefficients the residual sums cancel by less
# than 1e4, and the meat squares them: 1e-6 of the diagonal scale
@pytest.mark.parametrize("counts", ["u16", "float"])
@pytest.mark.parametrize("n,cuts", [
    (40001, [1, 2, 3, 32768, 32769, 40000, 40001]),
    (70000, [20, 21, 69999, 70000]),
    (3000, list(range(30, 3001, 30))),
])
def test_meat_pieces_match_oracle(dv, orc, counts, n, cuts):
    P = synthetic.make("binary", seed=n, G=9, n=n)
    val = P.val if counts == "u16" else P.val.astype(np.float32)
    b, th, sf = P.beta_true, P.theta_true, P.sf_true
    ends = np.asarray(cuts, np.int32)
    meat = dv.compute_clustered_meat(P.X, (P.rowptr, P.col, val, P.n), b, th, sf, ends)
    assert dv.context().engine(3) == "groups"
    ref = np.stack([orc.clustered_meat_fast(P.X, y, bb, t, sf, ends) for y, bb, t in zip(P.dense(), b, th)])
    check_mats(meat, ref, np.ones(P.G, bool), 1e-6, "meat")
