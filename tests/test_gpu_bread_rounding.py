"""Rounding of the FP64 bread of continuous designs against 80-bit sums: runs of
cells are summed apart, so the error stays that of short sums."""
import numpy as np
import pytest

from devil_b200 import synthetic

pytestmark = pytest.mark.gpu


# One FP64 rounding is u = 2^-53 / sqrt(3) = 6.4e-17 rms.  2,000 cells in runs of
# 64 added up per 1,024: sqrt((64 / 1024) * 64 / 3 + 16 / 3) / sqrt(2) = 1.8 u on an
# entry of H, and about as much again from the inverse: 2.3 u = 1.5e-16 rms of the
# diagonal scale (one sum over 1,024 cells: 13 u on an entry of H).
@pytest.mark.parametrize("p", [9, 12, 16])
def test_bread_rounds_like_short_sums(dv, p):
    G, n, ld = 16, 2000, np.longdouble
    P = synthetic.make("continuous", seed=7, G=G, n=n, p=p)
    b, th, sf = P.beta_true, P.theta_true, P.sf_true
    got = dv.compute_hessian(b, th, (P.rowptr, P.col, P.val, n), P.X, sf)
    X, Y, err = P.X.astype(ld), P.dense(), []
    for g in range(G):
        mu = np.exp(X @ b[g].astype(ld) + np.log(sf).astype(ld))
        H = (X * ((Y[g] * ld(th[g]) + 1) * mu / (1 + ld(th[g]) * mu) ** 2)[:, None]).T @ X
        B = np.linalg.inv(H.astype(np.float64)).astype(ld)
        for _ in range(3):  # Newton steps of the inverse in 80 bits
            B = B @ (2 * np.eye(p, dtype=ld) - H @ B)
        s = np.sqrt(np.diag(B))
        err.append((got[g] - B) / np.outer(s, s))
    assert np.sqrt(np.mean(np.square(err))) <= 1.5e-16
