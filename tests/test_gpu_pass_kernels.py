"""The kernel that a pass ran on, by design and size."""
import numpy as np
import pytest

from devil_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [9, 16, 32])
def test_wide_continuous_steps(dv, p):
    P = synthetic.make("continuous", seed=p, G=5, n=700, p=p)
    csr = (P.rowptr, P.col, P.val, P.n)
    dv.estimate_mom_dispersion(csr, P.X, P.beta_true, P.sf_true)
    dv.compute_hessian(P.beta_true, P.theta_true, csr, P.X, P.sf_true)
    ctx = dv.context()
    assert [ctx.kernel(k) for k in (1, 3)] == ["mom_cells", "cell64"]
    dv.compute_clustered_meat(P.X, csr, P.beta_true, P.theta_true, P.sf_true, np.array([300, 700], np.int32))
    assert ctx.kernel(3) == "cell64"


def test_fits(dv):
    P = synthetic.make("binary", seed=1, G=30, n=3000)
    x = (P.rowptr, P.col, P.val, P.n)
    dv.fit_devil(x, P.X, overdispersion="MLE", size_factors=P.sf_true)
    ctx = dv.context()
    assert [ctx.kernel(k) for k in range(4)] == ["grp_slices"] * 4
    dv.fit_devil(x, P.X, overdispersion="MLE", size_factors=P.sf_true, form="plain")
    assert [ctx.kernel(k) for k in range(4)] == ["gen_pass"] * 4
    dv.fit_devil(x, P.X, clusters=np.repeat([1, 2, 3], 1000), size_factors=P.sf_true)
    assert ctx.kernel(3) == "grp_pass"
    P = synthetic.make("continuous", seed=2, G=30, n=3000, p=12)
    dv.fit_devil((P.rowptr, P.col, P.val, P.n), P.X, overdispersion="MLE", size_factors=P.sf_true)
    assert [ctx.kernel(k) for k in range(4)] == ["tcw_pass", "mom_cells", "tcw_pass", "cell64"]
