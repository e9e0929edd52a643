"""Preparation of grouped designs: Gauss rules built by one, two, four and
eight blocks per rule (groups around 8,192, 16,384 and 65,536 cells, one of
them tiny), X'X from the distinct rows, size factors and theta_0 in passes."""
import numpy as np
import pytest

from devil_b200 import synthetic

pytestmark = pytest.mark.gpu


# the rules hold 1e-11 and a term's reciprocal 1e-12 relative; a converged
# step's conditioning amplifies them by 1e3 at most on these designs: 1e-8.
# The bread is the inverse of sums with the same bounds: 1e-8 of its scale.
@pytest.mark.parametrize("n,first", [(3000, 40), (16383, 8191), (16384, 8192), (32770, 16385), (131074, 65537),
                                     (131080, 37)])
def test_group_sizes_match_oracle(dv, orc, n, first):
    P = synthetic.make("binary", seed=n, G=5, n=n)
    X = P.X.copy()
    X[:, 1] = (np.arange(n) >= first).astype(float)
    sf = P.sf_true * np.where(np.arange(n) % 97 == 0, 9.0, 1.0)  # several offset bins
    Y = P.csr_f64()
    off = orc.offset_vector(0.0, n, sf)
    th0, b0 = orc.estimate_dispersion(Y, off), orc.init_beta(Y, X, off)
    ref = orc.cpu_fit(Y, X, off, th0, b0, orc.OD_MOM, 200, 1e-3)
    fit = dv.fit_devil((P.rowptr, P.col, P.val, n), X, overdispersion="MOM", size_factors=sf)
    assert dv.context().engine(0) == "groups"
    np.testing.assert_array_equal(fit["iterations"]["beta_iters"], ref["iters"])
    conv = ref["iters"] < 200
    assert conv.any()
    assert np.abs(fit["beta"] - ref["beta"])[conv].max() <= 1e-8
    d = np.sqrt(np.abs(np.einsum("gii->gi", ref["bread"])))
    r = np.abs(fit["beta_sandwiches_null"] - ref["bread"]) / (d[:, :, None] * d[:, None, :])
    assert r[conv].max() <= 1e-8


@pytest.mark.parametrize("n", [5, 1023, 1024, 16385, 40001])
def test_size_factors_match_oracle(dv, orc, n):
    rng = np.random.default_rng(n)
    Y = rng.poisson(3.0, (12, n)).astype(np.float64)
    Y[0] += 1.0
    # sums of n terms in another order than the oracle's: n * 2^-53 at most
    np.testing.assert_allclose(dv.calculate_sf(Y, "normed_sum"), orc.calculate_sf(Y, "normed_sum"), rtol=1e-12)
