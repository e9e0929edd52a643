"""Fits with a search for theta ("MLE", "new") keep the order of every sum
before it: on grouped designs with groups large enough for several blocks per
Gauss rule, and in clusters, both give the same coefficients bit for bit."""
import numpy as np
import pytest

from devil_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config,seed,G,n", [("binary", 1, 150, 40000), ("clustered", 2, 80, 30000)])
def test_new_and_mle_fits_share_beta(dv, config, seed, G, n):
    P = synthetic.make(config, seed=seed, G=G, n=n)
    seen = np.diff(P.rowptr) / n
    # (the "new" search stops the call on genes that are hardly seen)
    P = P.subset_genes(np.flatnonzero((seen > 0.02) & (seen < 0.7)))
    fits = [dv.fit_devil((P.rowptr, P.col, P.val, P.n), P.X, clusters=P.clusters, overdispersion=od,
                         size_factors=P.sf_true) for od in ("MLE", "new")]
    assert dv.context().engine(0) == "groups"
    np.testing.assert_array_equal(fits[0]["beta"], fits[1]["beta"])
