"""Two-sided t tails of test_de around the switch between the large-df series
and the continued fraction (df = 60, log(1 + t^2/df) = 1), for gene counts
around the genes a warp takes, plain and clustered.  The reference is the
incomplete beta in 30 digits: the oracle's continued fraction drifts by 7e-12
near t = 2 at df = 10^5."""
import mpmath
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def two_sided(t, df):
    with mpmath.workdps(30):
        t, d = mpmath.mpf(float(t)), mpmath.mpf(df)
        return float(mpmath.betainc(d / 2, mpmath.mpf(1) / 2, 0, d / (d + t * t), regularized=True))


# exp(-z), z up to 700, carries about z * 2^-52: 1e-12 relative
@pytest.mark.parametrize("G,p,clustered", [(1, 1, False), (7, 2, True), (8, 32, False), (257, 5, True)])
@pytest.mark.parametrize("n", [12, 61, 62, 63, 200, 100002])
def test_tails_match_oracle(dv, orc, G, p, clustered, n):
    rng = np.random.default_rng([G, n])
    # t from 1e-6 to beyond the switch at t^2 = (e - 1) df, its two sides included
    edge = np.sqrt((np.e - 1.0) * (n - 2.0))
    t = np.concatenate([[0.0, 1e-6, edge * (1 - 1e-9), edge * (1 + 1e-9), 36.0],
                        10.0 ** rng.uniform(-3, 1.5, max(0, G - 5))])[:G]
    bread = np.zeros((G, p, p)) + np.eye(p) * rng.lognormal(0, 1, (G, 1, 1))
    sw = bread * rng.lognormal(0, 0.5, (G, 1, 1)) if clustered else None
    beta = rng.normal(size=(G, p))
    beta[:, 0] = t * np.sqrt(bread[:, 0, 0])
    c = np.zeros(p)
    c[0] = 1.0
    fit = dict(beta=beta, beta_sandwiches_null=bread, beta_sandwiches=sw, design_matrix=np.ones((n, p)))
    got = dv.test_de(fit, c, pval_adjust_method="none")
    _, _, lfc = orc.test_de(beta, bread, sw, n, c)
    np.testing.assert_array_equal(got["lfc"], lfc)
    sd = [np.sqrt(m[:, 0, 0]) for m in ([bread] if sw is None else [bread, sw])]
    pv = np.array([max(two_sided(abs(b) / s[g], n - 2.0) for s in sd) for g, b in enumerate(beta[:, 0])])
    ok = pv > 1e-300
    assert np.abs(got["pval"] / np.where(ok, pv, 1.0) - 1.0)[ok].max() <= 1e-12
    assert np.all(got["pval"][~ok] <= 1e-299)
