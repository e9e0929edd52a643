"""The wide tensor-core passes without the products' image (it does not fit the
free memory): products formed in the block, the same split, the same sums."""
import numpy as np
import pytest

from devil_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", ["u16", "float"])
@pytest.mark.parametrize("p,n", [(9, 31), (9, 2501), (16, 4001), (18, 1000), (32, 3001)])
def test_same_bits_without_the_image(dv, monkeypatch, p, n, counts):
    P = synthetic.make("continuous", seed=p + n, G=150, n=n, p=p)
    val = P.val if counts == "u16" else P.val.astype(np.float32)
    fits = []
    for image, kernel in (("1", "tcw_pass"), ("0", "tcw_pass without image")):
        monkeypatch.setenv("DEVIL_TCW_IMAGE", image)
        # (one segmentation: the tuner picks by time)
        monkeypatch.setenv("DEVIL_AUTOTUNE", "0")
        fits.append(dv.fit_devil((P.rowptr, P.col, val, n), P.X, overdispersion="MLE", size_factors=P.sf_true,
                                 max_iter=20))
        assert [dv.context().kernel(k) for k in (0, 2)] == [kernel, kernel]
    for k in ("beta", "overdispersion", "beta_sandwiches_null"):
        np.testing.assert_array_equal(fits[0][k], fits[1][k])
