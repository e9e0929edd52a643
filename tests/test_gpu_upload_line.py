"""Host arrays around the size from which they go to the device through pinned
chunks, and around the number of chunks at which a third thread fills them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LINE, CHUNK = 8 << 20, 512 << 10


@pytest.mark.parametrize("nbytes", [LINE - 8, LINE, LINE + 8, 32 * CHUNK - 8, 32 * CHUNK + 8, 129 * CHUNK])
def test_upload_is_exact(dv, nbytes):
    p = np.random.default_rng(nbytes).random(nbytes // 8)
    for _ in range(2):
        np.testing.assert_array_equal(dv.p_adjust(p, "none"), p)
