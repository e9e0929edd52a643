"""Host arrays on both sides of the staged upload's size and chunk edges, and
devil_fit_batch over workers kept from call to call, from several threads, and
after a problem that fails."""
import threading

import numpy as np
import pytest

from devil_b200 import synthetic

pytestmark = pytest.mark.gpu

MIN, CHUNK = 4 << 20, 512 << 10


@pytest.mark.parametrize("nbytes", [MIN - 8, MIN, MIN + 8, MIN + CHUNK, 9 * CHUNK + 8, 40 * CHUNK - 8])
def test_upload_is_exact(dv, nbytes):
    rng = np.random.default_rng(nbytes)
    for _ in range(2):
        p = rng.random(nbytes // 8)
        np.testing.assert_array_equal(dv.p_adjust(p, "none"), p)


def _problems(seeds):
    ps = [synthetic.make("binary", seed=s, G=200, n=400 + 300 * s) for s in seeds]
    return [((P.rowptr, P.col, P.val, P.n), P.X) for P in ps]


def _check(dv, problems, fits):
    for (x, X), f in zip(problems, fits):
        r = dv.fit_devil(x, X, overdispersion="MLE", size_factors="normed_sum")
        for k in ("beta", "overdispersion", "beta_sandwiches_null"):
            np.testing.assert_array_equal(f[k], r[k])


def _batch(dv, problems, workers=4):
    return dv.fit_devil_batch(problems, overdispersion="MLE", size_factors="normed_sum", workers=workers)


def test_batches_on_kept_workers(dv):
    for seeds, workers in (([1, 2], 2), ([3, 4, 5, 6, 7], 4), ([1], 1)):
        problems = _problems(seeds)
        _check(dv, problems, _batch(dv, problems, workers))
    x, X = _problems([2])[0]
    with pytest.raises(Exception):
        _batch(dv, [(x, X), (x, np.repeat(X[:, :1], 2, 1))])  # a rank-deficient design
    problems = _problems([5, 2, 3])
    _check(dv, problems, _batch(dv, problems))


def test_batches_of_several_threads(dv):
    sets = [_problems([1, 2, 3]), _problems([4, 5]), _problems([6, 1])]
    out = [None] * 3

    def run(i):
        for _ in range(3):
            out[i] = _batch(dv, sets[i], 2)

    th = [threading.Thread(target=run, args=(i,)) for i in range(3)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for s, o in zip(sets, out):
        _check(dv, s, o)
