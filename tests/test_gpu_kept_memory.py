"""Device memory that a context keeps between calls does not take it from another
caller: idle batch workers are given back to any context that runs short."""
import ctypes as C

import numpy as np
import pytest

from devil_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture
def own(dv):
    """A context of its own as the process's default one."""
    kept = dict(dv._lib._contexts)
    dv._lib._contexts.clear()
    yield dv.context()
    dv.context().close()
    dv._lib._contexts.clear()
    dv._lib._contexts.update(kept)


def _free():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _adjust(dv, ctx, p):
    out = np.empty(len(p))
    at = lambda a: a.ctypes.data_as(C.c_void_p)
    return dv.load_library().devil_p_adjust(ctx.h, len(p), at(p), 1, at(out))


def test_idle_batch_workers_are_given_back(dv, own):
    import torch
    rng = np.random.default_rng(1)
    p = rng.random(1 << 24)
    # what the other context's call takes
    a = _free()
    ctx = dv._lib.Context(0)
    assert _adjust(dv, ctx, p) == 0
    takes = a - _free()
    ctx.close()
    # two workers with dense matrices of 80 MB
    P = synthetic.make("binary", seed=2, G=1000, n=10000)
    b = _free()
    for _ in range(2):
        dv.fit_devil_batch([(P.dense(), P.X)] * 2, overdispersion="MOM", workers=2)
    held = b - _free()
    assert 150 << 20 < held < 700 << 20
    # all but half of what the workers hold is missing
    ctx = dv._lib.Context(0)
    fill = torch.empty(_free() - takes + held // 2, dtype=torch.uint8, device="cuda")
    try:
        assert _adjust(dv, ctx, p) == 0
    finally:
        del fill
        ctx.close()
    assert _free() > b - (64 << 20)  # (the workers are gone)


def test_a_second_fit_takes_the_same_engine(dv, own):
    """A wide continuous fit whose count image (4 GB) just fits half of the free
    memory: the first call's images are the second call's."""
    import torch
    G, n, p = 4000, 500000, 9
    rng = np.random.default_rng(3)
    X = np.column_stack([np.ones(n), rng.normal(size=(n, p - 1))])
    cols = [np.unique(rng.integers(0, n, 400)).astype(np.int32) for _ in range(G)]
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int64)
    x = (ptr, np.concatenate(cols), np.ones(int(ptr[-1]), np.uint16), n)
    run = lambda: dv.fit_devil(x, X, overdispersion=False, max_iter=2)["beta"]
    fill = torch.empty(_free() - (11 << 30), dtype=torch.uint8, device="cuda")
    try:
        first = run()
        assert own.kernel(0) == "tcw_pass"
        np.testing.assert_array_equal(run(), first)
        assert own.kernel(0) == "tcw_pass"
    finally:
        del fill
