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
