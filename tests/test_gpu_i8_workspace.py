"""The workspace that a context keeps for the integer GEMM: given back when a
capture begins and with the context's last tensor."""
import gc
import os

import numpy as np
import pytest

from tests.device_pool import used_bytes

pytestmark = pytest.mark.gpu


def _ctx(sb, **env):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update({k: str(v) for k, v in env.items()})
    try:
        return sb.Context(0)
    finally:
        for k, v in old.items():
            os.environ.pop(k, None) if v is None else os.environ.__setitem__(k, v)


def _product(sb, ctx, n=512):
    rng = np.random.Generator(np.random.PCG64(2))
    A = sb.NewBlockSparseSorted((1, 1, n, n), 2, [(1, 1)], None, rng.standard_normal(n * n), ctx=ctx)
    B = sb.NewBlockSparseSorted((1, 1, n, n), 2, [(1, 1)], None, rng.standard_normal(n * n), ctx=ctx)
    C = sb.NewBlockSparseSorted.empty((1, 1, n, n), 2, ctx=ctx)

    def call():
        sb.contract_(C, ["i", "j", "m", "n"], A, ["i", "q", "m", "k"], B, ["q", "j", "k", "n"])

    return call, (A, B, C)


PLANES = 2 * 7 * 512 * 512  # of both operands: at least this much workspace


def test_given_back_when_a_capture_begins():
    import sparsebackends_b200 as sb
    ctx = _ctx(sb, SPARSEB_GEMM_I8=1)
    call, (A, B, C) = _product(sb, ctx)
    call()
    want, held = C.data, used_bytes(ctx)
    g = ctx.capture(lambda: sb.scale_(C, 1.0), keep=[C])
    assert held - used_bytes(ctx) >= PLANES
    call()  # and made anew
    assert np.array_equal(C.data, want) and used_bytes(ctx) >= held - (1 << 20)
    del g


def test_given_back_with_the_last_tensor():
    import sparsebackends_b200 as sb
    ctx = _ctx(sb, SPARSEB_GEMM_I8=1)
    gc.collect()
    base = used_bytes(ctx)
    call, tensors = _product(sb, ctx)
    call()
    assert used_bytes(ctx) - base >= 3 * 8 * 512 * 512 + PLANES
    del call, tensors
    gc.collect()
    assert used_bytes(ctx) - base < PLANES  # the plan's arrays stay
    call, tensors = _product(sb, ctx)
    call()
    a, b, c = (t.data.reshape(512, 512, order="F") for t in tensors)
    assert np.allclose(c, a @ b, rtol=0, atol=1e-11)
