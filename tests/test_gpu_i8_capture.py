"""The integer GEMM's plans made inside a capture (image lists and row tables
written by the host, a workspace of the graph's own), and its launches when the
workspace finds no memory.  Bit for bit: against eager calls on the integer path,
and, where that path gives way, against DMMA in one K loop per tile."""
import gc
import os

import numpy as np
import pytest

from tests.device_pool import limited

pytestmark = pytest.mark.gpu


def _ctx(sb, **env):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update({k: str(v) for k, v in env.items()})
    try:
        return sb.Context(0)
    finally:
        for k, v in old.items():
            os.environ.pop(k, None) if v is None else os.environ.__setitem__(k, v)


def _operands(rng, ms, ks, n):
    """Blocks A(i, q) and B(q, 1), block (last i, 1) of A missing."""
    A = {(i, q): rng.standard_normal((m, k)) for i, m in enumerate(ms, 1) for q, k in enumerate(ks, 1)
         if (i, q) != (len(ms), 1)}
    return A, {(q, 1): rng.standard_normal((k, n)) for q, k in enumerate(ks, 1)}


def _tensor(sb, ctx, bl):
    keys = sorted(bl, key=lambda k: k[::-1])
    dims = tuple(max(k[a] for k in bl) for a in (0, 1)) + tuple(max(b.shape[a] for b in bl.values()) for a in (0, 1))
    return sb.NewBlockSparseSorted(dims, 2, keys, None, np.concatenate([bl[k].reshape(-1, order="F") for k in keys]),
                                   ctx=ctx, block_dims=[bl[k].shape for k in keys])


def _call(sb, ctx, a, b):
    C = sb.NewBlockSparseSorted.empty((a.dims[0], 1, a.dims[2], b.dims[3]), 2, ctx=ctx)
    return C, lambda: sb.contract_(C, ["i", "j", "m", "n"], a, ["i", "q", "m", "k"], b, ["q", "j", "k", "n"])


@pytest.mark.parametrize("ms,ks,n", [((127, 2, 130), (70, 130), 150), ((64, 64, 128), (900, 65), 90),
                                     ((70, 200), (1900, 700), 33)], ids=["strips", "k_tiles", "split"])
@pytest.mark.parametrize("first", [True, False])
def test_replay_on_new_values(ms, ks, n, first):
    """first: the plan is made in the capture, nothing ran before it."""
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(sum(ms)))
    values = [_operands(rng, ms, ks, n) for _ in range(3)]
    values[1][0][1, 1][0, 3] = np.inf  # the flag is set in this replay and cleared in the next
    eager, ctx = (_ctx(sb, SPARSEB_GEMM_I8=1, SPARSEB_GEMM_THIN=0) for _ in range(2))
    a, b = (_tensor(sb, ctx, x) for x in values[0])
    C, call = _call(sb, ctx, a, b)
    if not first:
        call()
    g = ctx.capture(call, keep=[a, b, C])
    for A, B in values:
        for t, x in ((a, A), (b, B)):
            sb.map_(t, _tensor(sb, ctx, x), sb.MAP_COPY)
        g.launch()
        W, want = _call(sb, eager, _tensor(sb, eager, A), _tensor(sb, eager, B))
        want()
        assert np.array_equal(C.data, W.data, equal_nan=True)
    del g


K, SIDE = 40000, 128  # operands 82 MB, planes 72 MB, partial tiles 7 MB


def _long():
    rng = np.random.Generator(np.random.PCG64(4))
    return {(1, 1): rng.standard_normal((SIDE, K))}, {(1, 1): rng.standard_normal((K, SIDE))}


def _result(sb, A, B, **env):
    ctx = _ctx(sb, **env)
    C, call = _call(sb, ctx, _tensor(sb, ctx, A), _tensor(sb, ctx, B))
    call()
    return C.data


def test_dmma_without_memory_for_the_workspace():
    import sparsebackends_b200 as sb
    A, B = _long()
    want = _result(sb, A, B, SPARSEB_GEMM_I8=0, SPARSEB_GEMM_SPLITK=1, SPARSEB_GEMM_TILE="64x64")
    i8 = _result(sb, A, B, SPARSEB_GEMM_I8=1)
    assert not np.array_equal(want, i8)
    with limited(128 << 20):
        got = _result(sb, A, B, SPARSEB_GEMM_I8=1)
        gc.collect()
    assert np.array_equal(got, want)


def test_workspace_given_back_to_an_allocation():
    """Another tensor of the context takes the kept workspace's place; the call
    runs on DMMA while it does, and on the integer path when it is gone."""
    import sparsebackends_b200 as sb
    A, B = _long()
    dmma = _result(sb, A, B, SPARSEB_GEMM_I8=0, SPARSEB_GEMM_SPLITK=1, SPARSEB_GEMM_TILE="64x64")
    i8 = _result(sb, A, B, SPARSEB_GEMM_I8=1)
    with limited(256 << 20):
        ctx = _ctx(sb, SPARSEB_GEMM_I8=1)
        C, call = _call(sb, ctx, _tensor(sb, ctx, A), _tensor(sb, ctx, B))
        call()
        assert np.array_equal(C.data, i8)
        x = np.arange(17 << 20, dtype=np.float64)
        T = sb.DenseTensor(x, ctx=ctx)
        assert np.array_equal(T.to_numpy(), x)
        call()
        assert np.array_equal(C.data, dmma)
        del T
        gc.collect()
        call()
        assert np.array_equal(C.data, i8)
        del C, call, ctx
        gc.collect()
