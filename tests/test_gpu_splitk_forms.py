"""Split-K in clusters of 16 and through partial tiles (operands beyond twice
L2), every tile shape, uneven K loops and both operand orders, against numpy in
extended precision.  The tolerance is the sum's own rounding bound: K additions
of relative error 2^-53 on the sum of magnitudes."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILES = [None, "64x64", "128x32", "32x128", "64x32", "128x64", "64x128"]


def _ctx(sb, **env):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update({k: str(v) for k, v in env.items()})
    try:
        return sb.Context(0)
    finally:
        for k, v in old.items():
            os.environ.pop(k, None) if v is None else os.environ.__setitem__(k, v)


def _blocks(ms, ks, n, missing):
    rng = np.random.Generator(np.random.PCG64(16))
    A = {(i, q): rng.standard_normal((m, k)) for i, m in ms.items() for q, k in ks.items() if (i, q) not in missing}
    return A, {(q, 1): rng.standard_normal((k, n)) for q, k in ks.items()}


def _check(sb, ctx, A, B, rows, launches=None):
    ms, ks = {k[0]: a.shape[0] for k, a in A.items()}, {k[0]: b.shape[0] for k, b in B.items()}
    n, mm, kk = B[1, 1].shape[1], max(ms.values()), max(ks.values())

    def tensor(bl, dims):
        keys = sorted(bl, key=lambda k: k[::-1])
        return sb.NewBlockSparseSorted(dims, 2, keys, None, np.concatenate([bl[k].reshape(-1, order="F") for k in keys]),
                                       ctx=ctx, block_dims=[bl[k].shape for k in keys])

    a_t, b_t = tensor(A, (len(ms), len(ks), mm, kk)), tensor(B, (len(ks), 1, kk, n))
    for tail, dims in ((["m", "n"], (mm, n)), (["n", "m"], (n, mm))):
        C = sb.NewBlockSparseSorted.empty((len(ms), 1) + dims, 2, ctx=ctx)

        def call():
            sb.contract_(C, ["i", "j"] + tail, a_t, ["i", "q", "m", "k"], b_t, ["q", "j", "k", "n"])

        call()
        before = ctx.launch_count
        call()  # the plan is there: the GEMM's own launches
        if launches is not None:
            assert ctx.launch_count - before == launches
        got, ext = C.blocks_by_key(), dict(zip(C.keys, C.block_dims))
        for i in ms:
            qs = [q for q in ks if (i, q) in A]
            a = np.concatenate([A[i, q][:rows] for q in qs], 1)
            b = np.concatenate([B[q, 1] for q in qs], 0)
            c = got[i, 1].reshape(ext[i, 1], order="F")
            c = (c if tail[0] == "m" else c.T)[:rows]
            want = a.astype(np.longdouble) @ b.astype(np.longdouble)
            assert np.all(np.abs(c - want) <= a.shape[1] * 2.0 ** -53 * (np.abs(a) @ np.abs(b))), (i, tail)


@pytest.mark.parametrize("tile", TILES)
def test_clusters_of_sixteen(tile):
    import sparsebackends_b200 as sb
    env = dict(SPARSEB_GEMM_SPLITK=16, SPARSEB_GEMM_THIN=0, **({"SPARSEB_GEMM_TILE": tile} if tile else {}))
    A, B = _blocks({1: 70, 2: 3, 3: 133}, {1: 5, 2: 200, 3: 17}, 66, ((2, 2), (2, 3)))
    _check(sb, _ctx(sb, **env), A, B, 200, launches=1)


def test_one_tile_with_a_long_k():
    """Chosen by the launch rule: a single tile, 16 segments."""
    import sparsebackends_b200 as sb
    A, B = _blocks({1: 64}, {1: 8192}, 64, ())
    _check(sb, sb.Context(0), A, B, 64, launches=1)


@pytest.fixture(scope="module")
def large():
    return _blocks({1: 70, 2: 130}, {1: 99990, 2: 1, 3: 40000}, 66, ((1, 2),))


@pytest.mark.parametrize("tile", TILES)
def test_partial_tiles_of_operands_beyond_l2(tile, large):
    import sparsebackends_b200 as sb
    ctx = _ctx(sb, **({"SPARSEB_GEMM_TILE": tile} if tile else {}))
    _check(sb, ctx, *large, 4, launches=2)
