"""Split-K over a thread-block cluster: every split factor, fewer k-tiles than
segments, uneven K loops over the C blocks, and each tile shape, against numpy
in extended precision.  The tolerance is the sum's own rounding bound: K
additions of relative error 2^-53 on the sum of magnitudes."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ctx(sb, **env):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update({k: str(v) for k, v in env.items()})
    try:
        return sb.Context(0)
    finally:
        for k, v in old.items():
            os.environ.pop(k, None) if v is None else os.environ.__setitem__(k, v)


@pytest.mark.parametrize("tile", [None, "64x64", "128x32", "32x128", "64x32", "128x64"])
@pytest.mark.parametrize("splitk", [1, 2, 5, 8])
def test_cluster_split_sums(splitk, tile):
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(splitk))
    env = dict(SPARSEB_GEMM_SPLITK=splitk, SPARSEB_GEMM_I8=0, SPARSEB_GEMM_THIN=0, SPARSEB_POISON_OUTPUT=1)
    if tile:
        env["SPARSEB_GEMM_TILE"] = tile
    ctx = _ctx(sb, **env)
    ms, ks, n = {1: 70, 2: 3, 3: 133}, {1: 5, 2: 200, 3: 17}, 66
    A = {(i, q): rng.standard_normal((m, k)) for i, m in ms.items() for q, k in ks.items() if (i, q) not in ((2, 2), (2, 3))}
    B = {(q, 1): rng.standard_normal((k, n)) for q, k in ks.items()}

    def tensor(bl, dims):
        keys = sorted(bl, key=lambda k: k[::-1])
        return sb.NewBlockSparseSorted(dims, 2, keys, None, np.concatenate([bl[k].reshape(-1, order="F") for k in keys]),
                                       ctx=ctx, block_dims=[bl[k].shape for k in keys])

    for tail, dims in ((["m", "n"], (133, n)), (["n", "m"], (n, 133))):
        C = sb.NewBlockSparseSorted.empty((3, 1) + dims, 2, ctx=ctx)
        sb.contract_(C, ["i", "j"] + tail, tensor(A, (3, 3, 133, 200)), ["i", "q", "m", "k"],
                     tensor(B, (3, 1, 200, n)), ["q", "j", "k", "n"])
        got, ext = C.blocks_by_key(), dict(zip(C.keys, C.block_dims))
        for i in ms:
            qs = [q for q in ks if (i, q) in A]
            a = np.concatenate([A[i, q] for q in qs], 1).astype(np.longdouble)
            b = np.concatenate([B[q, 1] for q in qs], 0).astype(np.longdouble)
            c = got[i, 1].reshape(ext[i, 1], order="F")
            c = c if tail[0] == "m" else c.T
            assert np.all(np.abs(c - a @ b) <= a.shape[1] * 2.0 ** -53 * (np.abs(a) @ np.abs(b))), (i, splitk, tile)
