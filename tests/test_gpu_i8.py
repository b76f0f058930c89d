"""FP64 block GEMMs on the integer tensor cores (SPARSEB_GEMM_I8=1 takes them
at every size) at the edges of their tiles, k-tiles and chunks.

Reference: numpy's extended precision (64-bit mantissa).  Tolerance, against
|row| |column| (2-norms): an element's rounding to its row's scale is at most
2^-55 of the row's largest magnitude and random in sign, so each side adds at
most 2^-55 / sqrt(3) (root mean square, attained when one element carries the
row), the digit products left out less, and each FP64 addition of a pass
2^-53 of the partial sum.  Eight times 2^-55 is above six standard deviations
of their sum.
"""
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


def _run(sb, ctx, A, B, order, capfd=None):
    """C(i, j | m, n) = sum_{q, k} A(i, q | m, k) B(q, j | k, n): A and B dicts
    of blocks; order "AB" asks for tails (m, n), "BA" for (n, m)."""
    nq = max(k[1] for k in A)
    ni, nj = max(k[0] for k in A), max(k[1] for k in B)
    mx = [max(b.shape[0] for b in A.values()), max(b.shape[1] for b in A.values()), max(b.shape[1] for b in B.values())]

    def tensor(bl, dims):
        keys = sorted(bl, key=lambda k: k[::-1])
        return sb.NewBlockSparseSorted(dims, 2, keys, None, np.concatenate([bl[k].reshape(-1, order="F") for k in keys]),
                                       ctx=ctx, block_dims=[bl[k].shape for k in keys])

    a, b = tensor(A, (ni, nq, mx[0], mx[1])), tensor(B, (nq, nj, mx[1], mx[2]))
    tail = ["m", "n"] if order == "AB" else ["n", "m"]
    dims = (ni, nj) + ((mx[0], mx[2]) if order == "AB" else (mx[2], mx[0]))
    C = sb.NewBlockSparseSorted.empty(dims, 2, ctx=ctx)
    sb.contract_(C, ["i", "j"] + tail, a, ["i", "q", "m", "k"], b, ["q", "j", "k", "n"])
    out = {}
    got, ext = C.blocks_by_key(), dict(zip(C.keys, C.block_dims))
    for k, v in got.items():
        x = v.reshape(ext[k], order="F")
        out[k] = x if order == "AB" else x.T
    return out


def _blocks(rng, m, n, ks, fill=None):
    f = fill or (lambda shape: rng.standard_normal(shape))
    A = {(1, q + 1): f((m, k)) for q, k in enumerate(ks)}
    B = {(q + 1, 1): f((k, n)) for q, k in enumerate(ks)}
    return A, B


def _worst(got, A, B):
    """Largest |error| over |row| |column|, both over all pairs."""
    ld = np.longdouble
    want = sum(A[1, q].astype(ld) @ B[q, 1].astype(ld) for q in range(1, len(B) + 1))
    ra = np.sqrt(sum((A[1, q] ** 2).sum(1) for q in range(1, len(B) + 1)))
    cb = np.sqrt(sum((B[q, 1] ** 2).sum(0) for q in range(1, len(B) + 1)))
    err = np.abs(got[1, 1].astype(ld) - want).astype(float)
    return float(np.max(err / np.maximum(np.outer(ra, cb), 1e-300))), err


SIZES = [(1, 1, (17,)), (16, 17, (63,)), (127, 128, (64,)), (128, 129, (65,)), (129, 127, (1, 40)), (300, 33, (1535,)),
         (40, 300, (1536,)), (65, 257, (1537,)), (130, 144, (3100, 7)), (257, 130, (200, 64, 129))]


@pytest.mark.parametrize("order", ["AB", "BA"])
@pytest.mark.parametrize("m,n,ks", SIZES)
def test_edges_of_tiles_and_chunks(m, n, ks, order):
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(m * 7 + n))
    A, B = _blocks(rng, m, n, ks)
    got = _run(sb, _ctx(sb, SPARSEB_GEMM_I8=1, SPARSEB_GEMM_THIN=0, SPARSEB_POISON_OUTPUT=1), A, B, order)
    assert _worst(got, A, B)[0] <= 8 * 2.0 ** -55


@pytest.mark.parametrize("order", ["AB", "BA"])
@pytest.mark.parametrize("m,n,ks", [(15, 16, (768, 1)), (17, 31, (767,)), (33, 129, (769, 5)), (145, 47, (64, 703))])
def test_edges_of_strips(m, n, ks, order):
    """Packing in strips of 16 rows while every K is at most 768."""
    test_edges_of_tiles_and_chunks(m, n, ks, order)


@pytest.mark.parametrize("kind", ["gaussian", "graded_k", "graded_rows", "one_large", "opposed", "positive"])
def test_error_not_above_dmma(kind):
    """Root-mean-square error against |row| |column|, next to the DMMA path's,
    on inputs whose magnitudes vary along every index."""
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(11))
    m, n, ks = 150, 170, (400, 333)
    A, B = _blocks(rng, m, n, ks)
    for q, k in enumerate(ks, 1):
        s = 10.0 ** np.linspace(0, -6, k)
        if kind == "graded_k":
            A[1, q] *= s[None, :]
            B[q, 1] *= s[:, None]
        elif kind == "opposed":
            A[1, q] *= s[None, :] ** 0.5
            B[q, 1] *= s[::-1, None] ** 0.5
        elif kind == "graded_rows":
            A[1, q] *= 10.0 ** np.linspace(0, -9, m)[:, None]
            B[q, 1] *= 10.0 ** np.linspace(5, -5, n)[None, :]
        elif kind == "one_large":
            A[1, q][:, 3] *= 1e5
        elif kind == "positive":
            A[1, q], B[q, 1] = np.abs(A[1, q]), np.abs(B[q, 1])
    rms = {}
    for v in (0, 1):
        got = _run(sb, _ctx(sb, SPARSEB_GEMM_I8=v), A, B, "AB")
        ra = np.sqrt(sum((A[1, q] ** 2).sum(1) for q in (1, 2)))
        cb = np.sqrt(sum((B[q, 1] ** 2).sum(0) for q in (1, 2)))
        rms[v] = float(np.sqrt(np.mean((_worst(got, A, B)[1] / np.outer(ra, cb)) ** 2)))
    print(kind, rms)
    assert rms[1] <= max(rms[0], 2.0 ** -55)


@pytest.mark.parametrize("what", ["inf", "nan", "huge", "tiny", "subnormal", "zero_rows", "zero_block"])
def test_values_outside_the_scale_range(what):
    """Rows that the integer path does not take are recomputed with DMMA in one
    K loop per tile: the values, infinities and NaN of the DMMA path unsplit."""
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(3))
    A, B = _blocks(rng, 140, 150, (90, 70))
    if what == "inf":
        A[1, 1][5, 7] = np.inf
    elif what == "nan":
        B[2, 1][5, 7] = np.nan
    elif what == "huge":
        A[1, 2][9, :] *= 1e200
    elif what == "tiny":
        B[1, 1][:, 4] *= 1e-200
    elif what == "subnormal":
        A[1, 1][3, :] = 5e-324
    elif what == "zero_rows":
        A[1, 1][3, :] = 0.0
        A[1, 2][3, :] = 0.0
        B[1, 1][:, 149] = 0.0
    else:
        A[1, 1][:] = 0.0
    x = _run(sb, _ctx(sb, SPARSEB_GEMM_I8=1), A, B, "AB")[1, 1]
    y = _run(sb, _ctx(sb, SPARSEB_GEMM_I8=0, SPARSEB_GEMM_SPLITK=1), A, B, "AB")[1, 1]
    assert np.array_equal(np.isnan(x), np.isnan(y)) and np.array_equal(np.isinf(x), np.isinf(y))
    f = np.isfinite(y)
    if what in ("zero_rows", "zero_block"):
        assert np.array_equal(x == 0.0, y == 0.0)
        assert _worst({(1, 1): x}, A, B)[0] <= 8 * 2.0 ** -55
    else:
        assert np.array_equal(x[f], y[f])


def test_split_tiles_and_many_blocks():
    """Few tiles with a long K (k-segments summed from partial tiles) beside
    blocks of other extents, and a graph replay on new values."""
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(8))
    ks = (1900, 700, 1200)
    A = {(i, q + 1): rng.standard_normal((m, k)) for i, m in ((1, 70), (2, 200), (3, 1)) for q, k in enumerate(ks)
         if (i, q) != (2, 1)}
    B = {(q + 1, j): rng.standard_normal((k, n)) for j, n in ((1, 90), (2, 33)) for q, k in enumerate(ks)}
    got = _run(sb, _ctx(sb, SPARSEB_GEMM_I8=1), A, B, "AB")
    for (i, j), c in got.items():
        qs = [q for q in (1, 2, 3) if (i, q) in A]
        a = np.concatenate([A[i, q] for q in qs], 1)
        b = np.concatenate([B[q, j] for q in qs], 0)
        want = (a.astype(np.longdouble) @ b.astype(np.longdouble)).astype(float)
        scale = np.outer(np.sqrt((a ** 2).sum(1)), np.sqrt((b ** 2).sum(0)))
        assert np.max(np.abs(c - want) / scale) <= 8 * 2.0 ** -55, (i, j)


@pytest.mark.parametrize("ms", [(1, 1, 1), (127, 2, 130), (64, 64, 128), (5, 251, 17)])
@pytest.mark.parametrize("order", ["AB", "BA"])
def test_rows_stacked_over_output_blocks(ms, order):
    """Output blocks that read the same Y blocks share row tiles: stacks whose
    joints fall anywhere in a tile, beside a block with another list of pairs
    and an extent of its own, either operand order."""
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(sum(ms)))
    ks = (70, 130)
    A = {(i + 1, q + 1): rng.standard_normal((m, k)) for i, m in enumerate(ms) for q, k in enumerate(ks)}
    A[4, 2] = rng.standard_normal((77, 130))
    B = {(q + 1, j): rng.standard_normal((k, n)) for j, n in ((1, 90), (2, 150)) for q, k in enumerate(ks)}
    got = _run(sb, _ctx(sb, SPARSEB_GEMM_I8=1, SPARSEB_POISON_OUTPUT=1), A, B, order)
    assert set(got) == {(i, j) for i in (1, 2, 3, 4) for j in (1, 2)}
    for (i, j), c in got.items():
        qs = [q for q in (1, 2) if (i, q) in A]
        a = np.concatenate([A[i, q] for q in qs], 1)
        b = np.concatenate([B[q, j] for q in qs], 0)
        want = (a.astype(np.longdouble) @ b.astype(np.longdouble)).astype(float)
        scale = np.outer(np.sqrt((a ** 2).sum(1)), np.sqrt((b ** 2).sum(0)))
        assert np.max(np.abs(c - want) / scale) <= 8 * 2.0 ** -55, (i, j)


def test_workspace_across_structures():
    """The kept workspace grows, shrinks in use and serves other structures; every
    result equals a fresh context's."""
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(5))
    env = dict(SPARSEB_GEMM_I8=1, SPARSEB_GEMM_THIN=0, SPARSEB_POISON_OUTPUT=1)
    ctx = _ctx(sb, **env)
    for m, n, ks in [(40, 50, (70,)), (300, 260, (900, 65)), (33, 16, (20,)), (300, 260, (900, 65)), (301, 17, (64,))]:
        A, B = _blocks(rng, m, n, ks)
        got, want = _run(sb, ctx, A, B, "AB"), _run(sb, _ctx(sb, **env), A, B, "AB")
        assert np.array_equal(got[1, 1], want[1, 1])
