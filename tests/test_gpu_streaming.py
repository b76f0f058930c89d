"""The streaming kernels at the sizes where their work split changes: run
copies cut into segments, and scaled accumulation with four elements per
thread.  Both only move or add values in a fixed order, so results equal the
oracle's bit for bit."""
import numpy as np
import pytest

from oracle import sparse_oracle as so

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nblocks", [1, 2, 7])
@pytest.mark.parametrize("tail", [(31, 1), (32, 3), (1023, 2), (2049, 1), (4999, 7), (70001, 1)])
def test_prefix_reorder_copies_long_runs(nblocks, tail):
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(tail[0] + nblocks))
    pre = (3, 3)
    keys = sorted([(1 + i % 3, 1 + i // 3) for i in range(nblocks)], key=lambda k: k[::-1])
    data = rng.standard_normal(nblocks * tail[0] * tail[1])
    A = sb.NewBlockSparseSorted(pre + tail, 2, keys, None, data)
    R = so.BS(pre + tail, 2, keys, list(range(1, nblocks + 1)), data)
    P, W = sb.permutedims(A, [2, 1, 3, 4]), so.bs_permutedims(R, [2, 1, 3, 4])
    assert P.keys == W.keys
    got, want = P.blocks_by_key(), W.blocks_by_key()
    assert all(np.array_equal(got[k], np.ravel(want[k], order="F")) for k in want)


@pytest.mark.parametrize("length", [1, 255, 1023, 1024, 1025, 4097])
@pytest.mark.parametrize("first", [True, False])  # the reduced label last in the prefix, or reordered by a view
def test_coo_times_blocks_bit_exact(length, first):
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(length))
    ck = [(a, s) for s in (1, 2, 3) for a in (1, 2, 4)]
    cv = rng.standard_normal(len(ck))
    bk = [(q, s) for s in (1, 2, 3) for q in (1, 2)]
    data = rng.standard_normal(len(bk) * length)
    A, RA = sb.COOTensor((4, 3), ck, cv), so.COO((4, 3), ck, cv)
    B = sb.NewBlockSparseSorted((2, 3, length), 1, bk, None, data)
    RB = so.BS((2, 3, length), 1, bk, list(range(1, len(bk) + 1)), data)
    lB = ["q", "s", "x"]
    if not first:
        B, RB, lB = sb.permutedims(B, [2, 1, 3]), so.bs_permutedims(RB, [2, 1, 3]), ["s", "q", "x"]
    C = sb.NewBlockSparseSorted.empty((4, 2, length), 1)
    sb.contract_(C, ["a", "q", "x"], A, ["a", "s"], B, lB)
    W = so.contract(so.BS.empty((4, 2, length), 1), ["a", "q", "x"], RA, ["a", "s"], RB, lB)
    assert C.keys == W.keys
    got, want = C.blocks_by_key(), W.blocks_by_key()
    assert all(np.array_equal(got[k], np.ravel(want[k], order="F")) for k in want)


@pytest.mark.parametrize("tail", [(7,), (9000,), (3, 2, 5, 4, 6), (5, 7, 6, 11), (1, 1), (31, 70), (32, 5), (33, 600), (600, 33), (5000, 1), (9, 40, 21), (515, 515)])
@pytest.mark.parametrize("nblocks", [1, 6])
def test_zero_padding_scan_extents(tail, nblocks):
    """Extents found by the scan, for every form of its tasks (rows of one
    column, runs of columns, a lane per column), with one nonzero entry on each
    block's true corner and none at all in the last block."""
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(sum(tail) + nblocks))
    keys = [(i + 1,) for i in range(nblocks)]
    blocks, want = [], []
    for i in range(nblocks):
        b = np.zeros(tail)
        e = (1,) * len(tail)
        if i + 1 < nblocks or nblocks == 1:
            e = tuple(int(rng.integers(1, t + 1)) for t in tail)
            b[tuple(x - 1 for x in e)] = 1e-300
            b[tuple(int(rng.integers(0, x)) for x in e)] = 2.0
        blocks.append(b.reshape(-1, order="F"))
        want.append(e)
    A = sb.NewBlockSparseSorted((nblocks,) + tail, len(tail), keys, None, np.concatenate(blocks))
    assert sb.crop_padding(A).block_dims == want


@pytest.mark.parametrize("tperm", [(2, 1, 3), (2, 3, 1), (3, 1, 2), (3, 2, 1), (1, 3, 2)])
@pytest.mark.parametrize("top", [(1, 1, 1), (2, 3, 2), (64, 64, 1), (64, 64, 9), (65, 130, 3), (33, 1, 200), (33, 1, 900), (7, 150, 90)])
def test_ragged_permute_tiles(tperm, top):
    """Ragged tail permutes through tiles: partial tiles on either side, blocks
    with extents of one, a short contiguous axis; bit-exact against numpy."""
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(sum(top) + tperm[0]))
    keys = [(i + 1, 1) for i in range(40)]
    exts = [top] + [tuple(int(rng.integers(1, t + 1)) for t in top) for _ in keys[1:]]
    blocks = [rng.standard_normal(e) for e in exts]
    A = sb.NewBlockSparseSorted((40, 1) + top, 3, keys, None,
                                np.concatenate([b.reshape(-1, order="F") for b in blocks]), block_dims=exts)
    P = sb.permutedims(A, [2, 1] + [2 + t for t in tperm])
    want = {(1, i + 1): np.transpose(b, [t - 1 for t in tperm]).reshape(-1, order="F") for i, b in enumerate(blocks)}
    got = P.blocks_by_key()
    assert set(got) == set(want) and all(np.array_equal(got[k], want[k]) for k in want)


def test_crop_of_short_rows_stays_off_the_tiles():
    """Cropping blocks whose first axis is short (axis 0 contiguous on both
    sides): one row of it would be a whole tile, so the gather keeps them."""
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(5))
    tail, ext = (14, 60, 90), (11, 51, 77)
    b = np.zeros((3,) + tail)
    b[(slice(None),) + tuple(slice(0, e) for e in ext)] = rng.standard_normal((3,) + ext)
    A = sb.NewBlockSparseSorted((3,) + tail, 3, [(1,), (2,), (3,)], None,
                                np.concatenate([x.reshape(-1, order="F") for x in b]))
    R = sb.to_ragged(A, [ext] * 3)
    got = R.blocks_by_key()
    for i in range(3):
        assert np.array_equal(got[(i + 1,)], b[i][tuple(slice(0, e) for e in ext)].reshape(-1, order="F"))


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 262144, 1048577, 3000000])
def test_dot_and_norm_lengths(n):
    """One launch per scalar: chunk edges, more partials than the final sum's
    1024 strands, and repeated calls on growing and shrinking vectors.  The
    pairwise-like sum is compared with numpy's extended precision at n eps."""
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(n))
    x, y = rng.standard_normal(n), rng.standard_normal(n)
    X, Y = sb.DenseTensor(x), sb.DenseTensor(y)
    want = float(np.sum(x.astype(np.longdouble) * y))
    tol = n * np.finfo(float).eps * float(np.sum(np.abs(x * y))) / np.sqrt(n)
    first = sb.dot(X, Y)
    assert abs(first - want) <= tol
    assert abs(sb.norm(X) - float(np.sqrt(np.sum(x.astype(np.longdouble) ** 2)))) <= n * np.finfo(float).eps * np.sqrt(n)
    assert sb.dot(sb.DenseTensor(x[:1]), sb.DenseTensor(y[:1])) == x[0] * y[0]
    assert sb.dot(X, Y) == first
