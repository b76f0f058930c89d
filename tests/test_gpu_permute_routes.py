"""Ragged tail permutes where the route changes between tiles and the gather
(rows of 1 to 3 elements, tiles below half their capacity, many short batches)
and inside them (tile rows shorter than a warp, one and four gathered elements
per thread).  They only move values: bit-exact against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tperm", [(2, 3, 1), (3, 1, 2), (3, 2, 1), (2, 1, 3)])
@pytest.mark.parametrize("top", [(2, 40, 900), (3, 40, 900), (31, 30, 70), (32, 30, 70), (33, 30, 70), (5, 2500, 2),
                                 (6, 700, 20), (7, 333, 33)])
@pytest.mark.parametrize("blocks", [1, 5, 33])
def test_routes(top, tperm, blocks):
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(sum(top) + tperm[0]))
    exts = [tuple(max(1, t - (i + 2 * a) % 4) for a, t in enumerate(top)) for i in range(blocks)]
    vals = [rng.standard_normal(e) for e in exts]
    A = sb.NewBlockSparseSorted((blocks,) + top, 3, [(i + 1,) for i in range(blocks)], None,
                                np.concatenate([v.reshape(-1, order="F") for v in vals]), block_dims=exts)
    got = sb.permutedims(A, [1] + [1 + t for t in tperm]).blocks_by_key()
    for i, v in enumerate(vals):
        assert np.array_equal(got[(i + 1,)], np.transpose(v, [t - 1 for t in tperm]).reshape(-1, order="F")), i


@pytest.mark.parametrize("tail,kept", [((3, 900, 50), (2, 800, 41)), ((7, 5, 3000), (6, 5, 2801)), ((15, 15), (9, 8))])
@pytest.mark.parametrize("blocks", [1, 40])
def test_crops_and_pads_through_the_gather(tail, kept, blocks):
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(sum(tail)))
    full = [np.zeros(tail) for _ in range(blocks)]
    for f in full:
        f[tuple(slice(0, e) for e in kept)] = rng.standard_normal(kept)
    A = sb.NewBlockSparseSorted((blocks,) + tail, len(tail), [(i + 1,) for i in range(blocks)], None,
                                np.concatenate([f.reshape(-1, order="F") for f in full]))
    R = sb.to_ragged(A, [kept] * blocks)
    got, back = R.blocks_by_key(), sb.to_uniform(R).blocks_by_key()
    for i, f in enumerate(full):
        assert np.array_equal(got[(i + 1,)], f[tuple(slice(0, e) for e in kept)].reshape(-1, order="F"))
        assert np.array_equal(back[(i + 1,)], f.reshape(-1, order="F"))


@pytest.mark.parametrize("length", [32, 33, 63, 64, 65, 255, 256, 257, 511, 513, 2047, 2048])
def test_run_copies(length):
    """Runs around a warp's batch of loads, whole and with a rest."""
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(length))
    v = [rng.standard_normal((length, 3, 5)) for _ in range(4)]
    A = sb.NewBlockSparseSorted((4, length, 3, 5), 3, [(i + 1,) for i in range(4)], None,
                                np.concatenate([x.reshape(-1, order="F") for x in v]))
    got = sb.permutedims(A, [1, 2, 4, 3]).blocks_by_key()
    for i, x in enumerate(v):
        assert np.array_equal(got[(i + 1,)], np.transpose(x, (0, 2, 1)).reshape(-1, order="F")), i
