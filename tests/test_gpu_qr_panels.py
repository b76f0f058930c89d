"""Blockwise QR at the edges of its panels (32 reflectors up to 512 rows, 16 up
to 1024, one at a time beyond): M = Q R, Q^T Q = 1 and R's signs as LAPACK's.

Tolerance: the backward error of k Householder reflectors of length m is a
small multiple of m k eps at worst and of sqrt(m) k eps in practice; 4 k eps
times the norm of M leaves out only the constant of the latter."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 5), (2, 2), (31, 40), (32, 32), (33, 31), (40, 33), (128, 65), (129, 64), (256, 97), (257, 200),
         (384, 33), (385, 20), (511, 70), (512, 32), (513, 17), (700, 33), (1024, 40), (1025, 6), (60, 300)]


@pytest.mark.parametrize("m,n", SIZES)
@pytest.mark.parametrize("kind", ["random", "deficient"])
def test_panels(m, n, kind):
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(m * 1000 + n))
    M = rng.standard_normal((m, n))
    if kind == "deficient" and n > 1:
        M[:, n // 2] = 0.0
        M[: m // 2, n - 1] = M[: m // 2, 0]
    keys = [(i + 1, j + 1) for j in range(n) for i in range(m)]
    A = sb.NewBlockSparseSorted((m, n, 1), 1, keys, None, M.reshape(-1, order="F"))
    Q, R, lv, rv = sb.blocksparse_left_qr(A)
    k = min(m, n)
    q = np.zeros((m, k))
    for key, b in Q.blocks_by_key().items():
        q[key[0] - 1] = b
    r = R.to_numpy()
    eps = np.finfo(float).eps
    assert np.linalg.norm(q @ r - M) <= 4 * k * eps * np.linalg.norm(M)
    assert np.linalg.norm(q.T @ q - np.eye(k)) <= 4 * k * eps * np.sqrt(k)
    assert np.array_equal(r, np.triu(r))
    if kind == "random":
        want = np.linalg.qr(M)[1]
        d = np.abs(np.diag(want)) > 1e-6
        assert np.array_equal(np.sign(np.diag(r))[d], np.sign(np.diag(want))[d])
