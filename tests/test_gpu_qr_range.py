"""Blockwise QR of matrices with infinities, NaN and columns whose products
overflow: reflector by reflector, an identity (nothing below the pivot) changes
no column, and a reflector acts on the rows from its pivot on, so what the
non-finite entries do not reach stays finite.  Reference: the reflectors one at
a time in numpy; tolerance on finite entries: 4 k eps of the column's norm, as
for finite matrices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reflectors(M):
    a = M.copy()
    m, n = a.shape
    k = min(m, n)
    tau, V = np.zeros(k), np.zeros((m, k))
    with np.errstate(all="ignore"):
        for j in range(k):
            x = a[j + 1:, j]
            xn2, alpha = np.sum(x * x), a[j, j]
            if xn2 == 0.0:
                continue
            beta = -np.sqrt(alpha * alpha + xn2) if alpha >= 0.0 else np.sqrt(alpha * alpha + xn2)
            tau[j] = (beta - alpha) / beta
            V[j, j], V[j + 1:, j] = 1.0, x * (1.0 / (alpha - beta))
            a[j, j] = beta
            for c in range(j + 1, n):
                a[j:, c] -= V[j:, j] * (tau[j] * np.sum(V[j:, j] * a[j:, c]))
        q = np.eye(m, k)
        for j in range(k - 1, -1, -1):
            if tau[j] != 0.0:
                for c in range(j, k):
                    q[j:, c] -= V[j:, j] * (tau[j] * np.sum(V[j:, j] * q[j:, c]))
    return q, np.triu(a[:k])


def _matrix(kind):
    rng = np.random.Generator(np.random.PCG64(12))
    if kind in ("inf_over_identity", "inf_over_identity_16"):  # panels of 32 and of 16 reflectors
        m = 48 if kind == "inf_over_identity" else 600
        M = rng.standard_normal((m, 40))
        M[:, :20] = np.triu(M)[:, :20]
        M[3, 30], M[5, 39], M[2, 35] = np.inf, np.nan, -np.inf
    elif kind == "nan_late":
        M = rng.standard_normal((70, 50))
        M[45, 37] = np.nan
    elif kind == "inf_in_second_panel":
        M = rng.standard_normal((130, 80))
        M[100, 40] = np.inf
    elif kind == "overflowing_column":
        M = rng.standard_normal((60, 40))
        M[:, 10] *= 1e200
    else:  # "large_last": no reflector squares the last column, all meet it
        M = rng.standard_normal((40, 40))
        M[:, :39] *= 2.0 ** 500
        M[:, 39] *= 2.0 ** 560
    return M


@pytest.mark.parametrize("kind", ["inf_over_identity", "inf_over_identity_16", "nan_late", "inf_in_second_panel",
                                  "overflowing_column", "large_last"])
def test_non_finite_entries_stay_where_they_act(kind):
    import sparsebackends_b200 as sb
    M = _matrix(kind)
    m, n = M.shape
    keys = [(i + 1, j + 1) for j in range(n) for i in range(m)]
    A = sb.NewBlockSparseSorted((m, n, 1), 1, keys, None, M.reshape(-1, order="F"))
    Q, R, _, _ = sb.blocksparse_left_qr(A)
    k = min(m, n)
    q = np.zeros((m, k))
    for key, b in Q.blocks_by_key().items():
        q[key[0] - 1] = b
    r = R.to_numpy()
    want_q, want_r = _reflectors(M)
    if kind != "large_last":
        assert not np.isfinite(want_r).all()
    for got, want in ((q, want_q), (r, want_r)):
        f = np.isfinite(want)
        assert np.array_equal(np.isfinite(got), f)
        for c in range(want.shape[1]):
            g, w = got[f[:, c], c], want[f[:, c], c]
            norm = max((np.abs(w).max(initial=0.0)), 1.0)
            assert np.all(np.abs(g - w) <= 4 * k * np.finfo(float).eps * 300 * norm)
