"""Worst-case error of the integer tensor-core GEMM against |row| |column|
(2-norms), on operands whose roundings and low digits all have one sign.

Tolerance.  An element is rounded by at most 2^(E-55) where its row's largest
magnitude is at least 0.995 * 2^E, so each side adds at most 1.01 sqrt(K) 2^-55
(Cauchy-Schwarz).  Digits are at most 128, so the products left out, of weights
256^4 (five of them), 256^3 (four), ..., add at most K 2^14 (5 * 2^32 + 4 * 2^24
+ ...) 2^(E+F-108) < K 2^-59.6 of the two largest magnitudes.  The FP64 additions:
two per accumulation chunk and one per k-segment, of 64 * 12 terms at least, each
2^-53 of a sum below |row| |column|."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C127 = sum(127 * 256.0 ** (6 - s) for s in range(2, 7)) / 2.0 ** 54  # digits 0, 0, 127, ..., 127 beside a 1


def _ctx(sb, **env):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update({k: str(v) for k, v in env.items()})
    try:
        return sb.Context(0)
    finally:
        for k, v in old.items():
            os.environ.pop(k, None) if v is None else os.environ.__setitem__(k, v)


@pytest.mark.parametrize("K", [64, 700, 1500, 4000])
@pytest.mark.parametrize("tails", [(2.0 ** -20 / 3, None), (C127, C127), (2.0 ** -20 / 3, C127)])
def test_constant_tails(tails, K):
    import sparsebackends_b200 as sb
    m, n = 33, 20

    def operand(shape, tail):  # (rows or columns, K): one entry of 1, the rest the tail; signs by row
        x = np.ones(shape) if tail is None else np.full(shape, tail)
        x[np.arange(shape[0]), np.arange(shape[0]) % K] = 1.0
        return x * np.where(np.arange(shape[0]) % 2, -1.0, 1.0)[:, None]

    a, b = operand((m, K), tails[0]), operand((n, K), tails[1]).T.copy()
    b = b if tails[1] is None else np.roll(b, 7, axis=0)
    ctx = _ctx(sb, SPARSEB_GEMM_I8=1, SPARSEB_GEMM_THIN=0)
    A = sb.NewBlockSparseSorted((1, 1, m, K), 2, [(1, 1)], None, a.reshape(-1, order="F"), ctx=ctx)
    B = sb.NewBlockSparseSorted((1, 1, K, n), 2, [(1, 1)], None, b.reshape(-1, order="F"), ctx=ctx)
    C = sb.NewBlockSparseSorted.empty((1, 1, m, n), 2, ctx=ctx)
    sb.contract_(C, ["i", "j", "m", "n"], A, ["i", "q", "m", "k"], B, ["q", "j", "k", "n"])
    c = C.data.reshape(m, n, order="F")
    want = a.astype(np.longdouble) @ b.astype(np.longdouble)
    scale = np.outer(np.sqrt((a ** 2).sum(1)), np.sqrt((b ** 2).sum(0)))
    worst = float(np.max(np.abs(c - want) / scale))
    adds = 2 * -(-K // (64 * 12)) + -(-K // (64 * 12))
    print(K, worst * 2.0 ** 55)
    assert worst <= 2.02 * np.sqrt(K) * 2.0 ** -55 + K * 2.0 ** -59.6 + adds * 2.0 ** -53
