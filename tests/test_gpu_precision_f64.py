"""What the FP64 precisions promise.

"f64" (the default): every output element within the rounding of its own sum,
K 2^-53 sum_k |a_k| |b_k| (K products and additions of relative error 2^-53),
whatever the sizes: also where large entries of a row meet zeros or small
entries of the other operand, on operands large enough for every launch rule.
"f64i8", which a caller chooses: the integer tensor cores for large launches,
the same bits as a context that is held to them."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1536  # 7.2 GFLOP: well inside the range where the integer path is the faster one


def _env_ctx(sb, **env):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update({k: str(v) for k, v in env.items()})
    try:
        return sb.Context(0)
    finally:
        for k, v in old.items():
            os.environ.pop(k, None) if v is None else os.environ.__setitem__(k, v)


def _operands(kind, n=N):
    rng = np.random.Generator(np.random.PCG64(5))
    a, b = rng.standard_normal((n, n)), rng.standard_normal((n, n))
    if kind == "large_meets_zero":
        a[:, 1:] *= 1e-14
        b[0, :] = 0.0
    elif kind == "identity":  # an environment's identity channel times a state with decaying weights
        a = np.eye(n)
        b *= (10.0 ** np.linspace(0, -16, n))[:, None]
    elif kind == "opposed":
        a *= (10.0 ** np.linspace(0, -12, n))[None, :]
        b *= (10.0 ** np.linspace(-12, 0, n))[:, None]
    return a, b


def _product(sb, ctx, a, b):
    (m, k), n = a.shape, b.shape[1]
    A = sb.NewBlockSparseSorted((1, 1, m, k), 2, [(1, 1)], None, a.reshape(-1, order="F"), ctx=ctx)
    B = sb.NewBlockSparseSorted((1, 1, k, n), 2, [(1, 1)], None, b.reshape(-1, order="F"), ctx=ctx)
    C = sb.NewBlockSparseSorted.empty((1, 1, m, n), 2, ctx=ctx)
    sb.contract_(C, ["i", "j", "m", "n"], A, ["i", "q", "m", "k"], B, ["q", "j", "k", "n"])
    return C.data.reshape(m, n, order="F")


@pytest.mark.parametrize("kind", ["gaussian", "large_meets_zero", "identity", "opposed"])
def test_default_precision_is_elementwise(kind):
    import sparsebackends_b200 as sb
    ctx = sb.Context(0)
    assert ctx.precision == "f64"
    a, b = _operands(kind)
    c = _product(sb, ctx, a, b)
    rows = np.r_[0:8, N // 2:N // 2 + 8, N - 8:N]
    want = a[rows].astype(np.longdouble) @ b.astype(np.longdouble)
    assert np.all(np.abs(c[rows] - want) <= N * 2.0 ** -53 * (np.abs(a[rows]) @ np.abs(b)))
    assert np.array_equal(c, _product(sb, _env_ctx(sb, SPARSEB_GEMM_I8=0), a, b))


def test_chosen_integer_path():
    """"f64i8" takes the integer path at this size and DMMA for small launches;
    "f64" is back after it, with plans of its own."""
    import sparsebackends_b200 as sb
    ctx = sb.Context(0)
    a, b = _operands("gaussian")
    ctx.set_precision("f64i8")
    assert ctx.precision == "f64i8"
    x = _product(sb, ctx, a, b)
    assert np.array_equal(x, _product(sb, _env_ctx(sb, SPARSEB_GEMM_I8=1), a, b))
    y = _product(sb, ctx, a[:100, :90], b[:90, :100])
    ctx.set_precision("f64")
    assert np.array_equal(y, _product(sb, ctx, a[:100, :90], b[:90, :100]))
    d = _product(sb, ctx, a, b)
    assert np.array_equal(d, _product(sb, _env_ctx(sb, SPARSEB_GEMM_I8=0), a, b)) and not np.array_equal(d, x)


def test_heff_operator_in_f64i8():
    """The precision reaches the chain, with FP64 intermediates."""
    import sparsebackends_b200 as sb
    from sparsebackends_b200 import qn
    from tests.test_gpu_graph import _setup
    _, _, lay, ctx, T, psi, _ = _setup(True)
    want = qn.HeffOperator(lay, T["L"], T["W1"], T["W2"], T["R"], ctx)(psi).data
    op = qn.HeffOperator(lay, T["L"], T["W1"], T["W2"], T["R"], ctx, precision="f64i8")
    got = op(psi).data
    assert ctx.precision == "f64" and op.accuracy == 0.0
    assert np.array_equal(got, want)  # launches this small stay on DMMA


def test_f64i8_refuses_fp32_storage_as_f64_does():
    import sparsebackends_b200 as sb
    from sparsebackends_b200 import qn
    from tests.test_gpu_graph import _setup
    _, _, lay, ctx, T, psi, _ = _setup(True)
    for precision in ("f64", "f64i8"):
        with pytest.raises(sb.SparseBackendsError):
            qn.HeffOperator(lay, T["L"], T["W1"], T["W2"], T["R"], ctx, precision=precision,
                            f32_intermediates=True)(psi)
        assert ctx.precision == "f64"
