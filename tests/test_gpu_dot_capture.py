"""norm and dot inside a stream capture are refused, abandon the capture and
leave nothing behind: the eager calls that follow on the context return the
values of their own operands.  Device memory that the refused call could have
taken holds non-zero words, so a counter that nobody zeroed shows."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _leave_nonzero_memory():
    """Free every other one of many small device buffers filled with 0xFF; the
    others are returned and keep the pages in use."""
    cu = ctypes.CDLL("libcuda.so.1")
    kept = []
    for i, p in enumerate([_alloc(cu) for _ in range(512)]):
        if i % 2:
            assert cu.cuMemFree_v2(p) == 0
        else:
            kept.append(p)
    return cu, kept


def _alloc(cu, size=4096):
    p = ctypes.c_uint64()
    assert cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(size)) == 0
    assert cu.cuMemsetD8_v2(p, ctypes.c_ubyte(0xFF), ctypes.c_size_t(size)) == 0
    return p


@pytest.mark.parametrize("first", [False, True])
def test_refused_dot_leaves_no_state(first):
    """The refused call is the context's first dot product (first), or a longer
    one than its scratch was made for."""
    import sparsebackends_b200 as sb
    ctx = sb.Context(0)
    rng = np.random.Generator(np.random.PCG64(7))

    def vector(n):
        return sb.NewBlockSparseSorted((1, n), 1, [(1,)], None, rng.standard_normal(n), ctx=ctx)

    x, y, z = vector(90000), vector(40000), vector(3)
    if not first:
        assert np.isclose(sb.norm(z), np.linalg.norm(z.data), rtol=1e-14)
    cu, kept = _leave_nonzero_memory()
    for call in (lambda: sb.norm(x), lambda: sb.dot(x, x)):
        with pytest.raises(sb.SparseBackendsError):
            ctx.capture(call)
    for v in (x, y, z, x):
        want = np.linalg.norm(v.data)
        assert np.isclose(sb.norm(v), want, rtol=1e-13)
        assert np.isclose(sb.dot(v, v), want * want, rtol=1e-13)
    for p in kept:
        assert cu.cuMemFree_v2(p) == 0


def test_norm_of_an_empty_tensor_is_refused_too():
    import sparsebackends_b200 as sb
    ctx = sb.Context(0)
    e = sb.NewBlockSparseSorted.empty((2, 3), 1, ctx=ctx)
    assert sb.norm(e) == 0.0
    with pytest.raises(sb.SparseBackendsError):
        ctx.capture(lambda: sb.norm(e))
    assert sb.norm(e) == 0.0
