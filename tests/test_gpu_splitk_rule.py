"""Where split-K goes from clusters (one launch) to partial tiles (two): mean K
loops of 256 k-tiles of 16, 12 tiles' worth of them (64x64 tiles) and no more than
148 tiles, operands within L2.  Sums held to their rounding bound, both operand orders."""
import numpy as np
import pytest

from tests.test_gpu_splitk_forms import _check, _ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles,ks,launches,m", [(11, (4112,), 1, 64), (12, (4080,), 1, 64), (12, (4096,), 2, 64),
                                                 (40, (5000, 1, 2999), 2, 64), (100, (1400, 2800), 2, 64),
                                                 (148, (4200,), 2, 8), (149, (4200,), 1, 8)])
def test_rule(tiles, ks, launches, m):
    import sparsebackends_b200 as sb
    rng = np.random.Generator(np.random.PCG64(tiles))
    A = {(i, q): rng.standard_normal((m, k)) for i in range(1, tiles + 1) for q, k in enumerate(ks, 1)}
    B = {(q, 1): rng.standard_normal((k, 64)) for q, k in enumerate(ks, 1)}
    _check(sb, _ctx(sb, SPARSEB_GEMM_TILE="64x64"), A, B, 3, launches=launches)
