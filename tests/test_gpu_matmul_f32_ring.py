"""fp32 matmul, B by TMA: blocks of the depth that wrap the rings of six stages and four parts of A at every offset, with one tile a
CTA and with several, ragged columns and depth."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from nncv_b200._lib import F32  # noqa: E402
import gpu_util as G  # noqa: E402


@pytest.mark.parametrize("m,n,k", [(1, 32, 32), (129, 132, 36), (2500, 260, 100), (9600, 252, 164), (20000, 132, 228), (9500, 640, 388), (130, 9600, 420)])
def test_matmul_f32_ring(m, n, k):
    r = np.random.default_rng(m + n + k)
    a = r.uniform(-1, 1, (m, k)).astype(np.float32)
    b = r.uniform(-1, 1, (k, n)).astype(np.float32)
    c, _, _ = G.matmul(a, b, F32, F32, None, False)
    ref = a.astype(np.float64) @ b.astype(np.float64)
    # two tf32 parts keep 22 bits of an operand; every one of the k / 8 accumulations cuts up to 2^-23 of the sum
    assert G.rel_l2(c, ref) <= 2.0 ** -21 + k / 8 * 2.0 ** -23
    # every value by itself: no neighbour's column or row, no value left from another tile
    assert np.abs(c - ref).max() <= 2.0 ** -18 * np.sqrt(k) * 4
