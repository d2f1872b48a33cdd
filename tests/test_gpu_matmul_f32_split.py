"""fp32 matmul whose tiles are shared by clusters of two, four or eight CTAs: unequal shares of the depth, ragged rows,
columns and depth, the most tiles that still split and one more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from nncv_b200._lib import F32  # noqa: E402
import gpu_util as G  # noqa: E402


@pytest.mark.parametrize("m,n,k", [(128, 128, 252), (128, 128, 256), (1, 32, 2048), (100, 36, 512), (256, 132, 1028), (300, 500, 2020),
                                   (1024, 1024, 324), (9472, 100, 256), (9473, 128, 292)])
@pytest.mark.parametrize("epilogue", [False, True])
def test_matmul_f32_split(m, n, k, epilogue):
    r = np.random.default_rng(m + n + k)
    a = r.uniform(-1, 1, (m, k)).astype(np.float32)
    b = r.uniform(-1, 1, (k, n)).astype(np.float32)
    bias = r.standard_normal(n).astype(np.float32) if epilogue else None
    c, _, _ = G.matmul(a, b, F32, F32, bias, epilogue)
    ref = a.astype(np.float64) @ b.astype(np.float64)
    if epilogue:
        ref = np.maximum(ref + bias, 0)
    assert np.isfinite(c).all()
    # two tf32 parts keep 22 bits of an operand; every one of the k / 8 accumulations cuts up to 2^-23 of the sum
    bound = 2.0 ** -21 + k / 8 * 2.0 ** -23
    assert G.rel_l2(c, ref) <= bound
    c2, _, _ = G.matmul(a, b, F32, F32, bias, epilogue)
    assert np.array_equal(c, c2)
