"""fp32 depthwise convolution with a folded batch-norm: filter, scale and shift are each used as they are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from nncv_b200._lib import F32, check, lib  # noqa: E402
import gpu_util as G  # noqa: E402


@pytest.mark.parametrize("n,h,w,c,k", [(1, 9, 7, 8, 3), (2, 30, 33, 72, 5)])
def test_scale_and_shift_are_one_multiply_add(n, h, w, c, k):
    """A filter with a centre tap only, ones for input: the result is round(filter * scale + shift), the shift here being
    minus the rounded product, so that what is left is the product's own rounding error."""
    g = np.random.default_rng(c)
    f, scale = g.uniform(0.5, 2.0, c).astype(np.float32), g.uniform(0.5, 2.0, c).astype(np.float32)
    shift = -(f * scale)
    wt = np.zeros((c, k, k), np.float32)
    wt[:, k // 2, k // 2] = f
    X, W, S, B = torch.ones((n, h, w, c), device="cuda"), G.dev(wt), G.dev(scale), G.dev(shift)
    Y = torch.full_like(X, float("nan"))
    check(lib().nncv_b200_depthwise_conv_nhwc(G.p(X), G.p(W), F32, G.p(S), G.p(B), G.p(Y), F32, n, h, w, c, k, k, 1, k // 2, 0, G.stream_ptr()))
    G.sync_check()
    want = (f.astype(np.float64) * scale + shift).astype(np.float32)   # 48 bits of product: exact in 64
    assert np.count_nonzero(want) > c // 2
    assert np.array_equal(G.host(Y), np.broadcast_to(want, (n, h, w, c)))
