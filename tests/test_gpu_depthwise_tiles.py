"""The depthwise kernel's splits of a map (one or two columns a thread, any block size) at the edges of tiles: against the oracle."""
import numpy as np
import pytest

from nncv_b200._lib import BF16, F16, F32, check, lib
from oracle import binding as ob
from tests import gpu_util as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,h,w", [
    (1, 16, 1, 1), (2, 16, 9, 5), (3, 24, 7, 7), (1, 72, 17, 33), (2, 96, 16, 112), (1, 200, 8, 2), (5, 264, 13, 14), (1, 32, 65, 129), (40, 16, 12, 15),
])
@pytest.mark.parametrize("k,stride", [(3, 1), (3, 2), (5, 1), (5, 2)])
@pytest.mark.parametrize("dtype", [F16, BF16, F32])
def test_depthwise_tiles(n, c, h, w, k, stride, dtype):
    g = np.random.default_rng(n + c + h + w + k + stride)
    x = g.standard_normal((n, c, h, w)).astype(np.float32)
    wt = (g.standard_normal((c, k, k)) / k).astype(np.float32)
    scale, shift = g.uniform(0.5, 1.5, c).astype(np.float32), (g.standard_normal(c) * 0.1).astype(np.float32)
    oh, ow = (h + 2 * (k // 2) - k) // stride + 1, (w + 2 * (k // 2) - k) // stride + 1
    X = G.dev(np.ascontiguousarray(x.transpose(0, 2, 3, 1)), dtype)
    guard = 64
    Y = G.dev(np.full(n * oh * ow * c + guard, -77.0, np.float32), dtype)
    W, S, H = G.dev(wt), G.dev(scale), G.dev(shift)
    check(lib().nncv_b200_depthwise_conv_nhwc(G.p(X), G.p(W), F32, G.p(S), G.p(H), G.p(Y), dtype, n, h, w, c, k, k, stride, k // 2, 1,
                                              G.stream_ptr()))
    G.sync_check()
    got = G.host(Y)
    assert (got[-guard:] == -77.0).all()
    got = got[:-guard].reshape(n, oh, ow, c).transpose(0, 3, 1, 2)
    xq = G.host(X).transpose(0, 3, 1, 2)
    ref = ob.depthwise_conv2d(xq, wt, stride, k // 2, acc64=True) * scale[None, :, None, None] + shift[None, :, None, None]
    ref = np.where(ref > 0, ref, 0)
    # one rounding of the result: half of 2^-10, 2^-7 or, with the sums of 25 products in 32 bits, some 2^-24
    assert G.rel_l2(got, ref) <= {F16: 1e-3, BF16: 8e-3, F32: 1e-6}[dtype]
    assert lib().nncv_b200_device_status() == 0
