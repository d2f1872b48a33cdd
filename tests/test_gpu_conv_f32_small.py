"""fp32 convolutions on 64 x 32 tiles (few pixels): edges of tiles, split sums, and the error of a sum against 64 bits."""
import numpy as np
import pytest
import torch

from nncv_b200._lib import F32, check, lib
from oracle import binding as ob
from tests import gpu_util as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    # n, c, h, w, k, r, stride: one block; two of a CTA; more blocks than stages; split over 2, 4 and 8; ragged channels, columns, maps
    (1, 64, 8, 8, 32, 1, 1), (1, 72, 3, 5, 36, 1, 1), (1, 64, 56, 56, 64, 3, 1), (2, 128, 28, 28, 128, 3, 1), (1, 256, 14, 14, 256, 3, 1),
    (1, 512, 8, 8, 512, 3, 1), (3, 512, 7, 7, 100, 3, 2), (1, 8, 9, 9, 4, 3, 1), (1, 2048, 7, 7, 512, 1, 1), (5, 40, 6, 10, 240, 1, 1), (1, 1024, 1, 1, 1000, 1, 1),
])
@pytest.mark.parametrize("res,relu", [(True, True), (False, False)])
def test_small_tiles(case, res, relu):
    n, c, h, w, k, r, stride = case
    g = np.random.default_rng(sum(case))
    x = g.standard_normal((n, c, h, w)).astype(np.float32)
    wt = (g.standard_normal((k, c, r, r)) * np.sqrt(2.0 / (c * r * r))).astype(np.float32)
    scale, shift = g.uniform(0.5, 1.5, k).astype(np.float32), (g.standard_normal(k) * 0.1).astype(np.float32)
    oh, ow = (h + 2 * (r // 2) - r) // stride + 1, (w + 2 * (r // 2) - r) // stride + 1
    rs = g.standard_normal((n, k, oh, ow)).astype(np.float32) if res else None
    conv = G.Conv(wt, stride, r // 2, F32)
    try:
        y, _ = conv.run(x, scale, shift, rs, relu)
        again, _ = conv.run(x, scale, shift, rs, relu)
    finally:
        conv.close()
    assert np.array_equal(y, again)
    ref = ob.conv2d(x, wt, stride, r // 2, acc64=True) * scale[None, :, None, None] + shift[None, :, None, None]
    ref = ref + rs if res else ref
    ref = np.maximum(ref, 0) if relu else ref
    # the large products' steps are cut to 24 bits (2^-23 of a step), their sums and the parts' rounded (2^-24 each)
    bound = 2.0 ** -23 + 2.0 ** -24 * (np.sqrt(4 * r * r * np.ceil(c / 64)) + 8 + 3)
    assert np.isfinite(y).all() and G.rel_l2(y, ref) <= bound
    assert lib().nncv_b200_device_status() == 0


def test_small_tiles_have_no_bias():
    """What the tensor core cuts off every step is given back: the mean error along the result, over 2 M outputs."""
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    along = norm = 0.0
    for _ in range(40):
        x, w = torch.randn((1, 14, 14, 512), device="cuda", generator=g), torch.randn((256, 512), device="cuda", generator=g)
        conv = G.Conv(w.cpu().numpy()[:, :, None, None], 1, 0, F32)
        y = torch.zeros((1, 14, 14, 256), device="cuda")
        try:
            check(lib().nncv_b200_conv_run(conv.h, G.p(x), G.p(y), 1, 14, 14, None, None, None, 0, G.stream_ptr()))
            G.sync_check()
        finally:
            conv.close()
        ref = (x.double().view(-1, 512) @ w.double().T).flatten()
        along += float((y.double().flatten() - ref) @ ref)
        norm += float(ref @ ref)
    assert abs(along / norm) <= 0.25 * 2.0 ** -24
