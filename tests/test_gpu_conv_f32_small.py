"""fp32 convolutions on 64 x 32 tiles (few pixels): edges of tiles, split sums, and the error of a sum against 64 bits."""
import numpy as np
import pytest
import torch

from nncv_b200 import runtime as rt
from nncv_b200._lib import F32, check, lib
from nncv_b200.split_params import random_input, random_state_dict, to_flat_array
from oracle import binding as ob
from tests import gpu_util as G

pytestmark = pytest.mark.gpu


def _tile_of(run):
    """What `run` returns, and tile * 10 + CTAs of a tile of the tensor-core launch that it made."""
    check(lib().nncv_b200_profile(1))
    try:
        y = run()
        made = [r["bn"] for r in rt.profile_records() if r["kind"] == 1]
    finally:
        check(lib().nncv_b200_profile(0))
    assert len(made) == 1
    return y, made[0]


@pytest.mark.parametrize("splits", [1, 2, 4, 8])
@pytest.mark.parametrize("case", [
    # n, c, h, w, k, r, stride: one block (one CTA), two; more blocks than stages; ragged channels, columns, maps
    (1, 64, 8, 8, 128, 1, 1), (1, 72, 3, 5, 36, 1, 1), (1, 64, 56, 56, 64, 3, 1), (2, 128, 28, 28, 128, 3, 1), (1, 256, 14, 14, 256, 3, 1),
    (1, 512, 8, 8, 512, 3, 1), (3, 512, 7, 7, 100, 3, 2), (1, 8, 9, 9, 4, 3, 1), (1, 2048, 7, 7, 512, 1, 1), (5, 40, 6, 10, 240, 3, 1), (1, 1024, 1, 1, 1000, 1, 1),
])
@pytest.mark.parametrize("res,relu", [(True, True), (False, False)])
def test_small_tiles(case, splits, res, relu):
    n, c, h, w, k, r, stride = case
    blocks = r * r * -(-c // 64)
    if splits > blocks:
        pytest.skip("more CTAs than blocks of 64 channels")
    g = np.random.default_rng(sum(case))
    x = g.standard_normal((n, c, h, w)).astype(np.float32)
    wt = (g.standard_normal((k, c, r, r)) * np.sqrt(2.0 / (c * r * r))).astype(np.float32)
    scale, shift = g.uniform(0.5, 1.5, k).astype(np.float32), (g.standard_normal(k) * 0.1).astype(np.float32)
    oh, ow = (h + 2 * (r // 2) - r) // stride + 1, (w + 2 * (r // 2) - r) // stride + 1
    rs = g.standard_normal((n, k, oh, ow)).astype(np.float32) if res else None
    conv = G.Conv(wt, stride, r // 2, F32)
    try:
        check(lib().nncv_b200_conv_set_tile(conv.h, 32, splits, 0))
        (y, _), made = _tile_of(lambda: conv.run(x, scale, shift, rs, relu))
        assert made == 320 + splits
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


@pytest.mark.parametrize("case,small", [
    # two rounds of 64 x 32 tiles, or one that is slower than wide tiles that share their reduction: 3 to 41 % slower
    ((11, 168, 12, 8, 192, 3, 1), False), ((2, 112, 22, 67, 416, 3, 1), False), ((50, 32, 10, 59, 24, 3, 1), False),
    ((4, 64, 56, 56, 128, 1, 2), False), ((12, 1024, 14, 14, 256, 1, 1), False),
    # 12 to 30 % faster on 64 x 32 tiles
    ((1, 256, 14, 14, 256, 3, 1), True), ((2, 512, 7, 7, 2048, 1, 1), True), ((1, 512, 28, 28, 128, 1, 1), True), ((1, 256, 56, 56, 64, 1, 1), True),
])
def test_small_tiles_are_taken_where_they_are_faster(case, small):
    """The lines between tile widths, at layers a good way from them (a GPU of 148 SMs)."""
    n, c, h, w, k, r, stride = case
    conv = G.Conv(np.ones((k, c, r, r), np.float32), stride, r // 2, F32)
    try:
        _, made = _tile_of(lambda: conv.run(np.zeros((n, c, h, w), np.float32)))
    finally:
        conv.close()
    assert (made // 10 == 32) == small


@pytest.mark.parametrize("bn,splits", [(64, 1), (64, 8), (128, 2), (32, 4), (32, 8), (32, 16), (256, 1)])
def test_a_forced_tile_that_does_not_fit_is_the_modelled_one(bn, splits):
    """Tiles of 64 and 128 columns are forced the same way; more CTAs than there are blocks, or a tile there is none of: as modelled."""
    g = np.random.default_rng(1)
    x, wt = g.standard_normal((1, 128, 9, 7)).astype(np.float32), g.standard_normal((160, 128, 1, 1)).astype(np.float32)
    conv = G.Conv(wt, 1, 0, F32)
    try:
        (want, _), modelled = _tile_of(lambda: conv.run(x))
        check(lib().nncv_b200_conv_set_tile(conv.h, bn, splits, 0))
        (y, _), made = _tile_of(lambda: conv.run(x))
    finally:
        conv.close()
    if bn == 256:
        assert made == modelled
    else:
        assert made // 10 == bn and (made % 10 == splits if splits <= 2 else made % 10 in (1, 2))
    assert G.rel_l2(y, want) <= 1e-6


@pytest.mark.parametrize("h,w", [(64, 64), (97, 75)])
def test_a_network_of_one_image_on_small_tiles(h, w):
    """Residuals and results as planes: most layers of ResNet-18 take the small tiles at one image, blocks with residual among them."""
    blob = to_flat_array(18, random_state_dict(18, 0)).blob()
    rt.load_blob("resnet18", blob, F32)
    x, y = random_input(1, h, w, 3, "normal"), np.zeros((1, 1000), np.float32)
    rt.forward(y, x)
    rt.profile(True)
    rt.forward(y, x)
    layers = [r for r in rt.profile_records() if r["kind"] == 1]
    rt.profile(False)
    rt.unload()
    small = [r for r in layers if r["bn"] // 10 == 32]
    assert len(small) >= len(layers) // 2 and any(r["bn"] % 10 > 1 for r in small)
    assert G.rel_l2(y, ob.resnet_forward(18, x, blob)) <= 1e-5


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
