"""GPU parity of the fp32 convolution on the tensor cores (three bf16 planes per operand) against the fp64-accumulated
oracle, at the edges of its tiles: ragged pixel tiles and channel blocks, one and several Kout tiles, split reductions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from oracle import binding as ob  # noqa: E402
from nncv_b200._lib import F32, check, lib  # noqa: E402
import gpu_util as G  # noqa: E402


@pytest.mark.parametrize("case", [
    # n, c, h, w, kout, r, stride
    (1, 72, 5, 7, 4, 1, 1),          # one block of 64 and a ragged one of 8, four output channels
    (1, 8, 9, 9, 64, 3, 1),          # eight channels a tap
    (3, 64, 13, 11, 68, 3, 1),       # a second Kout tile of four channels
    (2, 64, 15, 17, 136, 3, 2),      # stride 2, ragged wide tile
    (1, 512, 7, 7, 512, 3, 1),       # 72 blocks, split over a cluster
    (9, 128, 28, 28, 128, 3, 1),     # more tiles than SMs hold at once
    (5, 256, 14, 14, 64, 1, 2),
    (1, 40, 130, 3, 240, 1, 1),
])
@pytest.mark.parametrize("res,relu", [(True, True), (False, False)])
def test_conv_f32(case, res, relu):
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
    finally:
        conv.close()
    ref = ob.conv2d(x, wt, stride, r // 2, acc64=True) * scale[None, :, None, None] + shift[None, :, None, None]
    ref = ref + rs if res else ref
    ref = np.maximum(ref, 0) if relu else ref
    # at most four accumulations of a block are cut to 24 bits (2^-23 each, 4.8e-7), the blocks' sums are rounded (2^-24 of the
    # running sum each, adding up like a random walk) and so are scale, shift and residual
    bound = 4 * 2.0 ** -23 + 2.0 ** -24 * (np.sqrt(r * r * np.ceil(c / 64)) + 3)
    assert np.isfinite(y).all() and G.rel_l2(y, ref) <= bound
    assert lib().nncv_b200_device_status() == 0


def test_conv_f32_keeps_all_24_bits_of_its_operands():
    """1x1 filter that copies one channel: every fp32 value comes through unchanged."""
    g = np.random.default_rng(3)
    x = (g.standard_normal((2, 128, 6, 6)) * np.exp2(g.integers(-30, 30, (2, 128, 6, 6)))).astype(np.float32)
    wt = np.eye(128, dtype=np.float32)[:, :, None, None]
    conv = G.Conv(wt, 1, 0, F32)
    try:
        y, _ = conv.run(x, None, None, None, False)
    finally:
        conv.close()
    assert np.array_equal(y, x)


@pytest.mark.parametrize("kind", ["normal", "relu", "positive"])
@pytest.mark.parametrize("c", [64, 72, 512])
def test_conv_f32_sums_have_no_bias(kind, c):
    """The tensor core cuts its sums: an error of one sign, which a network's layers add up where a rounding error would
    average out.  Its share of the result, over 16 M outputs of a 1x1 filter."""
    g = torch.Generator(device="cuda")
    g.manual_seed(c)
    x, w = torch.randn((64, 16, 16, c), device="cuda", generator=g), torch.randn((1024, c), device="cuda", generator=g)
    x, w = (x.abs(), w.abs()) if kind == "positive" else (x.clamp_min(0) if kind == "relu" else x, w)
    conv = G.Conv(w.cpu().numpy()[:, :, None, None], 1, 0, F32)
    y = torch.zeros((64, 16, 16, 1024), device="cuda")
    try:
        check(lib().nncv_b200_conv_run(conv.h, G.p(x), G.p(y), 64, 16, 16, None, None, None, 0, G.stream_ptr()))
        G.sync_check()
    finally:
        conv.close()
    ref = (x.double().view(-1, c) @ w.double().T).flatten()
    off = y.double().flatten() - ref
    # a step of 16 channels takes 0.09 (half of the operands zero) to 0.28 (all of one sign) times 2^-24 off its sum, of which
    # 0.19 are given back; with four steps in one accumulator 0.46 to 1.3 were missing
    assert abs(float(off @ ref / (ref @ ref))) <= 0.25 * 2.0 ** -24
