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


@pytest.mark.parametrize("r,c,k", [(1, 128, 64), (1, 72, 128), (3, 64, 64), (3, 512, 8)])   # 3x3 over 512 channels: split over a cluster
def test_conv_f32_infinities_nan_and_the_largest_values(r, c, k):
    """Non-finite inputs and weights end where IEEE arithmetic puts them, and finite values above the largest bf16 stay finite."""
    g = np.random.default_rng(r * c)
    n, h, w = 1, 9, 12
    x = g.standard_normal((n, c, h, w)).astype(np.float32)
    wt = g.standard_normal((k, c, r, r)).astype(np.float32)
    wt[::2] = np.round(wt[::2] * 4) / 4              # exact in bf16, zeros among them: the remainders are zero
    x[0, 3, 1, 1], x[0, 5, 4, 9], x[0, 7, 7, 2], x[0, c - 1, 7, 9] = np.inf, -np.inf, np.nan, np.inf
    x[0, 0, 7, 9] = -np.inf                          # meets the +inf of another channel
    wt[3 % k, 1, 0, 0] = np.inf
    big = np.float32(3.4e38)
    x[0, :, 4, 5] = 0
    x[0, 2, 4, 5] = big
    wt[:, 2] = np.where(np.abs(wt[:, 2]) > 0.9, np.float32(1.0), np.float32(0.25))
    conv = G.Conv(wt, 1, r // 2, F32)
    try:
        y, _ = conv.run(x, None, None, None, False)
    finally:
        conv.close()
    with np.errstate(all="ignore"):
        ref64 = torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(wt).double(), None, 1, r // 2).numpy()
        ref = np.where(np.abs(ref64) > np.finfo(np.float32).max, np.sign(ref64) * np.inf, ref64)
    sure = ~(np.abs(np.abs(ref64) / np.finfo(np.float32).max - 1) < 1e-5)   # the border to infinity itself
    assert np.array_equal(np.isnan(y[sure]), np.isnan(ref[sure]))
    inf = np.isinf(ref) & sure
    assert inf.any() and np.isnan(ref).any() and (np.abs(ref[np.isfinite(ref)]) > 3e38).any()
    assert np.array_equal(y[inf], ref[inf].astype(np.float32))
    fin = np.isfinite(ref) & sure
    size = torch.nn.functional.conv2d(torch.from_numpy(np.nan_to_num(np.abs(x), posinf=0)).double(),
                                      torch.from_numpy(np.nan_to_num(np.abs(wt), posinf=0)).double(), None, 1, r // 2).numpy()
    assert (np.abs(y[fin] - ref[fin]) <= 4e-6 * size[fin]).all()   # 2^-24 for each of at most 64 partial sums of the magnitudes


def test_conv_f32_tiny_values():
    """Below 2^-110 the third plane runs out of bf16's range: a value is kept to half of 2^-133."""
    g = np.random.default_rng(8)
    x = (g.standard_normal((1, 128, 6, 6)) * 2.0 ** -116).astype(np.float32)
    conv = G.Conv(np.eye(128, dtype=np.float32)[:, :, None, None], 1, 0, F32)
    try:
        y, _ = conv.run(x, None, None, None, False)
    finally:
        conv.close()
    assert np.abs(y.astype(np.float64) - x).max() <= 2.0 ** -134


def _plan_and_maps(sizes, c=128, k=128, r=3):
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    w = torch.randn((k, c, r, r), device="cuda", generator=g) / (c * r * r) ** 0.5
    conv = G.Conv(w.cpu().numpy(), 1, r // 2, F32)
    xs = [torch.randn((n, 28, 28, c), device="cuda", generator=g) for n in sizes]

    def run(x, y):
        check(lib().nncv_b200_conv_run(conv.h, G.p(x), G.p(y), x.shape[0], 28, 28, None, None, None, 1, G.stream_ptr()))
        return y

    want = [run(x, torch.zeros((x.shape[0], 28, 28, k), device="cuda")) for x in xs]
    G.sync_check()
    return conv, xs, want, run


def test_conv_f32_one_plan_on_two_streams():
    """Calls of one plan on different streams share nothing that they write."""
    conv, xs, want, run = _plan_and_maps([16, 16, 3])
    try:
        streams = [torch.cuda.Stream() for _ in xs]
        got = [[torch.zeros_like(w) for w in want] for _ in range(20)]
        G.sync_check()
        for ys in got:
            for s, x, y in zip(streams, xs, ys):
                with torch.cuda.stream(s):
                    run(x, y)
        G.sync_check()
        for ys in got:
            assert all(torch.equal(y, w) for y, w in zip(ys, want))
    finally:
        conv.close()
    assert lib().nncv_b200_device_status() == 0


def test_conv_f32_captured_calls_keep_their_workspace():
    """A graph of a plan's calls gives the same after larger calls of the plan, on another stream, and with two graphs in turn."""
    conv, xs, want, run = _plan_and_maps([2, 5, 40])
    try:
        graphs, ys = [], [torch.zeros_like(w) for w in want[:2]]
        for x, y in zip(xs, ys):
            graphs.append(torch.cuda.CUDAGraph())
            with torch.cuda.graph(graphs[-1]):
                run(x, y)
        assert torch.equal(run(xs[2], torch.zeros_like(want[2])), want[2])
        for y in ys:
            y.zero_()
        G.sync_check()
        streams = [torch.cuda.Stream() for _ in graphs]
        for _ in range(10):
            for s, gr in zip(streams, graphs):
                with torch.cuda.stream(s):
                    gr.replay()
        G.sync_check()
        assert all(torch.equal(y, w) for y, w in zip(ys, want))
        del graphs
    finally:
        conv.close()
    assert lib().nncv_b200_device_status() == 0
