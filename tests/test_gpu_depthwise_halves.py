"""Depthwise convolution of fp16 maps (converted by multiply-adds with 1) with a filter in fp16 and in fp32: against torch in 64 bits,
at edges of tiles, in one tile an SM and in several, with subnormals, infinities and NaN; the same bits in every batch."""
import pytest

torch = pytest.importorskip("torch")
from nncv_b200._lib import F16, F32, check, lib  # noqa: E402
from tests import gpu_util as G  # noqa: E402

pytestmark = pytest.mark.gpu


def _run(x, wt, scale, shift, stride, act):
    n, h, w, c = x.shape
    k = wt.shape[1]
    oh, ow = (h + 2 * (k // 2) - k) // stride + 1, (w + 2 * (k // 2) - k) // stride + 1
    y = torch.full((n * oh * ow * c + 64,), -77.0, device="cuda", dtype=torch.float16)
    check(lib().nncv_b200_depthwise_conv_nhwc(G.p(x), G.p(wt), F16 if wt.dtype == torch.float16 else F32, G.p(scale), G.p(shift), G.p(y), F16, n, h, w,
                                              c, k, k, stride, k // 2, act, G.stream_ptr()))
    G.sync_check()
    assert (y[-64:] == -77).all()
    ref = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), wt.double().unsqueeze(1), None, stride, k // 2, 1, c).permute(0, 2, 3, 1)
    ref = ref * scale.double() + shift.double()
    return y[:-64].reshape(n, oh, ow, c), ref.clamp_min(0) if act == 1 else ref


def _inputs(n, c, h, w, k, half):
    g = torch.Generator(device="cuda")
    g.manual_seed(n + c + h + w + k)
    x = torch.randn((n, h, w, c), device="cuda", generator=g).half()
    wt = torch.randn((c, k, k), device="cuda", generator=g) / k
    return x, wt.half() if half else wt, torch.rand(c, device="cuda", generator=g) + 0.5, torch.randn(c, device="cuda", generator=g) * 0.1


@pytest.mark.parametrize("n,c,h,w", [(1, 16, 1, 1), (1, 240, 14, 14), (300, 16, 1, 1), (200, 24, 7, 7), (64, 72, 17, 33), (160, 16, 9, 5), (40, 264, 13, 14),
                                     (8, 200, 65, 30)])
@pytest.mark.parametrize("k,stride", [(3, 1), (3, 2), (5, 1), (5, 2)])
@pytest.mark.parametrize("half", [True, False])
def test_depthwise_halves(n, c, h, w, k, stride, half):
    x, wt, scale, shift = _inputs(n, c, h, w, k, half)
    got, ref = _run(x, wt, scale, shift, stride, 1)
    # one rounding of the result (2^-11 of it, or half of fp16's smallest step), and 25 of 2^-24 of sums whose terms come to some 5
    bound = ref.abs() * 2.0 ** -11 + 2.0 ** -25 + 25 * 2.0 ** -24 * 5
    assert ((got.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("k,stride", [(3, 1), (3, 2), (5, 1), (5, 2)])
@pytest.mark.parametrize("half", [True, False])
@pytest.mark.parametrize("n", [1, 64])
def test_depthwise_halves_special(n, k, stride, half):
    x, wt, scale, shift = _inputs(n, 32, 17, 19, k, half)
    x[:, ::3, ::2, 4:8] *= 2.0 ** -15          # subnormal fp16
    got, ref = _run(x, wt * 1.0, scale, shift * 0, stride, 0)
    assert ((got.double() - ref).abs() <= ref.abs() * 2.0 ** -11 + 2.0 ** -25 + 25 * 2.0 ** -24 * 5).all()
    # only subnormals: results are small enough that their own rounding shows what was lost
    y = (torch.randint(-1023, 1024, x.shape, device="cuda").double() * 2.0 ** -24).half()
    got, ref = _run(y, wt, scale * 2.0 ** 12, shift * 0, stride, 0)
    assert ref.abs().max() > 0.1 and ((got.double() - ref).abs() <= ref.abs() * 2.0 ** -11 + 2.0 ** -25 + 25 * 2.0 ** -24 * 2.0 ** -2).all()
    x[n // 2, 5, 7, 3], x[0, 11, 2, 9], x[n - 1, 0, 18, 20], x[0, 16, 0, 1] = float("inf"), float("-inf"), float("nan"), 65504.0
    got, ref = _run(x, wt, scale, shift, stride, 0)
    nan = ref.isnan()
    assert (got.isnan() == nan).all()
    big = ref.abs() >= 65504   # fp16 results saturate
    fine = ~nan & ~big
    assert ((got.double() - ref).abs()[fine] <= (ref.abs() * 2.0 ** -11 + 2.0 ** -25 + 25 * 2.0 ** -24 * 65504)[fine]).all()
    assert (got.double()[big & ~nan] == ref[big & ~nan].sign() * 65504).all()


@pytest.mark.parametrize("c,o,k,stride", [(288, 7, 5, 2), (120, 14, 5, 1), (144, 14, 5, 1), (576, 7, 5, 1), (88, 28, 3, 1)])
@pytest.mark.parametrize("half", [True, False])
def test_an_image_does_not_depend_on_its_batch(c, o, k, stride, half):
    x, wt, scale, shift = _inputs(64, c, o * stride, o * stride, k, half)
    whole, _ = _run(x, wt, scale, shift, stride, 1)
    for n in (1, 16, 32, 48):
        assert torch.equal(_run(x[:n], wt, scale, shift, stride, 1)[0], whole[:n])
    # nor on what holds the filter
    assert torch.equal(_run(x, wt.float(), scale, shift, stride, 1)[0], whole)
