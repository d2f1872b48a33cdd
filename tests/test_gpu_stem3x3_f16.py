"""The 3x3 stride-2 first layer on fp16 images and an fp16 filter, behind a global average pool and a FC layer: ragged rows and
columns, every activation, every pixel by itself; the same bits as with the same values in fp32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from nncv_b200 import runtime as rt  # noqa: E402
from nncv_b200._lib import BF16, F16, lib  # noqa: E402
import gpu_util as G  # noqa: E402


def _run(x, cout, act, compute, w=None):
    """Logits of conv (+ act) -> average pool -> FC that copies the channels, and the same in 64 bits (before any rounding to 16, but
    saturated like 16-bit maps)."""
    g = np.random.default_rng(cout + act)
    wt = ((g.standard_normal((cout, 3, 3, 3)) * 0.3) if w is None else w).astype(np.float16)
    b = (g.standard_normal(cout) * 0.2).astype(np.float16) if w is None else np.zeros(cout, np.float16)
    off = 27 * cout
    blob = np.concatenate([wt.ravel(), b, np.eye(cout, dtype=np.float16).ravel(), np.zeros(cout, np.float16)])
    plan = (f"plan:nncv_b200_plan 1\nparams {blob.size} out {cout}\n"
            f"conv id=1 in=0 res=-1 cin=3 cout={cout} k=3 stride=2 pad=1 relu={int(act == 1)} act={act} w=0 b={off}\n"
            f"avgpool id=2 in=1\nfc id=3 in=2 cin={cout} cout={cout} w={off + cout} b={off + cout + cout * cout}\n")
    got = {}
    for io in (np.float16, np.float32):   # what fp16 holds, fp32 holds too: the element type of file and images changes no sum
        rt.load_blob(plan, blob.astype(io), compute)
        try:
            got[io] = np.zeros((x.shape[0], cout), io)
            rt.forward(got[io], x.astype(io))
            assert lib().nncv_b200_device_status() == 0
        finally:
            rt.unload()
    got = got[np.float16], got[np.float32]
    assert np.array_equal(got[0], got[1].astype(np.float16), equal_nan=True)
    got = got[0]
    y = torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(wt).double(), torch.from_numpy(b).double(), stride=2, padding=1)
    y = {0: lambda v: v, 1: torch.relu, 3: torch.nn.functional.hardswish, 5: torch.nn.functional.silu}[act](y).clamp(-65504, 65504)
    return got, y.mean((2, 3)).numpy()


@pytest.mark.parametrize("n,h,w", [(1, 224, 224), (2, 33, 40), (3, 8, 8), (1, 1, 16), (2, 2, 24), (1, 65, 104), (1, 40, 440), (1, 16, 456), (100, 64, 64), (2, 32, 42)])
@pytest.mark.parametrize("cout,act,compute", [(16, 3, F16), (16, 0, BF16), (32, 1, F16), (64, 5, F16), (16, 3, BF16)])
def test_first_layer(n, h, w, cout, act, compute):
    g = np.random.default_rng(n * h + w)
    x = g.standard_normal((n, 3, h, w)).astype(np.float16)
    got, ref = _run(x, cout, act, compute)
    # roundings to 16 bits: of the map (averaged), of the pooled vector and of the logits
    assert G.rel_l2(got.astype(np.float64), ref) <= (3 * 2.0 ** -11 if compute == F16 else 2 * 2.0 ** -8 + 2.0 ** -11)


@pytest.mark.parametrize("h,w", [(5, 8), (8, 24), (6, 42)])
def test_every_pixel(h, w):
    """One image for each pixel and channel, zero elsewhere: its logits are the filter values that meet this pixel, added up, and no
    other pixel hides what an output at the wrong place, missed or done twice makes of them."""
    x = np.zeros((3 * h * w, 3, h, w), np.float16)
    x.reshape(3 * h * w, -1)[np.arange(3 * h * w), np.arange(3 * h * w)] = 64
    got, ref = _run(x, 16, 0, F16, w=np.random.default_rng(5).uniform(0.5, 1.5, (16, 3, 3, 3)))
    # up to four products of 64 and a filter value, each rounded to 16 bits; their mean and the logit once more
    assert (np.abs(got - ref) <= 3 * 2.0 ** -11 * ref + 2.0 ** -24).all() and (ref > 0).all()


@pytest.mark.parametrize("col", [0, 2, 3, 6, 7, 15])
def test_an_infinite_pixel_reaches_its_window_only(col):
    """Output x reads columns 2 x - 1 .. 2 x + 1.  Of the eight outputs, each that an infinity reaches adds an eighth of the largest
    16-bit value to the mean."""
    x = np.ones((1, 3, 2, 16), np.float16)
    x[0, 1, 0, col] = np.inf
    got, ref = _run(x, 16, 0, F16, w=np.full((16, 3, 3, 3), 0.25))
    assert (np.abs(ref / 8188 - (1 if col % 2 == 0 or col == 15 else 2)) < 0.01).all() and (np.abs(got - ref) <= 2 * 2.0 ** -11 * ref).all()
