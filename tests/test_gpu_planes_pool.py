"""fp32 networks: the convolution that only a max-pool reads writes plain fp32, and the pool splits its maxima into bf16 planes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from nncv_b200 import runtime as rt  # noqa: E402
from nncv_b200._lib import F32, lib  # noqa: E402
import gpu_util as G  # noqa: E402


@pytest.mark.parametrize("k,stride,pad", [(3, 2, 1), (3, 1, 1), (2, 2, 0), (5, 2, 2)])
@pytest.mark.parametrize("shape", [(1, 64, 64), (2, 61, 45), (3, 22, 150)])
@pytest.mark.parametrize("relu", [0, 1])
def test_pool_behind_a_convolution(shape, k, stride, pad, relu):
    n, h, w = shape
    c, out = 40, 12
    sizes = [("w", c * 147), ("b", c), ("fw", out * c), ("fb", out)]
    at, off = {}, 0
    for name, size in sizes:
        at[name] = off
        off += size
    plan = (f"plan:nncv_b200_plan 1\nparams {off} out {out}\n"
            f"conv id=1 in=0 res=-1 cin=3 cout={c} k=7 stride=2 pad=3 relu={relu} w={at['w']} b={at['b']}\n"
            f"maxpool id=2 in=1 k={k} stride={stride} pad={pad}\navgpool id=3 in=2\nfc id=4 in=3 cin={c} cout={out} w={at['fw']} b={at['fb']}\n")
    g = np.random.default_rng(h * w + k)
    blob = (g.standard_normal(off) * 0.1).astype(np.float32)
    x = g.standard_normal((n, 3, h, w)).astype(np.float32)
    rt.load_blob(plan, blob, F32)
    try:
        got = np.zeros((n, out), np.float32)
        rt.forward(got, x)
        assert lib().nncv_b200_device_status() == 0
    finally:
        rt.unload()
    t = {name: torch.from_numpy(blob[at[name]:at[name] + size]).double() for name, size in sizes}
    y = torch.nn.functional.conv2d(torch.from_numpy(x).double(), t["w"].view(c, 3, 7, 7), t["b"], stride=2, padding=3)
    y = torch.nn.functional.max_pool2d(y.relu() if relu else y, k, stride, pad)
    ref = (y.mean((2, 3)) @ t["fw"].view(out, c).T + t["fb"]).numpy()
    # a rounding (2^-24) or a cut step (2^-23) of each of the few sums one after another
    assert G.rel_l2(got, ref) <= 8 * 2.0 ** -23
