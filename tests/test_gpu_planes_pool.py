"""fp32 networks: the convolution that only a max-pool reads writes plain fp32, and the pool splits its maxima into bf16 planes.  A map
with another reader, and what a pool writes, are planes that a pool reads."""
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


def _run(lines, sizes, x, out, seed):
    """Logits of the plan of these lines ({name} for a parameter's place), and its parameters in 64 bits."""
    at, off = {}, 0
    for name, size in sizes:
        at[name] = off
        off += size
    blob = (np.random.default_rng(seed).standard_normal(off) * 0.1).astype(np.float32)
    rt.load_blob(f"plan:nncv_b200_plan 1\nparams {off} out {out}\n" + "\n".join(lines).format(**at) + "\n", blob, F32)
    try:
        got = np.zeros((x.shape[0], out), np.float32)
        rt.forward(got, x)
        assert lib().nncv_b200_device_status() == 0
    finally:
        rt.unload()
    return got, {name: torch.from_numpy(blob[at[name]:at[name] + size]).double() for name, size in sizes}


@pytest.mark.parametrize("k,stride,pad", [(3, 2, 1), (3, 1, 1), (2, 2, 0), (5, 2, 2)])
@pytest.mark.parametrize("shape", [(1, 64, 64), (2, 61, 45)])
def test_pool_behind_a_pool(shape, k, stride, pad):
    n, h, w = shape
    c, out = 40, 12
    x = np.random.default_rng(h).standard_normal((n, 3, h, w)).astype(np.float32)
    got, t = _run(["conv id=1 in=0 res=-1 cin=3 cout=40 k=7 stride=2 pad=3 relu=0 w={w} b={b}", "maxpool id=2 in=1 k=3 stride=2 pad=1",
                   f"maxpool id=3 in=2 k={k} stride={stride} pad={pad}", "avgpool id=4 in=3", "fc id=5 in=4 cin=40 cout=12 w={fw} b={fb}"],
                  [("w", c * 147), ("b", c), ("fw", out * c), ("fb", out)], x, out, k)
    pool = torch.nn.functional.max_pool2d
    y = torch.nn.functional.conv2d(torch.from_numpy(x).double(), t["w"].view(c, 3, 7, 7), t["b"], stride=2, padding=3)
    ref = (pool(pool(y, 3, 2, 1), k, stride, pad).mean((2, 3)) @ t["fw"].view(out, c).T + t["fb"]).numpy()
    assert G.rel_l2(got, ref) <= 8 * 2.0 ** -23   # as above


@pytest.mark.parametrize("how", ["convolution", "residual", "two pools", "residual in plain"])
@pytest.mark.parametrize("shape", [(1, 64, 64), (3, 41, 45)])
def test_a_pooled_map_with_another_reader(shape, how):
    """The map that a max-pool reads is a convolution's input, too, or a residual, or another pool's."""
    n, h, w = shape
    c, out = 40, 12
    x = np.random.default_rng(h).standard_normal((n, 3, h, w)).astype(np.float32)
    third = {"convolution": "conv id=3 in=1 res=2 cin=40 cout=40 k=3 stride=1 pad=1 relu=0 w={w2} b={b2}",
             "residual": "conv id=3 in=2 res=1 cin=40 cout=40 k=3 stride=1 pad=1 relu=0 w={w2} b={b2}",
             "two pools": "maxpool id=3 in=1 k=5 stride=1 pad=2",
             # a convolution that adds planes and writes plain fp32 to its only reader
             "residual in plain": "conv id=7 in=2 res=1 cin=40 cout=40 k=3 stride=1 pad=1 relu=0 w={w2} b={b2}\nmaxpool id=3 in=7 k=3 stride=1 pad=1"}[how]
    got, t = _run(["conv id=1 in=0 res=-1 cin=3 cout=40 k=7 stride=2 pad=3 relu=0 w={w} b={b}", "maxpool id=2 in=1 k=3 stride=1 pad=1", third,
                   "conv id=4 in=3 res=2 cin=40 cout=40 k=1 stride=1 pad=0 relu=0 w={w3} b={b2}", "avgpool id=5 in=4", "fc id=6 in=5 cin=40 cout=12 w={fw} b={fb}"],
                  [("w", c * 147), ("b", c), ("w2", c * c * 9), ("w3", c * c), ("b2", c), ("fw", out * c), ("fb", out)], x, out, 3)
    conv, pool = torch.nn.functional.conv2d, torch.nn.functional.max_pool2d
    a = conv(torch.from_numpy(x).double(), t["w"].view(c, 3, 7, 7), t["b"], stride=2, padding=3)
    b = pool(a, 3, 1, 1)
    w2 = t["w2"].view(c, c, 3, 3)
    d = {"convolution": lambda: conv(a, w2, t["b2"], padding=1) + b, "residual": lambda: conv(b, w2, t["b2"], padding=1) + a, "two pools": lambda: pool(a, 5, 1, 2),
         "residual in plain": lambda: pool(conv(b, w2, t["b2"], padding=1) + a, 3, 1, 1)}[how]()
    y = conv(d, t["w3"].view(c, c, 1, 1), t["b2"]) + b
    ref = (y.mean((2, 3)) @ t["fw"].view(out, c).T + t["fb"]).numpy()
    assert G.rel_l2(got, ref) <= 16 * 2.0 ** -23   # two layers more
