"""The convolutions on 64 x 32 tiles (small batches) against the 128-row kernels, bit for bit, and against the oracle."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from nncv_b200._lib import BF16, F16, check, lib
from oracle import binding as ob
from tests import gpu_util as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    # n, c, h, w, k, r, stride: one block, more blocks than stages, ragged channels and columns, tiles of several images, odd maps
    (1, 8, 5, 7, 8, 1, 1), (1, 64, 8, 8, 32, 1, 1), (1, 512, 7, 7, 512, 3, 1), (3, 72, 7, 9, 40, 3, 1), (2, 24, 17, 19, 88, 3, 2),
    (5, 128, 28, 28, 24, 1, 1), (1, 64, 56, 56, 64, 3, 1), (9, 64, 4, 4, 72, 1, 2), (1, 16, 3, 130, 48, 3, 1), (2, 256, 14, 14, 1000, 1, 1),
])
@pytest.mark.parametrize("dtype,res,relu", [(F16, False, False), (F16, True, True), (BF16, True, False), (BF16, False, True)])
def test_small_tiles(case, dtype, res, relu):
    n, c, h, w, k, r, stride = case
    g = np.random.default_rng(n + c + h + w + k + r)
    x = g.standard_normal((n, c, h, w)).astype(np.float32)
    wt = (g.standard_normal((k, c, r, r)) * np.sqrt(2.0 / (r * r * c))).astype(np.float32)
    scale, shift = g.uniform(0.5, 1.5, k).astype(np.float32), (g.standard_normal(k) * 0.1).astype(np.float32)
    pad = r // 2
    oh, ow = (h + 2 * pad - r) // stride + 1, (w + 2 * pad - r) // stride + 1
    rs = g.standard_normal((n, k, oh, ow)).astype(np.float32) if res else None
    conv = G.Conv(wt, stride, pad, dtype)
    try:
        check(lib().nncv_b200_conv_set_tile(conv.h, 32, 1, 0))
        small, xq = conv.run(x, scale, shift, rs, relu)
        check(lib().nncv_b200_conv_set_tile(conv.h, 64, 1, 0))
        want, _ = conv.run(x, scale, shift, rs, relu)
    finally:
        conv.close()
    assert np.array_equal(small, want)
    q = lambda a: torch.from_numpy(a).to(G.TORCH_DT[dtype]).float().numpy()
    ref = ob.conv2d(xq, q(wt), stride, pad, acc64=True) * scale[None, :, None, None] + shift[None, :, None, None]
    ref = ref + q(rs) if res else ref
    ref = np.where(ref > 0, ref, 0) if relu else ref
    assert G.rel_l2(small, ref) <= (2e-3 if dtype == F16 else 8e-3)
    assert lib().nncv_b200_device_status() == 0


@pytest.mark.parametrize("n,c,h,w,k", [(1, 64, 56, 56, 128), (3, 256, 14, 14, 512), (1, 64, 9, 13, 128)])
def test_small_tiles_with_branch(n, c, h, w, k):
    g = np.random.default_rng(n + c + h)
    x = g.standard_normal((n, c, h, w)).astype(np.float32)
    w3 = (g.standard_normal((k, c, 3, 3)) * np.sqrt(2.0 / (9 * c))).astype(np.float32)
    w1 = (g.standard_normal((k, c, 1, 1)) * np.sqrt(2.0 / c)).astype(np.float32)
    cols = [G.dev(a.astype(np.float32)) for a in (g.uniform(0.5, 1.5, k), g.standard_normal(k), g.uniform(0.5, 1.5, k), g.standard_normal(k))]
    X = G.dev(np.ascontiguousarray(x.transpose(0, 2, 3, 1)), F16)
    oh, ow = (h - 1) // 2 + 1, (w - 1) // 2 + 1
    main, branch = G.Conv(w3, 2, 1, F16), G.Conv(w1, 2, 0, F16)
    got = []
    try:
        for bn in (32, 128):
            check(lib().nncv_b200_conv_set_tile(main.h, bn, 1, 0))
            Y = [torch.full((n, oh, ow, k), float("nan"), device="cuda", dtype=torch.float16) for _ in range(2)]
            check(lib().nncv_b200_conv_run_fused(main.h, branch.h, G.p(X), G.p(Y[0]), G.p(Y[1]), n, h, w, *map(G.p, cols), 1, G.stream_ptr()))
            G.sync_check()
            got.append(Y)
    finally:
        main.close()
        branch.close()
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and not got[0][0].isnan().any()


def _off(a, floats):
    """A device copy of the vector that starts `floats` floats past a 256-byte boundary."""
    t = torch.zeros(a.size + 8, device="cuda")
    t[floats:floats + a.size] = torch.from_numpy(a).cuda()
    return t[floats:floats + a.size]


@pytest.mark.parametrize("bn", [0, 32, 64])
@pytest.mark.parametrize("algo", [0, 2])
def test_scale_and_shift_on_any_float_boundary(algo, bn):
    """A shape's kernel is settled (bn 0: by timing) with aligned vectors; the same call then takes vectors one to three floats on."""
    n, c, h, w, k = 1, 128, 7, 9, 64
    g = np.random.default_rng(3)
    wt = (g.standard_normal((k, c, 3, 3)) * np.sqrt(2.0 / (9 * c))).astype(np.float32)
    scale, shift = g.uniform(0.5, 1.5, k).astype(np.float32), g.standard_normal(k).astype(np.float32)
    X = G.dev(g.standard_normal((n, h, w, c)).astype(np.float32), F16)
    conv, got = G.Conv(wt, 1, 1, F16, algo), []
    try:
        check(lib().nncv_b200_conv_set_tile(conv.h, bn, 1, 0))
        for off in (0, 1, 2, 3):
            S, H = _off(scale, off), _off(shift, (off + 1) % 4 if off else 0)
            Y = torch.full((n, h, w, k), float("nan"), device="cuda", dtype=torch.float16)
            check(lib().nncv_b200_conv_run(conv.h, G.p(X), G.p(Y), n, h, w, G.p(S), G.p(H), None, 1, G.stream_ptr()))
            G.sync_check()
            got.append(Y)
    finally:
        conv.close()
    assert not got[0].isnan().any() and all(torch.equal(y, got[0]) for y in got[1:])


@pytest.mark.parametrize("bn", [0, 32, 128])
def test_branch_scale_and_shift_on_any_float_boundary(bn):
    n, c, h, w, k = 1, 64, 9, 13, 128
    g = np.random.default_rng(4)
    w3 = (g.standard_normal((k, c, 3, 3)) * np.sqrt(2.0 / (9 * c))).astype(np.float32)
    w1 = (g.standard_normal((k, c, 1, 1)) * np.sqrt(2.0 / c)).astype(np.float32)
    cols = [a.astype(np.float32) for a in (g.uniform(0.5, 1.5, k), g.standard_normal(k), g.uniform(0.5, 1.5, k), g.standard_normal(k))]
    X = G.dev(g.standard_normal((n, h, w, c)).astype(np.float32), F16)
    oh, ow = (h - 1) // 2 + 1, (w - 1) // 2 + 1
    main, branch, got = G.Conv(w3, 2, 1, F16), G.Conv(w1, 2, 0, F16), []
    try:
        check(lib().nncv_b200_conv_set_tile(main.h, bn, 1, 0))
        for off in (0, 1):
            v = [_off(a, off) for a in cols]
            Y = [torch.full((n, oh, ow, k), float("nan"), device="cuda", dtype=torch.float16) for _ in range(2)]
            check(lib().nncv_b200_conv_run_fused(main.h, branch.h, G.p(X), G.p(Y[0]), G.p(Y[1]), n, h, w, *map(G.p, v), 1, G.stream_ptr()))
            G.sync_check()
            got.append(Y)
    finally:
        main.close()
        branch.close()
    assert not got[0][0].isnan().any() and torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


FORWARD = """
import sys
sys.path.insert(0, {root!r})
import numpy as np
from nncv_b200 import runtime as rt
from nncv_b200.split_params import random_input, random_state_dict, to_flat_array
from tests import plan_util as P
name, compute, silu, out = sys.argv[1], int(sys.argv[2]), sys.argv[3] == "1", sys.argv[4]
if name == "mobilenetv3":
    text = open({root!r} + "/tests/golden/mobilenetv3_from_mlir.plan").read()
    if silu:
        text = "\\n".join(l.replace("act=3", "act=5") if l.startswith("conv") else l for l in text.splitlines())
    total, classes, nodes = P.parse_plan_text(text)
    rt.load_blob("plan:" + text, P.random_blob(total, nodes, seed=4), compute)
else:
    rt.load_blob(name, to_flat_array(18, random_state_dict(18, 0)).blob(), compute)
x = random_input(2, 97, 75, 5, "normal")
y = np.zeros((2, 1000), np.float32)
rt.forward(y, x)
rt.profile(True)
rt.forward(y, x)
tiles = [r["bn"] for r in rt.profile_records() if r["kind"] == 5]
rt.profile(False)
np.savez(out, y=y, small=sum(t == 320 for t in tiles), launches=len(tiles))
"""


@pytest.mark.parametrize("name,compute,silu", [("resnet18", F16, False), ("resnet18", BF16, False), ("mobilenetv3", F16, False), ("mobilenetv3", F16, True)])
def test_networks_on_small_tiles_throughout(tmp_path, name, compute, silu):
    """Every convolution of a network on 64 x 32 tiles, by a cache of decisions that says so, against 64-column tiles: bit for bit.
    ResNet-18 has maps with pad slots, residuals, branches and fp32 logits; the mobile network fused hard-swish (or SiLU) and odd
    channel counts."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    cache, got = tmp_path / "tune.txt", {}
    for kind in ("timed", "9 32 1 0", "5 64 1 0"):
        if kind != "timed":
            # (a launch fused with a branch exists for 128 columns)
            cache.write_text("".join(f"{k} = {kind if not (k.split()[-2] in ('res2', 'res3') and kind[0] == '5') else '5 128 1 0'}\n" if k.startswith("conv c") else f"{k} = {v}\n"
                                     for k, v in (line.split(" = ") for line in decisions)))
        out = str(tmp_path / "out.npz")
        r = subprocess.run([sys.executable, "-c", FORWARD.format(root=root), name, str(compute), str(int(silu)), out], capture_output=True, text=True,
                           timeout=600, env=dict(os.environ, NNCV_B200_TUNE_CACHE=str(cache)))
        assert r.returncode == 0, r.stderr[-2000:]
        if kind == "timed":
            decisions = cache.read_text().splitlines()
        got[kind] = dict(np.load(out))
    small, wide = got["9 32 1 0"], got["5 64 1 0"]
    assert small["launches"] > 15 and small["small"] == small["launches"] and wide["small"] == 0
    assert np.isfinite(small["y"]).all() and np.array_equal(small["y"], wide["y"])


CANDIDATES = """
import sys
sys.path.insert(0, {root!r})
import numpy as np
from nncv_b200._lib import F16
from tests import gpu_util as G
n, c, h, w, k = map(int, sys.argv[1:])
conv = G.Conv(np.ones((k, c, 1, 1), np.float32), 1, 0, F16)
conv.run(np.ones((n, c, h, w), np.float32))
conv.close()
"""


@pytest.mark.parametrize("n,c,h,w,k,timed", [
    (128, 64, 1, 1, 1000, True), (5, 64, 7, 7, 512, True),     # one matrix of 64 tiles (as images of one pixel 512); the same of 7 x 7
    (64, 64, 7, 7, 512, False), (2048, 64, 1, 1, 1000, False),
])
def test_the_launched_shape_decides_whether_small_tiles_are_timed(n, c, h, w, k, timed):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, NNCV_B200_LOG="2")
    env.pop("NNCV_B200_TUNE_CACHE", None)
    r = subprocess.run([sys.executable, "-c", CANDIDATES.format(root=root), *map(str, (n, c, h, w, k))], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    log = r.stdout + r.stderr
    assert "kernel 5 tile 64" in log and ("kernel 9 tile 32" in log) == timed
