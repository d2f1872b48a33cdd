"""3x3 plans for the shifted-view kernel on dense tensors: the way that is chosen by timing (converted to shared-pad form, or
straight from the dense tensor) changes no bit, and a result laid over an operand is still right."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from nncv_b200._lib import BF16, F16, check, lib  # noqa: E402
import gpu_util as G  # noqa: E402


CASES = [(1, 64, 7, 7, 64), (3, 64, 56, 40, 64), (5, 128, 17, 23, 192), (2, 256, 14, 14, 256), (9, 64, 64, 64, 64)]


@pytest.mark.parametrize("n,c,h,w,k", CASES)
@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("res", [False, True])
def test_ways_agree(n, c, h, w, k, dtype, res):
    r = np.random.default_rng(n * c + h)
    wt = (r.standard_normal((k, c, 3, 3)) / np.sqrt(9 * c)).astype(np.float32)
    X, R = (G.dev(r.standard_normal((n, h, w, ch)).astype(np.float32), dtype) for ch in (c, k))
    S, B = torch.rand(k, device="cuda") + 0.5, torch.randn(k, device="cuda")
    chosen, forced = G.Conv(wt, 1, 1, dtype, algo=2), G.Conv(wt, 1, 1, dtype, algo=2)
    check(lib().nncv_b200_conv_set_tile(forced.h, 64, 1, 0))   # a forced tile is the shifted-view kernel's

    def run(conv, x, y, residual):
        check(lib().nncv_b200_conv_run(conv.h, G.p(x), G.p(y), n, h, w, G.p(S), G.p(B), G.p(residual), 1, G.stream_ptr()))
        G.sync_check()
        return y

    want = run(forced, X, torch.zeros_like(R), R if res else None)
    for _ in range(2):
        assert torch.equal(run(chosen, X, torch.zeros_like(R), R if res else None), want)
    if res:
        over = R.clone()
        assert torch.equal(run(chosen, X, over, over), want)
    if c == k:
        over = X.clone()
        assert torch.equal(run(chosen, over, over, R if res else None), want)


@pytest.mark.parametrize("first", ["aligned", "offset"])
def test_a_residual_at_sixteen_bytes(first):
    """The conversions take a residual on any 16-byte boundary; the direct kernel wants 32 bytes and is then no candidate,
    whichever came first."""
    n, c, h, w = 4, 64, 56, 56
    r = np.random.default_rng(2)
    wt = (r.standard_normal((c, c, 3, 3)) / np.sqrt(9 * c)).astype(np.float32)
    X = G.dev(r.standard_normal((n, h, w, c)).astype(np.float32), F16)
    room = G.dev(r.standard_normal(X.numel() + 8).astype(np.float32), F16)
    off = room[8:].view(n, h, w, c)
    even = off.clone()
    assert off.data_ptr() % 32 == 16 and even.data_ptr() % 32 == 0
    conv = G.Conv(wt, 1, 1, F16, algo=2)
    got = []
    for res in (even, off, even) if first == "aligned" else (off, even, off):
        y = torch.zeros_like(X)
        check(lib().nncv_b200_conv_run(conv.h, G.p(X), G.p(y), n, h, w, None, None, G.p(res), 1, G.stream_ptr()))
        got.append(y)
    G.sync_check()
    conv.close()
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


def test_the_trial_leaves_no_trace_in_the_profile():
    """A profile around the first call of a shape, which times both ways, holds what a later call's holds."""
    n, c, h, w = 2, 128, 30, 26
    conv = G.Conv(np.random.default_rng(4).standard_normal((c, c, 3, 3)).astype(np.float32), 1, 1, F16, algo=2)
    X = torch.randn((n, h, w, c), device="cuda", dtype=torch.float16)
    Y = torch.zeros_like(X)
    counts = []
    for _ in range(2):
        check(lib().nncv_b200_profile(1))
        check(lib().nncv_b200_conv_run(conv.h, G.p(X), G.p(Y), n, h, w, None, None, None, 0, G.stream_ptr()))
        G.sync_check()
        counts.append(lib().nncv_b200_profile_count())
        check(lib().nncv_b200_profile(0))
    conv.close()
    assert counts[0] == counts[1] == 1


ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def in_a_process_of_its_own(cache, function):
    """Runs a function of this module where the tuning cache is read from `cache`."""
    code = f"import sys; sys.path[:0] = [{ROOT!r}, {os.path.join(ROOT, 'tests')!r}]; import test_gpu_conv3x3_dense as t; t.{function}()"
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, NNCV_B200_TUNE_CACHE=str(cache)), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


def capture_one_image_after_a_call_of_two():
    x = torch.randn((2, 16, 16, 64), device="cuda", dtype=torch.float16)
    wt = np.random.default_rng(3).standard_normal((64, 64, 3, 3)).astype(np.float32) / 24
    conv, forced = G.Conv(wt, 1, 1, F16, algo=2), G.Conv(wt, 1, 1, F16, algo=2)
    check(lib().nncv_b200_conv_set_tile(forced.h, 64, 1, 0))

    def run(c, n, y):
        check(lib().nncv_b200_conv_run(c.h, G.p(x), G.p(y), n, 16, 16, None, None, None, 0, G.stream_ptr()))
        return y

    run(conv, 2, torch.zeros_like(x))
    want = run(forced, 1, torch.zeros_like(x[:1]))
    got = torch.zeros_like(want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(conv, 1, got)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)


def test_capture_with_a_cache_that_knows_the_tiles_only(tmp_path):
    """A tuning cache from before there were two ways names a shape's tile and no way: its call can be captured all the same."""
    cache = tmp_path / "tuned"
    key = "conv c64 k64 r3 s3 st1 p1 dt1 a2 n%d h16 w16 res0 o1 = 2 64 1 0\n"
    cache.write_text(key % 1 + key % 2 + "conv3x3 way c64 k64 dt1 n2 h16 w16 res0 = 0\n")
    in_a_process_of_its_own(cache, "capture_one_image_after_a_call_of_two")


def compare_with_a_forced_tile():
    for n, c, h, w, k in CASES:
        for dtype in (F16, BF16):
            for res in (False, True):
                test_ways_agree(n, c, h, w, k, dtype, res)


@pytest.mark.parametrize("way", ["0", "1"])
def test_either_way_gives_the_same_bits(tmp_path, way):
    """test_ways_agree compares the way that happens to be faster; here either is named by the tuning cache."""
    cache = tmp_path / "tuned"
    lines = [f"conv3x3 way c{c} k{k} dt{dt} n{n} h{h} w{w} res{res} = {way}\n" for n, c, h, w, k in CASES for dt in (F16, BF16) for res in (0, 1)]
    cache.write_text("".join(lines))
    in_a_process_of_its_own(cache, "compare_with_a_forced_tile")
    text = cache.read_text()
    assert text.startswith("".join(lines)) and "conv3x3 way" not in text[len("".join(lines)):]   # nothing was tried
    direct = text.count(" res4 ") + text.count(" res5 ")   # tiles tuned for the direct kernel on dense tensors
    assert (direct > 0) == (way == "1")
