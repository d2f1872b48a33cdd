"""Batches in host memory: the number of parts a batch runs in -- one, two or four, by its bytes, the way of the largest settled
by their first eight calls -- changes no logit; pinned and pageable images (small enough for one staged copy, and large enough
for the pinned ring, with a ragged last piece); a smaller batch in the workspace of a larger one; a call that fails."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from nncv_b200 import runtime as rt  # noqa: E402
from nncv_b200._lib import F16  # noqa: E402
from nncv_b200.split_params import random_input, random_state_dict, to_flat_array  # noqa: E402


@pytest.mark.parametrize("n,h,w", [(15, 64, 64), (17, 64, 40), (67, 32, 64), (35, 224, 220)])
@pytest.mark.parametrize("pinned", [False, True])
def test_parts_change_nothing(n, h, w, pinned):
    x = torch.from_numpy(random_input(n, h, w, 7, "normal"))
    if pinned:
        x = x.pin_memory()
    rt.load_blob("resnet18", to_flat_array(18, random_state_dict(18, 0)).blob(), F16)
    try:
        want = torch.zeros((n, 1000), device="cuda")
        rt.forward(want, x.cuda())
        for call in range(20):
            got = torch.full((n, 1000), float("nan"), pin_memory=pinned)
            rt.forward(got, x)
            assert torch.equal(got, want.cpu()), call
        rt.forward(got[:3], x[:3])
        assert torch.equal(got[:3], want[:3].cpu())
    finally:
        rt.unload()


@pytest.mark.parametrize("n,pinned", [(97, True), (97, False), (141, True), (257, False)])   # 29 MB: whole and halves in turn; 42 and 77: halves and quarters
def test_the_calls_that_settle_the_way(n, pinned):
    x = torch.from_numpy(random_input(n, 224, 224, 3, "normal").astype(np.float16))
    x = x.pin_memory() if pinned else x
    rt.load_blob("resnet18", to_flat_array(18, random_state_dict(18, 0), np.float16).blob(), F16)
    try:
        want = torch.zeros((n, 1000), device="cuda", dtype=torch.float16)
        rt.forward(want, x.cuda())
        for call in range(11):
            got = torch.full((n, 1000), float("nan"), dtype=torch.float16, pin_memory=pinned)
            rt.forward(got, x)
            assert torch.equal(got, want.cpu()), call
    finally:
        rt.unload()


ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FORCED = [(16, 64, 64), (17, 64, 40), (67, 32, 64), (101, 224, 220)]   # the last: 60 MB of fp32 images, quarters of 15 MB


def each_in_the_forced_way():
    for n, h, w in FORCED:
        for pinned in (False, True):
            test_parts_change_nothing(n, h, w, pinned)


@pytest.mark.parametrize("parts", [1, 2, 4])
def test_every_way_gives_the_same_logits(tmp_path, parts):
    """The way named by the tuning cache, in a process of its own."""
    total = to_flat_array(18, random_state_dict(18, 0)).blob().size
    cache = tmp_path / "tuned"
    lines = "".join(f"host parts resnet18 {total} dt1 e4 n{n} h{h} w{w} pinned{p} = {parts}\n" for n, h, w in FORCED for p in (0, 1))
    cache.write_text(lines)
    code = f"import sys; sys.path[:0] = [{ROOT!r}, {os.path.join(ROOT, 'tests')!r}]; import test_gpu_host_batches as t; t.each_in_the_forced_way()"
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, NNCV_B200_TUNE_CACHE=str(cache)), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    text = cache.read_text()
    assert all(f" n{n // parts} h{h // 4} " in text for n, h, w in FORCED[:1])   # layers tuned for the parts' batch


def test_a_call_that_fails_has_no_copy_in_flight():
    """Rows 4 GB apart are more than a copy engine's pitch can say: the copy of the first logits is refused when the images are
    already on their way.  The call returns the error when nothing reads or writes the caller's memory any more."""
    import time
    from nncv_b200._lib import lib
    from nncv_b200.memref import make_descriptor
    n = 256
    rt.load_blob("resnet18", to_flat_array(18, random_state_dict(18, 0)).blob(), F16)
    try:
        x = torch.randn((n, 3, 224, 224)).pin_memory()   # 154 MB: 2.8 ms of copying at the link's rate
        out = torch.full((n, 1000), float("nan")).pin_memory()
        rt.forward(out, x)
        good = out.clone()
        s, far = make_descriptor(x.data_ptr(), x.shape), make_descriptor(out.data_ptr(), out.shape, [1 << 30, 1])
        after = []
        for _ in range(5):
            out.fill_(float("nan"))
            torch.cuda.synchronize()
            lib()._mlir_ciface_forward(ctypes.byref(far), ctypes.byref(s), None)
            t = time.perf_counter()
            torch.cuda.synchronize()
            after.append(time.perf_counter() - t)
            assert lib().nncv_b200_last_status() == 4 and torch.isnan(out).all()
        assert sorted(after)[2] < 0.5e-3
        rt.forward(out, x)
        assert torch.equal(out, good)
    finally:
        rt.unload()
