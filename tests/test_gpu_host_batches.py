"""Batches in host memory: the way a batch is cut into parts, which the first calls of a shape vary, changes no logit; pinned
and pageable images (small enough for one staged copy, and large enough for the pinned ring, with a ragged last piece); a
smaller batch in the workspace of a larger one."""
import ctypes

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
        for call in range(20):   # more than the calls that try the ways
            got = torch.full((n, 1000), float("nan"), pin_memory=pinned)
            rt.forward(got, x)
            assert torch.equal(got, want.cpu()), call
        rt.forward(got[:3], x[:3])
        assert torch.equal(got[:3], want[:3].cpu())
    finally:
        rt.unload()


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
