"""Batches in host memory: the way a batch is cut into parts, which the first calls of a shape vary, changes no logit; pinned
and pageable images (small enough for one staged copy, and large enough for the pinned ring, with a ragged last piece); a
smaller batch in the workspace of a larger one."""
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
