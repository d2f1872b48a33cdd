"""Where logits go: straight into device memory of the caller's (any boundary, with or without gaps between rows), or by way of the
library's pinned memory to any host memory.  The same bits everywhere, and nothing beside the rows."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from nncv_b200 import runtime as rt  # noqa: E402
from nncv_b200._lib import BF16, F16, F32, check_last, lib  # noqa: E402
from nncv_b200._lib import check as check_status  # noqa: E402
from nncv_b200.memref import make_descriptor  # noqa: E402
from nncv_b200.split_params import random_state_dict, to_flat_array  # noqa: E402


def _call(out, x, stream=None):
    """`_mlir_ciface_forward`, or with a stream `nncv_b200_forward_device`, on rows out.stride(0) elements apart."""
    d, s = make_descriptor(out.data_ptr(), tuple(out.shape)), make_descriptor(x.data_ptr(), tuple(x.shape))
    d.strides[0] = out.stride(0)
    if stream is None:
        lib()._mlir_ciface_forward(ctypes.byref(d), ctypes.byref(s), None)
        check_last()
    else:
        check_status(lib().nncv_b200_forward_device(ctypes.byref(d), ctypes.byref(s), ctypes.c_void_p(stream)))


@pytest.mark.parametrize("compute,params", [(F32, np.float32), (F16, np.float16), (BF16, np.float32), (F32, np.float16)], ids=str)
@pytest.mark.parametrize("n", [1, 3, 40])
def test_logits_arrive_the_same_everywhere(n, compute, params):
    rt.load_blob("resnet18", to_flat_array(18, random_state_dict(18, 0)).blob().astype(params), compute)
    try:
        dt = torch.float32 if params == np.float32 else torch.float16
        x = torch.randn((n, 3, 40, 40), generator=torch.Generator().manual_seed(n)).to(dt)
        xd = x.cuda()
        stream = torch.cuda.current_stream().cuda_stream
        want = torch.zeros((n, 1000), device="cuda", dtype=dt)
        rt.forward_device(want, xd, stream)
        torch.cuda.synchronize()
        want = want.cpu()
        assert torch.isfinite(want.float()).all() and want.float().abs().sum() > 0

        def check(flat, offset, pitch, run):
            flat.fill_(-3.0)
            out = flat[offset:offset + (n - 1) * pitch + 1000].as_strided((n, 1000), (pitch, 1), offset)
            run(out)
            torch.cuda.synchronize()
            assert torch.equal(out.cpu(), want)
            rest = flat.clone().cpu()
            rest.as_strided((n, 1000), (pitch, 1), offset).fill_(-3.0)
            assert (rest == -3.0).all()

        for offset, pitch in ((0, 1000), (1, 1000), (8, 1000), (16, 1000), (0, 1008), (3, 1001)):
            room = offset + n * pitch + 64
            check(torch.empty(room, device="cuda", dtype=dt), offset, pitch, lambda o: _call(o, xd, stream))
            check(torch.empty(room, device="cuda", dtype=dt), offset, pitch, lambda o: _call(o, x))
            check(torch.empty(room, dtype=dt), offset, pitch, lambda o: _call(o, x))
            check(torch.empty(room, dtype=dt).pin_memory(), offset, pitch, lambda o: _call(o, x))
            check(torch.empty(room, dtype=dt).pin_memory(), offset, pitch, lambda o: _call(o, xd))
        assert lib().nncv_b200_device_status() == 0
    finally:
        rt.unload()
