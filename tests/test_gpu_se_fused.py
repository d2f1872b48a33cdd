"""Squeeze-and-excitation as one kernel (pool, gate and scaling by a cluster of CTAs that owns one, two or four images,
chosen by the batch): through a small imported mobile network, at batches on either side of each choice and with a last,
partly filled cluster."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from oracle import binding as ob  # noqa: E402
from nncv_b200 import runtime as rt  # noqa: E402
from nncv_b200._lib import BF16, F16, F32  # noqa: E402
import gpu_util as G  # noqa: E402
import plan_util as P  # noqa: E402


@pytest.mark.parametrize("compute", [F16, BF16, F32])
def test_images_do_not_depend_on_the_batch_they_came_in(golden_dir, compute):
    path = os.path.join(golden_dir, "mobilenetv3_from_mlir.plan")
    total, out, nodes = P.parse_plan_text(open(path).read())
    blob = P.random_blob(total, nodes, seed=4)
    rt.load_blob("plan:" + open(path).read(), blob, compute)
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(5)
        x = torch.randn((225, 3, 40, 72), device="cuda", generator=g)
        full = torch.zeros((225, out), device="cuda")
        rt.forward(full, x)
        for lo, hi in ((0, 1), (7, 25), (100, 213)):    # one image a cluster, staged and not; two; the whole batch: four
            part = torch.zeros((hi - lo, out), device="cuda")
            rt.forward(part, x[lo:hi].contiguous())
            if compute != F32:
                assert torch.equal(part, full[lo:hi])
            else:   # fp32 convolutions split their reduction by the batch: the sums of 46 layers are rounded in another order
                assert G.rel_l2(part.cpu().numpy(), full[lo:hi].cpu().numpy()) <= 46 * 2.0 ** -22
        ref = P.run_plan_cpu(nodes, blob, x[223:].cpu().numpy(), ob, acc64=compute == F32)
        # as for the network at other sizes: the layers' roundings to the compute type, 46 of them
        assert G.rel_l2(full[223:].cpu().numpy(), ref) <= {F32: 1e-4, F16: 1e-2, BF16: 5e-2}[compute]
    finally:
        rt.unload()
