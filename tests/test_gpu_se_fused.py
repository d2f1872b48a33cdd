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


@pytest.mark.parametrize("compute,io", [(F16, torch.float32), (BF16, torch.float32), (F32, torch.float32), (F16, torch.float16), (BF16, torch.float16)])
def test_images_do_not_depend_on_the_batch_they_came_in(golden_dir, compute, io):
    path = os.path.join(golden_dir, "mobilenetv3_from_mlir.plan")
    total, out, nodes = P.parse_plan_text(open(path).read())
    blob = P.random_blob(total, nodes, seed=4)
    if io == torch.float16:
        blob = blob.astype(np.float16)
    rt.load_blob("plan:" + open(path).read(), blob, compute)
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(5)
        x = torch.randn((225, 3, 40, 72), device="cuda", generator=g).to(io)
        full = torch.zeros((225, out), device="cuda", dtype=io)
        rt.forward(full, x)
        # one image a cluster, staged and not; two; the whole batch: four.  Depthwise layers with one tile an SM and with several.
        for lo, hi in ((0, 1), (7, 25), (50, 82), (150, 198), (100, 213)):
            part = torch.zeros((hi - lo, out), device="cuda", dtype=io)
            rt.forward(part, x[lo:hi].contiguous())
            if compute != F32:
                assert torch.equal(part, full[lo:hi])
            else:   # fp32 convolutions split their reduction by the batch: the sums of 46 layers are rounded in another order
                assert G.rel_l2(part.cpu().numpy(), full[lo:hi].cpu().numpy()) <= 46 * 2.0 ** -22
        ref = P.run_plan_cpu(nodes, blob.astype(np.float32), x[223:].float().cpu().numpy(), ob, acc64=compute == F32)
        # as for the network at other sizes: the layers' roundings to the compute type, 46 of them
        assert G.rel_l2(full[223:].cpu().numpy(), ref) <= {F32: 1e-4, F16: 1e-2, BF16: 5e-2}[compute]
    finally:
        rt.unload()


def test_the_type_of_the_file_changes_no_sum(golden_dir):
    """An fp16 file on fp16 images, and the same values in fp32: the arithmetic is that of the network, not of what holds its numbers."""
    path = os.path.join(golden_dir, "mobilenetv3_from_mlir.plan")
    total, out, nodes = P.parse_plan_text(open(path).read())
    blob = P.random_blob(total, nodes, seed=6).astype(np.float16)
    for n, h, w in ((1, 224, 224), (48, 64, 96)):
        x = np.random.default_rng(n).standard_normal((n, 3, h, w)).astype(np.float16)
        got = []
        for io in (np.float16, np.float32):
            rt.load_blob("plan:" + open(path).read(), blob.astype(io), F16)
            try:
                logits = np.zeros((n, out), io)
                rt.forward(logits, x.astype(io))
                got.append(logits.astype(np.float16))
            finally:
                rt.unload()
        assert np.array_equal(*got)


def test_host_batches_in_halves_from_an_fp16_file(golden_dir):
    """A batch in host memory that runs whole and in halves in turn, until one of them is settled."""
    path = os.path.join(golden_dir, "mobilenetv3_from_mlir.plan")
    total, out, nodes = P.parse_plan_text(open(path).read())
    rt.load_blob("plan:" + open(path).read(), P.random_blob(total, nodes, seed=4).astype(np.float16), F16)
    try:
        x = torch.randn((64, 3, 224, 224)).half().pin_memory()   # 19 MB
        want = torch.zeros((64, out), device="cuda", dtype=torch.float16)
        rt.forward(want, x.cuda())
        for call in range(10):
            got = torch.full((64, out), float("nan"), dtype=torch.float16).pin_memory()
            rt.forward(got, x)
            assert torch.equal(got, want.cpu()), call
    finally:
        rt.unload()
