"""What a user of nncv_b200 has it do, as cases that can be timed and compared.

Three kinds of work, all through the public entry points (`nncv_b200.runtime` and the C ABI):

  net   a whole network: `_mlir_ciface_forward` on tensors in host memory (what nncv's example driver does: images in,
        logits out, the call returns when they are there) or `nncv_b200_forward_device` on tensors in device memory.
        ResNet-18 and ResNet-50 are built in; MobileNetV3-small is the plan imported from nncv's fixture.
  gemm  linalg.matmul on row-major matrices, 16-bit or fp32, optional bias and ReLU.
  op    single operators on NHWC maps: convolutions with a fused epilogue, depthwise convolutions, pools, activations,
        the squeeze-and-excitation chain, concat and upsampling.

A network is loaded once and kept while images change, as a program does that serves it: weights belong to the network
(seed 0), images to the seed.  The library holds one model per device, so a state of another network loads it again.
"""
import ctypes
import math
import os

import numpy as np
import torch

import nncv_b200
from nncv_b200 import runtime as rt
from nncv_b200._lib import BF16, F16, F32, check, lib
from nncv_b200.split_params import random_state_dict, to_flat_array

DT = {"f32": F32, "f16": F16, "bf16": BF16}
TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZE = {"f32": 4, "f16": 2, "bf16": 2}
ACT = {"none": 0, "relu": 1, "hard_sigmoid": 2, "hard_swish": 3, "sigmoid": 4, "silu": 5}


# --------------------------------------------------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------------------------------------------------
def net(net, compute, batch, h, w, where, params="f32", name=None):
    """params: element type of the parameter file and with it of images and logits."""
    c = dict(kind="net", net=net, compute=compute, params=params, batch=batch, h=h, w=w, where=where)
    return dict(c, name=name) if name else c


def gemm(m, n, k, ab, c, epilogue=False, name=None):
    d = dict(kind="gemm", m=m, n=n, k=k, ab=ab, c=c, epilogue=epilogue)
    return dict(d, name=name) if name else d


def op(what, dtype, n, h, w, c, name=None, **more):
    d = dict(kind="op", op=what, dtype=dtype, n=n, h=h, w=w, c=c, **more)
    return dict(d, name=name) if name else d


def listed():
    return [
        # nncv's example program: one 256 x 256 picture in ordinary host memory, fp32 file, fp32 arithmetic
        net("resnet18", "f32", 1, 256, 256, "host", name="r18 f32 1x256 host"),
        # the same file and no option set (fp32 follows the file), a small batch of 224 x 224 images
        net("resnet18", "f32", 8, 224, 224, "host", name="r18 f32 8x224 host"),
        # one image at a time from another stage on the GPU: latency of a 16-bit forward
        net("resnet18", "f16", 1, 224, 224, "device", params="f16", name="r18 f16 1x224 device"),
        # images of an odd size and an odd batch, bf16 arithmetic on an fp32 file, pinned host buffers
        net("resnet18", "bf16", 13, 225, 301, "pinned", name="r18 bf16 13x225x301 pinned"),
        # the throughput configuration, device-resident and end to end from pinned host memory
        net("resnet18", "f16", 256, 224, 224, "device", params="f16", name="r18 f16 256x224 device"),
        net("resnet18", "f16", 256, 224, 224, "pinned", params="f16", name="r18 f16 256x224 pinned"),
        # the deeper network at its largest batch
        net("resnet50", "f16", 512, 224, 224, "device", params="f16", name="r50 f16 512x224 device"),
        # the mobile network, many small memory-bound layers: a serving batch
        net("mobilenetv3", "f16", 256, 224, 224, "device", params="f16", name="mbv3 f16 256x224 device"),
        # matmul: 16-bit at the largest size of the sweep, fp32 at an ordinary one with the fused epilogue
        gemm(4096, 4096, 4096, "f16", "f32", name="matmul f16 4096"),
        gemm(1024, 1024, 1024, "f32", "f32", epilogue=True, name="matmul f32 1024 bias relu"),
        # one 3x3 layer of the convolution sweep with scale / shift and ReLU
        op("conv3x3", "f16", 32, 16, 16, 256, residual=False, name="conv3x3 f16 32x16x256"),
        # the widest depthwise layer of a mobile network, batch-norm and hard-swish fused
        op("depthwise", "f16", 64, 112, 112, 96, k=3, stride=1, act="hard_swish", name="depthwise f16 64x112x96"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("net", "gemm", "op"), (0.6, 0.2, 0.2))[0]
    if kind == "net":
        name = rng.choices(("resnet18", "resnet50", "mobilenetv3"), (0.5, 0.25, 0.25))[0]
        # bf16's 8 mantissa bits are too few for MobileNetV3's 46 layers: nobody runs it so
        compute = rng.choices(("f16", "bf16", "f32"), (0.55, 0.2 if name != "mobilenetv3" else 0.0, 0.25))[0]
        side = 224 if rng.random() < 0.5 else _log(rng, 64, 384)
        h = w = side
        if rng.random() < 0.3:
            w = _log(rng, 64, 384)
        # bounds on the work: about 2 TFLOP in 16 bits, 40 GFLOP in fp32, 2 GB of activations for the mobile network
        per_image = {"resnet18": 3.63e9, "resnet50": 8.18e9, "mobilenetv3": 0.12e9}[name] * h * w / (224 * 224)
        most = 2.0e12 if compute != "f32" else 4.0e10
        top = int(min(256, max(1, most / per_image), 256 * 224 * 224 // (h * w) + 1))
        batch = _log(rng, 1, top)
        where = rng.choice(("device", "pinned", "host") if batch <= 16 else ("device", "pinned"))
        params = "f16" if compute == "f16" and rng.random() < 0.6 else "f32"
        return net(name, compute, batch, h, w, where, params)
    if kind == "gemm":
        ab = rng.choices(("f16", "bf16", "f32"), (0.5, 0.25, 0.25))[0]
        top = 4096 if ab != "f32" else 2048
        step = 8 if ab != "f32" else 4
        m, n, k = _log(rng, 16, top), _log(rng, 64, top), _log(rng, 64, top)
        n = n if ab != "f32" and rng.random() < 0.15 else max(64, n // 8 * 8)
        k = k // step * step
        c = "f32" if ab == "f32" or rng.random() < 0.5 else ab
        return gemm(m, n, k, ab, c, rng.random() < 0.5)
    what = rng.choices(("conv3x3", "conv", "depthwise", "maxpool", "avgpool", "activation", "se", "concat", "upsample2x"),
                       (3, 3, 2, 1, 1, 1, 1, 1, 1))[0]
    dtype = rng.choices(("f16", "bf16", "f32"), (0.6, 0.2, 0.2))[0]
    h, w = _log(rng, 7, 112), _log(rng, 7, 112)
    if what == "conv3x3":
        dtype = dtype if dtype != "f32" else "f16"
        c = rng.choice((64, 128, 192, 256, 512))
    elif what == "conv":
        c = 8 * _log(rng, 2, 64)
    else:
        c = 8 * _log(rng, 1, 72)
    # bounds: 100 MB an input map, and 40 GFLOP a convolution (4 in fp32)
    top = 100e6 / (h * w * c * SIZE[dtype])
    more = {}
    if what == "conv3x3":
        more = dict(residual=rng.random() < 0.5)
        top = min(top, 4.0e10 / (18.0 * h * w * c * c))
    elif what == "conv":
        r = rng.choice((1, 1, 3))
        more = dict(kout=8 * _log(rng, 2, 64), r=r, stride=rng.choice((1, 2)), residual=rng.random() < 0.3)
        top = min(top, (4.0e10 if dtype != "f32" else 4.0e9) / (2.0 * r * r * h * w * c * more["kout"]))
    elif what == "depthwise":
        more = dict(k=rng.choice((3, 5)), stride=rng.choice((1, 2)), act=rng.choice(("none", "relu", "hard_swish")))
    elif what == "maxpool":
        more = rng.choice((dict(k=3, stride=2), dict(k=5, stride=1), dict(k=2, stride=2)))
    elif what == "activation":
        more = dict(act=rng.choice(("relu", "hard_swish", "silu", "sigmoid")))
    elif what == "se":
        more = dict(cr=8 * max(1, c // 32))
    elif what == "concat":
        more = dict(c2=8 * _log(rng, 1, 32))
    n = _log(rng, 1, max(1, min(64, int(top))))
    return op(what, dtype, n, h, w, c, **more)


# --------------------------------------------------------------------------------------------------------------------
# networks
# --------------------------------------------------------------------------------------------------------------------
_plans = {}      # network -> (name for load(), nodes of its plan, parameters)
_loaded = None   # (network, compute, params) that the library holds


def _plan(name):
    if name not in _plans:
        if name == "mobilenetv3":
            root = os.path.dirname(os.path.dirname(os.path.abspath(nncv_b200.__file__)))
            with open(os.path.join(root, "tests", "golden", "mobilenetv3_from_mlir.plan")) as f:
                text = f.read()
            load_as = "plan:" + text
        else:
            load_as = name
            n = lib().nncv_b200_plan_text(name.encode(), None, 0)
            buf = ctypes.create_string_buffer(n + 1)
            lib().nncv_b200_plan_text(name.encode(), buf, n + 1)
            text = buf.value.decode()
        nodes, total = [], 0
        for line in text.splitlines():
            t = line.split("#")[0].split()
            if t and t[0] == "params":
                total = int(t[1])
            elif t and t[0] != "nncv_b200_plan":
                nodes.append((t[0], {k: int(v) for k, v in (f.split("=") for f in t[1:])}))
        _plans[name] = (load_as, nodes, total)
    return _plans[name]


def _weights(name):
    """The network's parameters, fp32, in file order: Kaiming-normal filters, batch-norm statistics around one."""
    if name != "mobilenetv3":
        depth = int(name[len("resnet"):])
        return to_flat_array(depth, random_state_dict(depth, 0)).blob()
    _, nodes, total = _plan(name)
    g = np.random.default_rng(0)
    blob = (g.standard_normal(total) * 0.05).astype(np.float32)
    for kind, f in nodes:
        if kind in ("conv", "dwconv"):
            cout, fan = f.get("cout", f.get("c")), (f["cin"] if kind == "conv" else 1) * f["k"] ** 2
            blob[f["w"]:f["w"] + cout * fan] = g.standard_normal(cout * fan) * math.sqrt(2.0 / fan)
            for role in ("gamma", "var"):
                if role in f:
                    blob[f[role]:f[role] + cout] = g.uniform(0.5, 1.5, cout)
        elif kind == "se":
            for role in ("w1", "w2"):
                blob[f[role]:f[role] + f["c"] * f["cr"]] = g.standard_normal(f["c"] * f["cr"]) * math.sqrt(1.0 / f["c"])
        elif kind == "fc":
            blob[f["w"]:f["w"] + f["cin"] * f["cout"]] = g.standard_normal(f["cin"] * f["cout"]) * math.sqrt(1.0 / f["cin"])
    return blob


def _load(key):
    global _loaded
    if _loaded != key:
        name, compute, params = key
        blob = _weights(name)
        rt.load_blob(_plan(name)[0], blob.astype(np.float16) if params == "f16" else blob, DT[compute])
        _loaded = key


def _net_flops(name, h, w):
    """Multiply-adds times two of one image: convolutions and FC layers, the direct count."""
    size, total = {0: (h, w)}, 0.0
    for kind, f in _plan(name)[1]:
        ih, iw = size.get(f["in"], (1, 1))
        out = (1, 1)
        if kind in ("conv", "dwconv", "maxpool"):
            out = ((ih + 2 * f["pad"] - f["k"]) // f["stride"] + 1, (iw + 2 * f["pad"] - f["k"]) // f["stride"] + 1)
            per = {"conv": f.get("cin", 0) * f.get("cout", 0), "dwconv": f.get("c", 0), "maxpool": 0}[kind] * f["k"] ** 2
            total += 2.0 * per * out[0] * out[1]
        elif kind == "se":
            out = (ih, iw)
            total += 4.0 * f["c"] * f["cr"]
        elif kind == "fc":
            total += 2.0 * f["cin"] * f["cout"]
        size[f["id"]] = out
    return total


# --------------------------------------------------------------------------------------------------------------------
# preparing and running
# --------------------------------------------------------------------------------------------------------------------
class Conv:
    """A convolution plan of the library, given back with the state that holds it."""

    def __init__(self, weights, stride, pad, dtype, algo):
        k, c, r, s = weights.shape
        self.h = lib().nncv_b200_conv_create(weights.data_ptr(), F32, k, c, r, s, stride, pad, dtype, algo)
        if not self.h:
            raise RuntimeError(lib().nncv_b200_last_error().decode())

    def __del__(self):
        lib().nncv_b200_conv_destroy(self.h)


def _out(i, k, stride, pad):
    return (i + 2 * pad - k) // stride + 1


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + 17)

    def normal(shape, dtype="f32", scale=1.0):
        return (torch.randn(shape, device="cuda", generator=g) * scale).to(TORCH[dtype])

    def uniform(shape, lo, hi, dtype="f32"):
        return (torch.rand(shape, device="cuda", generator=g) * (hi - lo) + lo).to(TORCH[dtype])

    if case["kind"] == "net":
        key = (case["net"], case["compute"], case["params"])
        _load(key)
        shape = (case["batch"], 3, case["h"], case["w"])
        x = uniform(shape, 0.0, 1.0, case["params"]) if case["compute"] == "f32" else normal(shape, case["params"])
        out = torch.zeros((case["batch"], 1000), device="cuda", dtype=x.dtype)
        if case["where"] != "device":
            x, out = x.cpu(), out.cpu()
            if case["where"] == "pinned":
                x, out = x.pin_memory(), out.pin_memory()
        return dict(kind="net", key=key, x=x, out=out, host=case["where"] != "device")
    if case["kind"] == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return dict(kind="gemm", dims=(m, n, k), ab=DT[case["ab"]], cd=DT[case["c"]], a=uniform((m, k), -1, 1, case["ab"]),
                    b=uniform((k, n), -1, 1, case["ab"]), c=torch.zeros((m, n), device="cuda", dtype=TORCH[case["c"]]),
                    bias=normal((n,)) if case["epilogue"] else None, relu=int(case["epilogue"]))
    n, h, w, c, dt, what = case["n"], case["h"], case["w"], case["c"], case["dtype"], case["op"]
    s = dict(kind="op", op=what, dims=(n, h, w, c), dtype=DT[dt], x=normal((n, h, w, c), dt))

    def empty(*shape):
        return torch.zeros(shape, device="cuda", dtype=TORCH[dt])

    if what in ("conv3x3", "conv"):
        k, r, stride = (c, 3, 1) if what == "conv3x3" else (case["kout"], case["r"], case["stride"])
        pad = r // 2
        oh, ow = _out(h, r, stride, pad), _out(w, r, stride, pad)
        s.update(conv=Conv(normal((k, c, r, r), scale=math.sqrt(2.0 / (c * r * r))), stride, pad, DT[dt], 2 if what == "conv3x3" else 0),
                 scale=uniform((k,), 0.5, 1.5), shift=normal((k,), scale=0.1), y=empty(n, oh, ow, k),
                 res=normal((n, oh, ow, k), dt) if case["residual"] else None)
    elif what == "depthwise":
        k, stride = case["k"], case["stride"]
        s.update(k=k, stride=stride, act=ACT[case["act"]], weights=normal((c, k, k), scale=math.sqrt(2.0) / k), scale=uniform((c,), 0.5, 1.5),
                 shift=normal((c,), scale=0.1), y=empty(n, _out(h, k, stride, k // 2), _out(w, k, stride, k // 2), c))
    elif what == "maxpool":
        k, stride = case["k"], case["stride"]
        pad = (k - 1) // 2
        s.update(k=k, stride=stride, pad=pad, y=empty(n, _out(h, k, stride, pad), _out(w, k, stride, pad), c))
    elif what == "avgpool":
        s.update(y=empty(n, c))
    elif what == "activation":
        s.update(act=ACT[case["act"]], y=empty(n, h, w, c))
    elif what == "se":
        cr = case["cr"]
        s.update(cr=cr, w1=normal((cr, c), scale=1 / math.sqrt(c)), b1=normal((cr,), scale=0.1), w2=normal((c, cr), scale=1 / math.sqrt(cr)),
                 b2=normal((c,), scale=0.1), pooled=empty(n, c), gate=empty(n, c), y=empty(n, h, w, c))
    elif what == "concat":
        s.update(x2=normal((n, h, w, case["c2"]), dt), y=empty(n, h, w, c + case["c2"]))
        s["ptrs"] = (ctypes.c_void_p * 2)(s["x"].data_ptr(), s["x2"].data_ptr())
        s["channels"] = (ctypes.c_int * 2)(c, case["c2"])
    elif what == "upsample2x":
        s.update(y=empty(n, 2 * h, 2 * w, c))
    return s


def _p(t):
    return None if t is None else t.data_ptr()


def run(s):
    stream = torch.cuda.current_stream().cuda_stream
    L = lib()
    if s["kind"] == "net":
        _load(s["key"])
        if s["host"]:
            rt.forward(s["out"], s["x"])
        else:
            rt.forward_device(s["out"], s["x"], stream)
        return s["out"]
    if s["kind"] == "gemm":
        m, n, k = s["dims"]
        check(L.nncv_b200_matmul(_p(s["a"]), _p(s["b"]), _p(s["c"]), m, n, k, s["ab"], s["cd"], _p(s["bias"]), s["relu"], stream))
        return s["c"]
    n, h, w, c = s["dims"]
    what, dt, x, y = s["op"], s["dtype"], _p(s["x"]), _p(s["y"])
    if what in ("conv3x3", "conv"):
        check(L.nncv_b200_conv_run(s["conv"].h, x, y, n, h, w, _p(s["scale"]), _p(s["shift"]), _p(s["res"]), 1, stream))
    elif what == "depthwise":
        check(L.nncv_b200_depthwise_conv_nhwc(x, _p(s["weights"]), F32, _p(s["scale"]), _p(s["shift"]), y, dt, n, h, w, c, s["k"], s["k"],
                                              s["stride"], s["k"] // 2, s["act"], stream))
    elif what == "maxpool":
        check(L.nncv_b200_maxpool_nhwc(x, y, dt, n, h, w, c, s["k"], s["stride"], s["pad"], stream))
    elif what == "avgpool":
        check(L.nncv_b200_avgpool_nhwc(x, y, dt, n, h * w, c, stream))
    elif what == "activation":
        check(L.nncv_b200_activation(x, y, dt, n * h * w * c, s["act"], stream))
    elif what == "se":
        check(L.nncv_b200_avgpool_nhwc(x, _p(s["pooled"]), dt, n, h * w, c, stream))
        check(L.nncv_b200_se_gate(_p(s["pooled"]), _p(s["w1"]), _p(s["b1"]), _p(s["w2"]), _p(s["b2"]), _p(s["gate"]), dt, n, c, s["cr"], stream))
        check(L.nncv_b200_scale_channels_nhwc(x, _p(s["gate"]), y, dt, n, h * w, c, stream))
        return s["pooled"], s["gate"], s["y"]
    elif what == "concat":
        check(L.nncv_b200_concat_channels_nhwc(s["ptrs"], s["channels"], 2, y, dt, n * h * w, stream))
    elif what == "upsample2x":
        check(L.nncv_b200_upsample2x_nhwc(x, y, dt, n, h, w, c, stream))
    return s["y"]


# --------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far two right answers lie apart
# --------------------------------------------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "net":
        es, n = SIZE[case["params"]], case["batch"]
        return {"bytes": float(es * (n * 3 * case["h"] * case["w"] + n * 1000 + _plan(case["net"])[2])),
                "flops": n * _net_flops(case["net"], case["h"], case["w"])}
    if case["kind"] == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": float(SIZE[case["ab"]] * (m * k + k * n) + SIZE[case["c"]] * m * n), "flops": 2.0 * m * n * k}
    n, h, w, c, es, what = case["n"], case["h"], case["w"], case["c"], SIZE[case["dtype"]], case["op"]
    x = n * h * w * c
    if what in ("conv3x3", "conv"):
        k, r, stride = (c, 3, 1) if what == "conv3x3" else (case["kout"], case["r"], case["stride"])
        pix = n * _out(h, r, stride, r // 2) * _out(w, r, stride, r // 2)
        # a 1x1 filter of stride 2 needs a quarter of the input
        read = x if r >= stride else pix * c
        return {"bytes": float(es * (read + pix * k * (2 if case["residual"] else 1) + k * c * r * r)), "flops": 2.0 * pix * k * c * r * r}
    if what == "depthwise":
        k, y = case["k"], n * _out(h, case["k"], case["stride"], case["k"] // 2) * _out(w, case["k"], case["stride"], case["k"] // 2) * c
        return {"bytes": float(es * (x + y)), "flops": 2.0 * y * k * k}
    if what == "maxpool":
        pad = (case["k"] - 1) // 2
        y = n * _out(h, case["k"], case["stride"], pad) * _out(w, case["k"], case["stride"], pad) * c
        return {"bytes": float(es * (x + y)), "flops": float(y * case["k"] ** 2)}
    y = {"avgpool": n * c, "activation": x, "se": x + 2 * n * c, "upsample2x": 4 * x}.get(what)
    if what == "concat":
        y = n * h * w * (c + case["c2"])
        x = y
    return {"bytes": float(es * (x + y)), "flops": float(x + (4 * n * c * case["cr"] if what == "se" else 0))}


def tolerance(case):
    if case["kind"] == "net":
        # tens of layers, each rounding its map to the compute type: 4e-4 to 1e-3 of the logits in fp16 through a ResNet,
        # 1e-3 to 2e-3 through MobileNetV3's 46 layers, 3e-3 to 5e-3 in bf16; fp32 sums of up to 4608 products a layer
        if case["compute"] == "f32":
            return {"rel": 1e-5}
        return {"rel": 1e-2 if case["compute"] == "bf16" or case["net"] == "mobilenetv3" else 4e-3}
    if case["kind"] == "gemm":
        return {"rel": {"f32": 1e-5, "f16": 1e-3, "bf16": 8e-3}[case["c"]]}
    if case["op"] in ("maxpool", "concat", "upsample2x"):
        return "exact"
    return {"rel": {"f32": 1e-5, "f16": 1e-3, "bf16": 8e-3}[case["dtype"]]}
