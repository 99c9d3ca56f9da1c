"""The work this framework is used for, as cases that can be timed one by one.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (inputs from the seed, handles,
weights), ``run`` is one pass through the public entry points, ``work`` the bytes and operations such a pass cannot do
without and ``tolerance`` how far another correct implementation may be off.  Seven kinds of work:

  resnet50     INT8 ResNet-50 through the graph executor (``module``), images on the device, logits out
  a16          one 4-bit-weight A16MatMul of a decoder's MLP through a device handle, decode to prefill
  matmul       tpu.MatMul INT8 on device tensors
  conv         tpu.Conv2D INT8 on device tensors, dense and depthwise, NCHW and channels-last
  operator     the interpreter's operator face: tpu.Conv2D / tpu.MatMul on host float buffers
  calibration  per-sample min / max, streaming histograms and KLD thresholds of a network's activations
  forward      the fp32 Top-dialect forward that calibration runs, through the graph executor
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

import tpu_mlir_b200._lib as L
from tpu_mlir_b200 import resnet50
from tpu_mlir_b200.calibration import CaliMathB200, ShardedCalibrator
from tpu_mlir_b200.module import module
from tpu_mlir_b200.ops import Conv2DOp, InferenceParameter, MatMulOp

DEV = "cuda"


def listed():
    return [
        # one image at a time: a camera or an interactive service, 75 small kernels whose latency is the whole cost
        dict(name="resnet50_b1", kind="resnet50", batch=1, channels_last=True, cuda_graph=True),
        # a ragged batch through the executor as it comes (NCHW tensors, op by op), the way the reference's tools drive it
        dict(name="resnet50_b23_default", kind="resnet50", batch=23, channels_last=False, cuda_graph=False),
        # the throughput configuration: accuracy evaluation over a data set, large-batch serving
        dict(name="resnet50_b256", kind="resnet50", batch=256, channels_last=True, cuda_graph=True),
        # token-by-token decoding of one sequence, the up projection of a 7B decoder's MLP
        dict(name="a16_decode_m1", kind="a16", M=1, N=11008, K=4096, group=64, f16=False),
        # a few dozen sequences decoded together (or a short prompt), f16 activations
        dict(name="a16_batch_m37_f16", kind="a16", M=37, N=11008, K=4096, group=64, f16=True),
        # prompt processing
        dict(name="a16_prefill_m2048", kind="a16", M=2048, N=11008, K=4096, group=64, f16=False),
        # a fully connected layer of ordinary size
        dict(name="matmul_512x1024x1024", kind="matmul", M=512, N=1024, K=1024, qdm=True, unsigned=False, relu=False),
        # a large convolution layer, the drop-in NCHW face
        dict(name="conv3x3_n32c256", kind="conv", n=32, c=256, h=56, w=56, oc=256, k=3, stride=1, depthwise=False, nhwc=False,
             qdm=True, unsigned=False),
        # a strided layer of a network that was not designed around multiples of 64, odd image sizes
        dict(name="conv3x3s2_ragged", kind="conv", n=3, c=72, h=57, w=61, oc=100, k=3, stride=2, depthwise=False, nhwc=False,
             qdm=False, unsigned=True),
        # the operator behind the unchanged CPU interpreter: float buffers on the host in and out
        dict(name="operator_conv_n8c256", kind="operator", op="conv", n=8, c=256, h=56, w=56, oc=256, k=3),
        # calibration statistics of ResNet-50's 73 activations over a few batches of samples
        dict(name="calibration_resnet50_s64", kind="calibration", samples=64, batch=16, tensors=73, scale=1.0),
        # the float forward behind calibration and threshold tuning
        dict(name="forward_resnet50_b32", kind="forward", batch=32),
    ]


# ------------------------------------------------------------------------------------------------ drawn cases
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["resnet50", "a16", "a16", "matmul", "conv", "conv", "operator", "calibration", "forward"])
    if kind == "resnet50":
        served = rng.random() < 0.7      # tuned options, else the defaults
        return dict(kind=kind, batch=_log(rng, 1, 256 if served else 64), channels_last=served, cuda_graph=served)
    if kind == "a16":
        N, K = rng.choice([(11008, 4096), (4096, 11008), (4096, 4096), (_log(rng, 2048, 16384), 256 * rng.randint(4, 48))])
        return dict(kind=kind, M=_log(rng, 1, 2048), N=N, K=K, group=rng.choice([64, 64, 128, 256]), f16=rng.random() < 0.3)
    if kind == "matmul":
        K = 16 * _log(rng, 8, 512) if rng.random() < 0.75 else _log(rng, 100, 4096)
        M, N = _log(rng, 1, 8192), _log(rng, 64, 8192)
        if K % 16:                      # rows that are not a multiple of 16 bytes: small classifier-like layers
            M, N = min(M, 512), min(N, 4096)
        return dict(kind=kind, M=M, N=N, K=K, qdm=rng.random() < 0.5, unsigned=rng.random() < 0.3, relu=rng.random() < 0.5)
    if kind == "conv":
        dw = rng.random() < 0.25
        hw = _log(rng, 7, 112)
        n = _log(rng, 1, 64)
        k = rng.choice([3, 3, 5]) if dw else rng.choice([1, 3, 3, 5])
        nhwc = not dw and rng.random() < 0.4
        c = 16 * _log(rng, 1, 32) if nhwc or rng.random() < 0.5 else _log(rng, 3, 512)
        oc = c if dw else (16 * _log(rng, 1, 32) if nhwc or rng.random() < 0.5 else _log(rng, 16, 512))
        stride = rng.choice([1, 1, 2])
        while n > 1 and (n * c * oc * hw * hw * k * k > (20e9 if not dw else 1e18) or n * max(c, oc) * hw * hw > 26e6):
            n = (n + 1) // 2
        return dict(kind=kind, n=n, c=c, h=hw, w=hw + rng.choice([0, 0, 1, 3]), oc=oc, k=k, stride=stride, depthwise=dw,
                    nhwc=nhwc, qdm=rng.random() < 0.5, unsigned=rng.random() < 0.5)
    if kind == "operator":
        if rng.random() < 0.4:
            return dict(kind=kind, op="matmul", M=_log(rng, 1, 2048), N=_log(rng, 256, 4096), K=16 * _log(rng, 16, 256))
        hw, c, n = _log(rng, 7, 56), 16 * _log(rng, 1, 32), _log(rng, 1, 32)
        oc = 16 * _log(rng, 1, 32)
        while n > 1 and n * max(c, oc) * hw * hw > 8e6:
            n = (n + 1) // 2
        return dict(kind=kind, op="conv", n=n, c=c, h=hw, w=hw, oc=oc, k=rng.choice([1, 3]))
    if kind == "calibration":
        samples = _log(rng, 2, 64)
        return dict(kind=kind, samples=samples, batch=rng.randint(1, samples), tensors=rng.randint(3, 73),
                    scale=round(rng.uniform(0.3, 8.0), 3))
    return dict(kind="forward", batch=_log(rng, 1, 32))


# ------------------------------------------------------------------------------------------------ shared pieces
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _p(t):
    return C.c_void_p(t.data_ptr())


class _Handle:
    """A device handle of the library, destroyed with its owner."""

    def __init__(self, destroy):
        self.h, self.destroy = C.c_void_p(), destroy

    def __del__(self):
        try:
            if self.h:
                self.destroy(C.byref(self.h))
        except Exception:
            pass


@functools.lru_cache(maxsize=None)
def _network():
    """Random-init ResNet-50 (fused fp32 ops) and its multiply-accumulates per image and weight count."""
    ops = resnet50.build_fp32(seed=3)
    graph, _ = resnet50.top_graph(ops, 1)
    macs = wts = 0
    for op in ops:
        if op["type"] in ("conv", "fc"):
            shape = graph["tensors"][op["name"]]["shape"]
            macs += int(np.prod(shape)) * int(np.prod(op["w"].shape[1:] if op["type"] == "conv" else op["w"].shape[:1]))
            wts += op["w"].size
    return ops, macs, wts


@functools.lru_cache(maxsize=None)
def _table():
    """Max-calibrated thresholds from two images through torch's CPU operators, to three digits: the quantised network does
    not depend on the last bits of any float kernel."""
    ops, _, _ = _network()
    x = torch.from_numpy(np.random.default_rng(7).standard_normal((2, 3, 224, 224), dtype=np.float32))
    table = {}
    for name, a in resnet50.fp32_forward_torch(ops, x).items():
        table[name] = (float("%.2e" % float(a.abs().max())), float("%.2e" % float(a.min())), float("%.2e" % float(a.max())))
    return table


@functools.lru_cache(maxsize=None)
def _int8_network():
    return resnet50.lower_int8(_network()[0], _table(), 1)


def _int8_graph(batch):
    """The lowered network at this batch size: only the tensors' first dimension depends on it."""
    graph, weights = _int8_network()
    tensors = {n: dict(t, shape=[batch] + list(t["shape"][1:])) for n, t in graph["tensors"].items()}
    return dict(graph, tensors=tensors), weights


def _shift_for(acc_std, multiplier):
    """A right shift that brings an accumulator of this spread to about the int8 range."""
    return max(1, int(round(math.log2(multiplier * acc_std * 3.0 / 127.0))))


def _requant(rng, channels, K, qdm, unsigned):
    """Multipliers and right shifts of one layer: the QDM form, or MultiplierShift as the lowering emits it."""
    if qdm:
        return rng.integers(2**30, 2**31, channels, dtype=np.int64), rng.integers(8, 21, channels, dtype=np.int64)
    acc = math.sqrt(K) * (147.0 if unsigned else 74.0) * 32.0
    mult = rng.integers(8000, 30000, channels, dtype=np.int64)
    return mult, np.array([_shift_for(acc, int(m)) for m in mult], dtype=np.int64)


def _out_hw(case):
    pad = case["k"] // 2
    s = case.get("stride", 1)
    return (case["h"] + 2 * pad - case["k"]) // s + 1, (case["w"] + 2 * pad - case["k"]) // s + 1


# ------------------------------------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed))


def run(state):
    return state["run"](state)


def _prepare_resnet50(case, seed):
    graph, weights = _int8_graph(case["batch"])
    m = module(channels_last=case["channels_last"], cuda_graph=case["cuda_graph"])
    m.load(graph, weights)
    x = torch.randn((case["batch"], 3, 224, 224), device=DEV, generator=_gen(seed))
    return dict(run=_run_graph, m=m, x=x)


def _prepare_forward(case, seed):
    graph, weights = resnet50.top_graph(_network()[0], case["batch"])
    m = module()
    m.load(graph, weights)
    x = torch.randn((case["batch"], 3, 224, 224), device=DEV, generator=_gen(seed))
    return dict(run=_run_graph, m=m, x=x)


def _run_graph(s):
    m = s["m"]
    m.set_tensor("input", s["x"])
    m.invoke()
    return m.tensors[m.output_names[0]]


def _prepare_a16(case, seed):
    M, N, K, g = case["M"], case["N"], case["K"], case["group"]
    gen = _gen(seed)
    dt = torch.float16 if case["f16"] else torch.bfloat16
    wq = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, device=DEV, generator=gen)
    sc = (torch.rand(N * K // g, device=DEV, generator=gen) * 0.019 + 0.001).to(dt)
    zp = torch.randint(0, 16, (N * K // g,), dtype=torch.uint8, device=DEV, generator=gen)
    x = torch.randn((M, K), device=DEV, generator=gen).to(dt)
    y = torch.empty((M, N), dtype=dt, device=DEV)
    lib = L.lib()
    h = _Handle(lib.b200q_a16_dev_destroy)
    L.check(lib.b200q_a16_dev_create_dt(_p(wq), _p(sc), _p(zp), None, N, K, g, L.DT_F16 if case["f16"] else L.DT_BF16, C.byref(h.h)))
    return dict(run=_run_a16, call=lib.b200q_a16_dev_run, h=h, M=M, xp=_p(x), yp=_p(y), y=y, keep=(wq, sc, zp, x))


def _run_a16(s):
    rc = s["call"](s["h"].h, s["xp"], s["yp"], s["M"], None)
    if rc:
        L.check(rc)
    return s["y"]


def _prepare_matmul(case, seed):
    M, N, K = case["M"], case["N"], case["K"]
    gen, rng = _gen(seed), np.random.default_rng(seed)
    if case["unsigned"]:
        a = torch.randint(0, 256, (M, K), dtype=torch.uint8, device=DEV, generator=gen)
    else:
        a = torch.randint(-128, 128, (M, K), dtype=torch.int8, device=DEV, generator=gen)
    b = torch.clamp(torch.round(torch.randn((N, K), device=DEV, generator=gen) * 32), -127, 127).to(torch.int8)
    bias = torch.randint(-2**16, 2**16, (N,), dtype=torch.int32, device=DEV, generator=gen)
    mult, rs = _requant(rng, N if case["qdm"] else 1, K, case["qdm"], case["unsigned"])
    mult_d = torch.from_numpy(mult.astype(np.int32)).to(DEV)
    shift_d = torch.from_numpy((-rs if case["qdm"] else rs).astype(np.int32)).to(DEV)
    out = torch.empty((M, N), dtype=torch.int8, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    e = L.Epilogue(dialect=L.RQ_QDM if case["qdm"] else L.RQ_MULTIPLIER_SHIFT,
                   round_mode=L.ROUND_HALF_AWAY_FROM_ZERO if case["qdm"] else L.ROUND_HALF_UP, per_channel=int(case["qdm"]),
                   out_zp=0, relu=L.RELU_BEFORE_REQUANT if case["relu"] else L.RELU_NONE, out_dtype=L.DT_I8, scale=0.0,
                   bias=bias.data_ptr(), multiplier=mult_d.data_ptr(), shift=shift_d.data_ptr())
    args = (_p(a), L.DT_U8 if case["unsigned"] else L.DT_I8, _p(b), L.DT_I8, M, N, K, C.byref(e), _p(out), _p(status), L.ALGO_AUTO, None)
    return dict(run=_run_matmul, call=L.lib().b200q_gemm_i8_dev, args=args, out=out, keep=(a, b, bias, mult_d, shift_d, status, e))


def _run_matmul(s):
    rc = s["call"](*s["args"])
    if rc:
        L.check(rc)
    return s["out"]


def _conv_op(case, rng):
    c, oc, k = case["c"], case["oc"], case["k"]
    dw = case.get("depthwise", False)
    kk = k * k * (1 if dw else c)
    mult, rs = _requant(rng, oc, kk, case.get("qdm", False), case.get("unsigned", False))
    if dw and case.get("qdm", False):
        rs = rs - 6                     # nine products instead of thousands: smaller accumulators
    pad = k // 2
    return Conv2DOp(input_shape=(case["n"], c, case["h"], case["w"]), oc=oc, kernel_shape=(k, k),
                    strides=(case.get("stride", 1),) * 2, pads=(pad,) * 4, group=c if dw else 1, do_relu=True,
                    input_dtype=L.DT_U8 if case.get("unsigned", False) else L.DT_I8,
                    out_dtype=L.DT_I8 if case.get("qdm", False) else L.DT_U8,
                    quant_mode=L.QM_QDM if case.get("qdm", False) else L.QM_MULTIPLIER_SHIFT, is_cv18xx=case.get("qdm", False),
                    multiplier=mult, rshift=rs)


def _prepare_conv(case, seed):
    gen, rng = _gen(seed), np.random.default_rng(seed)
    n, c, h, w, oc, k = (case[v] for v in ("n", "c", "h", "w", "oc", "k"))
    op = _conv_op(case, rng)
    shape = (n, h, w, c) if case["nhwc"] else (n, c, h, w)
    if case["unsigned"]:
        x = torch.randint(0, 256, shape, dtype=torch.uint8, device=DEV, generator=gen)
    else:
        x = torch.randint(-128, 128, shape, dtype=torch.int8, device=DEV, generator=gen)
    wt = torch.clamp(torch.round(torch.randn((oc, 1 if case["depthwise"] else c, k, k), device=DEV, generator=gen) * 32), -127, 127).to(torch.int8)
    bias = torch.randint(-2**12, 2**12, (oc,), dtype=torch.int32, device=DEV, generator=gen)
    oh, ow = op.out_shape[2:]
    y = torch.empty((n, oh, ow, oc) if case["nhwc"] else (n, oc, oh, ow), dtype=torch.int8 if case["qdm"] else torch.uint8, device=DEV)
    lib = L.lib()
    hd = _Handle(lib.b200q_conv2d_dev_destroy)
    L.check(lib.b200q_conv2d_dev_create(C.byref(op.desc), _p(wt), _p(bias), C.byref(hd.h)))
    layout = L.LAYOUT_NHWC if case["nhwc"] else L.LAYOUT_NCHW
    return dict(run=_run_conv, nhwc=case["nhwc"], lib=lib, h=hd, xp=_p(x), yp=_p(y), layout=layout, y=y, keep=(x, wt, bias, op))


def _run_conv(s):
    if s["nhwc"]:
        rc = s["lib"].b200q_conv2d_dev_run_layout(s["h"].h, s["xp"], s["layout"], s["yp"], s["layout"], None)
    else:
        rc = s["lib"].b200q_conv2d_dev_run(s["h"].h, s["xp"], s["yp"], None)
    if rc:
        L.check(rc)
    return s["y"]


def _prepare_operator(case, seed):
    rng = np.random.default_rng(seed)
    if case["op"] == "matmul":
        M, N, K = case["M"], case["N"], case["K"]
        a = rng.integers(-128, 128, (M, K), dtype=np.int8).astype(np.float32)
        b = rng.integers(-64, 65, (K, N), dtype=np.int8).astype(np.float32)
        bias = rng.integers(-2**12, 2**12, N).astype(np.float32)
        mult = 16384
        op = MatMulOp(M=M, K=K, N=N, with_bias=True, do_relu=True, quant_mode=L.QM_MULTIPLIER_SHIFT, multipliers=[mult],
                      rshifts=[_shift_for(math.sqrt(K) * 74.0 * 37.0, mult)])
        p = InferenceParameter(inputs=[a, b, bias, None, None], outputs=[np.zeros((M, N), np.float32)])
    else:
        n, c, h, w, oc, k = (case[v] for v in ("n", "c", "h", "w", "oc", "k"))
        op = _conv_op(case, rng)
        x = rng.integers(-128, 128, (n, c, h, w), dtype=np.int8).astype(np.float32)
        wt = rng.integers(-64, 65, (oc, c, k, k), dtype=np.int8).astype(np.float32)
        bias = rng.integers(-2**12, 2**12, oc).astype(np.float32)
        p = InferenceParameter(inputs=[x, wt, bias], outputs=[np.zeros(op.out_shape, np.float32)])
    op.init(p)
    return dict(run=_run_operator, op=op, p=p, done=_Deinit(op, p))


class _Deinit:
    def __init__(self, op, p):
        self.op, self.p = op, p

    def __del__(self):
        try:
            self.op.deinit(self.p)
        except Exception:
            pass


def _run_operator(s):
    s["op"].inference(s["p"])
    return s["p"].outputs[0]


def _calibration_shapes(case):
    """The first `tensors` activations of ResNet-50 (input included): name -> shape of one sample."""
    return {n: tuple(s) for n, s in list(_top_shapes().items())[:case["tensors"]]}


@functools.lru_cache(maxsize=None)
def _top_shapes():
    ops = _network()[0]
    graph, _ = resnet50.top_graph(ops, 1)
    return {n: t["shape"][1:] for n, t in graph["tensors"].items()}


def _prepare_calibration(case, seed):
    gen = _gen(seed)
    S = case["samples"]
    acts = {}
    for i, (name, shape) in enumerate(_calibration_shapes(case).items()):
        a = torch.randn((S,) + shape, device=DEV, generator=gen)
        a *= case["scale"] * (0.5 + 0.1 * (i % 13))
        if i % 4 != 0:                  # most activations come out of a ReLU
            a.clamp_(min=0)
        acts[name] = a
    batches = [(lo, min(lo + case["batch"], S)) for lo in range(0, S, case["batch"])]
    return dict(run=_run_calibration, acts=acts, batches=batches, samples=S, math=CaliMathB200())


def _run_calibration(s):
    acts = s["acts"]
    cal = ShardedCalibrator(lambda b: {n: a[b[0]:b[1]] for n, a in acts.items()}, math=s["math"])
    res = cal.run(s["batches"], s["samples"])
    return np.array([[r.min, r.max, r.abs_max, r.bins, r.width, r.kl, r.threshold] for r in res.values()], dtype=np.float64)


_PREPARE = dict(resnet50=_prepare_resnet50, a16=_prepare_a16, matmul=_prepare_matmul, conv=_prepare_conv,
                operator=_prepare_operator, calibration=_prepare_calibration, forward=_prepare_forward)


# ------------------------------------------------------------------------------------------------ work / tolerance
def work(case):
    kind = case["kind"]
    if kind in ("resnet50", "forward"):
        _, macs, wts = _network()
        eb = 1 if kind == "resnet50" else 4
        return dict(bytes=case["batch"] * (3 * 224 * 224 * 4 + 1000 * 4) + wts * eb, flops=2.0 * macs * case["batch"])
    if kind == "a16":
        M, N, K = case["M"], case["N"], case["K"]
        return dict(bytes=N * K // 2 + N * K // case["group"] * 3 + 2 * M * (N + K), flops=2.0 * M * N * K)
    if kind == "matmul":
        M, N, K = case["M"], case["N"], case["K"]
        return dict(bytes=M * K + N * K + M * N + 4 * N, flops=2.0 * M * N * K)
    if kind == "conv":
        oh, ow = _out_hw(case)
        cin = 1 if case["depthwise"] else case["c"]
        out = case["n"] * case["oc"] * oh * ow
        return dict(bytes=case["n"] * case["c"] * case["h"] * case["w"] + out + case["oc"] * cin * case["k"]**2,
                    flops=2.0 * out * cin * case["k"]**2)
    if kind == "operator":
        if case["op"] == "matmul":
            M, N, K = case["M"], case["N"], case["K"]
            return dict(bytes=4 * (M * K + M * N), flops=2.0 * M * N * K)
        oh, ow = _out_hw(case)
        out = case["n"] * case["oc"] * oh * ow
        return dict(bytes=4 * (case["n"] * case["c"] * case["h"] * case["w"] + out), flops=2.0 * out * case["c"] * case["k"]**2)
    elems = sum(int(np.prod(s)) for s in _calibration_shapes(case).values())
    # the histogram's bins follow from the extrema of all samples: two passes over the activations
    return dict(bytes=2 * 4 * elems * case["samples"], flops=0)


def tolerance(case):
    if case["kind"] == "a16":
        # 16-bit outputs of fp32 sums; the prefill form multiplies with the dequantised weight rounded to 16 bits
        return dict(rel=1e-2)
    if case["kind"] == "forward":
        return dict(rel=1e-5)           # fp32 sums of up to 4608 products, 53 layers deep
    return "exact"                      # integers; calibration's statistics are exact counts and their argmin
