"""The tensor-core form of the fp32 convolution (operands as three bf16 numbers) against 64-bit sums: the edges of its tiles and
k chunks, every row form, a batch that takes several image groups, K splits, results it has to recompute, stream capture.

Bound: 2^-21 * sum |x w| + 2^-23 * |ref|.  The product left out is below 2^-30 of a product, a chunk of 64 cuts off four times
(2^-23 of its sum each) and its two sums are rounded once into the fp32 total: together below 2^-21 of sum |x w|.
"""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tpu_mlir_b200 import _lib as L  # noqa: E402

ptr = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731


class Conv:
    def __init__(self, w, b, ih, iw, stride=1, pads=(0, 0, 0, 0), dil=1, relu=False, limit=-1.0):
        oc, ic, kh, kw = w.shape
        self.w, self.b, self.h = w, b, C.c_void_p()
        self.oh = (ih + pads[0] + pads[1] - dil * (kh - 1) - 1) // stride + 1
        self.ow = (iw + pads[2] + pads[3] - dil * (kw - 1) - 1) // stride + 1
        d = L.TopConvDesc(n=1, ic=ic, ih=ih, iw=iw, oc=oc, kh=kh, kw=kw, sh=stride, sw=stride, dh=dil, dw=dil, pht=pads[0], phb=pads[1],
                          pwl=pads[2], pwr=pads[3], groups=1, with_bias=int(b is not None), do_relu=int(relu), relu_limit=limit)
        L.check(L.lib().b200q_top_conv2d_dev_create(C.byref(d), ptr(w), ptr(b), C.byref(self.h)))

    def __call__(self, x):
        y = torch.full((x.shape[0], self.w.shape[0], self.oh, self.ow), float("nan"), device="cuda")
        s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        L.check(L.lib().b200q_top_conv2d_dev_run(self.h, ptr(x), ptr(y), x.shape[0], s))
        return y

    def __del__(self):
        L.lib().b200q_top_conv2d_dev_destroy(C.byref(self.h))


def ref64(x, w, b, stride, pads, dil):
    x = torch.nn.functional.pad(x.double(), (pads[2], pads[3], pads[0], pads[1]))
    return torch.nn.functional.conv2d(x, w.double(), None if b is None else b.double(), stride=stride, dilation=dil)


def draw(seed, n, ic, ih, iw, oc, kh, kw):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = lambda *s: torch.randn(s, device="cuda", generator=g)  # noqa: E731
    return r(n, ic, ih, iw), r(oc, ic, kh, kw) / np.sqrt(ic * kh * kw), r(oc)


CASES = [
    # n, ic, ih, iw, oc, kh, kw, stride, pads (t, b, l, r), dilation
    (1, 32, 1, 1, 32, 1, 1, 1, (0, 0, 0, 0), 1),          # smallest it takes: one row, half a chunk
    (2, 65, 9, 15, 65, 1, 1, 1, (0, 0, 0, 0), 1),         # one channel past a chunk and past a 64-wide tile; 270 rows
    (3, 40, 23, 21, 130, 3, 3, 1, (1, 1, 1, 1), 1),       # taps of a filter row share a block; ragged chunk, two past 128 wide
    (2, 72, 17, 19, 257, 3, 3, 1, (2, 2, 2, 2), 2),       # dilation: shifted rows without sharing; one past 256 wide
    (2, 96, 31, 33, 100, 5, 5, 2, (2, 2, 2, 2), 1),       # stride: a row holds all taps
    (4, 33, 20, 18, 64, 2, 3, 1, (0, 1, 2, 0), 1),        # even filter, uneven padding
    (9, 256, 7, 7, 512, 3, 3, 1, (1, 1, 1, 1), 1),        # long K on few tiles: splits
    (40, 256, 56, 56, 64, 1, 1, 1, (0, 0, 0, 0), 1),      # several groups of images, the last one smaller
    (16, 128, 28, 28, 512, 1, 1, 2, (0, 0, 0, 0), 1),     # strided 1x1
    (12, 64, 56, 56, 256, 3, 3, 1, (1, 1, 1, 1), 1),      # CTA pairs, wide tile
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("relu", [False, True])
def test_against_64_bits(case, relu):
    n, ic, ih, iw, oc, kh, kw, stride, pads, dil = case
    x, w, b = draw(11, n, ic, ih, iw, oc, kh, kw)
    if relu:
        b = None
    got = Conv(w, b, ih, iw, stride, pads, dil, relu, 0.75 if relu else -1.0)(x)
    ref = ref64(x, w, b, stride, pads, dil)
    mag = ref64(x.abs(), w.abs(), None, stride, pads, dil)
    if relu:
        ref = ref.clamp(0, 0.75)
    assert got.shape == ref.shape
    assert bool(((got.double() - ref).abs() <= mag * 2.0**-21 + ref.abs() * 2.0**-23).all())


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("kind", ["small integers", "wide integers", "one-hot", "power of two"])
def test_exact_sums_stay_exact(case, kind):
    """Sums that every order of fp32 additions gives exactly: integers whose partial sums stay below 2^24 (in 16 bits or more, so
    that all three parts take part), one filter value per channel (the input itself, or shifted by a power of two)."""
    n, ic, ih, iw, oc, kh, kw, stride, pads, dil = case
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    ints = lambda lim, *s: torch.randint(-lim, lim + 1, s, device="cuda", generator=g).float()  # noqa: E731
    b = ints(1000, oc)
    if kind == "small integers":
        x, w = ints(9, n, ic, ih, iw), ints(9, oc, ic, kh, kw)
    elif kind == "wide integers":       # at most four products of 21 bits and a bias
        x, w = ints(2**20, n, ic, ih, iw), torch.zeros((oc, ic, kh, kw), device="cuda")
        for _ in range(4):
            w[torch.arange(oc), torch.randint(ic, (oc,)), torch.randint(kh, (oc,)), torch.randint(kw, (oc,))] = float(1 - 2 * (_ & 1))
    else:
        x, w = torch.randn((n, ic, ih, iw), device="cuda", generator=g), torch.zeros((oc, ic, kh, kw), device="cuda")
        w[torch.arange(oc), torch.randint(ic, (oc,)), torch.randint(kh, (oc,)), torch.randint(kw, (oc,))] = 1.0 if kind == "one-hot" else 2.0**-7
        b = None
        x.view(-1)[0] = 3.4028234663852886e38       # its 6-bit part is infinite
    got = Conv(w, b, ih, iw, stride, pads, dil)(x)
    assert torch.equal(got.double(), ref64(x, w, b, stride, pads, dil))


def test_systematic_error_is_small():
    """The tensor core cuts off; that must not show in the mean (53 layers would add it up): 4e-9 measured."""
    x, w, _ = draw(5, 8, 256, 14, 14, 256, 3, 3)
    x.clamp_(min=0)
    b = torch.full((256,), 0.01, device="cuda")
    ref = ref64(x, w, b, 1, (1, 1, 1, 1), 1)
    e = Conv(w, b, 14, 14, 1, (1, 1, 1, 1))(x).double() - ref
    assert abs(float((e * ref.sign()).mean() / ref.abs().mean())) < 1.5e-8
    assert float(e.norm() / ref.norm()) < 2.2e-7            # a serial chain of fp32 FMAs: 2.2e-7 to 2.5e-7


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.0e38, 1e-30])
def test_values_outside_the_split(value):
    """Infinities, NaN, values whose bf16 is infinite and values whose low parts underflow give what fp32 FMAs give."""
    x, w, b = draw(3, 2, 64, 9, 9, 96, 3, 3)
    if value == 1e-30:
        x, b = x * 1e-30, b * 0
    else:
        x[1, 7, 4, 4] = value
        w[5] = 0
    got = Conv(w, b, 9, 9, 1, (1, 1, 1, 1))(x)
    ref = ref64(x, w, b, 1, (1, 1, 1, 1), 1).float()
    fin = torch.isfinite(ref)
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(got[torch.isinf(ref)], ref[torch.isinf(ref)])
    mag = ref64(torch.nan_to_num(x, 0, 0, 0).abs(), w.abs(), None, 1, (1, 1, 1, 1), 1)
    assert bool(((got - ref).abs()[fin] <= (mag * 2.0**-20)[fin] + ref.abs()[fin] * 2.0**-23).all())


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("stride", [1, 2])
def test_weights_that_are_not_finite_meet_the_border(value, stride):
    """The border counts as zeros: an infinite weight on it gives NaN, as it does in a sum over the padded image."""
    x, w, b = draw(3, 2, 64, 9, 9, 96, 3, 3)
    w[5, 3, 0, 2] = value
    got = Conv(w, b, 9, 9, stride, (1, 1, 1, 1))(x)
    ref = ref64(x, w, b, stride, (1, 1, 1, 1), 1).float()
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(got[torch.isinf(ref)], ref[torch.isinf(ref)])
    assert bool(torch.isnan(ref[:, 5, 0]).all())


@pytest.mark.parametrize("case", [CASES[i] for i in (0, 2, 4, 6, 9)])
@pytest.mark.parametrize("xs,ws", [(1e-36, 1e20), (1e-41, 1e20), (1e20, 1e-36), (1e-20, 1e-22), (1e-30, 1.0), (1.0, 1e-38)])
@pytest.mark.parametrize("part", [False, True])
def test_operands_near_underflow(case, xs, ws, part):
    """Small operands whose low parts underflow although the results do not, results that are subnormal, zeros that underflow made;
    everywhere, or in one image row and one channel only.  Beyond the bound of normal values, a product of fp32 FMAs is rounded to
    multiples of 2^-149, twice that allowed here."""
    n, ic, ih, iw, oc, kh, kw, stride, pads, dil = case
    x, w, _ = draw(13, n, ic, ih, iw, oc, kh, kw)
    if part:
        x[0, :, ih // 2] *= xs
        w[oc // 3] *= ws
    else:
        x, w = x * xs, w * ws
    got = Conv(w, None, ih, iw, stride, pads, dil)(x)
    ref = ref64(x, w, None, stride, pads, dil)
    mag = ref64(x.abs(), w.abs(), None, stride, pads, dil)
    assert bool(((got.double() - ref).abs() <= mag * 2.0**-21 + ref.abs() * 2.0**-23 + ic * kh * kw * 2.0**-148).all())


def test_time_does_not_hang_on_the_values():
    """Dead channels (weights near zero, biases that swallow what they give) cost nothing, an infinity or a tensor of NaN a bounded
    number of recomputed sums.  (Without the bias in the decision: 15 times; one sum after the other: 400 times.)"""
    x, w, b = draw(2, 32, 256, 14, 14, 256, 3, 3)

    def time_of(x, w):
        conv = Conv(w, b, 14, 14, 1, (1, 1, 1, 1))
        conv(x)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(8)]
        for e in ev:
            e.record()
            conv(x)
        torch.cuda.synchronize()
        return min(a.elapsed_time(z) for a, z in zip(ev, ev[1:]))
    plain = time_of(x, w)
    for scale in (1e-20, 1e-38):
        dead = w.clone()
        dead[::32] *= scale
        assert time_of(x, dead) < 3 * plain
    one = x.clone()
    one[0, 0, 5, 5] = float("inf")
    assert time_of(one, w) < 100 * plain
    assert time_of(x * float("nan"), w) < 100 * plain


def test_capture_and_two_streams():
    x, w, b = draw(9, 6, 64, 28, 28, 128, 3, 3)
    conv = Conv(w, b, 28, 28, 1, (1, 1, 1, 1))
    want = conv(x)
    x2 = x * 0.5
    want2 = conv(x2)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        captured = conv(x)
    for _ in range(3):
        captured.zero_()
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, want)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [[], []]
    for _ in range(10):                                    # one handle, two streams: each call has its own scratch
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                outs[i].append(conv(x if i == 0 else x2))
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs[0]) and all(torch.equal(o, want2) for o in outs[1])


@pytest.mark.parametrize("case", [CASES[i] for i in (0, 4, 6, 9)])       # 64 wide, strided, split, pair
def test_a_wait_that_runs_out_is_reported(case):
    """Failure detection without a fault: every stage's barrier is told to expect 16 bytes more than the loads deliver, so a bounded
    wait runs out after 1 ms.  With a split and a ReLU the lost sums end as zeros: only the status tells."""
    n, ic, ih, iw, oc, kh, kw, stride, pads, dil = case
    x, w, b = draw(1, n, ic, ih, iw, oc, kh, kw)
    conv = Conv(w, b, ih, iw, stride, pads, dil, True)
    want, lib = conv(x), L.lib()
    assert lib.b200q_top_conv2d_dev_status(conv.h, None) == L.OK
    lib.b200q_debug_set_wait_fault(16, 1_000_000)
    try:
        conv(x)
        rc = lib.b200q_top_conv2d_dev_status(conv.h, None)
    finally:
        lib.b200q_debug_set_wait_fault(0, 0)
    assert rc == L.ERR_TIMEOUT
    assert torch.equal(conv(x), want) and lib.b200q_top_conv2d_dev_status(conv.h, None) == L.OK


def test_executor_and_calibration_report_it():
    from tpu_mlir_b200.module import module
    from tpu_mlir_b200.run_calibration import run_calibration
    rng = np.random.default_rng(0)
    shape = dict(shape=[2, 32, 12, 12], dtype="f32")
    conv = dict(kernel_shape=[3, 3], pads=[1, 1, 1, 1], do_relu=True)
    graph = dict(inputs=["x"], outputs=["c2"], tensors=dict(x=shape, c1=shape, c2=shape), state="TOP_F32",
                 ops=[dict(type="top.Conv", name="c1", inputs=["x"], attrs=conv), dict(type="top.Conv", name="c2", inputs=["c1"], attrs=conv)])
    weights = {f"{c}_{k}": rng.standard_normal(s).astype(np.float32) for c in ("c1", "c2") for k, s in (("filter", (32, 32, 3, 3)), ("bias", (32,)))}
    samples = rng.standard_normal((4, 32, 12, 12)).astype(np.float32)
    m, lib = module(), L.lib()
    m.load(graph, weights)
    m.set_tensor("x", samples[:2])
    lib.b200q_debug_set_wait_fault(16, 1_000_000)
    try:
        m.invoke()
        with pytest.raises(L.B200QError) as e:
            m.check_status()
        assert e.value.code == L.ERR_TIMEOUT
        with pytest.raises(L.B200QError):
            run_calibration(graph, weights, samples)
    finally:
        lib.b200q_debug_set_wait_fault(0, 0)
    m.invoke()
    m.check_status()
    assert len(run_calibration(graph, weights, samples)) == 3
