"""INT8 products whose tiles are made narrower because they leave SMs idle: both sides of the line, ragged last tiles, and the
channels-last (per-row parameter) form at pixel counts around its tile widths, against the CUDA-core kernels bit for bit."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tpu_mlir_b200 import _lib as L  # noqa: E402
from tpu_mlir_b200.ops import Conv2DOp  # noqa: E402

ptr = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731


@pytest.mark.parametrize("M,N", [(1, 65), (128, 129), (130, 257), (513, 1000), (3072, 512), (3073, 512), (4736, 512), (4737, 512), (2368, 1024), (2369, 1025)])
@pytest.mark.parametrize("qdm", [False, True])
def test_matmul(M, N, qdm):
    K = 144
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N)
    a = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=g)
    b = torch.randint(-128, 128, (N, K), dtype=torch.int8, device="cuda", generator=g)
    bias = torch.randint(-2**12, 2**12, (N,), dtype=torch.int32, device="cuda", generator=g)
    rng = np.random.default_rng(1)
    mult = torch.from_numpy(rng.integers(2**30, 2**31, N).astype(np.int32) if qdm else rng.integers(8000, 30000, 1).astype(np.int32)).cuda()
    shift = torch.from_numpy(-rng.integers(7, 11, N).astype(np.int32) if qdm else np.array([23], np.int32)).cuda()
    e = L.Epilogue(dialect=L.RQ_QDM if qdm else L.RQ_MULTIPLIER_SHIFT, round_mode=L.ROUND_HALF_AWAY_FROM_ZERO if qdm else L.ROUND_HALF_UP,
                   per_channel=int(qdm), out_zp=0, relu=L.RELU_NONE, out_dtype=L.DT_I8, scale=0.0, bias=bias.data_ptr(),
                   multiplier=mult.data_ptr(), shift=shift.data_ptr())
    outs = []
    for algo in (L.ALGO_TENSOR_CORE, L.ALGO_CUDA_CORE):
        out = torch.full((M, N), 77, dtype=torch.int8, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        L.check(L.lib().b200q_gemm_i8_dev(ptr(a), L.DT_I8, ptr(b), L.DT_I8, M, N, K, C.byref(e), ptr(out), ptr(status), algo, None))
        torch.cuda.synchronize()
        assert int(status) == 0
        outs.append(out)
    assert torch.equal(*outs) and outs[0].float().std() > 10


@pytest.mark.parametrize("n,h,w", [(1, 1, 129), (1, 8, 24), (1, 5, 39), (1, 14, 14), (3, 19, 21), (2, 56, 56)])
@pytest.mark.parametrize("oc", [128, 384])
@pytest.mark.parametrize("qdm", [False, True])
def test_channels_last_conv(n, h, w, oc, qdm):
    c = 48
    rng = np.random.default_rng(n * h + oc)
    mult, rs = (rng.integers(2**30, 2**31, oc), rng.integers(6, 10, oc)) if qdm else (rng.integers(8000, 30000, oc), np.full(oc, 22))
    x = torch.from_numpy(rng.integers(-128, 128, (n, c, h, w), dtype=np.int8)).cuda()
    wt = torch.from_numpy(rng.integers(-128, 128, (oc, c, 1, 1), dtype=np.int8)).cuda()
    bias = torch.from_numpy(rng.integers(-2**12, 2**12, oc).astype(np.int32)).cuda()
    outs = []
    for algo, nhwc in ((L.ALGO_TENSOR_CORE, True), (L.ALGO_CUDA_CORE, False)):
        op = Conv2DOp(input_shape=(n, c, h, w), oc=oc, kernel_shape=(1, 1), strides=(1, 1), pads=(0, 0, 0, 0), do_relu=True,
                      input_dtype=L.DT_I8, out_dtype=L.DT_I8 if qdm else L.DT_U8, quant_mode=L.QM_QDM if qdm else L.QM_MULTIPLIER_SHIFT,
                      is_cv18xx=qdm, multiplier=mult.astype(np.int64), rshift=rs.astype(np.int64), algo=algo)
        hd = C.c_void_p()
        L.check(L.lib().b200q_conv2d_dev_create(C.byref(op.desc), ptr(wt), ptr(bias), C.byref(hd)))
        xi = x.permute(0, 2, 3, 1).contiguous() if nhwc else x
        y = torch.full((n, h, w, oc) if nhwc else (n, oc, h, w), 77, dtype=torch.uint8, device="cuda")
        layout = L.LAYOUT_NHWC if nhwc else L.LAYOUT_NCHW
        L.check(L.lib().b200q_conv2d_dev_run_layout(hd, ptr(xi), layout, ptr(y), layout, None))
        torch.cuda.synchronize()
        L.lib().b200q_conv2d_dev_destroy(C.byref(hd))
        outs.append(y.permute(0, 3, 1, 2) if nhwc else y)
    assert torch.equal(outs[0].contiguous(), outs[1]) and outs[1].float().std() > 10


@pytest.mark.parametrize("M,N", [(64, 4096), (128, 12544), (128, 12545), (100, 6145), (129, 6144), (129, 6400), (257, 300)])
@pytest.mark.parametrize("f16", [False, True])
def test_a16_prompts(M, N, f16):
    """The 16-bit products of a 4-bit-weight handle in tiles of every width.  Integer activations and power-of-two scales: every sum
    is exact in fp32, so the outputs are the reference's rounding bit for bit."""
    import oracle
    K, g = 192, 64
    rng = np.random.default_rng(M + N)
    q = rng.integers(0, 16, size=(N, K), dtype=np.uint8)
    wq = (q[:, 0::2] | (q[:, 1::2] << 4)).astype(np.uint8)
    sc = (2.0**-9 * rng.choice([1.0, 2.0, 4.0], N * K // g)).astype(np.float32)
    zp = rng.integers(0, 16, size=N * K // g, dtype=np.uint8)
    x = rng.integers(-3, 4, size=(M, K)).astype(np.float32)
    bits = (lambda a: a.astype(np.float16).view(np.uint16)) if f16 else (lambda a: (a.view(np.uint32) >> 16).astype(np.uint16))
    ref = oracle.a16matmul_w4(bits(x), wq, bits(sc), zp, group=g, f16=f16)
    d = [torch.from_numpy(a).cuda() for a in (bits(x).copy(), wq, bits(sc).copy(), zp)]
    y, h = torch.zeros((M, N), dtype=torch.uint16, device="cuda"), C.c_void_p()
    L.check(L.lib().b200q_a16_dev_create_dt(ptr(d[1]), ptr(d[2]), ptr(d[3]), None, N, K, g, L.DT_F16 if f16 else L.DT_BF16, C.byref(h)))
    L.check(L.lib().b200q_a16_dev_run(h, ptr(d[0]), ptr(y), M, None))
    L.check(L.lib().b200q_a16_dev_status(h, None))
    L.lib().b200q_a16_dev_destroy(C.byref(h))
    assert np.array_equal(y.cpu().numpy(), ref)
