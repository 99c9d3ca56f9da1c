"""The fp32 matrix product's split form: edges of its 32 x 64 tiles, of its 64-deep k slices and of the cluster's shares of K,
and both sides of the line to the convolution kernel.  Bound: K products summed in fp32 in any order, K * 2^-24 * sum |x w|, at
most 1e-5 of it, plus the result's rounding."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tpu_mlir_b200 import _lib as L  # noqa: E402

ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731


@pytest.mark.parametrize("M,K,N", [(1, 1, 1), (31, 127, 63), (32, 128, 64), (33, 129, 65), (1, 513, 1000), (32, 2048, 1000), (32, 520, 4096),
                                   (300, 1000, 257), (1152, 70, 1025), (1300, 96, 1000)])
@pytest.mark.parametrize("relu", [False, True])
def test_matmul_shapes(M, K, N, relu):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + K + N)
    x = torch.randn((M, K), device="cuda", generator=g)
    w = torch.randn((K, N), device="cuda", generator=g)
    b = torch.randn((N,), device="cuda", generator=g)
    y = torch.full((M, N), float("nan"), device="cuda")
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    L.check(L.lib().b200q_top_matmul_f32_dev(ptr(x), ptr(w), ptr(b), ptr(y), M, K, N, int(relu), 2.0, s))
    ref = x.double() @ w.double() + b.double()
    if relu:
        ref = ref.clamp(0, 2.0)
    bound = min(K * 2.0**-24, 1e-5) * (x.double().abs() @ w.double().abs()) + (ref.abs() + b.abs()) * 2.0**-23
    assert bool(((y.double() - ref).abs() <= bound).all())
