"""The operator face's staging: calls of one piece (converted by the calling thread or by the pool), of exactly one piece more,
of more pieces than staging slots, every storage type of the output, and several handles at once."""
import threading

import numpy as np
import pytest

import tpu_mlir_b200._lib as L
from tpu_mlir_b200.ops import Conv2DOp, InferenceParameter, MatMulOp

pytestmark = pytest.mark.gpu
PIECE = 512 * 1024      # values per piece


def _matmul(M, K, N, seed, out_dtype=L.DT_I8, signed=True):
    rng = np.random.default_rng(seed)
    a = rng.integers(-128, 128, (M, K)) if signed else rng.integers(0, 256, (M, K))
    b = rng.integers(-9, 10, (K, N))
    acc = a @ b
    if out_dtype == L.DT_I32:
        kw, want = dict(multipliers=(), rshifts=()), acc
    else:
        lo, hi = {L.DT_I8: (-128, 127), L.DT_U8: (0, 255), L.DT_I16: (-32768, 32767)}[out_dtype]
        kw, want = dict(multipliers=[3], rshifts=[7]), np.clip((acc * 3 + 64) >> 7, lo, hi)
    op = MatMulOp(M=M, K=K, N=N, quant_mode=L.QM_MULTIPLIER_SHIFT, input_dtype=L.DT_I8 if signed else L.DT_U8, out_dtype=out_dtype, **kw)
    f = lambda v: np.ascontiguousarray(v, dtype=np.float32)  # noqa: E731
    p = InferenceParameter(inputs=[f(a), f(b), None, None, None], outputs=[np.full((M, N), 7.0, np.float32)])
    return op, p, want.astype(np.float32)


@pytest.mark.parametrize("M,K,N", [(1, 16, 1), (3, 32, 33), (500, 96, 40), (PIECE // 1024, 1024, 8), (PIECE // 1024 + 1, 1024, 8),
                                   (5 * (PIECE // 2048) + 7, 2048, 24), (6 * 1024 + 1, 64, 512),
                                   # rows off 16 bytes: the pieces start anywhere, the products run on the CUDA cores
                                   (5 * (PIECE // 777) + 3, 777, 24), (9001, 33, 131), (PIECE // 1001 + 2, 1001, 40)])
def test_rows_over_pieces(M, K, N):
    op, p, want = _matmul(M, K, N, M)
    op.init(p)
    for _ in range(2):                      # the second call reuses staging, weights and requantisation arrays
        p.outputs[0][:] = 7.0
        op.inference(p)
        assert np.array_equal(p.outputs[0], want)
    op.deinit(p)


@pytest.mark.parametrize("dt,signed", [(L.DT_I8, False), (L.DT_U8, True), (L.DT_I16, True), (L.DT_I32, False)])
@pytest.mark.parametrize("M", [5, 9001])
def test_output_types(dt, signed, M):
    op, p, want = _matmul(M, 64, 131, 3, dt, signed)
    op.inference(p)
    assert np.array_equal(p.outputs[0], want)


def test_images_over_pieces_and_several_handles():
    def one(seed, out):
        rng = np.random.default_rng(seed)
        n, c, hw, oc = 9, 16, 47, 48
        x, w = rng.integers(-128, 128, (n, c, hw, hw)), rng.integers(-5, 6, (oc, c, 1, 1))
        acc = np.einsum("nchw,oc->nohw", x, w[:, :, 0, 0])
        want = np.clip((acc + 8) >> 4, 0, 127)
        op = Conv2DOp(input_shape=x.shape, oc=oc, kernel_shape=(1, 1), with_bias=False, do_relu=True, multiplier=[1], rshift=[4])
        p = InferenceParameter(inputs=[x.astype(np.float32), w.astype(np.float32)], outputs=[np.zeros(op.out_shape, np.float32)])
        op.init(p)
        for _ in range(3):
            op.inference(p)
            out.append(bool(np.array_equal(p.outputs[0], want)))
        op.deinit(p)
    results = [[] for _ in range(4)]
    threads = [threading.Thread(target=one, args=(i, r)) for i, r in enumerate(results)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert results == [[True] * 3] * 4
