"""ReLU between two convolutions: forward and backward each write the neighbouring convolution's packed operand."""
import numpy as np
import pytest

from tests.test_gpu_ops import env  # noqa: F401

pytestmark = pytest.mark.gpu


# the first convolution runs whole tiles, a split tail, a cluster, strided phases in its backward
@pytest.mark.parametrize("case", [(6, 32, 16, 15, 48, 3, 3, 1), (13, 64, 40, 40, 128, 1, 1, 1), (10, 384, 8, 8, 136, 1, 3, 1), (19, 256, 14, 14, 256, 3, 3, 1), (9, 64, 17, 17, 64, 3, 3, 2)])
@pytest.mark.parametrize("arith", ["3xfp16", "3xtf32"])
def test_relu_between_convolutions(env, case, arith):
    N, C, H, W, K, R, S, stride = case
    rng = np.random.RandomState(H + K)
    gpu, nd = env.gpu_op, env.nd
    f = lambda *shape: rng.randn(*shape).astype(np.float32)
    x, w1, w2 = f(N, C, H, W), f(K, C, R, S), f(256, K, 1, 1)
    mid, cell1 = gpu.convolution_2d_forward_get_out_shape(x.shape, w1.shape, "NCHW", "SAME", stride, stride)
    out, cell2 = gpu.convolution_2d_forward_get_out_shape(mid, w2.shape, "NCHW", "SAME", 1, 1)
    act = gpu.activation_get_cudnnlist(mid, "NCHW", "relu")
    X, W1, W2, DO = (nd.array(v, env.ctx) for v in (x, w1, w2, f(*out)))
    y1, a1, da, dy1 = (nd.empty(mid, env.ctx) for _ in range(4))
    y2, dx, dw1 = nd.empty(out, env.ctx), nd.empty(x.shape, env.ctx), nd.empty(w1.shape, env.ctx)
    results, fused = [], []
    gpu.set_contraction_path(2)
    gpu.set_tensor_arithmetic(arith)
    try:
        for step in range(4):
            before = gpu.fused_relu_pack_count()
            gpu.convolution_2d_forward(X, W1, y1, cell1, env.cudnn, env.stream)
            gpu.activation_forward(y1, a1, "relu", act, env.cudnn, env.stream)
            gpu.convolution_2d_forward(a1, W2, y2, cell2, env.cudnn, env.stream)
            fused.append(gpu.fused_relu_pack_count() - before)
            gpu.convolution_backward_data(a1, DO, W2, da, cell2, env.cudnn, env.stream)
            gpu.activation_backward(y1, dy1, a1, da, "relu", act, env.cudnn, env.stream)
            if step == 0:
                gpu.device_synchronize()          # the ReLU's backward runs on its own
            gpu.convolution_backward_filter(X, dy1, W1, dw1, cell1, env.cudnn, env.stream)
            gpu.convolution_backward_data(X, dy1, W1, dx, cell1, env.cudnn, env.stream)
            results.append([v.asnumpy() for v in (y1, a1, y2, da, dy1, dw1, dx)])
    finally:
        gpu.set_contraction_path(0)
        gpu.set_tensor_arithmetic("3xfp16")
    assert fused[0] == 0 and fused[2:] == [1, 1]          # the consumer is learned in the first pass, the bound in the second
    apart = results[0]
    for got in results:
        np.testing.assert_array_equal(got[1], np.maximum(got[0], 0))
        np.testing.assert_array_equal(got[4], np.where(got[0] > 0, got[3], np.float32(0)))
        for g, e in zip(got, apart):              # packs made with another power-of-two scale round their low halves differently
            assert np.max(np.abs(g - e)) <= 2e-6 * np.max(np.abs(e))
