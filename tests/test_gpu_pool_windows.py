"""Pooling kernels for particular windows: means of 3x3 at stride 1, maxima of 3x3 at stride 2 with padding."""
import numpy as np
import pytest

from tests.test_gpu_ops import env  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,C,H,W", [(1, 1, 1, 1), (1, 5, 1, 9), (3, 7, 9, 1), (2, 33, 8, 8), (2, 30, 17, 17), (1, 9, 35, 35), (1, 3, 32, 64), (1, 3, 46, 47)])
def test_mean_3x3_stride_1(env, N, C, H, W):
    rng = np.random.RandomState(H + W)
    x = rng.randn(N, C, H, W).astype(np.float32)
    out, cell = env.gpu_op.pooling_2d_forward_get_out_shape(x.shape, "NCHW", "mean", 1, 1, 1, 1, 3, 3)
    assert out == x.shape
    X, y, dx = env.nd.array(x, env.ctx), env.nd.empty(out, env.ctx), env.nd.empty(x.shape, env.ctx)
    env.gpu_op.pooling_2d_forward(X, y, cell, env.cudnn, env.stream)
    env.gpu_op.pooling_2d_backward(X, y, X, dx, cell, env.cudnn, env.stream)      # the gradient of a mean is the mean of the gradient
    pad = np.pad(x.astype(np.float64), ((0, 0), (0, 0), (1, 1), (1, 1)))
    want = sum(pad[:, :, r:r + H, c:c + W] for r in range(3) for c in range(3)) / 9
    for got in (y, dx):
        np.testing.assert_allclose(got.asnumpy(), want, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("N,C,H,W,ph,pw", [(1, 3, 2, 2, 1, 1), (2, 5, 7, 8, 1, 1), (1, 4, 56, 55, 1, 1), (1, 4, 9, 12, 1, 0), (2, 3, 12, 9, 0, 1)])
def test_max_3x3_stride_2_with_padding(env, N, C, H, W, ph, pw):
    rng = np.random.RandomState(H + W)
    x = rng.randn(N, C, H, W).astype(np.float32)
    out, cell = env.gpu_op.pooling_2d_forward_get_out_shape(x.shape, "NCHW", "max", ph, pw, 2, 2, 3, 3)
    dy = rng.randn(*out).astype(np.float32)
    X, DY, y, dx = env.nd.array(x, env.ctx), env.nd.array(dy, env.ctx), env.nd.empty(out, env.ctx), env.nd.empty(x.shape, env.ctx)
    env.gpu_op.pooling_2d_forward(X, y, cell, env.cudnn, env.stream)
    env.gpu_op.pooling_2d_backward(X, y, DY, dx, cell, env.cudnn, env.stream)
    want_y, want_dx = np.empty(out, np.float32), np.zeros((N, C, H, W), np.float64)
    for p in range(out[2]):
        for q in range(out[3]):
            h0, w0 = max(0, 2 * p - ph), max(0, 2 * q - pw)
            win = x[:, :, h0:2 * p - ph + 3, w0:2 * q - pw + 3]
            at = win.reshape(N, C, -1).argmax(axis=2)
            want_y[:, :, p, q] = win.max(axis=(2, 3))
            for n in range(N):
                for c in range(C):
                    want_dx[n, c, h0 + at[n, c] // win.shape[3], w0 + at[n, c] % win.shape[3]] += dy[n, c, p, q]
    np.testing.assert_array_equal(y.asnumpy(), want_y)
    np.testing.assert_allclose(dx.asnumpy(), want_dx, rtol=1e-6, atol=1e-6)
