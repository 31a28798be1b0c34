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


# a max pool between the ReLU and what comes behind (its gradient's maximum is the bound), first layers of few channels (patches) among them
@pytest.mark.parametrize("case", [(6, 3, 33, 40, 64, 3, 1, 2, 2), (9, 3, 75, 75, 32, 3, 2, 3, 2), (6, 32, 24, 22, 64, 3, 1, 3, 2), (5, 16, 23, 21, 36, 3, 1, 2, 2), (6, 32, 18, 18, 48, 3, 1, 3, 1)])
def test_relu_backward_behind_a_pool_writes_the_packed_gradient(env, case):
    N, C, H, W, K, R, stride, win, step = case
    rng = np.random.RandomState(H + K)
    gpu, nd = env.gpu_op, env.nd
    x, w = rng.randn(N, C, H, W).astype(np.float32), rng.randn(K, C, R, R).astype(np.float32)
    mid, cell = gpu.convolution_2d_forward_get_out_shape(x.shape, w.shape, "NCHW", "SAME", stride, stride)
    out, pool = gpu.pooling_2d_forward_get_out_shape(mid, "NCHW", "max", 0, 0, step, step, win, win)
    act = gpu.activation_get_cudnnlist(mid, "NCHW", "relu")
    X, Wd, DO = nd.array(x, env.ctx), nd.array(w, env.ctx), nd.array(rng.randn(*out).astype(np.float32), env.ctx)
    y, a, da, dy = (nd.empty(mid, env.ctx) for _ in range(4))
    o, dw = nd.empty(out, env.ctx), nd.empty(w.shape, env.ctx)
    results = []
    gpu.set_contraction_path(2)
    try:
        for apart in (True, False):
            gpu.convolution_2d_forward(X, Wd, y, cell, env.cudnn, env.stream)
            gpu.activation_forward(y, a, "relu", act, env.cudnn, env.stream)
            gpu.pooling_2d_forward(a, o, pool, env.cudnn, env.stream)
            gpu.pooling_2d_backward(a, o, DO, da, pool, env.cudnn, env.stream)
            before = gpu.launch_count()
            gpu.activation_backward(y, dy, a, da, "relu", act, env.cudnn, env.stream)
            if apart:
                gpu.device_synchronize()          # the ReLU's backward runs on its own
            gpu.convolution_backward_filter(X, dy, Wd, dw, cell, env.cudnn, env.stream)
            results.append([v.asnumpy() for v in (y, da, dy, dw)] + [gpu.launch_count() - before])
    finally:
        gpu.set_contraction_path(0)
    assert results[1][4] < results[0][4]          # one kernel less
    for got in results:
        np.testing.assert_array_equal(got[2], np.where(got[0] > 0, got[1], np.float32(0)))
        assert np.max(np.abs(got[3] - results[0][3])) <= 2e-6 * np.max(np.abs(results[0][3]))


# channel 0 in front of the ReLU is negative and large, and so is its gradient: the bounds that fused packs are scaled by lie 2^10 and more above what
# the ReLU lets through, so that a pack scaled by its own maximum differs from them in the low halves of most values
@pytest.mark.parametrize("readers", [(1,), (3,), (1, 3), (3, 1, 3)], ids=str)
@pytest.mark.parametrize("whole", [True, False], ids=["whole", "cut"])
def test_a_first_step_has_the_bits_of_later_ones(env, readers, whole):
    N, C, H, W, K = (40, 64, 22, 23, 64) if whole else (24, 96, 14, 15, 48)
    rng = np.random.RandomState(7)
    gpu, nd = env.gpu_op, env.nd
    f = lambda *shape: rng.randn(*shape).astype(np.float32)
    x, w1 = np.abs(f(N, C, H, W)), f(K, C, 3, 3)
    w1[0] = -300 * np.abs(w1[0])
    mid, cell1 = gpu.convolution_2d_forward_get_out_shape(x.shape, w1.shape, "NCHW", "SAME", 1, 1)
    act = gpu.activation_get_cudnnlist(mid, "NCHW", "relu")
    X, W1 = nd.array(x, env.ctx), nd.array(w1, env.ctx)
    y1, a1, da, dy1, dx, dw1 = (nd.empty(s, env.ctx) for s in (mid, mid, mid, mid, x.shape, w1.shape))
    behind = []
    for r in readers:
        w = f(64, K, r, r)
        w[:, 0] *= 2000
        out, cell = gpu.convolution_2d_forward_get_out_shape(mid, w.shape, "NCHW", "SAME", 1, 1)
        behind.append((nd.array(w, env.ctx), nd.array(f(*out), env.ctx), nd.empty(out, env.ctx), nd.empty(w.shape, env.ctx), cell))
    steps, fused = [], []
    gpu.set_contraction_path(2)
    try:
        for step in range(5):
            before = gpu.fused_relu_pack_count()
            gpu.convolution_2d_forward(X, W1, y1, cell1, env.cudnn, env.stream)
            gpu.activation_forward(y1, a1, "relu", act, env.cudnn, env.stream)
            for w, do, y, dw, cell in behind:
                gpu.convolution_2d_forward(a1, w, y, cell, env.cudnn, env.stream)
            fused.append(gpu.fused_relu_pack_count() - before)
            for w, do, y, dw, cell in behind:
                gpu.convolution_backward_filter(a1, do, w, dw, cell, env.cudnn, env.stream)
                gpu.convolution_backward_data(a1, do, w, da, cell, env.cudnn, env.stream)
            gpu.activation_backward(y1, dy1, a1, da, "relu", act, env.cudnn, env.stream)
            gpu.convolution_backward_filter(X, dy1, W1, dw1, cell1, env.cudnn, env.stream)
            gpu.convolution_backward_data(X, dy1, W1, dx, cell1, env.cudnn, env.stream)
            steps.append([v.asnumpy() for v in [y1, a1, da, dy1, dx, dw1] + [b[k] for b in behind for k in (2, 3)]])
    finally:
        gpu.set_contraction_path(0)
    assert fused[0] == 0 and fused[-1] == 1
    assert steps[0][0].min() < -2.0 ** 10 * steps[0][1].max() and np.abs(steps[0][2][:, 0]).max() > 2.0 ** 10 * np.abs(steps[0][3]).max()
    for later in steps[1:]:
        for a, b in zip(steps[0], later):
            np.testing.assert_array_equal(a, b)


# the mask takes away gradients 2^4, 2^10 and 2^14 times the largest that is left: the fused pack, scaled by the larger maximum, against the one on its own and 64 bits
@pytest.mark.parametrize("power", [4, 10, 14])
@pytest.mark.parametrize("case", [(6, 3, 33, 40, 64, 3, 1, 2, 2), (6, 32, 24, 22, 64, 3, 1, 3, 2)])
def test_a_bound_far_above_what_the_mask_leaves(env, case, power):
    import torch
    N, C, H, W, K, R, stride, win, step = case
    rng = np.random.RandomState(H + K)
    gpu, nd = env.gpu_op, env.nd
    x, w = np.abs(rng.randn(N, C, H, W)).astype(np.float32), rng.randn(K, C, R, R).astype(np.float32)
    w[0] = -np.abs(w[0])                          # channel 0 is never positive
    mid, cell = gpu.convolution_2d_forward_get_out_shape(x.shape, w.shape, "NCHW", "SAME", stride, stride)
    out, pool = gpu.pooling_2d_forward_get_out_shape(mid, "NCHW", "max", 0, 0, step, step, win, win)
    act = gpu.activation_get_cudnnlist(mid, "NCHW", "relu")
    do = rng.randn(*out).astype(np.float32)
    do[:, 0] *= 2.0 ** power
    X, Wd, DO = (nd.array(v, env.ctx) for v in (x, w, do))
    y, a, da, dy = (nd.empty(mid, env.ctx) for _ in range(4))
    o, dw = nd.empty(out, env.ctx), nd.empty(w.shape, env.ctx)
    got = []
    gpu.set_contraction_path(2)
    try:
        for apart in (True, False):
            gpu.convolution_2d_forward(X, Wd, y, cell, env.cudnn, env.stream)
            gpu.activation_forward(y, a, "relu", act, env.cudnn, env.stream)
            gpu.pooling_2d_forward(a, o, pool, env.cudnn, env.stream)
            gpu.pooling_2d_backward(a, o, DO, da, pool, env.cudnn, env.stream)
            before = gpu.launch_count()
            gpu.activation_backward(y, dy, a, da, "relu", act, env.cudnn, env.stream)
            if apart:
                gpu.device_synchronize()
            gpu.convolution_backward_filter(X, dy, Wd, dw, cell, env.cudnn, env.stream)
            got.append((gpu.launch_count() - before, dw.asnumpy()))
    finally:
        gpu.set_contraction_path(0)
    assert got[1][0] < got[0][0]
    grad = dy.asnumpy()
    bound, left = np.abs(da.asnumpy()).max(), np.abs(grad).max()
    assert bound > 2.0 ** (power - 1) * left
    # a kept value is off by 2^-22 of itself or 2^-25 / scale, scale >= 2^14 / bound, whichever is more; products are summed in fp32
    exact = lambda g: torch.nn.grad.conv2d_weight(torch.from_numpy(x).double(), w.shape, torch.from_numpy(g).double(), stride, R // 2).numpy()       # noqa: E731
    want, mag, each = exact(grad), exact(np.abs(grad)), exact(np.ones_like(grad))
    for _, dwv in got:
        assert np.all(np.abs(dwv - want) <= 8 * 2.0 ** -24 * mag + 2.0 ** -39 * bound * each)
    np.testing.assert_array_equal(got[1][1][0], 0)


# an operator call ahead of a recorded step writes what its first convolution packs: another bound by the next replay, or none
@pytest.mark.parametrize("how", ["relu", "copy"])
@pytest.mark.parametrize("arith", ["3xfp16", "3xtf32"])
def test_a_replay_packs_what_a_relu_wrote_since(env, how, arith):
    import ctypes
    from tinyflow_b200._base import _LIB, check_call, new_cell
    N, C, H, W, K = 24, 64, 14, 15, 48
    rng = np.random.RandomState(11)
    gpu, nd = env.gpu_op, env.nd
    f = lambda *shape: nd.array(rng.randn(*shape).astype(np.float32), env.ctx)       # noqa: E731
    X, W1, W2 = f(N, C, H, W), f(K, C, 3, 3), f(64, K, 3, 3)
    mid, cell1 = gpu.convolution_2d_forward_get_out_shape(X.shape, W1.shape, "NCHW", "SAME", 1, 1)
    out, cell2 = gpu.convolution_2d_forward_get_out_shape(mid, W2.shape, "NCHW", "SAME", 1, 1)
    act = gpu.activation_get_cudnnlist(mid, "NCHW", "relu")
    y1, a1, y2 = nd.empty(mid, env.ctx), nd.empty(mid, env.ctx), nd.empty(out, env.ctx)

    def ahead():
        gpu.convolution_2d_forward(X, W1, y1, cell1, env.cudnn, env.stream)
        gpu.activation_forward(y1, a1, "relu", act, env.cudnn, env.stream)

    def record():
        graph, on = ctypes.c_void_p(), new_cell(2)
        check_call(_LIB.TfStepRecordBegin(ctypes.byref(graph), on, env.stream))
        gpu.convolution_2d_forward(a1, W2, y2, cell2, env.cudnn, on)
        check_call(_LIB.TfStepRecordEnd(ctypes.byref(graph), 1))
        return graph
    gpu.set_contraction_path(2)
    gpu.set_tensor_arithmetic(arith)
    graph = None
    try:
        ahead()
        gpu.convolution_2d_forward(a1, W2, y2, cell2, env.cudnn, env.stream)
        ahead()
        graph = record()
        small = None
        for scale in (1.0, 2.0 ** 12):                       # a power of two: every bit but the exponent stays
            if scale > 1 and how == "relu":
                W1[:] = W1.asnumpy() * np.float32(scale)
                ahead()
            elif scale > 1:
                a1[:] = a1.asnumpy() * np.float32(scale)
            y2[:] = np.full(out, np.nan, np.float32)
            rc = _LIB.TfStepReplay(graph, None, 0, ctypes.c_float(0), ctypes.c_float(0), None, 0, env.stream)
            assert rc == 0 or (rc == 1 and scale > 1 and how == "copy")
            if rc == 1:                                      # nothing knows the new maximum: the caller records again
                _LIB.TfStepGraphFree(graph)
                graph = record()
                check_call(_LIB.TfStepReplay(graph, None, 0, ctypes.c_float(0), ctypes.c_float(0), None, 0, env.stream))
            got = y2.asnumpy()
            small = got if scale == 1 else small
            np.testing.assert_allclose(got, small * np.float32(scale), rtol=0, atol=2e-6 * scale * np.abs(small).max())
    finally:
        if graph is not None:
            _LIB.TfStepGraphFree(graph)
        gpu.set_contraction_path(0)
        gpu.set_tensor_arithmetic("3xfp16")
