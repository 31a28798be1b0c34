"""CUDA-core kernels for small sizes: products, convolutions of few channels, split reductions."""
import numpy as np
import pytest

from tests.test_gpu_ops import env  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N", [(1, 1, 1), (8, 33, 64), (7, 4100, 130), (9, 64, 31), (33, 127, 65), (32, 256, 32), (64, 3, 1029), (640, 65, 1030), (2, 2048, 1000)])
@pytest.mark.parametrize("tA,tB", [(False, False), (True, False), (False, True), (True, True)])
def test_simt_product_at_tile_edges(env, M, K, N, tA, tB):
    rng = np.random.RandomState(M + K + N)
    a, b = rng.randn(M, K).astype(np.float32), rng.randn(K, N).astype(np.float32)
    A, B = env.nd.array(np.ascontiguousarray(a.T) if tA else a, env.ctx), env.nd.array(np.ascontiguousarray(b.T) if tB else b, env.ctx)
    C = env.nd.empty((M, N), env.ctx)
    env.gpu_op.set_contraction_path(1)
    try:
        env.gpu_op.matrix_multiply(A, tA, B, tB, C, env.cublas, env.stream)
    finally:
        env.gpu_op.set_contraction_path(0)
    want, mag = a.astype(np.float64) @ b.astype(np.float64), np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)
    assert np.all(np.abs(C.asnumpy() - want) <= 1e-5 * np.abs(want) + 8 * 2.0 ** -24 * mag)


# few rows against a million weights and more: runs of K that are not whole, one and several CTAs, 8 and 16 rows, ragged columns
@pytest.mark.parametrize("M,K,N", [(7, 4608, 4096), (1, 1000, 1004), (9, 25088, 64), (16, 25090, 132), (13, 36, 40004), (3, 8200, 516), (8, 1024, 1024), (2, 2044, 4100)])
@pytest.mark.parametrize("tB", [False, True])
def test_few_rows_against_large_weights(env, M, K, N, tB):
    test_simt_product_at_tile_edges(env, M, K, N, False, tB)


@pytest.mark.parametrize("M,K,N", [(1000, 7, 1028), (4100, 16, 260), (1004, 1, 1000), (2052, 9, 516), (36, 8, 40000)])
def test_weight_gradients_of_few_rows(env, M, K, N):
    test_simt_product_at_tile_edges(env, M, K, N, True, False)


def _kernels(run):
    import ctypes
    import json
    from tinyflow_b200._base import _LIB
    report = ctypes.create_string_buffer(1 << 16)
    _LIB.TfKernelTimingEnable(1)
    try:
        run()
        _LIB.TfKernelTimingReport(report, len(report))
    finally:
        _LIB.TfKernelTimingEnable(0)
    return [r["name"] for r in json.loads(report.value.decode())]


# shapes that the kernels for a handful of rows take on 148 SMs: 8 and 16 rows to a block, runs of K and clusters that are not whole (clusters of
# 8, 4 and 1 CTAs, K of 4602, 2052, 2100, 1100 and 36; C = A B^T: 1, 2, 4 and 8 runs of a row), ragged columns
@pytest.mark.parametrize("M,K,N,tA,tB", [(7, 4608, 4096, False, False), (7, 4602, 4096, False, False), (16, 2052, 4096, False, False), (11, 2100, 2500, False, False), (13, 36, 40004, False, False),
                                         (9, 1100, 9004, False, False), (12, 1000, 4096, False, True), (16, 2052, 4098, False, True), (9, 4100, 2401, False, True), (5, 4604, 3000, False, True), (9, 4096, 1601, False, True),
                                         (15, 132, 9001, False, True), (1000, 7, 1028, True, False), (2052, 9, 516, True, False), (36, 16, 40000, True, False)])
def test_products_of_few_rows_take_their_kernels(env, M, K, N, tA, tB):
    assert _kernels(lambda: test_simt_product_at_tile_edges(env, M, K, N, tA, tB)) == ["rows_gemm"]


@pytest.mark.parametrize("case", [(3, 1, 28, 28, 6, 5, 5, "SAME"), (5, 6, 14, 14, 16, 5, 5, "VALID"), (2, 3, 9, 7, 5, 3, 3, "SAME"), (300, 2, 8, 8, 3, 7, 7, "SAME"),
                                  (2, 8, 11, 13, 32, 1, 3, "SAME"), (1, 5, 40, 33, 7, 3, 3, "VALID")])
def test_direct_convolution_of_few_channels(env, case):
    N, C, H, W, K, R, S, padding = case
    rng = np.random.RandomState(N + C)
    x, w = rng.randn(N, C, H, W).astype(np.float32), rng.randn(K, C, R, S).astype(np.float32)
    out, cell = env.gpu_op.convolution_2d_forward_get_out_shape(x.shape, w.shape, "NCHW", padding, 1, 1)
    dy = rng.randn(*out).astype(np.float32)
    X, Wd, DY = (env.nd.array(v, env.ctx) for v in (x, w, dy))
    got = {}
    for path in (0, 1):                      # the direct kernels, and the implicit product as the cross-check
        env.gpu_op.set_contraction_path(path)
        try:
            y, dx, dw = env.nd.empty(out, env.ctx), env.nd.empty(x.shape, env.ctx), env.nd.empty(w.shape, env.ctx)
            env.gpu_op.convolution_2d_forward(X, Wd, y, cell, env.cudnn, env.stream)
            env.gpu_op.convolution_backward_data(X, DY, Wd, dx, cell, env.cudnn, env.stream)
            env.gpu_op.convolution_backward_filter(X, DY, Wd, dw, cell, env.cudnn, env.stream)
            got[path] = [v.asnumpy() for v in (y, dx, dw)]
        finally:
            env.gpu_op.set_contraction_path(0)
    for a, b in zip(got[0], got[1]):
        np.testing.assert_allclose(a, b, rtol=1e-4, atol=3e-5 * np.abs(b).max())


@pytest.mark.parametrize("case", [(1, 16, 10, 10, 6, 5, 5, "SAME"), (300, 15, 6, 5, 12, 3, 3, "SAME"), (700, 4, 8, 9, 7, 3, 3, "VALID"),       # 4, 2 and 1 lanes an item
                                  (2, 2, 5, 3, 9, 3, 3, "SAME"), (4, 1, 7, 1, 4, 3, 3, "SAME"), (3, 13, 30, 31, 10, 7, 7, "VALID"), (5, 8, 12, 12, 16, 5, 5, "SAME")])
def test_direct_convolution_lanes_that_share_items(env, case):
    test_direct_convolution_of_few_channels(env, case)


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (256, 6, 28, 28), (3, 300, 5, 7), (64, 16, 10, 10), (1, 2, 129, 3)])
def test_channel_sums(env, shape):
    x = np.random.RandomState(1).randn(*shape).astype(np.float32)
    X, out = env.nd.array(x, env.ctx), env.nd.empty((shape[1],), env.ctx)
    env.gpu_op.broadcast_to_backward(X, out, "NCHW")
    want, mag = x.astype(np.float64).sum((0, 2, 3)), np.abs(x).astype(np.float64).sum((0, 2, 3))
    assert np.all(np.abs(out.asnumpy() - want) <= 1e-6 * mag)


def test_split_reductions_on_two_streams_at_once(env):
    """Every stream has partial sums and arrival counters of its own: two threads get the bits that one gets."""
    import threading
    nd, op, runs = env.nd, env.gpu_op, 150
    rng = np.random.RandomState(2)
    state = []
    for k in range(2):
        stream = op.create_cudaStream()
        logits = nd.array(rng.randn(2000 + k, 37).astype(np.float32), env.ctx)
        labels = nd.array(np.eye(37, dtype=np.float32)[rng.randint(0, 37, 2000 + k)], env.ctx)
        x = nd.array(rng.randn(64, 16, 33, 32 + k).astype(np.float32), env.ctx)
        plan = op.reduce_sum_get_cudnnlist(x.shape, (1, 16, 1, 1), "NCHW", env.cudnn)
        outs = [(nd.empty((1,), env.ctx), nd.empty((1, 16, 1, 1), env.ctx)) for _ in range(runs + 1)]
        state.append((stream, logits, labels, x, plan, outs))

    def work(k, which):
        stream, logits, labels, x, plan, outs = state[k]
        for loss, sums in which(outs):
            op.softmax_cross_entropy(logits, labels, loss, stream)
            op.reduce_sum_new(x, sums, plan, env.cudnn, stream)

    for k in range(2):
        work(k, lambda outs: outs[:1])
    op.device_synchronize()
    threads = [threading.Thread(target=work, args=(k, lambda outs: outs[1:])) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    op.device_synchronize()
    for k in range(2):
        want = [v.asnumpy() for v in state[k][-1][0]]
        for pair in state[k][-1][1:]:
            for got, one in zip(pair, want):
                np.testing.assert_array_equal(got.asnumpy(), one)
        mag = np.abs(state[k][3].asnumpy().astype(np.float64)).sum((0, 2, 3))
        assert np.all(np.abs(want[1].ravel() - state[k][3].asnumpy().astype(np.float64).sum((0, 2, 3))) <= 1e-6 * mag)


@pytest.mark.parametrize("call", ["axis_zero", "axis_1", "all", "broadcast_back_0", "broadcast_back_1", "all_backward", "axis_backward"])
def test_reductions_without_a_stream_read_a_sum_just_issued(env, call):
    """A large elementwise sum may be held back for one call; whoever reads it next launches it first."""
    nd, op = env.nd, env.gpu_op
    shape = {"all_backward": (1,), "axis_backward": (300, 5)}.get(call, (300, 5, 8, 9))
    rng = np.random.RandomState(4)
    if call in ("all_backward", "axis_backward"):                     # the result is what a held-back sum overwrites late
        big = (300, 5, 72)
        a, b, v = rng.randn(*big).astype(np.float32), rng.randn(*big).astype(np.float32), rng.randn(*shape).astype(np.float32)
        out, V = nd.empty(big, env.ctx), nd.array(v, env.ctx)
        A, B = nd.array(a, env.ctx), nd.array(b, env.ctx)
        op.matrix_elementwise_add(A, B, out, env.stream)
        op.reduce_sum_backward(V, out, -1 if call == "all_backward" else 2)
        want = np.broadcast_to(v if call == "all_backward" else v[:, :, None], big)
        np.testing.assert_array_equal(out.asnumpy(), want)
        return
    a, b = rng.randn(*shape).astype(np.float32), rng.randn(*shape).astype(np.float32)
    A, B, total = nd.array(a, env.ctx), nd.array(b, env.ctx), nd.empty(shape, env.ctx)
    axes, result = {"axis_zero": ((0,), (5, 8, 9)), "axis_1": ((1,), (300, 8, 9)), "all": ((0, 1, 2, 3), (1,)),
                    "broadcast_back_0": ((0, 1), (8, 9)), "broadcast_back_1": ((0, 2, 3), (5,))}[call]
    out = nd.empty(result, env.ctx)
    op.matrix_elementwise_add(A, B, total, env.stream)
    if call == "axis_zero":
        op.reduce_sum_axis_zero(total, out)
    elif call.startswith("broadcast"):
        op.broadcast_to_backward(total, out, "NHWC" if call.endswith("0") else "NCHW")
    else:
        op.reduce_sum(total, out, -1 if call == "all" else 1)
    s = (a + b).astype(np.float64)
    assert np.all(np.abs(out.asnumpy() - s.sum(axes).reshape(result)) <= 2e-6 * np.abs(s).sum(axes).reshape(result))


def test_split_reductions_in_a_capture_of_the_callers_own(env):
    """The scratch of a stream that is first used while its caller captures it is not part of the capture."""
    import ctypes
    import torch
    nd, op = env.nd, env.gpu_op
    rng = np.random.RandomState(6)
    logits, labels = nd.array(rng.randn(2000, 37).astype(np.float32), env.ctx), nd.array(np.eye(37, dtype=np.float32)[rng.randint(0, 37, 2000)], env.ctx)
    x, plan = nd.array(rng.randn(64, 16, 33, 32).astype(np.float32), env.ctx), op.reduce_sum_get_cudnnlist((64, 16, 33, 32), (1, 16, 1, 1), "NCHW", env.cudnn)
    want, got = ([nd.empty((1,), env.ctx), nd.empty((1, 16, 1, 1), env.ctx)] for _ in range(2))

    def work(out, stream):
        op.softmax_cross_entropy(logits, labels, out[0], stream)
        op.reduce_sum_new(x, out[1], plan, env.cudnn, stream)
    work(want, env.stream)
    op.device_synchronize()
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    cell = ctypes.pointer(ctypes.c_void_p(side.cuda_stream))
    with torch.cuda.graph(graph, stream=side):
        work(got, cell)
    op.release_cached_memory()
    op.set_memory_limit(sum(op.allocator_stats()))       # a full device: scratch is given up, but not what the graph names
    try:
        assert isinstance(nd.empty((1 << 28,), env.ctx), int)
    finally:
        op.set_memory_limit(0)
    for _ in range(3):
        for v in got:
            v[:] = np.zeros(v.shape, np.float32)
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a.asnumpy(), b.asnumpy())
    work(got, cell)                                      # and as ordinary calls on that stream
    op.device_synchronize()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a.asnumpy(), b.asnumpy())


@pytest.mark.parametrize("streams", [1, 2])
def test_products_of_two_threads(env, streams):
    """Packs and partial sums lie in the stream's scratch: two threads on one stream, or on two, do not disturb each other."""
    import threading
    nd, op, runs = env.nd, env.gpu_op, 40
    rng = np.random.RandomState(3)
    cells = [env.stream, env.stream if streams == 1 else op.create_cudaStream()]
    shapes = [(700, 2048, 900), (640, 1500, 520)]                    # tensor path, reductions split over CTAs
    state = [(nd.array(rng.randn(M, K).astype(np.float32), env.ctx), nd.array(rng.randn(K, N).astype(np.float32), env.ctx),
              [nd.empty((M, N), env.ctx) for _ in range(runs + 1)]) for M, K, N in shapes]

    def work(k, outs):
        a, b, _ = state[k]
        for c in outs:
            op.matrix_multiply(a, False, b, False, c, env.cublas, cells[k])
    for k in range(2):
        work(k, state[k][2][:1])
    op.device_synchronize()
    threads = [threading.Thread(target=work, args=(k, state[k][2][1:])) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    op.device_synchronize()
    for k in range(2):
        want = state[k][2][0].asnumpy()
        for c in state[k][2][1:]:
            np.testing.assert_array_equal(c.asnumpy(), want)


# The batches at which the number of sample groups and the samples of each change; features in whole and in ragged vectors.  (Not a
# batch of 2: there dx = inv * (g - mean(g) - xhat * mean(g * xhat)) cancels to eps / var ~ 1e-5 of its terms, whose fp32 rounding of
# 2^-24 is then 6e-3 of the result.)
@pytest.mark.parametrize("N", [5, 16, 17, 32, 33])
@pytest.mark.parametrize("plane", [(4, 5, 7), (3, 2, 7), (5, 3, 3)])
def test_batchnorm_at_group_edges(env, N, plane):
    from tests.test_gpu_ops import test_batchnorm, test_relu_backward_runs_inside_the_batchnorm_backward_that_follows as fused
    test_batchnorm(env, (N,) + plane, "pre_activation")
    if np.prod(plane) % 2 == 0:
        plane = (plane[0] * 2 ** 11 // N // 2 * 2,) + plane[1:]          # held back from 64 K elements on
        fused(env, (N,) + plane, True)
        fused(env, (N,) + plane, False)


# an image of no positions, no images: sums of nothing, not of what lies behind the array; one alone and among others that wait
@pytest.mark.parametrize("shape", [(3, 40, 0), (70, 5, 4, 0), (2, 300, 0, 6), (0, 7, 4, 4)], ids=str)
@pytest.mark.parametrize("held", [False, True])
def test_channel_sums_of_nothing(env, shape, held):
    gpu, nd = env.gpu_op, env.nd
    some = np.random.RandomState(3).randn(9, 6, 5).astype(np.float32)
    calls = []
    for x in (nd.empty(shape, env.ctx), nd.array(some, env.ctx)):
        ins, outs = gpu.reduce_sum_get_real_shape(x.shape, (x.shape[1],), "NCHW")
        calls.append((x, nd.array(np.full(x.shape[1], 7, np.float32), env.ctx), gpu.reduce_sum_get_cudnnlist(ins, outs, "NCHW", env.cudnn)))
    try:
        gpu.hold_products(held)
        for x, out, cell in calls:
            gpu.reduce_sum_new(x, out, cell, env.cudnn, env.stream)
        gpu.hold_products(False)
        gpu.launch_held(env.stream)
    finally:
        gpu.drop_held()
    np.testing.assert_array_equal(calls[0][1].asnumpy(), np.zeros(shape[1], np.float32))
    np.testing.assert_allclose(calls[1][1].asnumpy(), some.astype(np.float64).sum(axis=(0, 2)), rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("rows,cols", [(0, 5), (0, 70), (0, 1), (100, 0), (3, 0)])
def test_column_sums_of_nothing(env, rows, cols):
    gpu, nd = env.gpu_op, env.nd
    x, out = nd.empty((rows, cols), env.ctx), nd.array(np.full(cols, 7, np.float32), env.ctx) if cols else nd.empty((0,), env.ctx)
    ins, outs = gpu.reduce_sum_get_real_shape(x.shape, (cols,), "NHWC")
    gpu.reduce_sum_new(x, out, gpu.reduce_sum_get_cudnnlist(ins, outs, "NHWC", env.cudnn), env.cudnn, env.stream)
    np.testing.assert_array_equal(out.asnumpy(), np.zeros(cols, np.float32))
