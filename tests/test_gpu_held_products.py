"""Gradients of parameters that wait and share a launch: the bits of separate launches, whatever is held back together."""
import numpy as np
import pytest

from tests.test_gpu_step_graph import BUILDS, _same, _train

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", ["3xfp16", "3xtf32"])
@pytest.mark.parametrize("name", ["inceptionv3", "resnet50", "vgg16", "densenet121", "mlp", "lenet5"])
def test_products_held_back_have_the_bits_of_separate_launches(lib_path, monkeypatch, name, arith):
    from tinyflow_b200 import gpu_op
    build = BUILDS.get(name, lambda m: m.densenet121(batch=16, classes=10, image=96))
    gpu_op.set_tensor_arithmetic(arith)
    try:
        got = _train(monkeypatch, True, build, "sgd")
        with monkeypatch.context() as m:
            m.setattr(gpu_op, "hold_products", lambda on: None)
            want = _train(monkeypatch, False, build, "sgd")
    finally:
        gpu_op.set_tensor_arithmetic("3xfp16")
    assert got[2] and not want[2]
    _same(got, want)


# N, C, H, W, K, R, S, stride: with and without several taps a tile, odd numbers of 64-channel blocks, ragged tiles, cut and whole reductions
LAYERS = [(2, 64, 9, 9, 96, 3, 3, 1), (3, 160, 12, 7, 160, 7, 1, 1), (2, 33 * 4, 9, 9, 68, 1, 7, 1), (5, 64, 14, 14, 256, 1, 1, 1), (5, 256, 14, 14, 64, 1, 1, 1),
          (4, 288, 17, 17, 384, 3, 3, 2), (1, 48, 21, 21, 64, 5, 5, 1), (16, 96, 35, 35, 64, 1, 1, 1), (2, 768, 17, 17, 192, 1, 1, 1), (8, 128, 28, 28, 32, 3, 3, 1), (2, 3, 75, 75, 32, 3, 3, 2),
          # runs of 4 pieces: 9, 16, 17 and more of one tile, kept to a CTA's chunks among the others and dealt out one by one alone
          (2, 128, 17, 17, 128, 1, 1, 1), (4, 128, 16, 16, 128, 1, 1, 1), (17, 128, 8, 8, 128, 1, 1, 1), (9, 256, 17, 17, 96, 1, 1, 1)]


@pytest.mark.parametrize("arith", ["3xfp16", "3xtf32"])
@pytest.mark.parametrize("layers", [LAYERS, LAYERS[:1], LAYERS[7:8], LAYERS[-4:]], ids=["all", "one", "one cut", "runs"])
def test_layers_in_one_launch(lib_path, layers, arith):
    from tinyflow_b200 import gpu_op, ndarray as nd
    ctx, stream, rng = nd.gpu(0), gpu_op.create_cudaStream(), np.random.RandomState(1)
    handle = gpu_op.create_cudnnHandle(stream)
    gpu_op.set_tensor_arithmetic(arith)
    calls = []
    for N, C, H, W, K, R, S, u in layers:
        out, cell = gpu_op.convolution_2d_forward_get_out_shape((N, C, H, W), (K, C, R, S), "NCHW", "VALID" if u > 1 else "SAME", u, u)
        x, w, dy = (nd.array(rng.randn(*shape).astype(np.float32), ctx) for shape in ((N, C, H, W), (K, C, R, S), out))
        calls.append((x, dy, w, nd.empty((K, C, R, S), ctx), nd.array(np.full((K, C, R, S), np.nan, np.float32), ctx), cell))
    try:
        for x, dy, w, apart, _, cell in calls:
            gpu_op.convolution_backward_filter(x, dy, w, apart, cell, handle, stream)
        for again in range(2):                       # the second time on packs that are there
            gpu_op.hold_products(True)
            for x, dy, w, _, together, cell in calls:
                gpu_op.convolution_backward_filter(x, dy, w, together, cell, handle, stream)
            gpu_op.hold_products(False)
            gpu_op.launch_held(stream)
            for shape, (_, _, _, apart, together, _) in zip(layers, calls):
                np.testing.assert_array_equal(together.asnumpy(), apart.asnumpy(), err_msg=str(shape))
        # a pack that is written again lets what has to read it go first
        x, dy, w, apart, together, cell = calls[0]
        gpu_op.hold_products(True)
        gpu_op.convolution_backward_filter(x, dy, w, together, cell, handle, stream)
        other = nd.array(rng.randn(*x.shape).astype(np.float32), ctx)
        second = nd.empty(w.shape, ctx)
        gpu_op.convolution_backward_filter(other, dy, w, second, cell, handle, stream)
        gpu_op.hold_products(False)
        np.testing.assert_array_equal(together.asnumpy(), apart.asnumpy())
        gpu_op.launch_held(stream)
        assert not np.array_equal(second.asnumpy(), apart.asnumpy())
    finally:
        gpu_op.drop_held()
        gpu_op.set_tensor_arithmetic("3xfp16")


# more than one launch of each kind; reductions of one CTA up to a cluster of 8, sums of one block up to many, ragged tiles
@pytest.mark.parametrize("count", [1, 3, 37])
def test_dense_gradients_in_one_launch(lib_path, count):
    from tinyflow_b200 import gpu_op, ndarray as nd
    ctx, stream, rng = nd.gpu(0), gpu_op.create_cudaStream(), np.random.RandomState(count)
    cublas, cudnn = gpu_op.create_cublasHandle(stream), gpu_op.create_cudnnHandle(stream)
    calls = []
    for i in range(count):
        rows, a, b = (int(v) for v in (rng.choice([7, 64, 100, 1000, 1200]), rng.choice([9, 33, 120, 400]), rng.choice([10, 31, 84, 300])))
        x, dy = (nd.array(rng.randn(rows, n).astype(np.float32), ctx) for n in (a, b))
        image = nd.array(rng.randn(max(1, rows // 50), 6, 9, 1 + i % 5).astype(np.float32), ctx)
        cells = [gpu_op.reduce_sum_get_cudnnlist(*gpu_op.reduce_sum_get_real_shape(s, o, f), f, cudnn) for s, o, f in (((rows, b), (b,), "NHWC"), (image.shape, (6,), "NCHW"))]
        calls.append((x, dy, image, cells, [nd.empty((a, b), ctx), nd.empty((b,), ctx), nd.empty((6,), ctx)], [nd.empty((a, b), ctx), nd.empty((b,), ctx), nd.empty((6,), ctx)]))

    def run(into):
        for call in calls:
            x, dy, image, cells, out = call[:4] + (call[into],)
            gpu_op.matrix_multiply(x, True, dy, False, out[0], cublas, stream)
            gpu_op.reduce_sum_new(dy, out[1], cells[0], cudnn, stream)
            gpu_op.reduce_sum_new(image, out[2], cells[1], cudnn, stream)
    run(4)
    try:
        gpu_op.hold_products(True)
        run(5)
        gpu_op.hold_products(False)
        before = gpu_op.launch_count()
        gpu_op.launch_held(stream)
        assert gpu_op.launch_count() - before == (count + 15) // 16 + (2 * count + 31) // 32
    finally:
        gpu_op.drop_held()
    for x, dy, _, _, apart, together in calls:
        for one, other in zip(apart, together):
            np.testing.assert_array_equal(one.asnumpy(), other.asnumpy())
        np.testing.assert_allclose(together[0].asnumpy(), x.asnumpy().T.astype(np.float64) @ dy.asnumpy(), rtol=1e-4, atol=1e-2)


@pytest.mark.parametrize("count", [1, 2, 11])
def test_direct_filter_gradients_in_one_launch(lib_path, count):
    from tinyflow_b200 import gpu_op, ndarray as nd
    ctx, stream, rng = nd.gpu(0), gpu_op.create_cudaStream(), np.random.RandomState(count)
    handle = gpu_op.create_cudnnHandle(stream)
    calls = []
    for i in range(count):
        N, C, H, W, K, R, S, padding = [(3, 1, 28, 28, 6, 5, 5, "SAME"), (40, 6, 14, 14, 16, 5, 5, "VALID"), (300, 3, 9, 7, 5, 3, 3, "SAME"), (7, 2, 8, 8, 3, 7, 7, "SAME")][i % 4]
        out, cell = gpu_op.convolution_2d_forward_get_out_shape((N, C, H, W), (K, C, R, S), "NCHW", padding, 1, 1)
        x, w, dy = (nd.array(rng.randn(*shape).astype(np.float32), ctx) for shape in ((N, C, H, W), (K, C, R, S), out))
        calls.append((x, dy, w, nd.empty((K, C, R, S), ctx), nd.empty((K, C, R, S), ctx), cell))
    try:
        for k in (3, 4):
            gpu_op.hold_products(k == 4)
            for call in calls:
                gpu_op.convolution_backward_filter(call[0], call[1], call[2], call[k], call[5], handle, stream)
        gpu_op.hold_products(False)
        before = gpu_op.launch_count()
        gpu_op.launch_held(stream)
        assert gpu_op.launch_count() - before == 2 * len({call[2].shape[3] for call in calls})
    finally:
        gpu_op.drop_held()
    for call in calls:
        np.testing.assert_array_equal(call[4].asnumpy(), call[3].asnumpy())


DIRECT = [(300, 3, 9, 7, 5, 3, 3, 1), (40, 6, 14, 14, 16, 5, 5, 1), (200, 2, 8, 8, 8, 3, 3, 1), (64, 6, 11, 11, 16, 5, 5, 1), (30, 1, 28, 28, 6, 5, 5, 1)]


# the device has no byte left but the workspaces of separate launches: what waits is launched in parts, with the same bits
@pytest.mark.parametrize("recorded", [False, True])
@pytest.mark.parametrize("arith", ["3xfp16", "3xtf32"])
def test_a_full_device_launches_fewer_together(lib_path, arith, recorded):
    import ctypes
    from tinyflow_b200 import gpu_op, ndarray as nd
    from tinyflow_b200._base import _LIB, check_call, new_cell
    ctx, stream, rng = nd.gpu(0), gpu_op.create_cudaStream(), np.random.RandomState(5)
    handle = gpu_op.create_cudnnHandle(stream)
    gpu_op.set_tensor_arithmetic(arith)
    calls = []
    for N, C, H, W, K, R, S, u in LAYERS + DIRECT:
        out, cell = gpu_op.convolution_2d_forward_get_out_shape((N, C, H, W), (K, C, R, S), "NCHW", "VALID" if u > 1 else "SAME", u, u)
        x, w, dy = (nd.array(rng.randn(*shape).astype(np.float32), ctx) for shape in ((N, C, H, W), (K, C, R, S), out))
        sums = gpu_op.reduce_sum_get_cudnnlist(*gpu_op.reduce_sum_get_real_shape(out, (K,), "NCHW"), "NCHW", handle)
        calls.append((x, dy, w, cell, sums) + tuple(nd.array(np.full(s, np.nan, np.float32), ctx) for _ in range(2) for s in ((K, C, R, S), (K,))))

    def run(into, on):
        for call in calls:
            gpu_op.convolution_backward_filter(call[0], call[1], call[2], call[into], call[3], handle, on)
            gpu_op.reduce_sum_new(call[1], call[into + 1], call[4], handle, on)

    def hold_all():
        graph, on = ctypes.c_void_p(), stream
        if recorded:
            on = new_cell(2)
            check_call(_LIB.TfStepRecordBegin(ctypes.byref(graph), on, stream))
        before = gpu_op.launch_count()
        gpu_op.hold_products(True)
        run(7, on)
        gpu_op.hold_products(False)
        held = gpu_op.launch_count()
        gpu_op.launch_held(on)
        launches = gpu_op.launch_count() - held
        if recorded:
            check_call(_LIB.TfStepRecordEnd(ctypes.byref(graph), 1))
            before = gpu_op.launch_count()
            check_call(_LIB.TfStepReplay(graph, None, 0, ctypes.c_float(0), ctypes.c_float(0), None, 0, stream))
            gpu_op.device_synchronize()
            launches = gpu_op.launch_count() - before
            check_call(_LIB.TfStepGraphFree(graph))
        for call in calls:
            for apart, together in zip(call[5:7], call[7:9]):
                np.testing.assert_array_equal(together.asnumpy(), apart.asnumpy())
                together[:] = np.full(together.shape, np.nan, np.float32)
        return launches
    try:
        gpu_op.set_memory_limit(1)
        assert isinstance(nd.empty((1 << 30,), ctx), int)          # the scratch of every stream goes back
        gpu_op.set_memory_limit(0)
        run(5, stream)
        gpu_op.device_synchronize()
        gpu_op.release_cached_memory()
        gpu_op.set_memory_limit(sum(gpu_op.allocator_stats()) + (recorded << 20))        # a recording needs a little for itself
        in_parts = hold_all()
        gpu_op.set_memory_limit(0)
        assert hold_all() < in_parts
    finally:
        gpu_op.drop_held()
        gpu_op.set_memory_limit(0)
        gpu_op.set_tensor_arithmetic("3xfp16")


# what waits was called on one stream and goes there; calls on another stream do not wait, and do not overtake it
def test_products_wait_on_their_own_stream(lib_path):
    from tinyflow_b200 import gpu_op, ndarray as nd
    ctx, rng = nd.gpu(0), np.random.RandomState(2)
    one, two = gpu_op.create_cudaStream(), gpu_op.create_cudaStream()
    handle = gpu_op.create_cudnnHandle(one)
    calls = []
    for N, C, H, W, K, R, S, u in (LAYERS[9], LAYERS[4]):
        out, cell = gpu_op.convolution_2d_forward_get_out_shape((N, C, H, W), (K, C, R, S), "NCHW", "SAME", u, u)
        x, other, w, dy = (nd.array(rng.randn(*shape).astype(np.float32), ctx) for shape in ((N, C, H, W), (N, C, H, W), (K, C, R, S), out))
        calls.append([x, dy, w, cell, other] + [nd.array(np.full((K, C, R, S), np.nan, np.float32), ctx) for _ in range(3)])
    wgrad = lambda call, x, out, on: gpu_op.convolution_backward_filter(x, call[1], call[2], out, call[3], handle, on)       # noqa: E731
    try:
        for call in calls:
            wgrad(call, call[0], call[5], one)
        gpu_op.device_synchronize()
        gpu_op.hold_products(True)
        wgrad(calls[0], calls[0][0], calls[0][6], one)
        wgrad(calls[1], calls[1][0], calls[1][6], two)             # launched at once
        gpu_op.launch_held(two)
        gpu_op.device_synchronize()
        assert np.isnan(calls[0][6].asnumpy()).all()
        np.testing.assert_array_equal(calls[1][6].asnumpy(), calls[1][5].asnumpy())
        wgrad(calls[0], calls[0][4], calls[0][7], two)             # packs another input for the same plan, behind what still reads the first
        gpu_op.hold_products(False)
        gpu_op.device_synchronize()
        np.testing.assert_array_equal(calls[0][6].asnumpy(), calls[0][5].asnumpy())
        assert not np.isnan(calls[0][7].asnumpy()).any() and not np.array_equal(calls[0][7].asnumpy(), calls[0][5].asnumpy())
        gpu_op.launch_held(one)
    finally:
        gpu_op.drop_held()


def test_a_released_descriptor_lets_what_waits_go_first(lib_path):
    from tinyflow_b200 import gpu_op, ndarray as nd
    ctx, stream, rng = nd.gpu(0), gpu_op.create_cudaStream(), np.random.RandomState(4)
    handle = gpu_op.create_cudnnHandle(stream)
    N, C, H, W, K, R, S, u = LAYERS[4]
    out, cell = gpu_op.convolution_2d_forward_get_out_shape((N, C, H, W), (K, C, R, S), "NCHW", "SAME", u, u)
    x, w, dy = (nd.array(rng.randn(*shape).astype(np.float32), ctx) for shape in ((N, C, H, W), (K, C, R, S), out))
    apart, waits = (nd.array(np.full((K, C, R, S), np.nan, np.float32), ctx) for _ in range(2))
    try:
        gpu_op.convolution_backward_filter(x, dy, w, apart, cell, handle, stream)
        gpu_op.hold_products(True)
        gpu_op.convolution_backward_filter(x, dy, w, waits, cell, handle, stream)
        gpu_op.hold_products(False)
        gpu_op.release_descriptor(cell)
        # arrays of the packs' sizes, in whose place they come
        rows = N * H * W
        kept = [nd.array(np.full(rows * c // 2, np.nan, np.float32), ctx) for c in (C, K) for _ in range(4)]
        gpu_op.launch_held(stream)
        np.testing.assert_array_equal(waits.asnumpy(), apart.asnumpy())
        assert len(kept) == 8
    finally:
        gpu_op.drop_held()


def test_what_waits_goes_before_its_stream(lib_path):
    from tinyflow_b200 import gpu_op, ndarray as nd
    ctx, stream, later, rng = nd.gpu(0), gpu_op.create_cudaStream(), gpu_op.create_cudaStream(), np.random.RandomState(8)
    handle = gpu_op.create_cudnnHandle(later)
    N, C, H, W, K, R, S, u = LAYERS[4]
    out, cell = gpu_op.convolution_2d_forward_get_out_shape((N, C, H, W), (K, C, R, S), "NCHW", "SAME", u, u)
    x, w, dy = (nd.array(rng.randn(*shape).astype(np.float32), ctx) for shape in ((N, C, H, W), (K, C, R, S), out))
    sums = gpu_op.reduce_sum_get_cudnnlist(*gpu_op.reduce_sum_get_real_shape(out, (K,), "NCHW"), "NCHW", handle)
    apart, waits = ([nd.array(np.full(s, np.nan, np.float32), ctx) for s in ((K, C, R, S), (K,))] for _ in range(2))

    def run(into, on):
        gpu_op.convolution_backward_filter(x, dy, w, into[0], cell, handle, on)
        gpu_op.reduce_sum_new(dy, into[1], sums, handle, on)
    try:
        run(apart, later)
        gpu_op.device_synchronize()
        gpu_op.hold_products(True)
        run(waits, stream)
        gpu_op.destroy_cudaStream(stream)
        again = [nd.array(np.full(a.shape, np.nan, np.float32), ctx) for a in apart]
        run(again, later)                                          # waits in its turn
        gpu_op.hold_products(False)
        gpu_op.launch_held(later)
        for got in (waits, again):
            for a, b in zip(got, apart):
                np.testing.assert_array_equal(a.asnumpy(), b.asnumpy())
    finally:
        gpu_op.drop_held()


# called before the caller's own capture begins, launched inside: the graph names nothing that is gone when it is replayed
def test_what_waits_is_launched_in_a_capture(lib_path):
    import ctypes
    import torch
    from tinyflow_b200 import gpu_op, ndarray as nd
    ctx, rng = nd.gpu(0), np.random.RandomState(9)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    stream = ctypes.pointer(ctypes.c_void_p(side.cuda_stream))
    handle = gpu_op.create_cudnnHandle(stream)
    calls = []
    for N, C, H, W, K, R, S, u in LAYERS[1:5] + DIRECT[:2]:           # (tiles of 96 columns, LAYERS[0], do not wait)
        out, cell = gpu_op.convolution_2d_forward_get_out_shape((N, C, H, W), (K, C, R, S), "NCHW", "VALID" if u > 1 else "SAME", u, u)
        x, w, dy = (nd.array(rng.randn(*shape).astype(np.float32), ctx) for shape in ((N, C, H, W), (K, C, R, S), out))
        calls.append((x, dy, w, cell) + tuple(nd.array(np.full((K, C, R, S), np.nan, np.float32), ctx) for _ in range(2)))
    try:
        for call in calls:
            gpu_op.convolution_backward_filter(*call[:3], call[4], call[3], handle, stream)
        before = gpu_op.launch_count()
        gpu_op.hold_products(True)
        for call in calls:
            gpu_op.convolution_backward_filter(*call[:3], call[5], call[3], handle, stream)
        gpu_op.hold_products(False)
        assert gpu_op.launch_count() == before
        gpu_op.device_synchronize()
        with torch.cuda.graph(graph, stream=side):
            gpu_op.launch_held(stream)
        for _ in range(3):
            for call in calls:
                call[5][:] = np.full(call[5].shape, np.nan, np.float32)
            graph.replay()
            torch.cuda.synchronize()
            for call in calls:
                np.testing.assert_array_equal(call[5].asnumpy(), call[4].asnumpy())
    finally:
        gpu_op.drop_held()


def _half_way(monkeypatch, ex, node, feed):
    """A step that ends with an error at `node`, behind gradients that wait."""
    import random
    compute, draws, waiting = type(node.op).compute, random.getstate(), []

    def stop(op, n, *rest):
        if n is node:
            raise ArithmeticError("stopped")
        return compute(op, n, *rest)
    with monkeypatch.context() as m:
        from tinyflow_b200 import gpu_op
        m.setattr(type(node.op), "compute", stop)
        m.setattr(gpu_op, "launch_held", lambda stream: waiting.append("launched"))
        with pytest.raises(ArithmeticError):
            ex.run(feed)
    random.setstate(draws)
    assert not waiting


# a step that an operator stops: what waits is forgotten, and the step after it is the one that would have come
@pytest.mark.parametrize("name", ["inceptionv3", "lenet5", "mlp"])
def test_a_step_that_fails_leaves_nothing_behind(lib_path, monkeypatch, name):
    from tinyflow_b200 import gpu_op

    def fail(step, model, ex, feed, x):
        if step not in (2, 5):
            return
        last = [n for n in ex.topo_order if n in ex._patient]
        between = [n for n in ex.topo_order if n not in ex._patient and n.index > last[len(last) // 2].index and n.inputs and not n.issgd and type(n.op).__name__ != "AddOp"]
        _half_way(monkeypatch, ex, between[0], feed)
        from tinyflow_b200 import ndarray as nd
        a, b, c = (nd.array(np.full(s, v, np.float32), nd.gpu(0)) for s, v in (((100, 120), 1), ((100, 84), 1), ((120, 84), np.nan)))
        gpu_op.matrix_multiply(a, True, b, False, c, ex.cublasHandle, ex.cudaStream)       # the switch is off again
        gpu_op.device_synchronize()
        assert not np.isnan(c.asnumpy()).any()
    want = _train(monkeypatch, False, BUILDS[name], "sgd")
    got = _train(monkeypatch, False, BUILDS[name], "sgd", between=fail)
    _same(got, want)


def _shared_filter(m):
    """One filter and one bias that two layers share: their gradients are summed before the update reads them."""
    from tinyflow_b200 import autodiff as ad
    X, y_, w0, w, b, d = (ad.Placeholder("X"), ad.Placeholder("y_")) + tuple(ad.Variable(n) for n in ("w0", "w", "b", "d"))
    h = ad.activation_forward_op(ad.convolution_2d_forward_op(X, w0, "NCHW", "SAME", 1, 1), "NCHW", "relu")
    for _ in range(2):
        h = ad.activation_forward_op(ad.conv2withbias(h, w, b, "NCHW", "SAME", 1, 1), "NCHW", "relu")
    y = ad.matmul_op(ad.flatten_op(h), d)
    return m.Model("shared", X, y_, ad.softmaxcrossentropy_op(y, y_), y, {w0: (32, 16, 3, 3), w: (32, 32, 3, 3), b: (32,), d: (32 * 81, 10)}, (40, 16, 9, 9), (40, 10))


def test_a_gradient_that_something_reads_does_not_wait(lib_path, monkeypatch):
    from tinyflow_b200 import autodiff as ad, gpu_op, models
    ex = ad.Executor(*(lambda m: (m.loss, m.y))(_shared_filter(models)), 0.01, None, None, None, optimizer="sgd")
    gradients = [n for n in ex.topo_order if ex._is_parameter_gradient(n)]
    assert sorted(n in ex._patient for n in gradients) == [False] * 4 + [True] * 2        # w and b twice each; w0 and d
    got = _train(monkeypatch, True, _shared_filter, "sgd")
    with monkeypatch.context() as m:
        m.setattr(gpu_op, "hold_products", lambda on: None)
        want = _train(monkeypatch, False, _shared_filter, "sgd")
    _same(got, want)


# more than the stages that are launched together at the latest: some go while the rest is still being called
def test_much_work_does_not_wait_for_the_end(lib_path):
    from tinyflow_b200 import gpu_op, ndarray as nd
    ctx, stream, rng = nd.gpu(0), gpu_op.create_cudaStream(), np.random.RandomState(6)
    handle = gpu_op.create_cudnnHandle(stream)
    N, C, H, W, K = 16, 2048, 24, 24, 64                         # 16 tiles of 144 stages
    out, cell = gpu_op.convolution_2d_forward_get_out_shape((N, C, H, W), (K, C, 1, 1), "NCHW", "SAME", 1, 1)
    x, w, dy = (nd.array(rng.randn(*shape).astype(np.float32), ctx) for shape in ((N, C, H, W), (K, C, 1, 1), out))
    apart = nd.empty((K, C, 1, 1), ctx)
    gpu_op.convolution_backward_filter(x, dy, w, apart, cell, handle, stream)
    results = [nd.array(np.full((K, C, 1, 1), np.nan, np.float32), ctx) for _ in range(80)]          # 184,320 tile stages; 148 SMs take 151,552
    try:
        gpu_op.hold_products(True)
        counts = [gpu_op.launch_count()]
        for r in results:
            gpu_op.convolution_backward_filter(x, dy, w, r, cell, handle, stream)
            counts.append(gpu_op.launch_count())
        gpu_op.hold_products(False)
        assert sum(b > a for a, b in zip(counts, counts[1:])) == 1
        gpu_op.launch_held(stream)
        assert gpu_op.launch_count() > counts[-1]
    finally:
        gpu_op.drop_held()
    for r in results:
        np.testing.assert_array_equal(r.asnumpy(), apart.asnumpy())
