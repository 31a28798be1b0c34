"""Recorded steps: a replay has to give the bits the ordinary calls give, whatever the caller does between steps."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 9


def _train(monkeypatch, recorded, build, optimizer, between=None, fresh_batch=False):
    from tinyflow_b200 import autodiff as ad, gpu_op, models, ndarray, step_graph
    monkeypatch.setattr(step_graph, "ENABLED", recorded)
    random.seed(3)
    model = build(models)
    ex = ad.Executor(model.loss, model.y, 0.001, None, None, None, optimizer=optimizer)
    ctx = ndarray.gpu(0)
    feed = {n: ndarray.array(v, ctx) for n, v in model.init_params(seed=5).items()}
    for var in list(feed):
        for moment in ex.Variable_node_to_mv.get(var, ()):
            feed[moment] = ndarray.array(np.zeros(model.param_shapes[var], np.float32), ctx)
    all_feeds = dict(feed)
    X, Y = models.synthetic_batch(model, seed=8)
    x, y = ndarray.array(X, ctx), ndarray.array(Y, ctx)
    losses = []
    for step in range(STEPS):
        if fresh_batch:
            x = ndarray.array(np.roll(X, step, axis=0), ctx)
        all_feeds[model.X], all_feeds[model.y_] = x, y
        if between:
            between(step, model, ex, all_feeds, x)
        loss, _ = ex.run(all_feeds)
        losses.append(loss)
    gpu_op.device_synchronize()
    replayed = any(f.recording or any(b.recording for b in f.batches.values()) for f in ex._recordings.sets.values())
    return [v.asnumpy() for v in losses], {n.name: v.asnumpy() for n, v in all_feeds.items() if n.isw == 1}, replayed


def _same(a, b):
    for la, lb in zip(a[0], b[0]):
        np.testing.assert_array_equal(la, lb)
    for name in a[1]:
        np.testing.assert_array_equal(a[1][name], b[1][name], err_msg=name)


BUILDS = {
    "mlp": lambda m: m.mlp(batch=33),
    "lenet5": lambda m: m.lenet5(batch=9),
    "vgg16": lambda m: m.vgg16(batch=8, classes=20, image=32),                  # dropout: new seeds every step
    "resnet50": lambda m: m.resnet50(batch=16, classes=10, image=64),           # the fused and the held-back calls
    "inceptionv3": lambda m: m.inceptionv3(batch=2, classes=10, image=107),
}


@pytest.mark.parametrize("optimizer", ["sgd", "adam"])
@pytest.mark.parametrize("name", sorted(BUILDS))
def test_a_replayed_step_has_the_bits_of_the_ordinary_one(lib_path, monkeypatch, name, optimizer):
    want = _train(monkeypatch, False, BUILDS[name], optimizer)
    got = _train(monkeypatch, True, BUILDS[name], optimizer)
    assert got[2] and not want[2]
    _same(got, want)


def _overwrite_inputs(step, model, ex, feed, x):
    x[:] = np.random.RandomState(step).rand(*x.shape).astype(np.float32)


def _overwrite_a_parameter(step, model, ex, feed, x):
    if step in (5, 7):
        node = next(iter(model.param_shapes))
        feed[node][:] = (0.5 if step == 5 else 40.0) * feed[node].asnumpy()


def _change_the_rate(step, model, ex, feed, x):
    if step == 6:
        for node in ex.optimizer_nodes:
            node.learning_rate = 0.01


def _overwrite_inputs_late(step, model, ex, feed, x):
    if step >= 5:                                                    # the recording is made on a batch that nothing has rewritten
        _overwrite_inputs(step, model, ex, feed, x)


_held = []


def _hold_values(step, model, ex, feed, x):
    if step == 5:
        _held.append((ex.value_of(model.y), ex.value_of(model.y).asnumpy()))
    if step == 8:
        view, copy = _held.pop()
        np.testing.assert_array_equal(view.asnumpy(), copy)          # later steps left it alone


def _hold_and_write_gradients(step, model, ex, feed, x):
    if step in (4, 6):
        views = [ex.value_of(n) for n in ex.topo_order if n.name in ("+", "Zeroslike", "Oneslike")]
        copies = [v.asnumpy() for v in views]
        if step == 4:
            _held.extend(zip(views, copies))
        for n in ex.topo_order:
            if n.name == "Zeroslike":
                ex.value_of(n)[:] = np.full(ex.value_of(n).shape, 3.0, np.float32)
    if step == 8:
        for view, copy in _held:
            if copy.any():                                           # (the zeros were overwritten above)
                np.testing.assert_array_equal(view.asnumpy(), copy)
        del _held[:]


@pytest.mark.parametrize("between", [_overwrite_inputs, _hold_and_write_gradients, _overwrite_a_parameter, _change_the_rate, _hold_values])
@pytest.mark.parametrize("name", ["mlp", "resnet50"])
def test_what_a_caller_does_between_steps_reaches_the_replay(lib_path, monkeypatch, name, between):
    _same(_train(monkeypatch, True, BUILDS[name], "sgd", between), _train(monkeypatch, False, BUILDS[name], "sgd", between))


# Graphs whose first node is a tensor-path convolution: it packs its input, and the pack is only as good as the batch in it.
CONV_FIRST = {"vgg16": BUILDS["vgg16"], "inceptionv3": lambda m: m.inceptionv3(batch=8, classes=10, image=107)}


@pytest.mark.parametrize("name", sorted(CONV_FIRST))
def test_a_batch_rewritten_after_the_recording_reaches_the_replay(lib_path, monkeypatch, name):
    got = _train(monkeypatch, True, CONV_FIRST[name], "sgd", _overwrite_inputs_late)
    assert got[2]
    _same(got, _train(monkeypatch, False, CONV_FIRST[name], "sgd", _overwrite_inputs_late))


def _in_turn(order, held_from=None):
    """Feeds resident batch arrays in the order given by letters; from step `held_from` on the caller holds a view."""
    arrays = {}

    def between(step, model, ex, feed, x):
        from tinyflow_b200 import ndarray
        if step == 0:
            arrays.clear()
            for k, letter in enumerate(sorted(set(order))):
                arrays[letter] = ndarray.array(np.roll(x.asnumpy() * (1.0 + k), k, axis=0), ndarray.gpu(0))
        if step == held_from:
            _held.append(ex.value_of(model.y))
        if step == STEPS - 1:
            del _held[:]
        feed[model.X] = arrays[order[step]]
    return between


@pytest.mark.parametrize("order, held_from", [("AAAABAABA", None), ("AAABBBABA", 7), ("ABABABABA", 7), ("AAAABABAB", 6)])
@pytest.mark.parametrize("name", sorted(CONV_FIRST))
def test_resident_batches_in_turn(lib_path, monkeypatch, name, order, held_from):
    got = _train(monkeypatch, True, CONV_FIRST[name], "sgd", _in_turn(order, held_from))
    assert got[2]
    _same(got, _train(monkeypatch, False, CONV_FIRST[name], "sgd", _in_turn(order, held_from)))


def _column_sums_model(m):
    """A loss over ReduceSumAxisZero, which the reference runs without a stream."""
    from tinyflow_b200 import autodiff as ad
    X, y_, W = ad.Placeholder("X"), ad.Placeholder("y_"), ad.Variable("W")
    y = ad.matmul_op(X, W)
    sums = ad.reducesumaxiszero_op(ad.mul_op(y, y_))
    loss = ad.reduce_sum_op(ad.mul_op(sums, sums))
    return m.Model("column sums", X, y_, loss, y, {W: (20, 7)}, (33, 20), (33, 7))


@pytest.mark.parametrize("optimizer", ["sgd", "adam"])
def test_operators_without_a_stream_are_part_of_the_recording(lib_path, monkeypatch, optimizer):
    got = _train(monkeypatch, True, _column_sums_model, optimizer, _overwrite_inputs)
    assert got[2]
    _same(got, _train(monkeypatch, False, _column_sums_model, optimizer, _overwrite_inputs))


@pytest.mark.parametrize("name", ["mlp", "vgg16"])
def test_new_mini_batch_arrays_every_step(lib_path, monkeypatch, name):
    want = _train(monkeypatch, False, BUILDS[name], "sgd", fresh_batch=True)
    got = _train(monkeypatch, True, BUILDS[name], "sgd", fresh_batch=True)
    assert got[2]
    _same(got, want)


def test_a_step_that_cannot_be_recorded_says_so_and_runs(lib_path, monkeypatch):
    from tinyflow_b200 import autodiff as ad

    class HostCopyOp(ad.Op):
        name = "HostCopy"

        def __call__(self, node):
            return self._node([node])

        def compute(self, node, input_vals, output_val, cudnnHandle, cublasHandle, cudaStream, use_numpy=False):
            output_val[:] = input_vals[0].asnumpy()

        def gradient(self, node, output_grad):
            return [output_grad]

        def infer_shape(self, node, input_shapes, cudnnHandle):
            return input_shapes[0]

    def build(m):
        X, y_, W = ad.Placeholder("X"), ad.Placeholder("y_"), ad.Variable("W")
        y = HostCopyOp()(ad.matmul_op(X, W))
        return m.Model("host copy", X, y_, ad.l2loss_op(y, y_), y, {W: (20, 7)}, (33, 20), (33, 7))
    want = _train(monkeypatch, False, build, "sgd", _overwrite_inputs)
    with pytest.warns(RuntimeWarning, match="could not be recorded.*host waits") as said:
        got = _train(monkeypatch, True, build, "sgd", _overwrite_inputs)
    assert len(said) == 2 and "no further attempts" in str(said[1].message) and not got[2]
    _same(got, want)


def test_another_thread_waits_for_the_device_while_a_step_is_recorded(lib_path, monkeypatch):
    """Neither the recordings nor the waits fail, whichever library waits; the waiting thread shares no array with the step."""
    import threading
    import torch
    from tinyflow_b200 import gpu_op
    want = _train(monkeypatch, False, BUILDS["lenet5"], "sgd", fresh_batch=True)
    stop, errors, waits = threading.Event(), [], []

    def wait(synchronize):
        while not stop.is_set():
            try:
                synchronize()
                waits.append(1)
            except Exception as e:                                   # noqa: BLE001
                errors.append(e)
    threads = [threading.Thread(target=wait, args=(f,)) for f in (gpu_op.device_synchronize, torch.cuda.synchronize)]
    for t in threads:
        t.start()
    try:
        got = [_train(monkeypatch, True, BUILDS["lenet5"], "sgd", fresh_batch=True) for _ in range(8)]
    finally:
        stop.set()
        for t in threads:
            t.join()
    assert not errors and waits
    for run in got:
        assert run[2]
        _same(run, want)


def test_a_recording_packs_filters_for_its_own_plans_only(lib_path, monkeypatch):
    """Batches of other sizes build other plans; a step recorded after them has the launches it had before them."""
    from tinyflow_b200 import autodiff as ad, gpu_op, models, ndarray, step_graph
    monkeypatch.setattr(step_graph, "ENABLED", True)
    model = models.resnet50(batch=16, classes=10, image=64)          # 53 filters; one launch packs up to 128
    ex = ad.Executor(model.loss, model.y, 0.001, None, None, None, optimizer="sgd")
    ctx = ndarray.gpu(0)
    feed = {n: ndarray.array(v, ctx) for n, v in model.init_params(seed=5).items()}
    X, Y = models.synthetic_batch(model, seed=8)
    launches = []
    for batch in (16, 15, 14, 16):
        feed[model.X], feed[model.y_] = ndarray.array(X[:batch], ctx), ndarray.array(Y[:batch], ctx)
        for _ in range(5):
            before = gpu_op.launch_count()
            ex.run(feed)
        assert any(b.recording for f in ex._recordings.sets.values() for b in f.batches.values())
        launches.append(gpu_op.launch_count() - before)
    gpu_op.device_synchronize()
    assert launches[0] == launches[-1]


@pytest.mark.parametrize("name", ["vgg16", "resnet50", "inceptionv3"])
def test_filters_packed_ahead_have_the_bits_of_filters_packed_one_by_one(lib_path, monkeypatch, name):
    from tinyflow_b200 import gpu_op
    ahead = _train(monkeypatch, False, BUILDS[name], "sgd", _overwrite_a_parameter)
    monkeypatch.setattr(gpu_op, "pack_filters", lambda *args: None)
    _same(ahead, _train(monkeypatch, False, BUILDS[name], "sgd", _overwrite_a_parameter))


@pytest.mark.parametrize("held_by", ["recording", "scratch"])
def test_an_allocation_gets_the_memory_kept_for_later(lib_path, monkeypatch, held_by):
    """Blocks of recordings and scratch of streams are given up before an allocation fails; the steps go on as ever."""
    from tinyflow_b200 import autodiff as ad, gpu_op, ndarray
    ctx, kept = ndarray.gpu(0), []

    class WorkOp(ad.Op):
        name = "Work"

        def __call__(self, node):
            return self._node([node])

        def compute(self, node, input_vals, output_val, cudnnHandle, cublasHandle, cudaStream, use_numpy=False):
            work = ndarray.empty((2 << 20,), ctx)                    # 8 MB for the time of the call
            gpu_op.array_set(work, 1.0, cudaStream)
            gpu_op.matrix_elementwise_multiply_by_const(input_vals[0], 2.0, output_val, cudaStream)

        def gradient(self, node, output_grad):
            return [ad.mul_byconst_op(output_grad, 2.0)]

        def infer_shape(self, node, input_shapes, cudnnHandle):
            return input_shapes[0]

    def build(m):
        if held_by == "scratch":
            return m.mlp(batch=512, sizes=(784, 1500, 1000, 10))     # products on the tensor path: packs of both operands
        X, y_, W = ad.Placeholder("X"), ad.Placeholder("y_"), ad.Variable("W")
        y = WorkOp()(ad.matmul_op(X, W))
        return m.Model("work", X, y_, ad.l2loss_op(y, y_), y, {W: (20, 7)}, (33, 20), (33, 7))

    def between(step, model, ex, feed, x):
        if step == 6 and ex._recordings.sets and not kept:           # recorded in the fourth step
            gpu_op.device_synchronize()
            gpu_op.release_cached_memory()
            gpu_op.set_memory_limit(sum(gpu_op.allocator_stats()))
            try:
                kept.append(ndarray.empty((1 << 20,), ctx))
            finally:
                gpu_op.set_memory_limit(0)
    got = _train(monkeypatch, True, build, "sgd", between)
    assert got[2] and isinstance(kept[0], ndarray.NDArray)           # an int: the bytes that were short
    _same(got, _train(monkeypatch, False, build, "sgd"))


@pytest.mark.parametrize("recorded", [False, True])
@pytest.mark.parametrize("name", ["vgg16", "resnet50", "inceptionv3"])
def test_changes_of_the_batch_size_keep_no_memory(lib_path, monkeypatch, name, recorded):
    """A last, smaller batch comes with every epoch: what the descriptors of one size keep goes back with them."""
    from tinyflow_b200 import autodiff as ad, gpu_op, models, ndarray, step_graph
    monkeypatch.setattr(step_graph, "ENABLED", recorded)
    model = CONV_FIRST.get(name, BUILDS[name])(models)
    ex = ad.Executor(model.loss, model.y, 0.001, None, None, None, optimizer="sgd")
    ctx = ndarray.gpu(0)
    feed = {n: ndarray.array(v, ctx) for n, v in model.init_params(seed=5).items()}
    X, Y = models.synthetic_batch(model, seed=8)
    batches = {n: (ndarray.array(X[:n], ctx), ndarray.array(Y[:n], ctx)) for n in (X.shape[0], X.shape[0] - 3)}
    used = []
    for epoch in range(4):
        for n in sorted(batches, reverse=True):
            feed[model.X], feed[model.y_] = batches[n]
            for _ in range(5):
                ex.run(feed)
        gpu_op.device_synchronize()
        used.append(gpu_op.allocator_stats()[0])
    assert used[3] - used[1] <= 64 * 1024, used


@pytest.mark.parametrize("count", [1, 5, 400])
def test_many_updates_in_one_launch(lib_path, count):
    from tinyflow_b200 import gpu_op, ndarray as nd
    ctx, stream, rng = nd.gpu(0), gpu_op.create_cudaStream(), np.random.RandomState(count)
    sizes = [int(s) for s in rng.choice([1, 3, 4, 127, 4095, 4096, 4097, 20000], size=count)]
    host = [[rng.randn(n).astype(np.float32) for n in sizes] for _ in range(2)] + [[np.abs(rng.randn(n)).astype(np.float32) for n in sizes] for _ in range(2)]
    w, g, m, v = ([nd.array(a, ctx) for a in col] for col in host)
    w2, m2, v2 = ([nd.array(a, ctx) for a in host[k]] for k in (0, 2, 3))
    gpu_op.sgd_update_many(gpu_op.handle_array(w), gpu_op.handle_array(g), 0.1, stream)
    for a, b in zip(w2, g):
        gpu_op.sgd_update(a, b, 0.1, stream)
    for a, b in zip(w, w2):
        np.testing.assert_array_equal(a.asnumpy(), b.asnumpy())
    gpu_op.adam_update_many(*(gpu_op.handle_array(c) for c in (w, m, v, g)), 0.9, 0.999, 0.9, 0.999, 1e-8, 0.01, stream)
    for a, b, c, d in zip(w2, m2, v2, g):
        gpu_op.adam_mv(b, c, d, 0.9, 0.999, stream)
        gpu_op.adam_compute(a, b, c, 0.9, 0.999, 1e-8, 0.01, stream)
    for one, many in ((w, w2), (m, m2), (v, v2)):
        for a, b in zip(one, many):
            np.testing.assert_allclose(a.asnumpy(), b.asnumpy(), rtol=2e-6, atol=1e-7)
