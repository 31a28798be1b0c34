"""Performance cases: training steps through the public entry points.

A user of this framework builds a graph (``models`` or their own, with the ``ad`` operators), gives its loss to an
``ad.Executor`` and calls ``Executor.run`` once per mini-batch.  One pass here is that call: forward, backward and the
update of every parameter.  The outputs are the loss, all updated parameters and, with Adam, both moments.

The executor (graph, descriptors, streams) is kept from mini-batch to mini-batch and from one set of weights to the
next, as a training script keeps it; inputs, labels, weights and moments are what a pass is given.
"""
from __future__ import annotations

import gc
import queue
import random

import numpy as np
import torch

from tinyflow_b200 import autodiff as ad
from tinyflow_b200 import gpu_op, memory_plan, models, ndarray

# Dropout rates of the benchmark.  The softmax cross-entropy of the MLP and LeNet graphs has gradients summed over the
# batch, so their SGD rate is divided by it; the others' gradients are divided by batch * classes, and their rate is the
# benchmark's 0.01 at its 1000 classes.
DROPOUT = {"vgg16": 0.5, "resnet50": 0.5, "inceptionv3": 0.8, "inceptionv4": 0.8, "densenet121": 0.2}
SUMMED_LOSS = ("mlp", "lenet5")
MAX_BATCH_PIXELS = 64 * 224 * 224


def _case(name, model, batch, image=0, classes=1000, width=0, optimizer="sgd", arithmetic="3xfp16", plan="none"):
    c = {"model": model, "batch": batch, "image": image, "classes": classes, "width": width, "optimizer": optimizer,
         "arithmetic": arithmetic, "plan": plan}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest step: a small fully connected net on a small batch, with the executor's default optimiser
        _case("mlp b64 adam", "mlp", 64, classes=10, width=256, optimizer="adam"),
        # MNIST perceptron of the benchmark
        _case("mlp b1000", "mlp", 1000, classes=10, width=256),
        # LeNet-5 of the benchmark: channel counts too small for the tensor cores
        _case("lenet5 b256", "lenet5", 256, image=28, classes=10),
        # the smallest batch the reference's memory study trains: a deep graph of small kernels
        _case("inceptionv3 b2 adam", "inceptionv3", 2, image=299, optimizer="adam"),
        # ragged: odd batch, image and class counts
        _case("vgg16 b7 i97", "vgg16", 7, image=97, classes=101),
        _case("resnet50 b19 i161", "resnet50", 19, image=161, classes=37),
        # the benchmark's convolutional workloads at their own sizes
        _case("resnet50 b64", "resnet50", 64, image=224),
        _case("vgg16 b64", "vgg16", 64, image=224),
        _case("inceptionv3 b32", "inceptionv3", 32, image=299),
        _case("densenet121 b32", "densenet121", 32, image=224),
        # the other arithmetic of the tensor path
        _case("inceptionv4 b16 3xtf32", "inceptionv4", 16, image=299, arithmetic="3xtf32"),
        # a step under a swap plan: convolution inputs travel to pinned host memory and back
        _case("inceptionv3 b32 swap", "inceptionv3", 32, image=299, plan="vdnn-conv"),
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    model = rng.choice(("mlp", "lenet5", "vgg16", "resnet50", "inceptionv3", "densenet121", "inceptionv4"))
    optimizer = rng.choice(("sgd", "adam"))
    if model == "mlp":
        return _case(None, model, _log_int(rng, 16, 4096), classes=_log_int(rng, 5, 300), width=_log_int(rng, 32, 1500), optimizer=optimizer)
    if model == "lenet5":
        return _case(None, model, _log_int(rng, 8, 1024), image=28, classes=_log_int(rng, 5, 100), optimizer=optimizer)
    if model == "vgg16":
        image = rng.randint(64, 224)
    elif model == "inceptionv3":
        image = rng.randint(107, 299)
    elif model == "inceptionv4":
        image = rng.randint(123, 299)
    else:                                     # the residual and dense graphs pool over image // 32 positions at the end
        image = 32 * rng.randint(3, 7) + rng.randint(0, 1)
        image = min(image, 224)
    # layers normalised over the batch need one that is large enough for their statistics
    smallest = {"resnet50": 16, "densenet121": 16, "vgg16": 6}
    largest = min(64, MAX_BATCH_PIXELS // (image * image))
    if model in smallest:
        optimizer = "sgd"                     # Adam's first steps follow the signs of gradients that batch statistics make noisy
    return _case(None, model, _log_int(rng, smallest.get(model, 1), largest), image=image, classes=_log_int(rng, 10, 1000), optimizer=optimizer,
                 arithmetic="3xtf32" if rng.random() < 0.15 else "3xfp16")


def _model(case):
    kind = case["model"]
    if kind == "mlp":
        m = models.mlp(batch=case["batch"], sizes=(784, case["width"], 100, case["classes"]))
    elif kind == "lenet5":
        m = models.lenet5(batch=case["batch"], classes=case["classes"])
    else:
        m = models.BUILDERS[kind](batch=case["batch"], classes=case["classes"], image=case["image"])
    m.set_dropout(DROPOUT.get(kind, 0.0))
    return m


def _build(case):
    """The graph and its executor, with the plan (if any) waiting in the control queue."""
    model = _model(case)
    control = queue.Queue()
    if case["optimizer"] == "adam":
        rate = 0.00001
    else:
        rate = 0.1 / case["batch"] if case["model"] in SUMMED_LOSS else 0.00001 * case["classes"]
    ex = ad.Executor(model.loss, model.y, rate, control, None, None, optimizer=case["optimizer"])
    shapes = {model.X: model.input_shape, model.y_: model.label_shape}
    for node, shape in model.param_shapes.items():
        shapes[node] = tuple(shape)
        for moment in ex.Variable_node_to_mv.get(node, ()):
            shapes[moment] = tuple(shape)
    ex.infer_shape(shapes)
    if case["plan"] != "none":
        control.put(memory_plan.vdnn_plan(ex, policy=case["plan"].split("-")[1]))
    return model, ex


_kept = {}       # the executor of the model that is being trained


def _executor(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _kept:
        if _kept:                            # another model: the memory of the one before goes back
            _kept.clear()
            gc.collect()
            gpu_op.release_cached_memory()
        _kept[key] = _build(case)
    return _kept[key]


class _Shared(object):
    """Device memory for torch: float32, contiguous; ``owner`` keeps it alive."""

    def __init__(self, pointer, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": tuple(shape), "typestr": "<f4", "version": 2}


def _tensor(pointer, shape, owner):
    return torch.as_tensor(_Shared(pointer, shape, owner), device="cuda")


def _view(pointer, shape):
    """An NDArray over memory that something else owns."""
    import ctypes
    c = ndarray.DLArray()
    dims = (ctypes.c_int64 * len(shape))(*shape)
    c.data, c.ctx, c.ndim, c.shape = pointer, ndarray.gpu(0), len(shape), ctypes.cast(dims, ctypes.POINTER(ctypes.c_int64))
    arr = ndarray.NDArray(ctypes.pointer(c))
    arr.is_freed = True                      # its owner frees it
    return arr


def _put(source, target):
    """Copies a torch tensor into an NDArray through the library, as uploads go."""
    _view(source.data_ptr(), tuple(source.shape)).copyto(target)


def _size(shape):
    n = 1
    for d in shape:
        n *= int(d)
    return n


_ALIGN = 128      # floats between the starts of two parameters in the flat buffer: a multiple of 512 bytes, as arrays of their own have


def _flat(shapes, fill):
    """One array that holds a tensor of each shape, and the NDArrays over its parts."""
    offsets, total = [], 0
    for shape in shapes:
        offsets.append(total)
        total += -(-_size(shape) // _ALIGN) * _ALIGN
    whole = ndarray.empty((total,), ndarray.gpu(0))
    gpu_op.array_set(whole, 0.0, None)
    parts = [_view(whole.data_ptr + 4 * o, shape) for o, shape in zip(offsets, shapes)]
    for part, shape in zip(parts, shapes):
        _put(fill(shape), part)
    return whole, parts, _tensor(whole.data_ptr, (total,), whole)


def prepare(case, seed):
    gpu_op.set_tensor_arithmetic(case["arithmetic"])
    model, ex = _executor(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)

    def weight(shape):                       # He-normal weights, zero biases
        if len(shape) == 1:
            return torch.zeros(shape, device="cuda")
        fan_in = _size(shape[1:]) if len(shape) == 4 else shape[0]
        return torch.randn(shape, generator=gen, device="cuda").mul_((2.0 / fan_in) ** 0.5)

    shapes = [tuple(int(d) for d in s) for s in model.param_shapes.values()]
    whole, parts, view = _flat(shapes, weight)
    feed, out, held = dict(zip(model.param_shapes, parts)), {"weights": view}, [whole]
    if case["optimizer"] == "adam":
        for k, name in ((0, "m"), (1, "v")):
            whole, parts, view = _flat(shapes, lambda shape: torch.zeros(shape, device="cuda"))
            feed.update(zip((ex.Variable_node_to_mv[v][k] for v in model.param_shapes), parts))
            out[name] = view
            held.append(whole)
    if case["model"] in SUMMED_LOSS:
        x = torch.rand(model.input_shape, generator=gen, device="cuda")
    else:
        x = torch.randn(model.input_shape, generator=gen, device="cuda")
    labels = torch.randint(0, model.label_shape[1], (model.label_shape[0],), generator=gen, device="cuda")
    y = torch.zeros(model.label_shape, device="cuda")
    y.scatter_(1, labels[:, None], 1.0)
    for node, t in ((model.X, x), (model.y_, y)):
        feed[node] = ndarray.empty(tuple(t.shape), ndarray.gpu(0))
        _put(t, feed[node])
    random.seed(seed)                        # dropout draws its seeds from here
    ex.b1t[0], ex.b2t[0] = ex.b1, ex.b2      # training starts anew
    gpu_op.device_synchronize()
    return {"executor": ex, "feed": feed, "out": out, "held": held}


def run(state):
    loss, _ = state["executor"].run(state["feed"])
    return dict(state["out"], loss=_tensor(loss.data_ptr, loss.shape, loss))


def work(case):
    """Multiply-adds of every matrix product and convolution (forward, input gradient, filter gradient), two operations
    each; the mini-batch read, parameters (and moments) read and written once."""
    model, ex = _build(case)
    shape = ex.node_to_shape_map
    flops = 0
    for node in ex.topo_order:
        kind = type(node.op).__name__
        if kind == "MatMulOp":
            a = shape[node.inputs[0]]
            flops += 2 * _size(shape[node]) * (a[0] if node.matmul_attr_trans_A else a[1])
        elif kind in ("Convolution2DForwardOp", "Convolution2DBackwardOp"):
            filt = shape[node.inputs[1]]
            y = shape[node] if kind == "Convolution2DForwardOp" else shape[node.inputs[2]]
            flops += 2 * _size(y) * _size(filt[1:])
    params = sum(_size(s) for s in model.param_shapes.values())
    tensors = 3 if case["optimizer"] == "adam" else 1
    floats = _size(model.input_shape) + _size(model.label_shape) + 2 * tensors * params + 1
    return {"bytes": 4 * floats, "flops": flops}


def tolerance(case):
    """What exact-fp32 kernels, 3xFP16 and 3xTF32 differ by, over two steps: all of them are fp32 arithmetic with other
    orders of summation.  Deep graphs amplify that rounding: batch statistics of single activations in ResNet-50, and with
    Adam the moments (the gradients themselves) behind ReLUs and maxima that flip near ties."""
    if case["model"] == "resnet50":
        return {"rel": 5e-3, "max": 0.2}
    if case["optimizer"] == "adam" and case["model"] not in SUMMED_LOSS:
        return {"rel": 1e-2, "max": 0.95}
    return {"rel": 3e-5, "max": 1e-3}
