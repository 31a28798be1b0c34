"""Training-step executor; host-side mirror of ``autodiff.Executor`` (autodiff.py:2237-2890).

The executor builds the gradient graph of ``targetloss`` w.r.t. every ``Variable`` it reaches,
appends one optimiser node per parameter, moves each optimiser node to just after the last
reader of its parameter (so updates interleave with the backward pass, autodiff.py:3002-3021)
and then runs the nodes in that order, one C-ABI call per node, allocating each node's output
through ``DLArrayAlloc`` every step exactly as the reference does.

``run(feed_dict)`` takes ``{node: NDArray}`` for the data placeholders, every parameter and (for
Adam) its two moment tensors, and returns ``[loss NDArray, {node: NDArray}]`` where the dict is
the feed dict for the next step (parameters and moments, updated in place).

Memory-plan messages from a scheduler keep the reference's layout
(autodiff.py:2561-2590): ``top_control_queue.put((swap_list, release_list, recompute_list))`` with
``swap_list`` entries ``(tensor_index, start_time_ms, start_node_index, move_to_gpu)`` and release /
recompute entries ``(start_node_index, tensor_index)``.  Swaps run on a worker thread over a side
stream through ``DLArrayCopyFromTo`` into pinned host arrays.
"""
from __future__ import annotations

import queue
import random
import threading
import time
import warnings
import weakref

from . import gpu_op, ndarray, step_graph
from .graph import (AddOp, AdamOp, BNForwardOp, BroadcastToGradientOp, Convolution2DBackwardOp, Convolution2DForwardOp, MatMulOp, OnesLikeOp, Pooling2DForwardOp, SgdOp, Variable, ZerosLikeOp, adam_op, find_topo_sort, get_Variable_node_list, gradients, sgd_op)


def getcomputelist(Variable_node_list, Variable_node_grad_list, b1, b2, b1t, b2t, e, learning_rate):
    """One Adam node per parameter plus its moment Variables (autodiff.py:2985-2999)."""
    computelist, mv, var_to_mv = [], [], {}
    for var, grad in zip(Variable_node_list, Variable_node_grad_list):
        m, v = Variable(var.name + "m"), Variable(var.name + "v")
        mv += [m, v]
        var_to_mv[var] = (m, v)
        node = adam_op(var, m, v, grad, b1, b2, b1t, b2t, e, learning_rate)
        node.issgd = 1
        computelist.append(node)
    return computelist, mv, var_to_mv


def getsgdcomputelist(Variable_node_list, Variable_node_grad_list, learning_rate):
    """One SGD node per parameter (the wiring of TrainExecute.py:315-324)."""
    computelist = []
    for var, grad in zip(Variable_node_list, Variable_node_grad_list):
        node = sgd_op(var, grad, learning_rate)
        node.issgd = 1
        computelist.append(node)
    return computelist


def swapadam(topoorder):
    """Move each optimiser node to just after the last non-optimiser reader of its parameter."""
    order = list(topoorder)
    i = 0
    n = len(order)
    for i in range(n):
        node = order[i]
        if node.issgd == 1 and node.isw == 0:
            node.isw = 3
            param = node.inputs[0]
            j = n - 1
            while j > i:
                if order[j].issgd != 1 and param in order[j].inputs:
                    break
                j -= 1
            order.pop(i)
            order.insert(j, node)
    return order


class _SwapWorker(threading.Thread):
    """Executes the swap requests of ONE direction for the executor on its own side stream, in the order they were
    submitted.  Two workers (device -> host and host -> device) let the two copy engines run at the same time; a
    swap-in first waits for the queued swap-out of the same tensor.  A reader of a tensor that still has requests
    queued waits for them (``wait_for``): it must not pick up the device array of a tensor whose swap-out is about to
    free it."""

    def __init__(self, executor, to_gpu, other=None):
        super().__init__(daemon=True)
        self.ex = executor
        self.to_gpu = to_gpu
        self.other = other             # the swap-out worker, for the swap-in worker
        self.q = queue.Queue()
        self.stream = None
        self.cond = threading.Condition()
        self.pending = 0
        self.pending_for = {}          # tensor index -> queued or running requests

    def submit(self, wait_ms, index):
        with self.cond:
            self.pending += 1
            self.pending_for[index] = self.pending_for.get(index, 0) + 1
        self.q.put((wait_ms, index))

    def run(self):
        self.stream = gpu_op.create_cudaStream()
        while True:
            item = self.q.get()
            if item is None:
                return
            wait_ms, index = item
            try:
                if wait_ms > 0:
                    time.sleep(wait_ms / 1000.0)
                if self.other is not None:
                    self.other.wait_for(index)        # the tensor's way out has to be complete before its way back
                self.ex._do_swap(index, self.to_gpu, self.stream)
            finally:
                with self.cond:
                    self.pending -= 1
                    self.pending_for[index] -= 1
                    self.cond.notify_all()

    def wait_for(self, index):
        with self.cond:
            while self.pending_for.get(index, 0) > 0:
                self.cond.wait()

    def drain(self):
        with self.cond:
            while self.pending > 0:
                self.cond.wait()


class _SwapWorkers(object):
    """The pair of workers behind the executor's swap requests."""

    def __init__(self, executor):
        self.out = _SwapWorker(executor, False)
        self.back = _SwapWorker(executor, True, other=self.out)
        self.out.start()
        self.back.start()

    def submit(self, wait_ms, index, to_gpu):
        (self.back if to_gpu else self.out).submit(wait_ms, index)

    def wait_for(self, index):
        self.out.wait_for(index)
        self.back.wait_for(index)

    def drain(self):
        self.out.drain()
        self.back.drain()


class Executor(object):
    def __init__(self, targetloss, y, learning_rate, top_control_queue=None, top_message_queue=None, log_path=None,
                 optimizer="adam"):
        self.b1, self.b2, self.e = 0.9, 0.999, 0.00000001
        self.b1t, self.b2t = [0.9], [0.999]
        self.targetloss, self.y, self.learning_rate = targetloss, y, learning_rate
        self.log_path = log_path
        self.optimizer = optimizer

        variables = get_Variable_node_list(targetloss)
        variables.reverse()                      # last layer first: its gradient is ready first
        self.Variable_node_grad_list = gradients(targetloss, variables)
        self.Variable_node_to_grad = dict(zip(variables, self.Variable_node_grad_list))
        if optimizer == "adam":
            compute, self.mv, self.Variable_node_to_mv = getcomputelist(
                variables, self.Variable_node_grad_list, self.b1, self.b2, self.b1t, self.b2t, self.e, learning_rate)
        elif optimizer == "sgd":
            compute, self.mv, self.Variable_node_to_mv = getsgdcomputelist(variables, self.Variable_node_grad_list, learning_rate), [], {}
        else:
            raise ValueError("optimizer must be 'adam' or 'sgd'")
        self.optimizer_nodes = compute
        self.topo_order = swapadam(find_topo_sort(compute))
        variables.reverse()                      # back to network order
        self.Variable_node_list = variables
        self.eval_node_list = [targetloss] + variables + [self.Variable_node_to_mv[v][0] for v in variables if v in self.Variable_node_to_mv] \
            + [self.Variable_node_to_mv[v][1] for v in variables if v in self.Variable_node_to_mv] + [y]
        for i, node in enumerate(self.topo_order):
            node.index = i
        # a recorded step repeats the launches of the moment it was recorded: assignments to nodes outdate it
        self._changes = [0]
        for node in self.topo_order:
            node._changes = (node._changes or ()) + (self._changes,)
        self.total_node = len(self.topo_order)

        self.top_control_queue, self.top_message_queue = top_control_queue, top_message_queue
        # stream and handles are created on first use, so graph analysis works without a device
        self.cudaStream = self.cudnnHandle = self.cublasHandle = None
        self.ctx_cpu, self.ctx_gpu = ndarray.cpu(0), ndarray.gpu(0)
        self.node_to_shape_map = None
        self.feed_shapes = None
        # convolutions of a fed filter, and their descriptors as the library takes them (with the objects behind)
        self._convs = [n for n in self.topo_order if type(n.op) is Convolution2DForwardOp and not n.inputs[1].inputs]
        self._conv_cells = ([], None)
        # gradients of parameters that only the optimiser reads: they may wait and share launches
        readers = {}
        for node in self.topo_order:
            for i in node.inputs:
                readers.setdefault(i, []).append(node)
        self._patient = {n for n in self.topo_order if self._is_parameter_gradient(n) and all(type(r.op) in (SgdOp, AdamOp) for r in readers.get(n, ()))}
        self._values = {}          # node index -> NDArray on the GPU (None while swapped out)
        self._feed = {}            # what the most recent run was fed: node -> NDArray on the GPU
        self._leases = {}          # node index -> weak references to the views of its array that were handed out
        self._recordings = step_graph.Recordings()
        self._record_failures = 0
        self.recording_error = None          # why the last attempt to record a step failed
        self._constants = set()    # indices of the fill nodes whose array holds their constant already
        self.host_values = {}      # node index -> pinned host NDArray holding a swapped-out tensor
        self.have_plan = False
        self._swap_worker = None
        self._values_lock = threading.Lock()
        self.passive_swap_in = 0

    @staticmethod
    def _is_parameter_gradient(node):
        if type(node.op) is Convolution2DBackwardOp:
            return node.type == 1
        return type(node.op) is BroadcastToGradientOp or (type(node.op) is MatMulOp and node.matmul_attr_trans_A)

    @property
    def values(self):
        """Node index -> NDArray on the GPU.  Whoever holds this dict may hold any array of it, so none is written again."""
        self._forget_recordings()
        self._values, self._values_exposed = dict(self._values), True
        return self._values

    @values.setter
    def values(self, values):
        self._forget_recordings()
        self._values = values

    _values_exposed = False

    def _forget_recordings(self):
        self._recordings.clear()
        self._constants.clear()

    def _ensure_handles(self):
        if self.cudaStream is None:
            self.cudaStream = gpu_op.create_cudaStream()
            self.cudnnHandle = gpu_op.create_cudnnHandle(self.cudaStream)
            self.cublasHandle = gpu_op.create_cublasHandle(self.cudaStream)

    # ---- shape inference (autodiff.py:2318-2336): builds every descriptor exactly once ----------
    def infer_shape(self, feed_shapes):
        self._forget_recordings()
        self._record_failures = 0
        self.node_to_shape_map = dict(feed_shapes)
        for node in self.topo_order:
            if node in self.node_to_shape_map:
                continue
            input_shapes = [self.node_to_shape_map[i] for i in node.inputs]
            replaced = node.cudnnlist[0] if isinstance(node.op, (Convolution2DForwardOp, Pooling2DForwardOp, BNForwardOp)) else 0
            self.node_to_shape_map[node] = tuple(node.op.infer_shape(node, input_shapes, self.cudnnHandle))
            if replaced:                     # the descriptor of earlier shapes: what it keeps on the device goes back
                gpu_op.release_descriptor(replaced)

    # ---- memory-plan messages ---------------------------------------------------------------------
    def _apply_plan(self, swap_list, release_list, recompute_list):
        self._forget_recordings()
        for node in self.topo_order:
            node.control_message_out, node.control_message_out_time = [], 0
            node.release_list, node.recompute_list = [], []
        for tensor_index, start_time, start_node_index, move_to_gpu in swap_list:
            start = self.topo_order[start_node_index]
            wait = start_time if start.control_message_out_time == 0 else start_time - start.control_message_out_time
            start.control_message_out_time = start_time
            start.control_message_out.append((wait, tensor_index, move_to_gpu))
        for start_node_index, tensor_index in release_list:
            self.topo_order[start_node_index].release_list.append(tensor_index)
        for start_node_index, tensor_index in recompute_list:
            self.topo_order[start_node_index].recompute_list.append(tensor_index)
        self.have_plan = bool(swap_list or release_list or recompute_list)
        if swap_list and self._swap_worker is None:
            self._swap_worker = _SwapWorkers(self)

    def _do_swap(self, index, to_gpu, stream):
        shape = self.node_to_shape_map[self.topo_order[index]]
        if to_gpu:
            with self._values_lock:
                if self._values.get(index) is not None or index not in self.host_values:
                    return
            dev = ndarray.empty(shape, self.ctx_gpu)
            self.host_values[index].copyto(dev, stream)
            with self._values_lock:
                if self._values.get(index) is None:
                    self._values[index] = dev
        else:
            with self._values_lock:
                dev = self._values.get(index)
            if dev is None:
                return
            host = self.host_values.get(index)
            if host is None:
                host = ndarray.empty(shape, self.ctx_cpu)
            dev.copyto(host, stream)             # returns once the copy has completed
            with self._values_lock:
                self.host_values[index] = host
                self._values[index] = None
            dev.free_gpu()

    def _after_node(self, node):
        for wait, tensor_index, to_gpu in node.control_message_out:
            self._swap_worker.submit(wait, tensor_index, to_gpu)
        for tensor_index in node.release_list:
            with self._values_lock:
                arr = self._values.get(tensor_index)
                self._values[tensor_index] = None
            if arr is not None and self.topo_order[tensor_index].isw == 0:
                arr.free_gpu()

    def _resident(self, n):
        """The GPU array of node ``n``, swapping it in on demand (the reference's passive swap-in)."""
        if self._swap_worker is not None:
            self._swap_worker.wait_for(n.index)      # a queued swap-out would free the array under the reader
        arr = self._values.get(n.index)
        if arr is not None:
            return arr
        if not self.have_plan and n in self._feed:
            return self._feed[n]
        host = self.host_values.get(n.index)
        if host is None:
            raise RuntimeError("tensor of node %d (%s) is neither on the GPU nor swapped out" % (n.index, n.name))
        self.passive_swap_in += 1
        arr = ndarray.empty(self.node_to_shape_map[n], self.ctx_gpu)
        host.copyto(arr, self.cudaStream)
        self._values[n.index] = arr
        return arr

    def _lease(self, n):
        """A view of node ``n``'s array for the caller; the next step leaves the array alone while a view is alive."""
        view = self._resident(n).borrow()
        if n.index in self._constants:           # whoever looks may write: the constant is filled in anew
            self._forget_recordings()
        ref = weakref.ref(view)
        while n is not None:                     # a sum that is a view of its operand keeps that one's array, too
            self._leases.setdefault(n.index, []).append(ref)
            n = self._unchanged_operand(n) if type(n.op) is AddOp else None
        return view

    def _live_leases(self):
        if self._leases:
            self._leases = {i: live for i, live in ((i, [r for r in refs if r() is not None]) for i, refs in self._leases.items()) if live}
        return self._leases

    def _compute(self, node, out, stream):
        inputs = [self._resident(n) for n in node.inputs]
        if node.issgd:
            node.op.compute(node, inputs, None, self.cudnnHandle, self.cublasHandle, stream, False)
            return
        if out is None:
            out = ndarray.empty(self.node_to_shape_map[node], self.ctx_gpu)
        if isinstance(out, int):
            raise MemoryError("device out of memory allocating %d bytes for node %d (%s)" % (out, node.index, node.name))
        short = node.op.compute(node, inputs, out, self.cudnnHandle, self.cublasHandle, stream, False)
        if short:
            raise MemoryError("device out of memory inside node %d (%s): %d bytes short" % (node.index, node.name, short))
        self._values[node.index] = out

    def _unchanged_operand(self, node):
        """The operand a sum is equal to because the other one is a zeros node (the gradient of a broadcast's shape
        operand, which every bias adds to its layer's gradient), or None."""
        a, b = node.inputs
        shapes = self.node_to_shape_map
        if shapes[a] != shapes[b] or a in self._feed or b in self._feed:
            return None
        if type(b.op) is ZerosLikeOp:
            return a
        return b if type(a.op) is ZerosLikeOp else None

    def _update_parameters(self, nodes, stream):
        """The optimiser nodes of a step, one launch for all that share a rule (their place in the order is behind every
        reader of their parameter, so the end of the step will do)."""
        groups = {}
        for node in nodes:
            if type(node.op) is SgdOp:
                rule = (node.learning_rate,)
            else:
                rule = (node.b1, node.b2, node.b1t[0], node.b2t[0], node.e, node.learning_rate)
            groups.setdefault(rule, []).append([self._resident(n) for n in node.inputs])
        for rule, rows in groups.items():
            arrays = [gpu_op.handle_array(column) for column in zip(*rows)]
            if len(rule) == 1:
                gpu_op.sgd_update_many(arrays[0], arrays[1], rule[0], stream)
            else:
                gpu_op.adam_update_many(arrays[0], arrays[1], arrays[2], arrays[3], *rule, stream)

    def _pack_filters(self, stream):
        cells = [n.cudnnlist[0] for n in self._convs]
        if len(self._conv_cells[0]) != len(cells) or any(a is not b for a, b in zip(self._conv_cells[0], cells)):
            self._conv_cells = (cells, gpu_op.cell_array(cells))
        gpu_op.pack_filters([self._feed[n.inputs[1]] for n in self._convs], self._conv_cells[1], stream)

    def _issue(self, feed_dict, stream, recording=False):
        """Issues every node's calls on ``stream``.  Returns (arrays by node index, loss array)."""
        # Without a plan a node writes the array it wrote in the previous step, unless a caller still looks at that.  Under
        # a plan the arrays come and go: the previous step's go back to the pool one at a time, each just before its node
        # runs again (dropping all of them here would leave a synchronised GPU idle for a millisecond or two).
        previous = {} if self._values_exposed else dict(self._values)
        self._values, self._values_exposed = {}, False
        if self.have_plan:
            self._values = {n.index: v for n, v in self._feed.items()}        # a plan may move these too
        else:
            for index in self._live_leases():
                previous.pop(index, None)
        previous.pop(self.targetloss.index, None)        # the loss belongs to the caller
        shapes, timed = self.node_to_shape_map, self.top_message_queue is not None
        together = not (self.have_plan or timed or gpu_op.data_parallel_active())
        updates, holding = [], False
        if together and self._convs and all(n.inputs[1] in self._feed for n in self._convs):
            self._pack_filters(stream)
        for node in self.topo_order:
            if not node.inputs and node in self._feed:
                if self.have_plan:
                    self._after_node(node)
                continue
            if together and node.issgd and type(node.op) in (SgdOp, AdamOp):
                updates.append(node)
                continue
            out = previous.pop(node.index, None)
            if out is not None and (self.have_plan or out.is_freed or out.shape != shapes[node]):
                out = None
            if together and type(node.op) in (ZerosLikeOp, OnesLikeOp):
                # nobody else writes its array, so the constant of the first step is still there
                if out is None or node.index not in self._constants:
                    self._compute(node, out, stream)
                    self._constants.add(node.index)
                else:
                    self._values[node.index] = out
                continue
            if together and type(node.op) is AddOp:
                same = self._unchanged_operand(node)
                if same is not None:               # x + 0 is x: a view of it
                    self._values[node.index] = self._resident(same).borrow()
                    continue
            if self.have_plan:
                for idx in node.recompute_list:
                    self._compute(self.topo_order[idx], None, stream)
            if together and (node in self._patient) != holding:        # an error drops what is held, and the switch
                holding = not holding
                gpu_op.hold_products(holding)
            if timed:
                t0 = time.perf_counter()
                self._compute(node, out, stream)
                node.runtime = (time.perf_counter() - t0) * 1000.0
            else:
                self._compute(node, out, stream)
            if self.have_plan:
                self._after_node(node)
        if together:
            if holding:
                gpu_op.hold_products(False)
            gpu_op.launch_held(stream)
        if updates:
            self._update_parameters(updates, stream)
        previous.clear()
        return self._values, self._values.get(self.targetloss.index)

    # ---- one training step ----------------------------------------------------------------------------
    def run(self, feed_dict, convert_to_numpy_ret_vals=False):
        self._ensure_handles()
        loss = self._run_recorded(feed_dict)
        if loss is None:
            loss = self._run_nodes(feed_dict)
        self.b1t[0] *= self.b1
        self.b2t[0] *= self.b2
        if self.have_plan:
            next_feed = {n: self._values[n.index] for n in feed_dict if n.isw == 1}
        else:
            next_feed = {n: self._feed[n] for n in feed_dict if n.isw == 1}
        if convert_to_numpy_ret_vals:
            return [loss.asnumpy(), {n: v.asnumpy() for n, v in next_feed.items()}]
        return [loss, next_feed]

    def _run_nodes(self, feed_dict):
        self._feed = {}
        feed_shapes = {}
        for node, value in feed_dict.items():
            if not ndarray.is_gpu_ctx(value.ctx):
                value = value.copyto(self.ctx_gpu, None)
            self._feed[node] = value
            feed_shapes[node] = value.shape
        if self.feed_shapes != feed_shapes:
            self.infer_shape(feed_shapes)
            self.feed_shapes = feed_shapes
        if self.top_control_queue is not None and not self.top_control_queue.empty():
            self._apply_plan(*self.top_control_queue.get())
        try:
            self._issue(feed_dict, self.cudaStream)
        except BaseException:
            gpu_op.drop_held()
            raise
        if self._swap_worker is not None:
            self._swap_worker.drain()
        return self._resident(self.targetloss)

    # ---- the same step, recorded (step_graph.py) --------------------------------------------------------
    def _run_recorded(self, feed_dict):
        """The loss of this step if it could be replayed from a recording (made here once the feed has come often
        enough), else None."""
        if not step_graph.ENABLED or self.have_plan or self.top_message_queue is not None or self._record_failures > 1:
            return None
        if self.top_control_queue is not None and not self.top_control_queue.empty():
            return None
        entry, staged, wanted = self._recordings.choose(feed_dict)
        recording = entry.recording
        if recording is not None and recording.changes != self._changes[0]:
            recording = entry.recording = None
        if self._live_leases() or gpu_op.data_parallel_active():
            return None
        if recording is None:
            if not wanted or any(v.shape != self.feed_shapes.get(n) for n, v in feed_dict.items()):
                return None
            recording = self._record(feed_dict, staged)
            if recording is None:
                return None
            self._recordings.keep(entry, recording)
        self._feed = dict(feed_dict)
        if staged:
            for node, array in recording.staged:
                value = feed_dict[node]
                if value.shape != array.shape:
                    return None
                if ndarray.is_gpu_ctx(value.ctx):
                    gpu_op.copy_on_stream(value, array, self.cudaStream)
                else:
                    value.copyto(array, None)
                self._feed[node] = array
        rc = recording.replay(self, random.randint)
        if rc != 0:
            if rc == 1:
                entry.recording = None
            return None
        self._values = recording.values
        loss = ndarray.empty(recording.loss.shape, self.ctx_gpu)
        gpu_op.copy_on_stream(recording.loss, loss, self.cudaStream)
        recording.values[self.targetloss.index] = loss
        return loss

    def _record(self, feed_dict, staged):
        if any(not ndarray.is_gpu_ctx(v.ctx) for n, v in feed_dict.items() if not (staged and n.isw == 2)):
            return None
        feed, copies = dict(feed_dict), []
        if staged:
            for node in feed_dict:
                if node.isw == 2:
                    feed[node] = ndarray.empty(feed_dict[node].shape, self.ctx_gpu)
                    copies.append((node, feed[node]))
        draws = random.getstate()                # the recorded step is not run: its seeds have not been drawn
        before = self._feed, self._values
        self._feed = feed
        try:
            return step_graph.record(self, feed, copies)
        except RuntimeError as e:
            self._record_failures += 1
            self._feed, self._values = before
            self.recording_error = str(e)
            warnings.warn("this training step could not be recorded and runs as ordinary calls (%s)%s"
                          % (e, "; no further attempts for these shapes" if self._record_failures > 1 else ""), RuntimeWarning, stacklevel=4)
            return None
        finally:
            random.setstate(draws)

    # ---- inspection helpers (no counterpart in the reference) ---------------------------------------------
    def value_of(self, node):
        """GPU array computed for ``node`` in the most recent ``run``."""
        return self._lease(node)

    def gradient_of(self, variable):
        return self._lease(self.Variable_node_to_grad[variable])

    def synchronize(self):
        gpu_op.device_synchronize()
