"""Recorded training steps.

A step of a graph is the same sequence of launches every time, on the same arrays, as long as the caller feeds the same
ones.  The executor therefore records the step once it has seen the same feed repeatedly and replays it with one call
(``TfStepReplay``) from then on: the host work per step no longer grows with the number of nodes.

What is replayed is keyed by identity.  Parameters and moments (updated in place) are one key; the mini-batch arrays are a
second one below it.  A caller that brings new mini-batch arrays every step, or feeds several in turn, gets a *staged*
recording, whose inputs are copied into arrays of the executor's own first.  Entries disappear with the arrays they name.

A recording is paid for once, a staged input at every step.  ResNet-50 at batch 64: 5 ms of host time for the recording
(2.5-3.5 for the calls, the rest to instantiate the graph and to upload it), 15 us a step for the copies.  So arrays that come
in turn get recordings of their own only after RUNS_WITHOUT_STAGING steps, when the copies have cost about as much.
"""
from __future__ import annotations

import ctypes
import os
import weakref

from . import gpu_op, ndarray
from ._base import _LIB, check_call, last_error, new_cell

ENABLED = os.environ.get("TINYFLOW_STEP_GRAPH", "1") != "0"
RUNS_BEFORE_RECORDING = 2        # of the same arrays: the first calls of a plan still learn what follows what
RUNS_BEFORE_STAGING = 4          # of the same parameters with ever changing mini-batches
RUNS_WITHOUT_STAGING = 512       # of the same arrays, others in between
MAX_FEEDS = 4                    # parameter sets, and mini-batches per set, that keep a recording
MAX_KNOWN = 16                   # that are counted


class Recording(object):
    """A replayable step: the library's graph and the arrays it writes."""

    def __init__(self, graph, values, loss, kept, seed_nodes, arrays, staged, changes):
        self.graph, self.values, self.loss, self.kept, self.staged, self.changes = graph, values, loss, kept, staged, changes
        self.seed_nodes = seed_nodes
        self.seeds = (ctypes.c_uint * max(1, len(seed_nodes)))()
        self.arrays = gpu_op.handle_array(arrays)

    def __del__(self):
        if self.graph is not None and _LIB is not None:
            _LIB.TfStepGraphFree(self.graph)
            self.graph = None

    def replay(self, executor, draw):
        """0 when the step is on its way, else the library's reason (see ``TfStepReplay``)."""
        for i, node in enumerate(self.seed_nodes):
            node.seed[0] = self.seeds[i] = draw(0, 100)
        rc = _LIB.TfStepReplay(self.graph, self.seeds, len(self.seed_nodes), ctypes.c_float(executor.b1t[0]), ctypes.c_float(executor.b2t[0]),
                               self.arrays, len(self.arrays), executor.cudaStream)
        if rc < 0:
            check_call(rc)
        return rc


class _Table(dict):
    """Entries by key.  The entries refer to it weakly: a dropped one, and what was recorded for it, goes at once."""
    __slots__ = ("__weakref__",)


class _Feed(object):
    """How often a set of arrays was run, how often since another one, and what was recorded for it."""
    __slots__ = ("runs", "in_a_row", "refs", "recording", "batches", "latest", "__weakref__")

    def __init__(self):
        self.runs, self.in_a_row, self.refs, self.recording, self.batches, self.latest = 0, 0, None, None, _Table(), None

    def settled(self):
        """Worth a recording on the arrays themselves."""
        return self.in_a_row >= RUNS_BEFORE_RECORDING or self.runs >= RUNS_WITHOUT_STAGING


class Recordings(object):
    def __init__(self):
        self.sets = _Table()

    def clear(self):
        self.sets.clear()

    @staticmethod
    def _entry(table, key, arrays):
        entry = table.pop(key, None)
        if entry is None:
            entry = _Feed()
            # (bound here: at interpreter exit the module's names go before the arrays do)
            gone = lambda _ref, t=weakref.ref(table), e=weakref.ref(entry), k=key, forget=_forget: forget(t(), k, e())     # noqa: E731
            entry.refs = [weakref.ref(a, gone) for a in arrays]
            while len(table) >= MAX_KNOWN:
                del table[next(iter(table))]
        table[key] = entry                      # most recently used last
        return entry

    def choose(self, feed_dict):
        """(entry, staged, wanted): the entry whose recording serves this run, whether its inputs are staged, and whether
        the entry is due one if it has none.  Counts the run."""
        params, batch = [], []
        for node, value in feed_dict.items():
            (batch if node.isw == 2 else params).append((node, value))
        top = self._entry(self.sets, tuple((id(n), id(v)) for n, v in params), [v for _, v in params])
        key = tuple((id(n), id(v)) for n, v in batch)
        below = self._entry(top.batches, key, [v for _, v in batch])
        if top.latest != key:
            top.latest, below.in_a_row = key, 0
        staged = below.recording is None and not below.settled() and top.runs >= RUNS_BEFORE_STAGING
        wanted = staged or below.settled()
        top.runs += 1
        below.runs += 1
        below.in_a_row += 1
        return top if staged else below, staged, wanted

    def keep(self, entry, recording):
        """Attaches a recording to its entry.  The oldest ones beyond MAX_FEEDS go now, beside the cost of making one (dropping
        one takes 100-700 us), and not in front of the first step on new arrays."""
        entry.recording = recording
        for top in self.sets.values():
            self._trim(top.batches, lambda e: e.recording)
        self._trim(self.sets, lambda e: e.recording or any(b.recording for b in e.batches.values()))

    @staticmethod
    def _trim(table, recorded):
        keys = [k for k, e in table.items() if recorded(e)]
        for k in keys[:max(0, len(keys) - MAX_FEEDS)]:
            del table[k]


def _forget(table, key, entry):
    if table is not None and entry is not None and table.get(key) is entry:
        del table[key]


def record(executor, feed_dict, staged):
    """Records one step of ``executor`` on ``feed_dict`` (nothing is executed).  None if that is not possible just now
    (kernel timing, data-parallel exchange), RuntimeError with the reason if the step cannot be recorded."""
    graph, stream = ctypes.c_void_p(), new_cell(2)
    rc = _LIB.TfStepRecordBegin(ctypes.byref(graph), stream, executor.cudaStream)
    if rc != 0:
        if rc < 0:
            raise RuntimeError(last_error())
        return None
    values, loss, keep, stopped = {}, None, 0, None
    try:
        values, loss = executor._issue(feed_dict, stream, recording=True)
        keep = 1
    except Exception as e:                      # whatever stopped it: the caller runs the step as ordinary calls and says so
        stopped = e
    finally:
        rc = _LIB.TfStepRecordEnd(ctypes.byref(graph), keep)
    if rc != 0:
        raise RuntimeError("%s: %s" % (type(stopped).__name__, stopped) if stopped is not None else last_error()) from stopped
    kept = [n for n in feed_dict if n.isw == 1]
    seed_nodes = [n for n in executor.topo_order if hasattr(n, "seed")]
    return Recording(graph, values, loss, kept, seed_nodes, list(feed_dict.values()), staged, executor._changes[0])
