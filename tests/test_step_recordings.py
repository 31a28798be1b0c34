"""Which steps are recorded, and on whose arrays (no device code)."""
import gc
import weakref

import pytest

from tinyflow_b200 import step_graph


class _Node(object):
    def __init__(self, isw):
        self.isw = isw


class _Array(object):
    pass


def _replay(order):
    """The recordings that the runs of `order` make (run number, staged); a new letter is a new mini-batch array."""
    table, w, x = step_graph.Recordings(), _Node(1), _Node(2)
    weights, arrays, made = _Array(), {}, []
    for step, letter in enumerate(order):
        entry, staged, wanted = table.choose({w: weights, x: arrays.setdefault(letter, _Array())})
        if entry.recording is None and wanted:
            entry.recording = "staged" if staged else letter
            made.append((step, staged))
    return made


@pytest.mark.parametrize("order, made", [
    ("AAAAAAAA", [(2, False)]),                          # one resident batch, or one array that is overwritten
    ("ABABABABABABABABABAB", [(4, True)]),               # two upload buffers in turn: one recording, and none later on
    ("ABCDEFGHIJ", [(4, True)]),                         # ever new arrays
    ("AAAABABAB", [(2, False), (4, True)]),
    ("AAABBBABAB", [(2, False), (4, True), (5, False)]),  # each came often enough in a row
], ids=lambda v: v if isinstance(v, str) else "")
def test_recordings_that_a_sequence_of_batches_makes(order, made):
    assert _replay(order) == made


def test_arrays_that_keep_coming_in_turn_get_recordings_of_their_own():
    n = step_graph.RUNS_WITHOUT_STAGING
    assert _replay("AB" * (n + 2)) == [(4, True), (2 * n, False), (2 * n + 1, False)]


@pytest.mark.parametrize("drop", ["clear", "batch array", "parameter", "table full"])
def test_a_dropped_recording_goes_at_once(drop):
    """Its device memory does not wait for the garbage collector."""
    table, w, x = step_graph.Recordings(), _Node(1), _Node(2)
    weights, batch = _Array(), _Array()
    entry, _, _ = table.choose({w: weights, x: batch})
    recording = _Array()
    table.keep(entry, recording)
    gone = weakref.ref(recording)
    del entry, recording
    gc.collect()
    gc.disable()
    try:
        if drop == "clear":
            table.clear()
        elif drop == "batch array":
            del batch
        elif drop == "parameter":
            del weights
        else:
            kept = [_Array() for _ in range(step_graph.MAX_FEEDS)]
            for other in kept:
                assert gone() is not None
                entry = table.choose({w: other, x: batch})[0]
                table.keep(entry, _Array())
        assert gone() is None
    finally:
        gc.enable()
