"""Host logic of the batched paths without a GPU: the degree classes, the chunking of
HostBatchProver (consecutive runs of about equal bytes, none empty) and launches that fail."""

from __future__ import annotations

import random
from types import SimpleNamespace

import pytest

from zkduel_b200 import _lib
from zkduel_b200.batch import BatchProver, HostBatchProver, chunk_bounds, degree_class


def test_degree_classes():
    assert [degree_class(d) for d in range(1, 8)] == [2, 2, 4, 4, 7, 7, 7]


@pytest.mark.parametrize("chunks", [1, 2, 3, 8, 16, 100])
def test_chunk_bounds_cover_everything_in_order(chunks):
    rng = random.Random(chunks)
    sizes = [rng.choice([8, 32]) * 2 ** rng.randint(10, 20) * rng.randint(2, 8) for _ in range(64)]
    b = chunk_bounds(sizes, chunks)
    assert b[0] == 0 and b[-1] == len(sizes)
    assert all(x < y for x, y in zip(b, b[1:]))  # no empty chunk
    assert 1 <= len(b) - 1 <= min(chunks, len(sizes))
    if chunks <= 8:  # about equal bytes: no chunk beyond twice its share plus one proof
        share = sum(sizes) / (len(b) - 1)
        assert all(sum(sizes[x:y]) <= 2 * share + max(sizes) for x, y in zip(b, b[1:]))


def test_chunk_bounds_small_cases():
    assert chunk_bounds([5], 4) == [0, 1]
    assert chunk_bounds([1, 1, 1, 1], 2) == [0, 2, 4]
    assert chunk_bounds([100, 1, 1, 1], 2) == [0, 1, 4]


class _Chunk:
    def __init__(self, log, name, fails=False):
        self.log, self.name, self.fails = log, name, fails

    def _start(self):
        self.log.append(("start", self.name))
        if self.fails:
            raise RuntimeError("launch failed")

    def _join(self):
        self.log.append(("join", self.name))


def test_chunks_started_before_a_failing_one_are_joined():
    """The caller's stream waits for what runs, also when a later chunk cannot be started: the
    caller may free the tables next, in its own stream's order."""
    log = []
    p = HostBatchProver.__new__(HostBatchProver)
    p.stream, p.copy_streams = None, []
    p.chunks = [(0, 0, _Chunk(log, "a")), (0, 0, _Chunk(log, "b", fails=True)), (0, 0, _Chunk(log, "c"))]
    with pytest.raises(RuntimeError, match="launch failed"):
        p.launch()
    assert log[:2] == [("start", "a"), ("start", "b")] and {("join", "a"), ("join", "b")} <= set(log[2:])
    assert ("start", "c") not in log


def test_groups_started_before_a_failing_one_are_joined(monkeypatch):
    log = []

    class Lib:
        def sc_batch_launch(self, h):
            log.append(("start", h))
            return _lib.SC_ERR_CUDA if h == 2 else _lib.SC_OK

        def sc_batch_join(self, h):
            log.append(("join", h))
            return _lib.SC_OK

        def sc_last_error(self):
            return b"launch failed"

    monkeypatch.setattr(_lib, "load", lambda: Lib())
    p = BatchProver.__new__(BatchProver)
    p.groups = [SimpleNamespace(handle=h) for h in (1, 2, 3)]
    with pytest.raises(_lib.SumcheckError, match="launch failed"):
        p.launch()
    assert log[:2] == [("start", 1), ("start", 2)] and {("join", 1), ("join", 2)} <= set(log[2:])
    assert ("start", 3) not in log
    p.groups = []  # nothing for the prover's end to destroy
