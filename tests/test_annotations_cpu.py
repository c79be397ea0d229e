"""Entry points stay annotated under a profiler, and call through without one."""

from __future__ import annotations

from contextlib import contextmanager

import torch

from meshtryoshka_gb300 import record
from meshtryoshka_gb300.record import annotate


@annotate("annotated_sum")
def _sum(a, b=1):
    return a + b


def test_annotations_appear_only_while_profiling():
    assert _sum(1, b=2) == 3 and _sum.__name__ == "_sum"
    with annotate("outside"):
        pass
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        assert _sum(2) == 3
        with annotate("annotated_block"):
            pass
    names = {e.name for e in prof.events()}
    assert {"annotated_sum", "annotated_block"} <= names and "outside" not in names


def test_an_exception_passes_through():
    try:
        with annotate("raises"):
            raise KeyError("inside")
    except KeyError as e:
        assert e.args == ("inside",)


def test_the_cheap_form_unless_a_profiler_runs(monkeypatch):
    opened = []

    def form(kind):
        @contextmanager
        def opens(name):
            opened.append((kind, name))
            yield

        return opens

    monkeypatch.setattr(record, "record_function", form("dispatched"))
    monkeypatch.setattr(record, "_Fast", form("fast"))
    assert _sum(1) == 2
    with annotate("block"):
        pass
    assert opened == [("fast", "annotated_sum"), ("fast", "block")]
    opened.clear()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]):
        assert _sum(1) == 2
        with annotate("block"):
            pass
    assert opened == [("dispatched", "annotated_sum"), ("dispatched", "block")]
