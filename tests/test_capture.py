"""A capture holds the garbage collector off: a graph that dies while another one is captured
ends the capture."""
import contextlib
import gc
import threading

import pytest
import torch

from cretif_b200.engine.engine import capturing


@pytest.mark.parametrize("fails", [False, True])
@pytest.mark.parametrize("was_on", [False, True])
def test_collector_is_held_off_and_put_back(monkeypatch, fails, was_on):
    seen = []

    @contextlib.contextmanager
    def fake_graph(graph, pool=None, stream=None):
        seen.append((graph, pool, stream, gc.isenabled()))
        yield
        seen.append(gc.isenabled())

    monkeypatch.setattr(torch.cuda, "graph", fake_graph)
    (gc.enable if was_on else gc.disable)()
    try:
        with pytest.raises(RuntimeError) if fails else contextlib.nullcontext():
            with capturing("graph", "pool", "stream"):
                assert not gc.isenabled()
                if fails:
                    raise RuntimeError("a launch inside the capture failed")
        assert gc.isenabled() == was_on
    finally:
        gc.enable()
    assert seen[0] == ("graph", "pool", "stream", False)
    assert fails or seen[1] is False


def test_collector_stays_off_until_the_last_capture_ends(monkeypatch):
    """Two captures overlap in two threads; the first to begin is the first to end."""
    monkeypatch.setattr(torch.cuda, "graph",
                        lambda graph, pool=None, stream=None: contextlib.nullcontext())
    first_ends, first_ended, seen = threading.Event(), threading.Event(), []

    def first():
        with capturing("graph", "pool", "stream"):
            began.set()
            first_ends.wait(10)
        first_ended.set()

    gc.enable()
    began, thread = threading.Event(), threading.Thread(target=first)
    thread.start()
    try:
        assert began.wait(10)
        with capturing("another graph", "pool", "stream"):
            first_ends.set()
            assert first_ended.wait(10)
            seen.append(gc.isenabled())
        assert gc.isenabled()
    finally:
        first_ends.set()
        thread.join()
        gc.enable()
    assert seen == [False]
