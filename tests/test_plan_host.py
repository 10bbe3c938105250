"""LprPlan's capture on the CPU, with the CUDA objects replaced by stand-ins."""
import contextlib
import gc
from types import SimpleNamespace

import torch


def test_capture_frees_earlier_garbage_and_leaves_the_collector_on(monkeypatch):
    from fastlpr_b200 import plan as plan_mod
    log = []

    class Garbage:
        def __del__(self):
            log.append("freed")

    @contextlib.contextmanager
    def graph(_graph, stream=None):
        log.append("begin")
        yield

    stream = SimpleNamespace(wait_stream=lambda s: None)
    monkeypatch.setattr(torch.cuda, "graph", graph)
    monkeypatch.setattr(torch.cuda, "CUDAGraph", lambda: None)
    monkeypatch.setattr(torch.cuda, "Stream", lambda device=None: stream)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: stream)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)
    p = object.__new__(plan_mod.LprPlan)
    p.device, p.prop, p.order, p._finite = None, object(), [0], None
    p._issue = lambda idx: log.append(gc.isenabled()) or {}
    cycle = Garbage()
    cycle.itself = cycle
    del cycle
    enabled = gc.isenabled()
    gc.enable()
    try:
        p._capture()
        assert gc.isenabled()
    finally:
        if not enabled:
            gc.disable()
    # the eager pass and the captured one both ran with the collector on, and
    # nothing was left for it to free inside the capture
    assert [v for v in log if isinstance(v, bool)] == [True, True]
    assert log.index("freed") < log.index("begin") and len(p.segs) == 1
