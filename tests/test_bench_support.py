"""The timing helpers' order of calls (no GPU needed)."""
from types import SimpleNamespace

import torch

from nanoinfer_b200 import bench_support


def test_prefill_timing_leaves_the_hosts_packing_outside_the_events(monkeypatch):
    calls = []

    class Event:
        def __init__(self, enable_timing):
            pass

        def record(self):
            calls.append("record")

        def elapsed_time(self, other):
            return 1.0

    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: calls.append("wait"))
    monkeypatch.setattr(bench_support, "L2Flusher", lambda device: SimpleNamespace(flush=lambda: calls.append("flush")))
    monkeypatch.setattr(bench_support, "vocabulary", lambda eng: 100)
    monkeypatch.setattr(bench_support, "step_flops", lambda *a: 0.0)
    eng = SimpleNamespace(device="cpu", model=None, cache=SimpleNamespace(open_request=lambda: 0, close_request=lambda r: None),
                          runner=SimpleNamespace(use_graphs=False, step=lambda items: calls.append("step")))
    bench_support.time_prefill(eng, 2, 8, runs=2, warmup=1)
    # the device must be busy with the flush while the host prepares the step between the two events
    assert calls == ["wait", "flush", "record", "step", "record", "wait"] * 3
