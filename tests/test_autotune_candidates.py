"""The tuner's own candidates differ in what reaches a launch. CPU: the config calls and CUDA events are stand-ins."""
import types

from rocketgpu_b200 import autotune


def test_default_candidates_differ_in_arena_threads_or_graphs(monkeypatch):
    import torch
    event = types.SimpleNamespace(record=lambda s: None, synchronize=lambda: None, elapsed_time=lambda e: 1.0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: None)
    monkeypatch.setattr(torch.cuda, "Event", lambda enable_timing: event)
    tried, steps = [], []
    monkeypatch.setattr(autotune, "set_config", lambda sim, at, ct, g: tried.append((at, g)))
    best, results = autotune.autotune(None, lambda: steps.append(1))
    assert len(results) == len(set(tried[:-1])) == len(autotune.ARENA_THREADS) * 2
    assert len(steps) == len(results) * 4 and best in [c for c, _ in results]
