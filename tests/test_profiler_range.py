"""The range around a layer's write is recorded by every kind of profiler and observer."""

import json
import threading

import pytest
import torch
from torch.profiler import ExecutionTraceObserver, ProfilerActivity, profile

NAME = "echokv.write.step"


@pytest.fixture
def apply(monkeypatch):
    import echokv_b200.kernels.write as W
    from echokv_b200.tiered_cache import TieredKVCache

    calls = []
    monkeypatch.setattr(W, "write_step", lambda *a, **kw: calls.append(1))
    yield lambda: TieredKVCache.apply(None, None, None, None)
    assert calls


def _recorded(prof):
    return sum(e.name == NAME for e in prof.events())


def test_a_profiler_of_this_thread(apply):
    with profile(activities=[ProfilerActivity.CPU]) as prof:
        apply()
        apply()
    assert _recorded(prof) == 2


def test_a_profiler_of_all_threads(apply):
    from torch._C._profiler import _ExperimentalConfig

    with profile(activities=[ProfilerActivity.CPU], experimental_config=_ExperimentalConfig(profile_all_threads=True)) as prof:
        apply()
        worker = threading.Thread(target=apply)
        worker.start()
        worker.join()
    assert _recorded(prof) == 2


def test_an_execution_trace_observer(apply, tmp_path):
    observer = ExecutionTraceObserver().register_callback(str(tmp_path / "trace.json"))
    observer.start()
    apply()
    observer.stop()
    observer.unregister_callback()
    names = [n["name"] for n in json.loads((tmp_path / "trace.json").read_text())["nodes"]]
    assert names.count(NAME) == 1


def test_nothing_is_entered_when_nobody_looks(apply, monkeypatch):
    import echokv_b200.tiered_cache as T

    monkeypatch.setattr(T, "record_function", lambda name: pytest.fail("a range without an observer"))
    apply()
