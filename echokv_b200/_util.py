"""Helpers shared by the host-side modules."""

from __future__ import annotations

import ctypes
import os

import torch


def to_device(t: torch.Tensor, device) -> torch.Tensor:
    """Copy a host tensor to ``device`` without stalling the CPU.

    A copy from pageable memory makes the host wait for the stream; staging the
    source in pinned memory and copying with ``non_blocking=True`` lets the host
    run ahead (the caching pinned allocator keeps the staging buffer alive until
    the copy has run).  Same role as the reference's ``echokv_vllm/_util.py:8-20``.
    """
    device = torch.device(device)
    if device.type != "cuda":
        raise RuntimeError("echokv_b200 runs on CUDA devices only")
    return t.pin_memory().to(device, non_blocking=True)


def _callbacks_check():
    try:
        check = ctypes.PyDLL(os.path.join(os.path.dirname(torch.__file__), "lib", "libtorch_cpu.so"))._ZN2at12hasCallbacksEv
    except (OSError, AttributeError):  # another build of torch: ranges are always entered
        return lambda: True
    check.argtypes, check.restype = (), ctypes.c_bool
    return check


# ``at::hasCallbacks()``: whether a profiler or observer, of this thread or of all of them, sees a ``record_function`` range entered
# now.  torch gives it no name in Python; ``torch.autograd._profiler_enabled`` leaves out what observes all threads.  0.2 us, where the
# range itself costs 8 us whether anyone looks or not.
ranges_are_seen = _callbacks_check()
