"""Recording of CUDA graphs."""
from __future__ import annotations

import gc
import threading
from contextlib import contextmanager

import torch

_lock = threading.Lock()
_recordings = 0
_collect_after = False


@contextmanager
def recording(graph: "torch.cuda.CUDAGraph"):
    """`torch.cuda.graph(graph)` during which no cycles are collected. Engines and pipelines hold their graphs in cycles, and destroying a graph of one that
    nobody holds any more is an error in any recording of the process. Recordings of several threads may overlap: the collector
    is on again, if it was, when the last of them has ended."""
    global _recordings, _collect_after
    with _lock:
        if _recordings == 0:
            _collect_after = gc.isenabled()
            gc.disable()
        _recordings += 1
    try:
        with torch.cuda.graph(graph):
            yield
    finally:
        with _lock:
            _recordings -= 1
            if _recordings == 0 and _collect_after:
                gc.enable()
