"""Interval timer with the reference's semantics (src/qubo_lib/utils/perf_timer.py:4-39).

On a GPU every ``pick_time`` records a CUDA event on the current stream (or on ``stream``, a
torch stream, where one is given: looking the current one up costs 4 us per pick) and
synchronises it, so each interval covers the device work issued since the previous pick; on the
host it is a ``perf_counter`` interval.  ``get_time_from_start`` is the sum of all intervals in ms.
"""
from __future__ import annotations

import time


class PerformanceTimer:
    def __init__(self, use_gpu: bool = False, stream=None):
        self.times = []
        self.use_gpu = bool(use_gpu)
        self._stream = stream
        self._marks = []  # (event, label) of mark_time
        if self.use_gpu:
            import torch
            self._torch = torch
            self.start_event = torch.cuda.Event(enable_timing=True)
            self.start_event.record(stream)
            self.last_event = self.start_event
        else:
            self.start_time = time.perf_counter()

    def mark_time(self, label=None):
        """pick_time without waiting on a GPU: the interval is entered by the next pick_time."""
        if not self.use_gpu:
            self.pick_time(label)
            return
        ev = self._torch.cuda.Event(enable_timing=True)
        ev.record(self._stream)
        self._marks.append((ev, label))

    def pick_time(self, label=None):
        if self.use_gpu:
            ev = self._torch.cuda.Event(enable_timing=True)
            ev.record(self._stream)
            ev.synchronize()
            for mark, mark_label in self._marks:
                self.times.append((self.last_event.elapsed_time(mark), mark_label))
                self.last_event = mark
            self._marks.clear()
            ms = self.last_event.elapsed_time(ev)
            self.last_event = ev
        else:
            now = time.perf_counter()
            ms = (now - self.start_time) * 1000
            self.start_time = now
        self.times.append((ms, label))

    def get_time_from_start(self):
        return sum(t for t, _ in self.times)
