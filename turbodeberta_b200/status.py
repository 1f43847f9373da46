"""Device status words whose reading has been deferred (no host synchronisation at call time)."""
from __future__ import annotations

import threading

import torch


class PendingStatus:
    """Status words of calls made with ``check_status=False`` (no host sync at call time), kept until
    ``check_pending_status()`` reads them.  Nothing is ever dropped: once ``FOLD_AT`` blocks of a device have piled up
    they are folded into one block by an element-wise maximum on that device (a launch, not a synchronisation), so a
    caller that never checks holds a bounded number of small tensors and still sees every report when it does.

    Whoever reads them may be on another stream than the call was (a pass in another thread checks for all), so each block has an
    event behind its launch, which the reading stream waits for.  Words recorded into a graph have none: they are the replays'."""
    FOLD_AT = 256

    def __init__(self):
        self._by_dev: dict = {}
        self._lock = threading.Lock()

    def append(self, status: torch.Tensor) -> None:
        capturing = status.is_cuda and torch.cuda.is_current_stream_capturing()
        full = self._put(status, capturing)
        if full:                                     # not in a capture: folding would be recorded into the graph
            self._put(torch.stack(self._ready(full)).amax(dim=0), capturing)

    def drain(self) -> list:
        """All blocks, for the current stream of each device to read."""
        if not self._by_dev:                         # as after nearly every pass
            return []
        with self._lock:
            taken, self._by_dev = self._by_dev, {}
        return [st for blocks in taken.values() for st in self._ready(blocks)]

    def _put(self, status, capturing):
        event = torch.cuda.current_stream(status.device).record_event() if status.is_cuda and not capturing else None
        with self._lock:
            blocks = self._by_dev.setdefault(status.device, [])
            blocks.append((status, event))
            return self._by_dev.pop(status.device) if len(blocks) >= self.FOLD_AT and not capturing else None

    @staticmethod
    def _ready(blocks) -> list:
        for status, event in blocks:
            if event is not None:
                stream = torch.cuda.current_stream(status.device)
                stream.wait_event(event)
                status.record_stream(stream)
        return [status for status, _ in blocks]

    def __len__(self) -> int:
        return sum(len(v) for v in self._by_dev.values())


#: the one queue of the process: attention calls and table projections append, check_pending_status() drains
PENDING = PendingStatus()
