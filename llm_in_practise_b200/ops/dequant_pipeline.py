"""Expansion of 4-bit weights ahead of their GEMMs, on a side stream.

The expansion is HBM-bound (5 TB/s, 91 us for 34816 x 5120), the tcgen05 GEMMs are bound by the tensor pipe and leave most of
the DRAM bandwidth idle — so the next weights are expanded *while* the current GEMM runs: three blocks of the expansion fit on
an SM beside a block of the GEMM. Two ahead: the largest weight takes longer than the shortest GEMM before it.

The order of requests in a training step is the same every step (q|k|v, o, gate|up, down per layer, then the same ones in
reverse for the input gradients), so the pipeline simply remembers which (weight, direction) followed which last time and
expands the next two into the other buffers as soon as the current request has been served. A misprediction costs nothing but
the wasted expansion: every request checks that its buffer really holds what it asked for and otherwise expands in line.

Both directions read W as it is stored (the input gradient as an MN-major operand), so the backward takes what the forward
has just expanded where a buffer still holds it: the last three weights. The other way round a buffer is expanded afresh.

All expansions — predicted or not — run on the side stream (the compute stream waits on their event), which also gives
the ZeRO-3 shard prefetcher (parallel/zero.py) a single consumer stream.
"""
from __future__ import annotations

import os
from typing import Dict, Optional, Tuple

import torch

ENABLED = os.environ.get("B200_DEQUANT_AHEAD", "1") != "0"


class _Slot:
    __slots__ = ("buf", "key", "ready", "used")

    def __init__(self):
        self.buf: Optional[torch.Tensor] = None
        self.key = None
        self.ready = torch.cuda.Event()
        self.used = torch.cuda.Event()      # recorded on the compute stream once the consumer GEMM is enqueued


class DequantPipeline:
    def __init__(self, device: torch.device, nslots: int = 3):
        self.device = device
        self.stream = torch.cuda.Stream(device)
        self.slots = [_Slot() for _ in range(nslots)]
        self.next_of: Dict[tuple, Tuple[object, torch.dtype, bool]] = {}
        self.prev_key = None
        self.cur = -1                       # slot handed out by the last request
        self.open = False                   # its consumer may not be enqueued yet
        self.hits = self.misses = 0

    def _expand(self, i: int, q, dtype, key) -> None:
        slot, n = self.slots[i], q.N * q.K
        if slot.buf is None or slot.buf.dtype != dtype or slot.buf.numel() < n:
            slot.buf = torch.empty(n, dtype=dtype, device=self.device)
        self.stream.wait_event(slot.used)                                # the GEMM that last read this buffer is done
        with torch.cuda.stream(self.stream):
            q.dequantize(dtype, out=slot.buf[:n].view(q.N, q.K))
            slot.ready.record(self.stream)
        slot.key = key

    def _holds(self, key) -> Optional[int]:
        """The buffer that serves this request: expanded for it, or for the forward that it is the backward of."""
        forward = key[:2] + (False,)
        return next((i for i, s in enumerate(self.slots) if s.key in (key, forward)), None)

    def _ahead(self) -> None:
        """Expand the requests that are expected next where no buffer holds them."""
        chain, key = [], self.prev_key
        while len(chain) < len(self.slots) - 1 and key in self.next_of:
            q, dtype, backward = self.next_of[key]
            key = (id(q), dtype, backward)
            chain.append((q, dtype, key, self._holds(key)))
        taken = {self.cur} | {i for *_, i in chain}
        for q, dtype, key, i in chain:
            if i is None:
                i = next((j for j in range(len(self.slots)) if j not in taken), None)
                if i is None:
                    return
                self._expand(i, q, dtype, key)
                taken.add(i)

    def get(self, q, dtype: torch.dtype, backward: bool) -> torch.Tensor:
        key = (id(q), dtype, backward)
        comp = torch.cuda.current_stream(self.device)
        self.done()                                                      # previous consumer is enqueued before this point
        i = self._holds(key)
        if i is None:
            self.misses += 1
            i = (self.cur + 1) % len(self.slots)
            self._expand(i, q, dtype, key)
        else:
            self.hits += 1
        slot = self.slots[i]
        slot.key = key                                                   # from its backward on it serves no forward
        comp.wait_event(slot.ready)
        if self.prev_key is not None:
            self.next_of[self.prev_key] = (q, dtype, backward)
        self.prev_key, self.cur, self.open = key, i, True
        self._ahead()
        n = q.N * q.K
        return slot.buf[:n].view(q.N, q.K)

    def done(self) -> None:
        """The GEMM that reads the last request is enqueued on the current stream: its buffer is free after it."""
        if self.open:
            self.open = False
            self.slots[self.cur].used.record(torch.cuda.current_stream(self.device))


_pipes: Dict[int, DequantPipeline] = {}


def pipeline(device: torch.device) -> DequantPipeline:
    idx = device.index if device.index is not None else torch.cuda.current_device()
    p = _pipes.get(idx)
    if p is None:
        p = _pipes[idx] = DequantPipeline(torch.device("cuda", idx))
    return p


def reset() -> None:
    _pipes.clear()
