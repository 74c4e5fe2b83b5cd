"""Expansion of 4-bit weights one GEMM ahead, on a side stream.

The dequant kernels are HBM-bound (4.5 TB/s for ~0.1 ms), the tcgen05 GEMMs are bound by the tensor pipe and the
shared-memory port and leave most of the DRAM bandwidth idle — so the next weight is expanded *while* the current GEMM
runs. An SM has room for one dequant block of 256 threads and 32 registers beside a GEMM CTA (224 threads of 234), for one of 42 registers
none; the others wait for an SM that the GEMM has left. Only the next GEMM waits for them, and a GEMM's CTAs only for those that started before.

The order of requests in a training step is the same every step (q|k|v, o, gate|up, down per layer, then the transposed
ones in reverse), so the pipeline simply remembers which (weight, layout) followed which last time and expands that one
into the other buffer as soon as the current request has been served. A misprediction costs nothing but the wasted
expansion: every request checks that its buffer really holds what it asked for and otherwise expands in line.

All expansions — predicted or not — run on the side stream (the compute stream waits on their event), which also gives
the ZeRO-3 shard prefetcher (parallel/zero.py) a single consumer stream.
"""
from __future__ import annotations

import os
import weakref
from typing import Dict, Optional, Tuple

import torch

ENABLED = os.environ.get("B200_DEQUANT_AHEAD", "1") != "0"


def _stamp(q) -> tuple:
    """What changes when a weight's codes or scales are written or replaced."""
    return tuple((t.data_ptr(), 0 if t.is_inference() else t._version) for t in vars(q).values() if isinstance(t, torch.Tensor))


class _Slot:
    __slots__ = ("buf", "key", "ref", "stamp", "ready", "used", "home", "stream")

    def __init__(self):
        self.buf: Optional[torch.Tensor] = None
        self.key = self.stamp = None
        self.ref = lambda: None             # the weight it holds; an id alone may be another object's by now
        self.ready = torch.cuda.Event()
        self.used = torch.cuda.Event()      # recorded on the compute stream once the consumer GEMM is enqueued
        self.home = self.stream = None      # the streams whose pool the buffer is from, and that it was handed to

    def holds(self, q, key, stamp) -> bool:
        return self.key == key and self.ref() is q and self.stamp == stamp


class DequantPipeline:
    def __init__(self, device: torch.device, nslots: int = 2):
        self.device = device
        self.stream = torch.cuda.Stream(device)
        self.slots = [_Slot() for _ in range(nslots)]
        self.next_of: Dict[tuple, Tuple[object, torch.dtype, bool]] = {}     # weakly: a model that is gone leaves nothing here
        self.known: Dict[int, tuple] = {}   # id -> (weight, stamp) that the side stream has been ordered after
        self.prev_key = None
        self.cur = -1                       # slot handed out by the last request
        self.hits = self.misses = 0

    def release(self) -> None:
        """Before the buffers go back to their pools: what runs there next comes after their last expansions and products."""
        for slot in self.slots:
            self._give_back(slot)

    def _give_back(self, slot: _Slot) -> None:
        if slot.buf is not None:
            if slot.stream is not None:
                slot.used.record(slot.stream)
            slot.home.wait_event(slot.ready)
            slot.home.wait_event(slot.used)
            slot.buf = slot.key = None

    def _expand(self, slot: _Slot, q, dtype, transpose: bool, key, stamp, comp) -> None:
        n = q.N * q.K
        after = self.known.get(id(q))
        behind = after is None or after[0]() is not q or after[1] != stamp   # the weight may still be on its way on the compute stream
        if slot.buf is None or slot.buf.dtype != dtype or slot.buf.numel() < n:
            self._give_back(slot)
            slot.buf = torch.empty(n, dtype=dtype, device=self.device)
            slot.home = comp
            behind = True                                                # and so may what had this memory before
        if behind:
            self.stream.wait_stream(comp)
        self.stream.wait_event(slot.used)                                # the GEMM that last read this buffer is done
        with torch.cuda.stream(self.stream):
            shape = (q.K, q.N) if transpose else (q.N, q.K)
            q.dequantize(dtype, out=slot.buf[:n].view(shape), transpose=transpose)
            slot.ready.record(self.stream)
        stamp = _stamp(q)                                                # a first expansion may add a table to the weight
        if behind:
            self.known[id(q)] = (weakref.ref(q, lambda _, i=id(q): self._forget(i)), stamp)
        slot.key, slot.ref, slot.stamp = key, weakref.ref(q), stamp

    def _forget(self, i: int) -> None:
        entry = self.known.get(i)
        if entry is not None and entry[0]() is None:
            del self.known[i]

    def get(self, q, dtype: torch.dtype, transpose: bool) -> torch.Tensor:
        key, stamp = (id(q), dtype, transpose), _stamp(q)
        comp = torch.cuda.current_stream(self.device)
        if self.cur >= 0:
            last = self.slots[self.cur]
            last.used.record(last.stream)                                # previous consumer is enqueued before this point
        hit = next((i for i, s in enumerate(self.slots) if s.holds(q, key, stamp)), None)
        if hit is None:
            self.misses += 1
            hit = (self.cur + 1) % len(self.slots)
            self._expand(self.slots[hit], q, dtype, transpose, key, stamp, comp)
        else:
            self.hits += 1
        slot = self.slots[hit]
        slot.stream = comp
        comp.wait_event(slot.ready)
        if self.prev_key is not None:
            self.next_of[self.prev_key] = (weakref.ref(q), dtype, transpose)
        self.prev_key, self.cur = key, hit
        nref, ndt, ntr = self.next_of.get(key, (lambda: None, None, False))
        nq = nref()
        if nq is not None:
            nkey, nstamp = (id(nq), ndt, ntr), _stamp(nq)
            other = (hit + 1) % len(self.slots)
            if not self.slots[other].holds(nq, nkey, nstamp):
                self._expand(self.slots[other], nq, ndt, ntr, nkey, nstamp, comp)
        n = q.N * q.K
        return slot.buf[:n].view((q.K, q.N) if transpose else (q.N, q.K))


_pipes: Dict[int, DequantPipeline] = {}


def pipeline(device: torch.device) -> DequantPipeline:
    idx = device.index if device.index is not None else torch.cuda.current_device()
    p = _pipes.get(idx)
    if p is None:
        p = _pipes[idx] = DequantPipeline(torch.device("cuda", idx))
    return p


def reset() -> None:
    for p in _pipes.values():
        p.release()
    _pipes.clear()
