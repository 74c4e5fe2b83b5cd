"""Expansion of 4-bit weights ahead of their GEMMs: which work is ordered after which, on streams that only keep count."""
import contextlib
import gc

import pytest
import torch

from llm_in_practise_b200.ops import dequant_pipeline as dq


class Stream:
    def __init__(self, *_):
        self.done = set()                                    # work that this stream's next work comes after

    def work(self, name):
        self.done.add(name)

    def wait_event(self, e):
        self.done |= e.after

    def wait_stream(self, s):
        self.done |= s.done


class Event:
    def __init__(self, *_):
        self.after = set()

    def record(self, stream):
        self.after = set(stream.done)


class Weight:
    def __init__(self, name, comp, n=4):
        self.name, self.N, self.K = name, n, n
        self.packed = torch.full((n * n,), float(len(name)))
        self.runs = []                                       # what each expansion came after
        comp.work("made " + name)

    def dequantize(self, dtype, out, transpose):
        side = Stream.current
        self.runs.append(set(side.done))
        side.work("expanded %s %d" % (self.name, len(self.runs)))
        out.copy_(self.packed.view(out.shape))


@pytest.fixture
def pipe(monkeypatch):
    comp = Stream()

    @contextlib.contextmanager
    def on(stream):
        Stream.current = stream
        yield

    monkeypatch.setattr(torch.cuda, "Stream", Stream)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *_: comp)
    monkeypatch.setattr(torch.cuda, "stream", on)
    return dq.DequantPipeline(torch.device("cpu")), comp


def test_a_new_weight_is_there_before_it_is_expanded(pipe):
    p, comp = pipe
    ws = []
    for name in ("a", "bb", "ccc", "dddd"):
        ws.append(Weight(name, comp))
        w = ws[-1]
        assert torch.equal(p.get(w, torch.float32, False), w.packed.view(4, 4))
        assert "made " + name in w.runs[0]


def test_a_buffer_that_is_replaced_is_not_written_any_more(pipe):
    p, comp = pipe
    small, big = Weight("small", comp), Weight("big", comp, 8)
    p.get(small, torch.float32, False)
    p.get(small, torch.float32, True)                        # the other buffer
    comp.done.discard("expanded small 1")                    # as if nobody had asked for it: the side stream may still be at it
    comp.work("had the memory")
    p.get(big, torch.float32, False)
    assert "expanded small 1" in comp.done                   # before this stream's pool gives the old buffer to anyone
    assert "had the memory" in big.runs[0]                   # the new one may have been another's until now


def test_a_round_that_repeats_is_expanded_ahead(pipe):
    p, comp = pipe
    ws = [Weight(name, comp) for name in ("a", "bb", "ccc")]
    for _ in range(3):
        for w in ws:
            assert torch.equal(p.get(w, torch.float32, False), w.packed.view(4, 4))
            comp.work("product")
    assert p.misses == 4                                     # the first round, and the first step from its end to its beginning


def test_a_weight_that_changed_is_expanded_again(pipe):
    p, comp = pipe
    w = Weight("a", comp)
    p.get(w, torch.float32, False)
    w.packed.fill_(7.0)
    comp.work("filled")
    assert bool((p.get(w, torch.float32, False) == 7.0).all()) and "filled" in w.runs[1]


def test_an_id_is_not_a_weight(pipe):
    p, comp = pipe
    w = Weight("a", comp)
    old = id(w)
    p.get(w, torch.float32, False)
    del w
    gc.collect()
    assert not p.known                                       # nothing is kept of what is gone
    for _ in range(50):                                      # until one lies where the other did, on the same memory
        w = Weight("bb", comp)
        if id(w) == old:
            break
    assert bool((p.get(w, torch.float32, False) == 2.0).all())
    q = Weight("ccc", comp)
    p.slots[p.cur].key, p.slots[p.cur].stamp = (id(q), torch.float32, False), dq._stamp(q)
    assert bool((p.get(q, torch.float32, False) == 3.0).all())
