"""Prompts of the scan with a decay per key channel, tile by tile in products of split bf16, against the recurrence in float64: the edges of
blocks of 16 tokens, tiles of 64 and runs, and what is walked instead."""
import pytest
import torch

from llm_in_practise_b200.inference import ragged
from llm_in_practise_b200.inference.ragged import make_pieces
from llm_in_practise_b200.ops.linear_scan import linear_scan

pytestmark = pytest.mark.gpu


def walk(q, k, v, state, runs, H, G, D, g, u):
    q, k, v, g, state = (t.double() for t in (q, k, v, g, state))
    o, rep = torch.zeros(q.shape[0], H, D, dtype=torch.float64, device=q.device), H // G
    q, k = (t.reshape(-1, G, D).repeat_interleave(rep, 1) for t in (q, k))
    for first, n, p0, s in runs:
        S = state[s].clone() if p0 > 0 else torch.zeros_like(state[s])
        for t in range(first, first + n):
            kv = k[t][:, :, None] * v[t].view(H, 1, D)
            if u is not None:
                o[t] = torch.einsum("hde,hd->he", S + u.double().view(H, D, 1) * kv, q[t])
            S = S * g[t].view(H, D, 1) + kv
            if u is None:
                o[t] = torch.einsum("hde,hd->he", S, q[t])
        state[s] = S
    return o.reshape(-1, H * D), state


def case(lens, H, G, D, low, bonus, seed=7):
    r = torch.Generator(device="cuda").manual_seed(seed)
    T = sum(lens)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=r)                                   # noqa: E731
    x = rnd(T, 2 * G * D + H * D + 4)                     # strided rows, as a slice of a projection
    q, k, v = x[:, :G * D], x[:, G * D:2 * G * D], x[:, 2 * G * D:2 * G * D + H * D]
    g = torch.rand(T, H * D, device="cuda", generator=r) * (1.0 - low) + low
    runs, at = [], 0
    for i, n in enumerate(lens):
        runs.append([at, n, 0 if i % 2 == 0 else 5 + i, i])
        at += n
    return q, k, v, g, rnd(len(lens), H, D, D), runs, rnd(H, D) if bonus else None


def scan(q, k, v, g, state, runs, H, G, D, u):
    pieces = make_pieces(runs, "cuda")
    pos = slot = torch.zeros(q.shape[0], dtype=torch.int32, device="cuda")
    return linear_scan(q, k, v, state, pos, slot, pieces.runs, pieces.n_runs, H, G, D, D, "channel", g=g, pieces=pieces, u=u)


@pytest.mark.parametrize("lens,H,G,D", [([65], 2, 2, 64), ([64, 16, 79, 1], 2, 1, 128), ([200, 17], 4, 4, 64), ([97, 130, 15], 20, 5, 128)])
@pytest.mark.parametrize("low", [0.0, 0.9, 1e-30])
@pytest.mark.parametrize("bonus", [False, True])
def test_tiles(lens, H, G, D, low, bonus):
    q, k, v, g, state, runs, u = case(lens, H, G, D, low, bonus)
    g[3::29] = low                                        # decays of zero, and products that underflow, among them
    want_o, want_s = walk(q, k, v, state, runs, H, G, D, g, u)
    o = scan(q, k, v, g, state, runs, H, G, D, u)
    # a value is a sum over at most D channels and what the decays leave of 64 tokens and the state before, each term a product of up to 16 decays
    # a block and rounded a few times: D + 64 roundings of 2^-24 of the largest value on the way, four times over
    for got, want in ((o, want_o), (state, want_s)):
        assert ((got.double() - want).abs().max() / want.abs().max()).item() < 4 * (D + 64) * 2.0 ** -24


@pytest.mark.parametrize("what,value", [("v", float("nan")), ("v", float("inf")), ("k", float("nan")), ("q", float("inf")), ("g", float("nan")),
                                        ("g", 1e12), ("state", float("inf"))])
@pytest.mark.parametrize("at", [5, 70, 130])
@pytest.mark.parametrize("bonus", [False, True])
def test_not_finite_stays_behind_its_token(what, value, at, bonus):
    """A NaN or infinity reaches its token (a decay under a bonus: the one after it) and the ones after that, and growth of decays above one that
    ends in fp32's range is followed; both for a channel or column of one head."""
    H, G, D = 4, 2, 64
    q, k, v, g, state, runs, u = case([150], H, G, D, 0.5, bonus, seed=9)
    runs[0][2] = 3
    if what == "state":
        state[0, 1, 7, 9] = value
    elif value == 1e12:
        g[at - 4:at, 1] = value                           # 1e48 from one end of a block to the other, against decays that bring it back
        g[at - 5, 1] = 1e-30
        g[at, 1] = 1e-30
    else:
        {"v": v, "k": k, "q": q, "g": g}[what][at, 1] = value
    want_o, want_s = walk(q, k, v, state, runs, H, G, D, g, u)
    o = scan(q, k, v, g, state, runs, H, G, D, u)
    limit = 3.4028234663852886e38
    for got, want in ((o, want_o), (state, want_s)):
        finite = want.isfinite() & (want.abs() <= limit)
        if value != 1e12:
            assert torch.equal(got.isfinite(), finite)
        else:                                             # fp32 may leave its range where 64 bits do not; the other heads are as they were
            finite &= got.isfinite()
            cols = torch.ones_like(finite) if got is state else torch.ones_like(finite).view(-1, H, D)
            (cols[:, 0] if got is not state else cols[0, 0]).zero_()
            assert finite[cols.reshape(finite.shape)].all()
            finite &= cols.reshape(finite.shape)
        assert ((got.double() - want)[finite].abs().max() / want[finite].abs().max()).item() < 4 * (D + 64) * 2.0 ** -24


@pytest.mark.parametrize("rows,lens,H,G,D", [(65, [66, 200], 2, 2, 64), (128, [129, 384], 2, 1, 128), (200, [433, 30, 201], 4, 4, 64)])
@pytest.mark.parametrize("bonus", [False, True])
@pytest.mark.parametrize("bad", [None, 3, 90, 190])
def test_tiles_of_more_than_64_tokens(rows, lens, H, G, D, bonus, bad, monkeypatch):
    """A caller's own tiles, whose state waits in the scratch between 64 tokens and the next; with a NaN in a later part of one, too."""
    q, k, v, g, state, runs, u = case(lens, H, G, D, 0.9, bonus, seed=11)
    if bad is not None:
        k[bad, 1] = float("nan")
    want_o, want_s = walk(q, k, v, state, runs, H, G, D, g, u)
    monkeypatch.setattr(ragged, "TILE_Q", rows)
    pieces = make_pieces(runs, "cuda")
    pieces.tile_rows = rows
    assert pieces.n_tiles == sum(-(-n // rows) for n in lens)
    pos = slot = torch.zeros(q.shape[0], dtype=torch.int32, device="cuda")
    o = linear_scan(q, k, v, state, pos, slot, pieces.runs, pieces.n_runs, H, G, D, D, "channel", g=g, pieces=pieces, u=u)
    for got, want in ((o, want_o), (state, want_s)):
        finite = want.isfinite()
        assert torch.equal(got.isfinite(), finite)
        assert ((got.double() - want)[finite].abs().max() / want[finite].abs().max()).item() < 4 * (D + 64) * 2.0 ** -24


def test_a_state_that_only_the_products_lose(monkeypatch):
    """The last 16 tokens before the state is put by take it from one end of fp32's range towards the other: their own sum is outside it."""
    H = G = 1
    D = 64
    q, k, v, g, state, runs, u = case([256], H, G, D, 0.9, False, seed=12)
    runs[0][2] = 3
    g[:128, 5] = 1.0
    q[:64, 5] = 0.0
    q[64:, 5] = 1e-38
    k[:, 5] = 0.0
    k[48:64, 5] = 3.1e37
    v[48:64] = 0.0
    v[48:64, 9] = 1.0
    state[0, 0, 5] = 0.0
    state[0, 0, 5, 9] = -3e38
    want = walk(q, k, v, state.clone(), runs, H, G, D, g, u)[0][64:128]
    monkeypatch.setattr(ragged, "TILE_Q", 128)
    pieces = make_pieces(runs, "cuda")
    pieces.tile_rows = 128
    pos = slot = torch.zeros(256, dtype=torch.int32, device="cuda")
    got = linear_scan(q, k, v, state, pos, slot, pieces.runs, pieces.n_runs, H, G, D, D, "channel", g=g, pieces=pieces, u=u)[64:128]
    assert bool(got.isfinite().all()) and ((got.double() - want).abs().max() / want.abs().max()).item() < 4 * (D + 64) * 2.0 ** -24
