"""The delta rule in chunks of 64 tokens against the recurrence in float64, at the edges of chunks, runs and windows of chunks."""
import pytest
import torch

from llm_in_practise_b200.ops import linear_scan as scan_mod
from llm_in_practise_b200.ops.linear_scan import linear_scan

pytestmark = pytest.mark.gpu


def walk(q, k, v, state, runs, H, G, D, Dv, a, b):
    q, k, v, a, b, state = (t.double() for t in (q, k, v, a, b, state))
    o, rep = torch.zeros(q.shape[0], H, Dv, dtype=torch.float64, device=q.device), H // G
    q, k = (t.reshape(-1, G, D).repeat_interleave(rep, 1) for t in (q, k))
    for first, n, p0, s in runs:
        S = state[s].clone() if p0 > 0 else torch.zeros_like(state[s])
        for t in range(first, first + n):
            S = S * a[t].view(H, 1, 1)
            u = b[t].view(H, 1) * (v[t].view(H, Dv) - torch.einsum("hde,hd->he", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            o[t] = torch.einsum("hde,hd->he", S, q[t])
        state[s] = S
    return o.reshape(-1, H * Dv), state


@pytest.fixture
def took(monkeypatch):
    """Sizes here are for the edges and not for the clock: every call is offered to the chunked kernels; what they answered."""
    answers, real = [], scan_mod._delta_chunks
    monkeypatch.setattr(scan_mod, "_chunks_pay", lambda *a: True)
    monkeypatch.setattr(scan_mod, "_delta_chunks", lambda *a: answers.append(real(*a)) or answers[-1])
    return answers


@pytest.mark.parametrize("lens,H,G,D,Dv", [
    ([64], 2, 1, 64, 16), ([65, 17, 63], 4, 4, 128, 48), ([1, 130, 1, 200], 4, 2, 128, 32), ([300], 6, 1, 64, 64),
    ([64, 128, 90], 20, 4, 128, 128),                     # more (run, head, column block)s than SMs
    ([8300, 40], 1, 1, 64, 16), ([2500, 70], 2, 2, 128, 32),         # more chunks than the workspace holds: three windows, two
])
@pytest.mark.parametrize("decay", [(0.9, 1.0), (0.0, 1.0), (1e-6, 1e-3)])
def test_chunks(lens, H, G, D, Dv, decay, took):
    g = torch.Generator(device="cuda").manual_seed(7)
    T, C = sum(lens), 2 * G * D + H * Dv
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)                                   # noqa: E731
    x = rnd(T, C + 4)                                     # strided rows, as a slice of a projection
    q, k, v = x[:, :G * D], x[:, G * D:2 * G * D], x[:, 2 * G * D:C]
    for t in (q, k):
        t /= t.reshape(T, G, D).norm(dim=-1).repeat_interleave(D, 1) + 1e-6
    a = torch.rand(T, H, device="cuda", generator=g) * (decay[1] - decay[0]) + decay[0]
    a[0] = 0.0
    b = torch.rand(T, H, device="cuda", generator=g)
    runs, at = [], 0
    for i, n in enumerate(lens):
        runs.append([at, n, 0 if i % 2 == 0 else 5 + i, i])
        at += n
    state = rnd(len(lens), H, D, Dv)
    want_o, want_s = walk(q, k, v, state, runs, H, G, D, Dv, a, b)
    pos = slot = torch.zeros(T, dtype=torch.int32, device="cuda")
    o = linear_scan(q, k, v, state, pos, slot, torch.tensor(runs, dtype=torch.int32, device="cuda"), len(lens), H, G, D, Dv, "head_delta", g=a, beta=b)
    assert took == [True]
    # unit keys, beta < 1: nothing grows. A value is a sum over at most D keys and 64 tokens, each term rounded a few times: D + 64
    # roundings of 2^-24 of the largest value on the way, four times over for the solve and the carried state
    for got, want in ((o, want_o), (state, want_s)):
        assert ((got.double() - want).abs().max() / want.abs().max()).item() < 4 * (D + 64) * 2.0 ** -24


@pytest.mark.parametrize("what,value", [("v", float("nan")), ("v", float("inf")), ("k", float("nan")), ("q", float("inf")), ("beta", float("nan")),
                                        ("a", float("nan"))])
@pytest.mark.parametrize("at", [5, 63, 100])
def test_not_finite_stays_behind_its_token(what, value, at, took):
    """A NaN or infinity in one token reaches that token and the ones after it (of a value's column, of a head), never those before."""
    g = torch.Generator(device="cuda").manual_seed(9)
    n, H, G, D, Dv = 130, 4, 2, 64, 32
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)                                   # noqa: E731
    q, k, v = rnd(n, G * D) * D ** -0.5, rnd(n, G * D) * D ** -0.5, rnd(n, H * Dv)
    a, b = torch.rand(n, H, device="cuda", generator=g) * 0.5 + 0.5, torch.rand(n, H, device="cuda", generator=g)
    {"v": v, "k": k, "q": q, "beta": b, "a": a}[what][at, 1] = value
    runs, state = [[0, n, 3, 0]], rnd(1, H, D, Dv)
    want_o, want_s = walk(q, k, v, state, runs, H, G, D, Dv, a, b)
    pos = slot = torch.zeros(n, dtype=torch.int32, device="cuda")
    o = linear_scan(q, k, v, state, pos, slot, torch.tensor(runs, dtype=torch.int32, device="cuda"), 1, H, G, D, Dv, "head_delta", g=a, beta=b)
    assert took == [True]
    for got, want in ((o, want_o), (state, want_s)):
        finite = want.isfinite()
        assert torch.equal(got.isfinite(), finite)
        # the bound of test_chunks
        assert not finite.any() or ((got.double() - want)[finite].abs().max() / want[finite].abs().max()).item() < 4 * (D + 64) * 2.0 ** -24


def test_rows_off_the_16_bytes_take_the_walk(took):
    """Rows that start at any float are taken all the same, token by token."""
    g = torch.Generator(device="cuda").manual_seed(10)
    n, H, G, D, Dv = 100, 2, 1, 64, 16
    x = torch.randn(n, 2 * G * D + H * Dv + 4, device="cuda", generator=g) * D ** -0.5
    q, k, v = x[:, 1:1 + G * D], x[:, 1 + G * D:1 + 2 * G * D], x[:, 1 + 2 * G * D:1 + 2 * G * D + H * Dv]
    a, b = torch.rand(n, H, device="cuda", generator=g), torch.rand(n, H, device="cuda", generator=g)
    runs, state = [[0, n, 0, 0]], torch.zeros(1, H, D, Dv, device="cuda")
    want_o, want_s = walk(q, k, v, state, runs, H, G, D, Dv, a, b)
    pos = slot = torch.zeros(n, dtype=torch.int32, device="cuda")
    o = linear_scan(q, k, v, state, pos, slot, torch.tensor(runs, dtype=torch.int32, device="cuda"), 1, H, G, D, Dv, "head_delta", g=a, beta=b)
    assert took == [False]
    for got, want in ((o, want_o), (state, want_s)):               # the bound of test_chunks
        assert ((got.double() - want).abs().max() / want.abs().max()).item() < 4 * (D + 64) * 2.0 ** -24
