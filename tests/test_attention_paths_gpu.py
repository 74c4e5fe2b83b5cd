"""Attention kernels that a rule on sizes picks, at the sizes where they can go wrong (tile edges, remainders, single keys), against
the package's plain PyTorch path on the CPU."""
import pytest
import torch

from llm_in_practise_b200.ops.multimap_attention import multimap_attention

pytestmark = pytest.mark.gpu

# Both sides round to bf16, whose neighbours are up to 2^-7 of a value apart: two roundings of nearly the same number differ by at
# most one such step. What the kernels add on top (fp32 sums, 2^-17 of every probability, 2^-22 of every exponential) stays below
# 2^-12 of the largest value; the bound has twice that.
def close(got, want, vmax=4.0):
    got, want = got.float().cpu(), want.float()
    bound = 2.0 ** -7 * want.abs() + 2.0 ** -11 * vmax
    worst = ((got - want).abs() - bound).max().item()
    assert worst <= 0, f"{worst} over the bound"


def pools(rows, G, M, D, Dv, BS, seed=0):
    """Pools in shuffled pages for sequences of ``rows`` keys each; the table's unset entries point at page 0, which holds NaN."""
    g = torch.Generator().manual_seed(seed)
    per = [-(-n // BS) for n in rows]
    order = (torch.randperm(sum(per), generator=g) + 1).to(torch.int32)
    table = torch.zeros(len(rows), max(per), dtype=torch.int32)
    at = 0
    for i, n in enumerate(per):
        table[i, :n] = order[at:at + n]
        at += n
    ck = torch.randn(at + 1, G * M, BS, D, generator=g).to(torch.bfloat16)
    cv = torch.randn(at + 1, G, BS, Dv, generator=g).to(torch.bfloat16)
    ck[0] = cv[0] = float("nan")
    return ck, cv, table, g


@pytest.mark.parametrize("H,G,M,D,Dv", [(4, 4, 1, 128, 128), (16, 4, 1, 128, 128), (10, 2, 1, 64, 64), (24, 2, 1, 128, 128), (20, 1, 1, 64, 128),
                                        (8, 2, 2, 64, 128), (4, 1, 2, 128, 64)])
@pytest.mark.parametrize("opt", ["none", "window", "chunk"])
@pytest.mark.parametrize("BS", [16, 64])
def test_decode_batches(H, G, M, D, Dv, opt, BS):
    rows = [1, 2, 15, 16, 17, 64, 65, 129, 640, 777]              # keys of a tile, of a warp's round, of a range, and one beside each
    ck, cv, table, g = pools(rows, G, M, D, Dv, BS)
    T = len(rows)
    q = torch.randn(T, H * M * D, generator=g).to(torch.bfloat16)
    pos, slot = torch.tensor([n - 1 for n in rows], dtype=torch.int32), torch.arange(T, dtype=torch.int32)
    kw = {}
    if opt == "window":
        kw = dict(window=50, keep_first=3)
    if M == 1 and opt == "window":
        kw["sink"] = torch.randn(H, generator=g)
    if M == 1 and opt == "chunk":
        kw = dict(chunk=48, softcap=5.0, gate=torch.randn(T, H, generator=g))
    if M == 2:
        kw.update(combine=opt != "none", lam=0.3, post=0.8, eps=1e-5)
    args = (ck, cv, table, pos, slot, H, G, M, D, Dv, D ** -0.5)
    want = multimap_attention(q, *args, **kw)
    dev = lambda v: v.cuda() if isinstance(v, torch.Tensor) else v                                  # noqa: E731
    for max_pos in (0, 776):                                       # without and with the keys cut into ranges
        got = multimap_attention(q.cuda(), *map(dev, args), max_pos=max_pos, **{k: dev(v) for k, v in kw.items()})
        close(got, want)
