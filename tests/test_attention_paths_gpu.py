"""Attention kernels that a rule on sizes picks, at the sizes where they can go wrong (tile edges, remainders, single keys), against
the package's plain PyTorch path on the CPU."""
import pytest
import torch

from llm_in_practise_b200.ops.multimap_attention import multimap_attention

pytestmark = pytest.mark.gpu

@pytest.fixture
def entries(monkeypatch):
    """Names of the entry points that took a call (those that handed it back are not among them)."""
    from llm_in_practise_b200.ops import _native as nv
    names, real = set(), nv.proto

    def proto(name, argtypes):
        fn = real(name, argtypes)

        def call(*args):
            rc = fn(*args)
            if rc == 0:
                names.add(name)
            return rc
        return call
    monkeypatch.setattr(nv, "proto", proto)
    return names


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


@pytest.mark.parametrize("H,G,D", [(4, 2, 128), (8, 2, 64), (10, 2, 64), (2, 2, 128), (3, 1, 128)])
@pytest.mark.parametrize("opt", ["none", "window", "chunk"])
@pytest.mark.parametrize("BS", [8, 16, 64, 128])
def test_prompt_pieces(H, G, D, opt, BS, entries):
    """Pieces that start and end anywhere in pages and 64-key blocks, single tokens beside them, keys past the end that are NaN."""
    from llm_in_practise_b200.inference.ragged import make_pieces
    runs = [(65, 0), (1, 130), (9, 63), (130, 200), (64, 64), (1, 0)]                # (tokens, first position)
    ck, cv, table, g = pools([n + p for n, p in runs], G, 1, D, D, BS)
    pos = torch.cat([torch.arange(p, p + n) for n, p in runs]).to(torch.int32)
    slot = torch.cat([torch.full((n,), i) for i, (n, _) in enumerate(runs)]).to(torch.int32)
    T = pos.numel()
    for i, (n, p) in enumerate(runs):                                                # what lies behind a sequence in its last page
        if (n + p) % BS:
            ck[table[i, (n + p) // BS], :, (n + p) % BS:] = float("nan")
            cv[table[i, (n + p) // BS], :, (n + p) % BS:] = float("nan")
    q = torch.randn(T, H * D, generator=g).to(torch.bfloat16)
    kw = {}
    if opt == "window":
        kw = dict(window=70, keep_first=3, sink=torch.randn(H, generator=g))
    if opt == "chunk":
        kw = dict(chunk=100, softcap=5.0, gate=torch.randn(T, H, generator=g), post=0.7)
    args = (ck, cv, table, pos, slot, H, G, 1, D, D, D ** -0.5)
    want = multimap_attention(q, *args, **kw)
    dev = lambda v: v.cuda() if isinstance(v, torch.Tensor) else v                                  # noqa: E731
    firsts = [sum(n for n, _ in runs[:i]) for i in range(len(runs))]
    pieces = make_pieces([(f, n, p, i) for i, (f, (n, p)) in enumerate(zip(firsts, runs))], "cuda")
    wide = torch.zeros(T, H * D + 8, dtype=torch.bfloat16, device="cuda")
    for out in (None, wide[:, :H * D]):
        got = multimap_attention(q.cuda(), *map(dev, args), pieces=pieces, max_pos=329, out=out, **{k: dev(v) for k, v in kw.items()})
        # here P is rounded to bf16 before the product (as in the mma.sync kernel): 2^-9 of every term, which averages out over the
        # sum to well below 2^-9 of the largest value; the bound grants it in full
        close(got, want, vmax=16.0)
    assert entries == {"b200_paged_attn_tc"}


@pytest.mark.parametrize("H,Hkv,D", [(4, 2, 128), (6, 6, 64), (4, 1, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("causal", [True, False])
def test_packed_prompts(H, Hkv, D, dtype, causal, entries):
    """Lengths at the edges of key blocks and query tiles; a NaN in the sequence behind must not reach the one in front."""
    from llm_in_practise_b200.ops.flash import flash_attention_varlen
    lens = [1, 63, 64, 65, 128, 129, 200, 7]
    g = torch.Generator().manual_seed(3)
    qkv = torch.randn(sum(lens), (H + 2 * Hkv) * D, generator=g).to(dtype)
    qkv[-7:] = float("nan")
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).to(torch.int32)
    want = flash_attention_varlen(qkv, cu, max(lens), H, Hkv, D, D ** -0.5, causal)
    got = flash_attention_varlen(qkv.cuda(), cu.cuda(), max(lens), H, Hkv, D, D ** -0.5, causal)
    close(got[:-7], want[:-7], vmax=16.0)
    assert torch.isnan(got[-7:]).all()
    assert entries == {"b200_flash_attn_varlen_fwd_tc"}


@pytest.mark.parametrize("B,S,H,Hkv,D", [(2, 1, 2, 1, 64), (3, 65, 2, 2, 64), (2, 129, 4, 2, 64), (1, 300, 6, 2, 128), (2, 256, 3, 3, 64)])
@pytest.mark.parametrize("causal", [True, False])
def test_fused_qkv_forward(B, S, H, Hkv, D, causal, entries):
    """Forward with the log-sum-exp the backward reads; a batch entry whose last rows are NaN leaves the ones beside it alone."""
    from llm_in_practise_b200.ops.attention import _ref_attention
    from llm_in_practise_b200.ops.flash import _fwd
    g = torch.Generator().manual_seed(4)
    qkv = torch.randn(B * S, (H + 2 * Hkv) * D, generator=g).to(torch.bfloat16)
    want = _ref_attention(qkv, B, S, H, Hkv, D, causal, 0, D ** -0.5)
    got, lse = _fwd(qkv.cuda(), B, S, H, Hkv, D, causal, D ** -0.5)
    close(got, want, vmax=16.0)
    t = qkv.double().view(B, S, H + 2 * Hkv, D)
    k = t[:, :, H:H + Hkv].repeat_interleave(H // Hkv, 2)
    sc = torch.einsum("bqhd,bkhd->bhqk", t[:, :, :H], k) * D ** -0.5
    if causal:
        sc = sc.masked_fill(~torch.ones(S, S, dtype=torch.bool).tril(), float("-inf"))
    # products of bf16 numbers are exact in fp32, a sum of D of them is good to D 2^-24 of its terms: 1e-5 at these sizes
    assert (lse.double().cpu() - torch.logsumexp(sc, -1)).abs().max().item() < 1e-4
    if B > 1:
        qkv[-S:] = float("nan")
        again, _ = _fwd(qkv.cuda(), B, S, H, Hkv, D, causal, D ** -0.5)
        assert torch.equal(again[:-S], got[:-S])
    assert entries == {"b200_flash_attn_fwd_tc"}


@pytest.mark.parametrize("B,S,H,Hkv", [(2, 1, 2, 1), (2, 64, 3, 3), (1, 65, 4, 2), (2, 129, 4, 1), (1, 300, 6, 2)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_fused_qkv_backward(B, S, H, Hkv, D, causal, entries):
    """Gradient of the fused projection at the edges of key blocks, query tiles and groups of heads, against float64 autograd."""
    from llm_in_practise_b200.ops.flash import flash_attention
    g = torch.Generator(device="cuda").manual_seed(5)
    qkv = torch.randn(B * S, (H + 2 * Hkv) * D, device="cuda", generator=g).to(torch.bfloat16).requires_grad_()
    go = torch.randn(B * S, H * D, device="cuda", generator=g).to(torch.bfloat16)
    flash_attention(qkv, B, S, H, Hkv, D, causal, D ** -0.5).backward(go)
    x = qkv.detach().double().requires_grad_()
    t = x.view(B, S, H + 2 * Hkv, D).transpose(1, 2)
    q, k, v = t[:, :H], t[:, H:H + Hkv].repeat_interleave(H // Hkv, 1), t[:, H + Hkv:].repeat_interleave(H // Hkv, 1)
    sc = q @ k.transpose(-1, -2) * D ** -0.5
    if causal:
        sc = sc.masked_fill(~torch.ones(S, S, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    (sc.softmax(-1) @ v).transpose(1, 2).reshape(B * S, H * D).backward(go.double())
    # P, dS, the forward's output behind delta and the result are rounded to bf16 (2^-9 each, independent): four times their root sum
    for lo, hi in ((0, H * D), (H * D, (H + Hkv) * D), ((H + Hkv) * D, (H + 2 * Hkv) * D)):
        a, b = qkv.grad[:, lo:hi].double(), x.grad[:, lo:hi]
        assert (a - b).norm() <= 4 * 2 * 2.0 ** -9 * b.norm() + 2.0 ** -9 * go.double().norm() * (S == 1)
    assert entries == {"b200_flash_attn_fwd_tc", "b200_flash_attn_bwd_tc"}


def exact_fused(x, B, S, H, Hkv, D, causal, scale):
    """Context [B * S, H * D] of the fused projection ``x`` in its own precision (float64 here), differentiable."""
    t = x.view(B, S, H + 2 * Hkv, D).transpose(1, 2)
    q, k, v = t[:, :H], t[:, H:H + Hkv].repeat_interleave(H // Hkv, 1), t[:, H + Hkv:].repeat_interleave(H // Hkv, 1)
    sc = q @ k.transpose(-1, -2) * scale
    if causal:
        sc = sc.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=x.device).tril(), float("-inf"))
    return (sc.softmax(-1) @ v).transpose(1, 2).reshape(B * S, H * D)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("scale", [0.0, -0.1])
def test_scale_not_positive(D, scale, entries):
    """Equal weights (scale 0) and reversed ones under the causal mask: a masked score stays minus infinity whatever it is multiplied by."""
    from llm_in_practise_b200.ops.flash import flash_attention, flash_attention_varlen
    B, S, H, Hkv = 2, 130, 4, 2
    g = torch.Generator(device="cuda").manual_seed(6)
    qkv = torch.randn(B * S, (H + 2 * Hkv) * D, device="cuda", generator=g).to(torch.bfloat16).requires_grad_()
    go = torch.randn(B * S, H * D, device="cuda", generator=g).to(torch.bfloat16)
    out = flash_attention(qkv, B, S, H, Hkv, D, True, scale)
    out.backward(go)
    x = qkv.detach().double().requires_grad_()
    want = exact_fused(x, B, S, H, Hkv, D, True, scale)
    want.backward(go.double())
    close(out.detach(), want.detach().cpu(), vmax=16.0)
    for lo, hi in ((0, H * D), (H * D, (H + Hkv) * D), ((H + Hkv) * D, (H + 2 * Hkv) * D)):
        a, b = qkv.grad[:, lo:hi].double(), x.grad[:, lo:hi]       # the bound of test_fused_qkv_backward; exactly zero at scale 0
        assert (a - b).norm() <= 4 * 2 * 2.0 ** -9 * b.norm()
    cu = torch.tensor([0, S, 2 * S], dtype=torch.int32, device="cuda")
    close(flash_attention_varlen(qkv.detach(), cu, S, H, Hkv, D, scale), want.detach().cpu(), vmax=16.0)
    assert entries == {"b200_flash_attn_fwd", "b200_flash_attn_bwd", "b200_flash_attn_varlen_fwd"}


@pytest.mark.parametrize("S", [1, 65, 129, 200])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_backward_leaves_neighbours_alone(S, D, causal):
    """The last tile of a batch entry ends inside the entry behind it: NaN there (queries, keys, values, gradient) must not arrive."""
    from llm_in_practise_b200.ops.flash import flash_attention
    H, Hkv = 4, 2
    g = torch.Generator(device="cuda").manual_seed(7)
    qkv = torch.randn(2 * S, (H + 2 * Hkv) * D, device="cuda", generator=g).to(torch.bfloat16)
    go = torch.randn(2 * S, H * D, device="cuda", generator=g).to(torch.bfloat16)
    grads = []
    for poison in (False, True):
        x, d = qkv.clone(), go.clone()
        if poison:
            x[S:], d[S:] = float("nan"), float("nan")
        x.requires_grad_()
        flash_attention(x, 2, S, H, Hkv, D, causal, D ** -0.5).backward(d)
        grads.append(x.grad[:S])
    assert torch.equal(*grads)


@pytest.mark.parametrize("H,G,M,D,Dv", [(16, 4, 1, 128, 128), (12, 1, 1, 64, 64), (4, 2, 2, 64, 128)])
def test_decode_values_not_finite(H, G, M, D, Dv):
    """An infinite value weighted by a probability above zero is infinite, and it stays in its own column."""
    rows = [1, 5, 70, 300]
    ck, cv, table, g = pools(rows, G, M, D, Dv, 16)
    inf = float("inf")
    for i, n in enumerate(rows):                                   # (key, column, value): the first key, one inside and the last
        for key, col, v in ((0, 0, inf), (n // 2, 3, -inf), (n - 1, Dv - 1, inf), (n // 3, 8, float("nan")), (0, 9, inf), (n - 1, 9, -inf)):
            cv[table[i, key // 16], :, key % 16, col] = v
    T = len(rows)
    q = torch.randn(T, H * M * D, generator=g).to(torch.bfloat16)
    pos, slot = torch.tensor([n - 1 for n in rows], dtype=torch.int32), torch.arange(T, dtype=torch.int32)
    args = (ck, cv, table, pos, slot, H, G, M, D, Dv, D ** -0.5)
    want = multimap_attention(q, *args).float()
    dev = lambda v: v.cuda() if isinstance(v, torch.Tensor) else v                                  # noqa: E731
    for max_pos in (0, 299):
        got = multimap_attention(q.cuda(), *map(dev, args), max_pos=max_pos).float().cpu()
        finite = want.isfinite()
        assert torch.equal(got.isfinite(), finite)
        assert torch.equal(got[~finite].nan_to_num(nan=0.0), want[~finite].nan_to_num(nan=0.0))
        close(got[finite], want[finite])


@pytest.mark.parametrize("H,G,D", [(4, 2, 128), (3, 1, 64), (4, 2, 96)])
def test_capped_rows_do_not_see_what_lies_behind(H, G, D):
    """Which of the two forms of tanh a block's scores take must not depend on rows behind the sequence (large numbers or zeros there) nor on
    the other rows of the tile. 96: the mma.sync kernel."""
    from llm_in_practise_b200.inference.ragged import make_pieces
    n, BS, cap = 70, 64, 1000.0                                    # scores of about 10: x = score / cap is small, its error times cap is not
    ck, cv, table, g = pools([n], G, 1, D, D, BS)
    q = torch.randn(n, H * D, generator=g).to(torch.bfloat16)
    pos, slot = torch.arange(n, dtype=torch.int32), torch.zeros(n, dtype=torch.int32)
    pieces = make_pieces([(0, n, 0, 0)], "cuda")
    got = []
    for behind in (0.0, 100.0):
        ck[table[0, 1], :, n - BS:] = behind
        got.append(multimap_attention(q.cuda(), ck.cuda(), cv.cuda(), table.cuda(), pos.cuda(), slot.cuda(), H, G, 1, D, D, 10 * D ** -0.5,
                                      pieces=pieces, max_pos=n - 1, softcap=cap))
    assert torch.equal(*got)
    q[40] *= 64                                                    # one row with large scores leaves the others alone
    again = multimap_attention(q.cuda(), ck.cuda(), cv.cuda(), table.cuda(), pos.cuda(), slot.cuda(), H, G, 1, D, D, 10 * D ** -0.5,
                               pieces=pieces, max_pos=n - 1, softcap=cap)
    others = torch.arange(n) != 40
    assert torch.equal(again.cpu()[others], got[1].cpu()[others])


@pytest.mark.parametrize("form,D", [("dense", 64), ("packed", 64), ("packed", 128), ("paged", 64), ("paged", 128)])
def test_largest_weight_is_exact(form, D):
    """Keys far below but for one in the first block and a somewhat larger one in the second, whose weight is then 1 in 16 bits too: the
    first one's value is zero, so that the result is v / (1 + e^-d) with nothing rounded but the result."""
    from llm_in_practise_b200.inference.ragged import make_pieces
    from llm_in_practise_b200.ops.flash import flash_attention, flash_attention_varlen
    H, S, dtype = 8, 128, torch.bfloat16
    g = torch.Generator().manual_seed(8)
    q, k = torch.zeros(S, H, D, dtype=dtype), torch.zeros(S, H, D, dtype=dtype)
    v = torch.randn(S, H, D, generator=g).to(dtype)
    d = torch.linspace(0.3, 5.0, H).to(dtype)                      # below 2^8 in weight
    q[:, :, 0], k[:, :, 0] = 1.0, -100.0
    k[3, :, 0], k[70, :, 0], v[3] = 0.0, d, 0.0
    want = (v[70].double() / (1 + torch.exp(-d.double()))[:, None]).reshape(1, H * D)
    qkv = torch.cat([q, k, v], 1).reshape(S, 3 * H * D).cuda()
    if form == "dense":
        got = flash_attention(qkv, 1, S, H, H, D, True, 1.0)
    elif form == "packed":
        got = flash_attention_varlen(qkv, torch.tensor([0, S], dtype=torch.int32, device="cuda"), S, H, H, D, 1.0)
    else:
        pos, slot = torch.arange(S, dtype=torch.int32, device="cuda"), torch.zeros(S, dtype=torch.int32, device="cuda")
        page = lambda t: t.transpose(0, 1)[None].contiguous().cuda()                               # noqa: E731
        got = multimap_attention(q.reshape(S, -1).cuda(), page(k), page(v), torch.zeros(1, 1, dtype=torch.int32, device="cuda"), pos, slot,
                                 H, H, 1, D, D, 1.0, pieces=make_pieces([(0, S, 0, 0)], "cuda"), max_pos=S - 1)
    got = got[70:].double().cpu()
    half = 2.0 ** (torch.floor(torch.log2(want.abs())) - 8)        # half a step of bf16 at the result
    assert ((got - want).abs() <= half * (1 + 2.0 ** -8)).all()    # 2^-8 of it: 2^-16 of the result, far above fp32's part


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="two GPUs in one process")
def test_second_device():
    """The opt-in to large shared memory belongs to a device: one process that uses two of them, one after the other."""
    from llm_in_practise_b200.ops.flash import flash_attention, flash_attention_varlen
    for D in (64, 128):
        per = []
        for dev in ("cuda:0", "cuda:1"):
            with torch.cuda.device(dev):
                x = torch.randn(130, 3 * 2 * D, generator=torch.Generator().manual_seed(9)).to(torch.bfloat16).to(dev).requires_grad_()
                out = flash_attention(x, 1, 130, 2, 2, D, True, D ** -0.5)
                out.backward(out.detach())
                cu = torch.tensor([0, 130], dtype=torch.int32, device=dev)
                per.append([t.cpu() for t in (out.detach(), x.grad, flash_attention_varlen(x.detach(), cu, 130, 2, 2, D, D ** -0.5))])
        assert all(torch.equal(a, b) for a, b in zip(*per))
