"""Forward attention of more tiles than are resident at once, against the same sequences alone. A CTA goes on from tile to tile where there are more
than 592; the others here ([128] * 9) take a CTA each."""
import pytest
import torch

from llm_in_practise_b200.ops.flash import _fwd, flash_attention_varlen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Hkv,D", [(40, 8, 128), (48, 48, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("lens", [[1, 63, 700, 129, 65, 2, 300, 64], [128] * 9, [128] * 16, [5, 1300]])
def test_packed_tiles_in_turn(H, Hkv, D, dtype, causal, lens):
    """Tiles past a sequence's end, of one row to 128, of one key block to twenty: the bits of a call that one CTA a tile takes."""
    g = torch.Generator(device="cuda").manual_seed(len(lens))
    qkv = torch.randn(sum(lens), (H + 2 * Hkv) * D, device="cuda", generator=g).to(dtype)
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).to(torch.int32).cuda()
    assert len(lens) * H * -(-max(lens) // 128) > 296
    got = flash_attention_varlen(qkv, cu, max(lens), H, Hkv, D, D ** -0.5, causal)
    # a key head at a time: at most 55 tiles
    x, rep, at = qkv.view(-1, H + 2 * Hkv, D), H // Hkv, 0
    for n in lens:
        for j in range(0, Hkv, 7):
            one = torch.cat([x[at:at + n, j * rep:(j + 1) * rep], x[at:at + n, H + j:H + j + 1], x[at:at + n, H + Hkv + j:H + Hkv + j + 1]], 1).reshape(n, -1).contiguous()
            alone = flash_attention_varlen(one, torch.tensor([0, n], dtype=torch.int32, device="cuda"), n, rep, 1, D, D ** -0.5, causal)
            assert torch.equal(got[at:at + n].view(n, H, D)[:, j * rep:(j + 1) * rep].reshape(n, -1), alone)
        at += n


@pytest.mark.parametrize("B,S,H,Hkv,D", [(9, 300, 40, 8, 128), (100, 33, 12, 12, 64), (2, 2100, 24, 24, 64)])
def test_dense_tiles_in_turn(B, S, H, Hkv, D):
    """Outputs and log-sum-exps, and the same from a replayed graph."""
    g = torch.Generator(device="cuda").manual_seed(S)
    qkv = torch.randn(B * S, (H + 2 * Hkv) * D, device="cuda", generator=g).bfloat16()
    out, lse = _fwd(qkv, B, S, H, Hkv, D, True, D ** -0.5)
    assert B * H * -(-S // 128) > 296
    x, rep = qkv.view(B * S, H + 2 * Hkv, D), H // Hkv
    for b in range(0, B, 4):
        for j in range(0, Hkv, 5):
            r = slice(b * S, (b + 1) * S)
            one = torch.cat([x[r, j * rep:(j + 1) * rep], x[r, H + j:H + j + 1], x[r, H + Hkv + j:H + Hkv + j + 1]], 1).reshape(S, -1).contiguous()
            o, l = _fwd(one, 1, S, rep, 1, D, True, D ** -0.5)
            assert torch.equal(out[r].view(S, H, D)[:, j * rep:(j + 1) * rep].reshape(S, -1), o)
            assert torch.equal(lse[b, j * rep:(j + 1) * rep], l[0])
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        again, lse2 = _fwd(qkv, B, S, H, Hkv, D, True, D ** -0.5)
    for _ in range(2):
        again.zero_(); lse2.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(again, out) and torch.equal(lse2, lse)


@pytest.mark.parametrize("dtype,eps", [(torch.bfloat16, 2.0 ** -9), (torch.float16, 2.0 ** -12)])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("lens,H,Hkv,D", [([30, 700, 129, 64], 28, 7, 128), ([256] * 30, 12, 12, 64)])
def test_tiles_in_turn_against_fp64(lens, H, Hkv, D, dtype, eps, causal):
    """Packed, and where the lengths are equal dense as well. Weights and results are rounded to 16 bits, each by at most eps of itself."""
    g = torch.Generator(device="cuda").manual_seed(D)
    qkv = torch.randn(sum(lens), (H + 2 * Hkv) * D, device="cuda", generator=g).to(dtype)
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).to(torch.int32).cuda()
    assert len(lens) * H * -(-max(lens) // 128) > 592
    got = [flash_attention_varlen(qkv, cu, max(lens), H, Hkv, D, D ** -0.5, causal)]
    if len(set(lens)) == 1:
        got.append(_fwd(qkv, len(lens), lens[0], H, Hkv, D, causal, D ** -0.5)[0])
    x, at = qkv.double().view(-1, H + 2 * Hkv, D).transpose(0, 1), 0
    for n in lens:
        q, k, v = x[:H, at:at + n], x[H:H + Hkv, at:at + n], x[H + Hkv:, at:at + n]
        k, v = k.repeat_interleave(H // Hkv, 0), v.repeat_interleave(H // Hkv, 0)
        s = q @ k.transpose(1, 2) * D ** -0.5
        if causal:
            s = s.masked_fill(torch.ones(n, n, device="cuda").triu(1).bool(), float("-inf"))
        p = torch.softmax(s, -1)
        ref, most = (p @ v).transpose(0, 1).reshape(n, -1), (p @ v.abs()).transpose(0, 1).reshape(n, -1)
        for o in got:
            # eps for each weight and for the result, and as much again for the exponentials and the sums in fp32
            assert bool(((o[at:at + n].double() - ref).abs() <= 4 * eps * most + 2.0 ** -24).all())
        at += n
