"""Attention whose work is dealt out in an order: backward CTAs that take several items in turn, and forward tiles by groups of heads, give
each sequence what it gets alone."""
import pytest
import torch

from llm_in_practise_b200.ops import _native as nv
from llm_in_practise_b200.ops.flash import flash_attention, flash_attention_varlen, f32, i32, i64, vp


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,H,Hkv,D", [(5, 130, 40, 8, 128),      # three rounds of query tiles, one of key blocks; two rows in the last tile
                                         (24, 70, 8, 8, 64),        # a round and a part of one of single-tile items
                                         (3, 513, 24, 24, 64),      # items of one to nine pairs
                                         (38, 64, 4, 4, 128),       # four items more than SMs, a pair each
                                         (20, 321, 16, 8, 128)])    # keys that stay in shared memory: 480 items of 2 to 12 pairs, a third one for some
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("causal", [True, False])
def test_backward_items(B, S, H, Hkv, D, dtype, causal):
    g = torch.Generator(device="cuda").manual_seed(S)
    one = torch.randn(S, (H + 2 * Hkv) * D, device="cuda", generator=g).to(dtype)
    dout = torch.randn(S, H * D, device="cuda", generator=g).to(dtype)

    def grad(n):
        x = one.repeat(n, 1).requires_grad_()
        flash_attention(x, n, S, H, Hkv, D, causal, D ** -0.5).backward(dout.repeat(n, 1))
        return x.grad.view(n, S, -1)

    alone, many = grad(1), grad(B)
    assert torch.isfinite(alone).all()
    for b in range(B):
        assert torch.equal(many[b], alone[0])                        # no sum crosses items: the same bits
    ref = one.double().requires_grad_()
    q, k, v = ref.view(1, S, H + 2 * Hkv, D).transpose(1, 2).split([H, Hkv, Hkv], 1)
    k, v = k.repeat_interleave(H // Hkv, 1), v.repeat_interleave(H // Hkv, 1)
    o = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=causal)
    o.transpose(1, 2).reshape(S, H * D).backward(dout.double())
    err = (alone[0].double() - ref.grad).norm() / ref.grad.norm()
    # P and dS are rounded to 16 bits in front of the second products, and so are the output (in delta) and the result
    assert err < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.5, float(err)


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,H,Hkv,D", [(11, 1030, 24, 24, 128),   # 133 MB of keys and values: three groups
                                         (8, 4100, 40, 8, 128),     # the same with heads that share keys; four rows in the last tile
                                         (7, 2050, 12, 12, 64)])    # one group
@pytest.mark.parametrize("causal", [True, False])
def test_forward_by_groups_of_heads(B, S, H, Hkv, D, causal):
    g = torch.Generator(device="cuda").manual_seed(S)
    x = torch.randn(B * S, (H + 2 * Hkv) * D, device="cuda", generator=g).bfloat16()
    cu = torch.arange(0, (B + 1) * S, S, device="cuda", dtype=torch.int32)
    with torch.no_grad():
        many = flash_attention(x, B, S, H, Hkv, D, causal, D ** -0.5).view(B, S, -1)
        packed = flash_attention_varlen(x, cu, S, H, Hkv, D, D ** -0.5, causal).view(B, S, -1)
        for b in range(B):
            one = x.view(B, S, -1)[b].contiguous()
            assert torch.equal(many[b], flash_attention(one, 1, S, H, Hkv, D, causal, D ** -0.5))
            assert torch.equal(packed[b], flash_attention_varlen(one, cu[:2], S, H, Hkv, D, D ** -0.5, causal))
    q, k, v = x.view(B, S, H + 2 * Hkv, D)[-1].transpose(0, 1).double().split([H, Hkv, Hkv])
    rep = H // Hkv
    ref = torch.stack([torch.nn.functional.scaled_dot_product_attention(q[h][None], k[h // rep][None], v[h // rep][None], is_causal=causal)[0] for h in (0, H - 1)], 1)
    got = packed[-1].view(S, H, D)[:, [0, H - 1]].double()
    assert (got - ref).norm() / ref.norm() < 2.0 ** -8              # P and the result are rounded to 8 bits


@pytest.mark.gpu
def test_more_tiles_than_a_grid_dimension():
    """A bound on the lengths of 8.4 million tokens: the tensor-core kernel takes the call and gives what it gives with the true one."""
    lens, H, D = [300, 0, 129], 4, 64
    x = torch.randn(sum(lens), 3 * H * D, device="cuda").bfloat16()
    cu = torch.tensor([0, 300, 300, 429], device="cuda", dtype=torch.int32)
    want = flash_attention_varlen(x, cu, 300, H, H, D, D ** -0.5)
    out = torch.zeros_like(want)
    fn = nv.proto("b200_flash_attn_varlen_fwd_tc", [vp, vp, vp, i64, i32, i32, i32, i32, i32, i32, f32, i32, vp])
    for longest in (65535 * 128, 65535 * 128 + 1, 65600 * 128):
        out.zero_()
        assert fn(x.data_ptr(), out.data_ptr(), cu.data_ptr(), x.shape[0], 3, longest, H, H, D, 1, D ** -0.5, nv.DT_BF16, nv.stream()) == 0
        assert torch.equal(out, want)
