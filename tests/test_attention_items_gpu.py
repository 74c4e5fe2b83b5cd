"""Attention backward: CTAs that take several items in turn give each what it gets alone."""
import pytest
import torch

from llm_in_practise_b200.ops.flash import flash_attention


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,H,Hkv,D", [(5, 130, 40, 8, 128),      # three rounds of query tiles, one of key blocks; two rows in the last tile
                                         (24, 70, 8, 8, 64),        # a round and a part of one of single-tile items
                                         (3, 513, 24, 24, 64),      # items of one to nine pairs
                                         (38, 64, 4, 4, 128)])      # four items more than SMs, a pair each
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
