"""Numerics of every CUDA kernel vs a plain PyTorch fp32 reference of the same op: the oracle of every kernel is
the plain torch expression that the reference's script executes."""
import os

import pytest
import torch
import torch.nn.functional as F

from llm_in_practise_b200.ops import elementwise as ew
from llm_in_practise_b200.ops import norm as N
from llm_in_practise_b200.ops import loss as L
from llm_in_practise_b200.ops import w4 as W4
from llm_in_practise_b200.ops import lora as LR
from llm_in_practise_b200.ops.attention import attention, _ref_attention

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel(a, b):
    return ((a.float() - b.float()).abs().max() / (b.float().abs().max() + 1e-6)).item()


@pytest.mark.parametrize("layer_norm", [False, True])
@pytest.mark.parametrize("dtype,cols", [(torch.bfloat16, 5120), (torch.bfloat16, 768), (torch.float32, 128)])
def test_norm_fwd_bwd(layer_norm, dtype, cols):
    rows = 300
    x = torch.randn(rows, cols, device=DEV, dtype=dtype, requires_grad=True)
    r = torch.randn(rows, cols, device=DEV, dtype=dtype, requires_grad=True)
    w = (1 + 0.1 * torch.randn(cols, device=DEV)).to(dtype).requires_grad_()
    b = (0.1 * torch.randn(cols, device=DEV)).to(dtype).requires_grad_() if layer_norm else None
    f = N.layer_norm if layer_norm else N.rms_norm
    args = (x, w, b, 1e-5, r) if layer_norm else (x, w, 1e-6, r)
    y, h = f(*args)
    gy, gh = torch.randn_like(y), torch.randn_like(h)
    (y * gy).sum().backward(retain_graph=True)
    (h * gh).sum().backward()
    got = [y, h, x.grad, r.grad, w.grad] + ([b.grad] if layer_norm else [])
    # fp32 oracle
    xf, rf, wf = x.detach().float().requires_grad_(), r.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    bf = b.detach().float().requires_grad_() if layer_norm else None
    hf = (xf + rf)
    if layer_norm:
        yf = F.layer_norm(hf, (cols,), wf, bf, 1e-5)
    else:
        yf = hf * torch.rsqrt(hf.pow(2).mean(-1, keepdim=True) + 1e-6) * wf
    ((yf * gy.float()).sum() + (hf * gh.float()).sum()).backward()
    want = [yf, hf, xf.grad, rf.grad, wf.grad] + ([bf.grad] if layer_norm else [])
    tol = 2e-2 if dtype == torch.bfloat16 else 1e-4
    for g, wnt in zip(got, want):
        assert rel(g, wnt) < tol


@pytest.mark.parametrize("interleaved,D", [(False, 128), (True, 96), (False, 64)])
def test_qknorm_rope(interleaved, D):
    T, H, Hkv = 70, 4, 2
    qkv = torch.randn(T, (H + 2 * Hkv) * D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    qw = (1 + 0.1 * torch.randn(D, device=DEV)).bfloat16().requires_grad_()
    kw = (1 + 0.1 * torch.randn(D, device=DEV)).bfloat16().requires_grad_()
    cos, sin = ew.rope_tables(128, D, 10000.0, DEV)
    pos = torch.randint(0, 128, (T,), device=DEV, dtype=torch.int32)
    out = ew.qknorm_rope(qkv, qw, kw, cos, sin, pos, H, Hkv, D, interleaved)
    g = torch.randn_like(out)
    (out * g).sum().backward()
    # oracle in fp32
    q32 = qkv.detach().float().requires_grad_()
    qw32, kw32 = qw.detach().float().requires_grad_(), kw.detach().float().requires_grad_()
    ref_qk = ew._ref_qknorm_rope(q32[:, :(H + Hkv) * D], qw32, kw32, cos, sin, pos, H, Hkv, D, interleaved, 1e-6)
    ref = torch.cat([ref_qk, q32[:, (H + Hkv) * D:]], dim=1)
    (ref * g.float()).sum().backward()
    assert rel(out, ref) < 2e-2
    assert rel(qkv.grad, q32.grad) < 3e-2
    assert rel(qw.grad, qw32.grad) < 3e-2
    assert rel(kw.grad, kw32.grad) < 3e-2


def test_swiglu_gelu():
    gu = torch.randn(257, 2 * 1024, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    h = ew.swiglu(gu)
    g = torch.randn_like(h)
    (h * g).sum().backward()
    g32 = gu.detach().float().requires_grad_()
    ref = F.silu(g32[:, :1024]) * g32[:, 1024:]
    (ref * g.float()).sum().backward()
    assert rel(h, ref) < 2e-2 and rel(gu.grad, g32.grad) < 2e-2
    x = torch.randn(64, 768, device=DEV, requires_grad=True)
    y = ew.gelu(x)
    (y * 2).sum().backward()
    x2 = x.detach().clone().requires_grad_()
    (F.gelu(x2) * 2).sum().backward()
    assert rel(y, F.gelu(x2)) < 1e-5 and rel(x.grad, x2.grad) < 1e-4


def test_embedding_and_dropout():
    table = torch.randn(1000, 256, device=DEV, requires_grad=True)
    pos = torch.randn(64, 256, device=DEV, requires_grad=True)
    ids = torch.randint(0, 1000, (4, 64), device=DEV)
    out = ew.embedding(ids, table, pos)
    g = torch.randn_like(out)
    (out * g).sum().backward()
    t2, p2 = table.detach().clone().requires_grad_(), pos.detach().clone().requires_grad_()
    ref = F.embedding(ids, t2) + p2
    (ref * g).sum().backward()
    assert rel(out, ref) < 1e-6 and rel(table.grad, t2.grad) < 1e-5 and rel(pos.grad, p2.grad) < 1e-5
    x = torch.randn(1 << 20, device=DEV, requires_grad=True)
    y = ew.dropout(x, 0.1, True, seed=1234)
    keep = (y != 0).float().mean().item()
    assert abs(keep - 0.9) < 5e-3
    assert torch.allclose(y[y != 0], (x / 0.9)[y != 0])
    y.sum().backward()
    assert torch.equal(x.grad != 0, y != 0)


@pytest.mark.parametrize("dtype,V", [(torch.bfloat16, 151936), (torch.float32, 30528), (torch.bfloat16, 1000)])
def test_cross_entropy(dtype, V):
    M = 96
    logits = (3 * torch.randn(M, V, device=DEV)).to(dtype).requires_grad_()
    t = torch.randint(0, V, (M,), device=DEV)
    t[::7] = -100
    loss = L.cross_entropy(logits, t)
    loss.backward()
    l32 = logits.detach().float().requires_grad_()
    ref = F.cross_entropy(l32, t, ignore_index=-100)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 2e-3 * max(1, abs(ref.item()))
    assert rel(logits.grad, l32.grad) < (2e-2 if dtype == torch.bfloat16 else 1e-4)


def test_linear_cross_entropy():
    M, K, V = 300, 256, 5003
    x = torch.randn(M, K, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(V, K, device=DEV) / 16).bfloat16().requires_grad_()
    t = torch.randint(0, V, (M,), device=DEV)
    t[:10] = -100
    loss = L.linear_cross_entropy(x, w, t, chunk_tokens=128)
    loss.backward()
    x32, w32 = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    ref = F.cross_entropy(x32 @ w32.t(), t, ignore_index=-100)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 5e-3 * abs(ref.item())
    assert rel(x.grad, x32.grad) < 3e-2 and rel(w.grad, w32.grad) < 3e-2


@pytest.mark.parametrize("trainable_head", [False, True])
def test_linear_cross_entropy_vocab_chunked(trainable_head, monkeypatch):
    """K8 without a [tokens, vocab] tensor: one online-softmax pass for a frozen head (per-row-beta GEMM accumulation),
    two passes for a trainable one; vocabulary 20011 (not a multiple of the chunk nor of 8), per-row weights, ignored rows."""
    monkeypatch.setattr(L, "_VOCAB_CHUNK", 4096)
    monkeypatch.setattr(L, "_VOCAB_CHUNK_MIN_BYTES", 0)
    M, K, V = 300, 256, 20011
    x = torch.randn(M, K, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(V, K, device=DEV) / 16).bfloat16().requires_grad_(trainable_head)
    t = torch.randint(0, V, (M,), device=DEV)
    t[:10] = -100
    t[10] = V - 1                                   # a target in the last, partial chunk
    rs = L.micro_batch_row_scale(t, 2)
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    loss = L.linear_cross_entropy(x, w, t, row_scale=rs)
    loss.backward()
    peak = torch.cuda.max_memory_allocated() - base
    # frozen head: everything allocated stays below ONE bf16 [tokens, vocab] tensor; a trainable head also owns its
    # fp32 gradient (and the temporary it is formed in): allow those
    assert peak < M * V * 2 + (3 * V * K * 4 if trainable_head else 0), "a [tokens, vocab] tensor was allocated"
    x32, w32 = x.detach().float().requires_grad_(), w.detach().float().requires_grad_(trainable_head)
    rows = F.cross_entropy(x32 @ w32.t(), t, ignore_index=-100, reduction="none")
    ref = torch.dot(rows, rs)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 5e-3 * abs(ref.item())
    assert rel(x.grad, x32.grad) < 3e-2
    if trainable_head:
        assert rel(w.grad, w32.grad) < 3e-2


def test_linear_cross_entropy_main_grad_scaling_and_eval():
    """A head weight with a flat-arena ``main_grad``: evaluation under no_grad leaves it untouched, a declared upstream
    scale (engines: 1 / grad_accum) is folded into what forward accumulates, and an undeclared ``(loss * c).backward()``
    still lands ``c * dW`` there (gradient accumulation with ga = 2, an eval pass in between, vs the torch reference)."""
    M, K, V = 256, 128, 1000
    w = (torch.randn(V, K, device=DEV) / 8).bfloat16().requires_grad_()
    w.main_grad = torch.zeros(V, K, device=DEV, dtype=torch.float32)
    xs = [torch.randn(M, K, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    ts = [torch.randint(0, V, (M,), device=DEV) for _ in range(2)]

    def ref_grads(c):
        w32 = w.detach().float().requires_grad_()
        gx = []
        for x, t in zip(xs, ts):
            x32 = x.float().requires_grad_()
            (F.cross_entropy(x32 @ w32.t(), t) * c).backward()
            gx.append(x32.grad)
        return w32.grad, gx

    # (a) declared scale, as the ZeRO engine / pretrain loop do, with an evaluation pass between the micro-steps
    want_w, want_x = ref_grads(0.5)
    got_x = []
    for i, (x, t) in enumerate(zip(xs, ts)):
        xi = x.clone().requires_grad_()
        with L.grad_scale_context(0.5):
            loss = L.linear_cross_entropy(xi, w, t)
        (loss * 0.5).backward()
        got_x.append(xi.grad)
        if i == 0:
            before = w.main_grad.clone()
            with torch.no_grad():
                L.linear_cross_entropy(xs[1], w, ts[1])
            assert torch.equal(w.main_grad, before), "an eval pass must not touch the gradient arena"
    assert w.grad is None
    assert rel(w.main_grad, want_w) < 2e-2
    for g, r in zip(got_x, want_x):
        assert rel(g, r) < 2e-2
    # (b) nothing declared: the factor autograd delivers is applied in backward
    w.main_grad.zero_()
    want_w, _ = ref_grads(0.25)
    for x, t in zip(xs, ts):
        (L.linear_cross_entropy(x.clone().requires_grad_(), w, t) * 0.25).backward()
    assert rel(w.main_grad, want_w) < 2e-2


def test_nf4_roundtrip_and_double_quant():
    w = torch.randn(512, 1024, device=DEV, dtype=torch.bfloat16)
    packed, absmax = W4.nf4_quantize(w)
    p_ref, a_ref = W4._nf4_quantize_ref(w)
    assert torch.equal(absmax, a_ref)
    assert (packed != p_ref).float().mean().item() < 1e-3   # ties only
    deq = W4.w4_dequant(packed, absmax, None, 512, 1024, 64)
    ref = W4._w4_dequant_ref(packed, absmax, None, 512, 1024, 64, None, torch.bfloat16)
    assert torch.equal(deq, ref)
    assert rel(deq, w) < 0.2  # 4-bit quantisation error
    q = W4.NF4Weight.quantize(w, double_quant=True, keep_decoded=False)
    assert rel(q.scales(), absmax) < 0.02
    assert rel(q.dequantize(), w) < 0.25


def test_w4_dequant_transposed_and_dgrad():
    from llm_in_practise_b200.ops.linear import FusedLinear
    w = torch.randn(512, 1024, device=DEV, dtype=torch.bfloat16)
    q = W4.NF4Weight.quantize(w, double_quant=True)
    assert torch.equal(q.dequantize(transpose=True), q.dequantize().t().contiguous())
    # asymmetric W4A16 (zs, integer LUT, group 128) through the same kernel
    packed = torch.randint(0, 256, (256 * 384 // 2,), device=DEV, dtype=torch.uint8)
    scale = torch.rand(256 * 384 // 128, device=DEV) * 0.01 + 0.001
    lut = torch.arange(16, device=DEV, dtype=torch.float32)
    a = W4.w4_dequant(packed, scale, scale * 7, 256, 384, 128, lut, torch.float16)
    b = W4.w4_dequant(packed, scale, scale * 7, 256, 384, 128, lut, torch.float16, transpose=True)
    assert torch.equal(b, a.t().contiguous())
    # the frozen-base backward uses it: dX must match dY @ W
    lin = FusedLinear(1024, [("p", 512)], dtype=torch.bfloat16, device=DEV)
    lin.weight.data.copy_(w)
    lin.quantize_nf4(True)
    x = torch.randn(256, 1024, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(256, 512, device=DEV, dtype=torch.bfloat16)
    lin(x).backward(dy)
    assert rel(x.grad, dy.float() @ lin.nf4.dequantize().float()) < 1e-2


@pytest.mark.parametrize("r,K", [(32, 1024), (64, 512), (8, 1030)])
def test_lora_small_kernels_wide_ranks(r, K):
    M = 300
    x = torch.randn(M, K + 8, device=DEV, dtype=torch.bfloat16)[:, 2:K + 2] if K % 8 else torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    pm = torch.randn(M, r, device=DEV, dtype=torch.bfloat16)
    G = torch.zeros(r, K, device=DEV)
    LR.lora_wgrad(pm, x, G, 1.0, 5, 0.0)
    assert rel(G, pm.float().t() @ x.float()) < 2e-2
    if K % 8 == 0:
        a = (torch.randn(r, K, device=DEV) / 8).bfloat16()
        assert rel(LR.lora_down(x, a, 1.0, 5, 0.0), x.float() @ a.float().t()) < 2e-2


def test_w4_gemv_matches_dequant():
    N_, K, g = 1024, 2048, 128
    packed = torch.randint(0, 256, (N_ * K // 2,), device=DEV, dtype=torch.uint8)
    scale = torch.rand(N_ * K // g, device=DEV) * 0.01 + 0.001
    zs = scale * 8
    lut = torch.arange(16, device=DEV, dtype=torch.float32)
    x = torch.randn(3, K, device=DEV, dtype=torch.float16)
    y = W4.w4_gemv(x, packed, scale, zs, N_, K, g, lut)
    wd = W4.w4_dequant(packed, scale, zs, N_, K, g, lut, torch.float16)
    assert rel(y, x.float() @ wd.float().t()) < 5e-3


@pytest.mark.parametrize("r,p", [(8, 0.0), (16, 0.1)])
def test_lora_small_kernels(r, p):
    M, K = 1000, 1536
    x = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    a = (torch.randn(r, K, device=DEV) / 8).bfloat16()
    seed = 777
    mask = LR.keep_mask((M, K), seed, p, DEV).float() / (1 - p) if p > 0 else torch.ones(M, K, device=DEV)
    T = LR.lora_down(x, a, 0.5, seed, p)
    assert rel(T, 0.5 * (x.float() * mask) @ a.float().t()) < 2e-2
    pm = torch.randn(M, r, device=DEV, dtype=torch.bfloat16)
    G = torch.zeros(r, K, device=DEV)
    LR.lora_wgrad(pm, x, G, 2.0, seed, p)
    assert rel(G, 2.0 * pm.float().t() @ (x.float() * mask)) < 2e-2
    dx = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    dx0 = dx.clone()
    LR.lora_dx(pm, a, dx, 1.5, seed, p)
    assert rel(dx, dx0.float() + 1.5 * mask * (pm.float() @ a.float())) < 2e-2


def test_lora_down_tensor_core_edges():
    """mma.sync lora_down: token count not a multiple of 8, rank not a multiple of 8, strided activations, dropout."""
    M, K, r, p, seed = 1003, 2048, 12, 0.2, 4242
    x = torch.randn(M, K + 64, device=DEV, dtype=torch.bfloat16)[:, 32:K + 32]          # row stride K + 64, 16-byte aligned
    a = (torch.randn(r, K, device=DEV) / 8).bfloat16()
    mask = LR.keep_mask((M, K), seed, p, DEV).float() / (1 - p)
    T = LR.lora_down(x, a, 2.0, seed, p)
    assert T.shape == (M, r)
    assert rel(T, 2.0 * (x.float() * mask) @ a.float().t()) < 2e-2


@pytest.mark.parametrize("H,Hkv,D,S", [(8, 2, 128, 256), (12, 12, 64, 255), (4, 4, 64, 100), (4, 2, 128, 1536), (2, 2, 64, 1032)])
def test_attention_tiled(H, Hkv, D, S):
    B = 2
    Sp = (S + 7) // 8 * 8
    if Sp != S:
        pytest.skip("tiled path needs S % 8 == 0 (callers pad)")
    qkv = torch.randn(B * S, (H + 2 * Hkv) * D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    out = attention(qkv, B, S, H, Hkv, D, causal=True, impl="tiled")
    g = torch.randn_like(out)
    (out * g).sum().backward()
    q32 = qkv.detach().float().requires_grad_()
    ref = _ref_attention(q32, B, S, H, Hkv, D, True, 0, D ** -0.5)
    (ref * g.float()).sum().backward()
    assert rel(out, ref) < 2e-2
    assert rel(qkv.grad, q32.grad) < 3e-2


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (128, torch.float16), (32, torch.bfloat16), (96, torch.float16)])
def test_flash_attention_dropout(D, dtype, causal):
    """In-kernel attention-probability dropout: the mask is read back through one-hot values (q = k = 0 makes P uniform),
    then forward and backward with random inputs and the same seed must match the fp32 reference that uses that mask."""
    from llm_in_practise_b200.ops.flash import flash_attention
    B, H, Hkv, S, p, seed = 2, 4, 2, D, 0.25, 0x1234ABCD5678
    g = H // Hkv
    W = (H + 2 * Hkv) * D
    probe = torch.zeros(B, S, H + 2 * Hkv, D, device=DEV, dtype=dtype)
    probe[:, :, H + Hkv:] = torch.eye(S, device=DEV, dtype=dtype)[None, :, None, :]          # v[key] = one-hot(key)
    with torch.no_grad():
        o = flash_attention(probe.view(B * S, W), B, S, H, Hkv, D, False, D ** -0.5, p, seed)
    pm = o.view(B, S, H, D).permute(0, 2, 1, 3).float() * S                                  # [B, H, row, key] = mask / keep
    keep = (pm > 0)
    assert abs(keep.float().mean().item() - (1 - p)) < 0.02
    assert torch.allclose(pm[keep], torch.full_like(pm[keep], 1 / (1 - p)), rtol=2e-2)
    torch.manual_seed(5)
    qkv = torch.randn(B * S, W, device=DEV, dtype=dtype, requires_grad=True)
    out = flash_attention(qkv, B, S, H, Hkv, D, causal, D ** -0.5, p, seed)
    go = torch.randn_like(out)
    (out * go).sum().backward()
    q32 = qkv.detach().float().requires_grad_()
    t = q32.view(B, S, H + 2 * Hkv, D)
    q, k, v = t[:, :, :H].permute(0, 2, 1, 3), t[:, :, H:H + Hkv].permute(0, 2, 1, 3), t[:, :, H + Hkv:].permute(0, 2, 1, 3)
    sc = torch.matmul(q, k.repeat_interleave(g, 1).transpose(-1, -2)) * D ** -0.5
    if causal:
        i = torch.arange(S, device=DEV)
        sc = sc.masked_fill(i[None, :] > i[:, None], float("-inf"))
    ref = torch.matmul(torch.softmax(sc, -1) * keep.float() / (1 - p), v.repeat_interleave(g, 1))
    ref = ref.permute(0, 2, 1, 3).reshape(B * S, H * D)
    (ref * go.float()).sum().backward()
    assert rel(out, ref) < 2e-2
    assert rel(qkv.grad, q32.grad) < 3e-2


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("H,Hkv,D,S,dtype", [(8, 2, 128, 256, torch.bfloat16), (12, 12, 64, 255, torch.bfloat16),
                                             (5, 1, 128, 77, torch.float16), (4, 2, 128, 1100, torch.bfloat16),
                                             (40, 8, 128, 512, torch.bfloat16), (2, 2, 64, 64, torch.float16),
                                             (4, 4, 32, 256, torch.bfloat16), (8, 2, 96, 200, torch.bfloat16),
                                             (6, 3, 96, 130, torch.float16), (4, 1, 32, 77, torch.float16)])
def test_flash_attention(H, Hkv, D, S, dtype, causal):
    """csrc/flash_attn.cu forward + backward against the fp32 reference of the same op (any S, GQA, both mask modes)."""
    B = 2
    torch.manual_seed(S + H)
    qkv = torch.randn(B * S, (H + 2 * Hkv) * D, device=DEV, dtype=dtype, requires_grad=True)
    out = attention(qkv, B, S, H, Hkv, D, causal=causal, impl="flash")
    g = torch.randn_like(out)
    (out * g).sum().backward()
    q32 = qkv.detach().float().requires_grad_()
    ref = _ref_attention(q32, B, S, H, Hkv, D, causal, 0, D ** -0.5)
    (ref * g.float()).sum().backward()
    assert rel(out, ref) < 2e-2
    W = (H + 2 * Hkv) * D
    for name, lo, hi in (("dq", 0, H * D), ("dk", H * D, (H + Hkv) * D), ("dv", (H + Hkv) * D, W)):
        assert rel(qkv.grad[:, lo:hi], q32.grad[:, lo:hi]) < 3e-2, name
    with torch.no_grad():
        out2 = attention(qkv, B, S, H, Hkv, D, causal=causal)
    assert torch.equal(out2, out)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("gain", [1.0, 3.0])
@pytest.mark.parametrize("H,Hkv,S,dtype", [(8, 2, 512, torch.bfloat16), (4, 4, 77, torch.float16), (5, 1, 200, torch.bfloat16),
                                           (2, 2, 1000, torch.bfloat16), (2, 1, 128, torch.float16), (3, 3, 64, torch.bfloat16)])
def test_flash_attention_tcgen05_forward(H, Hkv, S, dtype, causal, gain, monkeypatch):
    """csrc/flash_tc.cu (tcgen05 / TMEM / TMA forward, head_dim 128): context vs the fp32 reference, log-sum-exp vs the
    mma.sync kernel (the backward kernel consumes it), sequence lengths that do not fill the 128 x 64 tiles, GQA.
    gain 3 spreads the scores over ~±40 (log2 units), so the running maximum is raised in late key blocks too and the
    O accumulator in TMEM is rescaled there."""
    from llm_in_practise_b200.ops import flash as FL
    B, D = 2, 128
    torch.manual_seed(S * 3 + H)
    qkv = (torch.randn(B * S, (H + 2 * Hkv) * D, device=DEV) * gain).to(dtype)
    monkeypatch.setattr(FL, "_TC", True)
    out, lse = FL._fwd(qkv, B, S, H, Hkv, D, causal, D ** -0.5, True)
    monkeypatch.setattr(FL, "_TC", False)
    out_old, lse_old = FL._fwd(qkv, B, S, H, Hkv, D, causal, D ** -0.5, True)
    ref = _ref_attention(qkv.float(), B, S, H, Hkv, D, causal, 0, D ** -0.5)
    assert rel(out, ref) < 2e-2, rel(out, ref)
    assert rel(out_old, ref) < 2e-2
    assert (lse - lse_old).abs().max().item() < 2e-2


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("H,Hkv,S,dtype", [(8, 2, 512, torch.bfloat16), (4, 4, 77, torch.float16), (5, 1, 200, torch.bfloat16),
                                           (2, 2, 1000, torch.bfloat16), (2, 1, 128, torch.float16), (3, 3, 64, torch.bfloat16)])
def test_flash_attention_tcgen05_backward(H, Hkv, S, dtype, causal, monkeypatch):
    """csrc/flash_bwd_tc.cu (dK/dV pass + dQ pass on tcgen05, no atomics): gradient of the fused projection against autograd
    through the fp32 reference attention, ragged sequence lengths, GQA groups accumulated inside one CTA."""
    from llm_in_practise_b200.ops import flash as FL
    B, D = 2, 128
    torch.manual_seed(S * 7 + H)
    qkv = torch.randn(B * S, (H + 2 * Hkv) * D, device=DEV).to(dtype).requires_grad_()
    g = torch.randn(B * S, H * D, device=DEV).to(dtype)
    monkeypatch.setattr(FL, "_TC", True)
    monkeypatch.setattr(FL, "_TC_BWD", True)
    out = FL.flash_attention(qkv, B, S, H, Hkv, D, causal, D ** -0.5)
    (dq,) = torch.autograd.grad(out, qkv, g)
    q32 = qkv.detach().float().requires_grad_()
    ref = _ref_attention(q32, B, S, H, Hkv, D, causal, 0, D ** -0.5)
    (dref,) = torch.autograd.grad(ref, q32, g.float())
    for name, lo, hi in (("dq", 0, H * D), ("dk", H * D, (H + Hkv) * D), ("dv", (H + Hkv) * D, (H + 2 * Hkv) * D)):
        assert rel(dq[:, lo:hi], dref[:, lo:hi]) < 3e-2, (name, rel(dq[:, lo:hi], dref[:, lo:hi]))


def test_adamw_and_8bit():
    from llm_in_practise_b200.optim import FusedAdamW, PagedAdamW8bit
    from llm_in_practise_b200.utils.arena import ParamArena
    n = 10000
    for cls, tol in [(FusedAdamW, 1e-5), (PagedAdamW8bit, 5e-2)]:
        arena = ParamArena(device=DEV)
        i = arena.request("w", (n,))
        arena.finalize()
        arena.data.normal_()
        ref = torch.nn.Parameter(arena.data.clone())
        opt = cls(arena, lr=1e-2, weight_decay=0.01)
        ropt = torch.optim.AdamW([ref], lr=1e-2, weight_decay=0.01)
        for _ in range(10):
            g = torch.randn(arena.numel, device=DEV)
            arena.grad.copy_(g)
            ref.grad = g.clone()
            opt.step()
            ropt.step()
        assert rel(arena.data, ref.data) < tol, cls.__name__


@pytest.mark.parametrize("M", [1, 8, 13, 40, 64])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_small_m_gemv_kernels(M, dtype):
    from llm_in_practise_b200.ops.gemm import gemv16
    torch.manual_seed(M)
    N_, K = 1000, 1024                      # N not a multiple of 16: the last row tile is partial
    x = torch.randn(M, K, device=DEV, dtype=dtype)
    w = (torch.randn(N_, K, device=DEV) / 32).to(dtype)
    b = torch.randn(N_, device=DEV, dtype=dtype)
    ref = x.float() @ w.float().t() + b.float()
    assert rel(gemv16(x, w, b), ref) < 1e-2
    assert rel(gemv16(x, w, None, out_dtype=torch.float32), x.float() @ w.float().t()) < 5e-3
    packed = torch.randint(0, 256, (N_ * K // 2,), device=DEV, dtype=torch.uint8)
    scale = torch.rand(N_ * K // 128, device=DEV) * 0.01 + 0.001
    lut = torch.arange(16, device=DEV, dtype=torch.float32)
    y = W4.w4_gemv(x, packed, scale, scale * 8, N_, K, 128, lut, b)
    wd = W4.w4_dequant(packed, scale, scale * 8, N_, K, 128, lut, dtype)
    assert rel(y, x.float() @ wd.float().t() + b.float()) < 1e-2
    # integer codes take the table-free kernel; a non-linear table (NF4, or this shuffled one) and symmetric int4 with the
    # offset inside the table (lut[c] = c - 8, no zero term) must agree with the dequantised product too
    assert W4.linear_lut(lut) == (1.0, 0.0)
    for tbl, zs in ((lut - 8, None), (lut.flip(0).contiguous() * 0.5, None), (torch.tensor([0.1 * (c % 5) - c * c / 100 for c in range(16)], device=DEV), scale * 0.3)):
        y2 = W4.w4_gemv(x, packed, scale, zs, N_, K, 128, tbl, None)
        wd2 = W4.w4_dequant(packed, scale, zs, N_, K, 128, tbl, dtype)
        assert rel(y2, x.float() @ wd2.float().t()) < 1e-2
    assert W4.linear_lut(lut - 8) == (1.0, 8.0) and W4.linear_lut(lut.flip(0).contiguous() * 0.5) == (-0.5, 15.0)


@pytest.mark.parametrize("kind", ["dense", "nf4", "int4"])
@pytest.mark.parametrize("M,K", [(1, 1024), (8, 1024), (33, 1024), (2, 128), (2, 256), (8, 384)])
def test_gemv_fused_tail_matches_separate_ops(kind, M, K):
    """b200_gemv_fused at TP 1: projection + residual add + RMSNorm in one launch vs the fp32 torch expression. The short
    contractions are what a row-parallel layer is left with at TP 8 on small models (K = 128: one quantisation group)."""
    from llm_in_practise_b200.ops import fused_decode as FD
    from llm_in_practise_b200.ops.linear import FusedLinear
    torch.manual_seed(5)
    N = 2048
    lin = FusedLinear(K, [("o_proj", N)], dtype=torch.bfloat16, device=DEV, init_std=0.05)
    wref = lin.weight.data.float().clone()
    if kind == "nf4":
        lin.quantize_nf4(True)
        wref = lin.nf4.dequantize(torch.float32).float()
    elif kind == "int4":
        from llm_in_practise_b200.quant.formats import quantize_rtn
        q = quantize_rtn(lin.weight.data, 128, True)
        lin.set_nf4(q)
        wref = W4._w4_dequant_ref(q.packed, q.scale, q.zs, N, K, 128, q._lut(), torch.float32)
    x = torch.randn(M, K, device=DEV).bfloat16()
    res = torch.randn(M, N, device=DEV).bfloat16()
    nw = (1 + 0.1 * torch.randn(N, device=DEV)).bfloat16()
    assert FD.supported(lin, x, N)
    tail = FD.FusedTail(N, torch.device(DEV))
    for rep in range(2):            # the second call starts from the first one's epoch / tickets
        out, res_out = FD.gemv_fused(lin, x, res, nw, 1e-6, tail)
    h = (x.float() @ wref.t()).bfloat16().float() + res.float()
    hb = h.bfloat16().float()
    want = hb * torch.rsqrt(hb.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.float()
    assert rel(res_out, hb) < 2e-2 and rel(out, want) < 2e-2


@pytest.mark.parametrize("T,E,k", [(1000, 8, 2), (77, 4, 1), (4096, 8, 2)])
def test_moe_grouped_gemm_matches_expert_loop(T, E, k):
    """K16 (ops/moe.py): device-side counting sort + ONE grouped tcgen05 GEMM per projection (b_map picks the expert's weight
    per 128-row tile, unused tiles skipped) against the per-expert loop in fp32, forward and all gradients."""
    from llm_in_practise_b200.ops.moe import moe_ffn
    from llm_in_practise_b200.ops import elementwise as ew
    torch.manual_seed(T + E)
    D, H = 256, 512
    dt = torch.bfloat16
    x = (torch.randn(T, D, device=DEV) * 0.5).to(dt).requires_grad_()
    w1 = (torch.randn(E, H, D, device=DEV) * D ** -0.5).to(dt).requires_grad_()
    b1 = (torch.randn(E, H, device=DEV) * 0.1).to(dt).requires_grad_()
    w2 = (torch.randn(E, D, H, device=DEV) * H ** -0.5).to(dt).requires_grad_()
    b2 = (torch.randn(E, D, device=DEV) * 0.1).to(dt).requires_grad_()
    logits = torch.randn(T, E, device=DEV)
    if E > 4:
        logits[:, 5] = -1e9                                # an expert without tokens
    top_v, top_i = torch.topk(logits, k, dim=-1)
    top_p = torch.softmax(top_v, -1)
    from llm_in_practise_b200.ops import _native as nvm
    n0 = nvm.launch_count
    out, d = moe_ffn(x, top_i, top_p.to(dt), w1, b1, w2, b2, ew.gelu)
    assert nvm.launch_count - n0 >= 2                         # the two grouped launches went through the native library
    xf, w1f, b1f, w2f, b2f = (t.detach().float().requires_grad_() for t in (x, w1, b1, w2, b2))
    ref = torch.zeros(T, D, device=DEV)
    for e in range(E):
        for s in range(k):
            m = top_i[:, s] == e
            if m.any():
                y = torch.nn.functional.gelu(xf[m] @ w1f[e].T + b1f[e]) @ w2f[e].T + b2f[e]
                ref = ref.index_add(0, m.nonzero().squeeze(1), y * top_p[m, s:s + 1])
    assert rel(out, ref) < 2e-2, rel(out, ref)
    g = torch.randn(T, D, device=DEV)
    grads = torch.autograd.grad(out, [x, w1, b1, w2, b2], g.to(dt))
    grads_ref = torch.autograd.grad(ref, [xf, w1f, b1f, w2f, b2f], g)
    for name, a, b in zip(("dx", "dw1", "db1", "dw2", "db2"), grads, grads_ref):
        assert rel(a, b) < 3e-2, (name, rel(a, b))


def test_deepseeklike_flash_mla_and_grouped_moe_match_fp32_model():
    """K16 + K17 in the model: bf16 DeepSeekLike on the native paths (latent attention on the flash kernels with the latent
    dim zero-padded to 32, grouped-GEMM MoE) against the SAME weights in fp32 on the batched-matmul / expert-loop paths."""
    from llm_in_practise_b200.models.deepseeklike import DeepSeekLike
    torch.manual_seed(1)
    kw = dict(vocab_size=512, block_size=128, n_layer=2, n_head=4, d_model=256, dropout=0.0, num_experts=8, top_k=2, num_shared=1)
    ref = DeepSeekLike(dtype=torch.float32, device="cpu", **kw)                 # plain torch paths (matmul attention, expert loop)
    m = DeepSeekLike(dtype=torch.bfloat16, device=DEV, **kw)
    m.load_state_dict({k: v.to(torch.bfloat16) for k, v in ref.state_dict().items()})
    ref.load_state_dict({k: v.float().cpu() for k, v in m.state_dict().items()})      # identical (bf16-representable) weights
    ids = torch.randint(0, 512, (4, 128), device=DEV)
    la, lb = m(ids, ids), ref(ids.cpu(), ids.cpu())
    assert abs(float(la) - float(lb)) < 3e-2 * abs(float(lb)), (float(la), float(lb))
    la.backward()
    lb.backward()
    ga = torch.cat([p.grad.float().reshape(-1).cpu() for p in m.parameters()])
    gb = torch.cat([p.grad.float().reshape(-1) for p in ref.parameters()])
    assert float((ga - gb).norm() / gb.norm()) < 8e-2


def test_dropout_seed_offset_from_device_memory():
    """b200_set_graph_state: a dropout launch captured in a CUDA graph drops different elements at every replay (the per-step
    part of the Philox seed is read from device memory), forward and backward of one replay use the same mask."""
    import ctypes
    from llm_in_practise_b200.ops import _native as nvm
    x = torch.ones(1 << 16, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    off = torch.zeros(1, dtype=torch.int64, device=DEV)
    fn = nvm.proto("b200_set_graph_state", [ctypes.c_void_p])
    nvm.check(fn(off.data_ptr()), "set_graph_state")
    try:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            y = ew.dropout(x, 0.25, True, seed=1234)
            y.sum().backward()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        x.grad = None
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            y = ew.dropout(x, 0.25, True, seed=1234)
            (gx,) = torch.autograd.grad(y.sum(), x)
        masks = []
        for step in range(3):
            off.fill_(step * 7919)
            g.replay()
            torch.cuda.synchronize()
            keep = y.detach() != 0
            assert torch.equal(keep, gx != 0)                      # backward regenerated the forward's mask
            assert abs(float(keep.float().mean()) - 0.75) < 0.02
            masks.append(keep.clone())
        assert not torch.equal(masks[0], masks[1]) and not torch.equal(masks[1], masks[2])
        off.fill_(0)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y.detach() != 0, masks[0])             # same offset, same mask
    finally:
        nvm.check(fn(None), "set_graph_state")


def test_graphed_train_step_matches_eager_and_trains_with_dropout():
    """utils/graph_step.GraphedTrainStep: forward + backward + AdamW + zero_grad of a small GPTLike replayed from ONE CUDA
    graph. Without dropout the parameters follow the eager run step for step (learning rate and bias corrections reach the
    captured optimizer kernel through device memory); with dropout the loss still falls and differs from replay to replay."""
    import ctypes
    from llm_in_practise_b200.models.gpt import GPTLike
    from llm_in_practise_b200.ops import _native as nvm
    from llm_in_practise_b200.parallel.ddp import DistributedDataParallel as DDP
    from llm_in_practise_b200.utils.graph_step import GraphedTrainStep

    def build(dropout):
        torch.manual_seed(3)
        ew.manual_seed(11)
        m = GPTLike(512, 64, 2, 4, 128, dropout=dropout, dtype=torch.bfloat16, device=DEV)
        d = DDP(m, mixed_precision=torch.bfloat16)
        return m, d, d.make_optimizer(lr=3e-3, weight_decay=0.01)

    def loss_of(d, x):
        o = d(x, x)
        return o[1] if isinstance(o, tuple) else o

    x = torch.randint(0, 512, (4, 64), device=DEV, generator=torch.Generator(device=DEV).manual_seed(1))
    try:
        # ---- parity without dropout: 3 warm-up steps inside GraphedTrainStep + 5 replays == 8 eager steps ----
        m1, d1, o1 = build(0.0)
        for _ in range(8):
            loss_of(d1, x).backward()
            o1.step()
            d1.zero_grad()
        m2, d2, o2 = build(0.0)
        gs = GraphedTrainStep(lambda t: loss_of(d2, t), o2, [x], zero_grad=d2.zero_grad, warmup=3)
        for _ in range(5):
            lg = gs(x)
        torch.cuda.synchronize()
        p1 = torch.cat([p.detach().float().reshape(-1) for p in m1.parameters()])
        p2 = torch.cat([p.detach().float().reshape(-1) for p in m2.parameters()])
        assert o2._step == 8 and float((p1 - p2).norm() / p1.norm()) < 2e-2      # bf16 + atomics in the embedding backward: not bit-reproducible
        # ---- with dropout: trains, and no two replays see the same loss (different masks) ----
        m3, d3, o3 = build(0.1)
        gs3 = GraphedTrainStep(lambda t: loss_of(d3, t), o3, [x], zero_grad=d3.zero_grad, warmup=3)
        losses = [float(gs3(x)) for _ in range(30)]
        assert losses[-1] < 0.7 * losses[0] and len(set(round(v, 5) for v in losses)) > 25
    finally:
        nvm.check(nvm.proto("b200_set_graph_state", [ctypes.c_void_p])(None), "set_graph_state")


@pytest.mark.parametrize("T,k,E,tile", [(1, 1, 1, 128), (32, 2, 8, 128), (37, 3, 5, 8), (700, 4, 64, 16), (4096, 2, 8, 128), (513, 6, 300, 32)])
def test_moe_dispatch_kernel_matches_the_sorted_layout(T, k, E, tile, monkeypatch):
    """The one-launch dispatch gives the layout of the stable sort by expert: destinations, tokens, tile map, counts; experts
    that receive nothing (one is forced) take no tile."""
    from llm_in_practise_b200.ops import _native as nv
    from llm_in_practise_b200.ops import moe
    g = torch.Generator().manual_seed(T + E)
    top_i = torch.randint(0, E, (T, k), generator=g)
    if E > 2:
        top_i[top_i == 1] = E - 1                                    # expert 1 receives nothing
    top_i = top_i.cuda()
    got = moe.dispatch(top_i, E, tile)
    real = nv.has
    monkeypatch.setattr(nv, "has", lambda name: name != "b200_moe_dispatch" and real(name))
    want = moe.dispatch(top_i, E, tile)
    assert got.rows == want.rows and got.num_experts == want.num_experts
    for a in ("dest", "tok", "tile_map", "counts"):
        assert torch.equal(getattr(got, a), getattr(want, a)), a
    assert got.host_counts() == want.counts.tolist()


@pytest.mark.parametrize("W", [64, 100, 2048])
@pytest.mark.parametrize("hd,wd", [(torch.bfloat16, torch.float32), (torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_router_logits_any_width(W, hd, wd):
    from llm_in_practise_b200.ops.moe import ROUTE_SOFTMAX_ALL, route_grouped, route_topk
    g = torch.Generator().manual_seed(W)
    T, E, top = 77, 11, 3
    h = torch.randn(T, W, generator=g).to(hd).cuda()
    w = (torch.randn(E, W, generator=g) * W ** -0.5 * 3).to(wd).cuda()
    s = torch.softmax(h.double() @ w.double().T, -1)
    wp, wi = torch.topk(s, top, dim=-1)
    for ti, tp in (route_topk(h, w, None, top, ROUTE_SOFTMAX_ALL)[:2], route_grouped(h, w, None, top, 1, 1, 1, softmax=True)[:2]):
        assert torch.equal(ti, wi)
        assert torch.allclose(tp.double(), wp, atol=1e-5, rtol=1e-4)
