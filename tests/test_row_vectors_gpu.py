"""Rotation with head norms and row norms where a row stays in registers, at the edges of the sizes that take those kernels."""
import pytest
import torch

from llm_in_practise_b200.ops.elementwise import qknorm_rope, rope_tables
from llm_in_practise_b200.ops.norm import layer_norm, rms_norm

UNIT = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -24}   # half of the step in [1, 2): 7, 10 and 23 bits are stored


@pytest.mark.gpu
@pytest.mark.parametrize("T,n_q,n_k,n_v,D,normed,dtype", [
    (1, 1, 1, 0, 64, True, torch.bfloat16),              # one block, most of it past the end
    (37, 5, 2, 2, 128, True, torch.float16),
    (37, 3, 1, 1, 64, False, torch.bfloat16),
    (130, 40, 8, 8, 128, True, torch.bfloat16),
])
def test_rotation_of_vectors(T, n_q, n_k, n_v, D, normed, dtype):
    gen = torch.Generator(device="cuda").manual_seed(T)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    qkv = rand(T, (n_q + n_k + n_v) * D).to(dtype).requires_grad_()
    qw, kw = ((1 + 0.2 * rand(D)).to(dtype), (1 + 0.2 * rand(D)).to(dtype)) if normed else (None, None)
    cos, sin = rope_tables(T + 3, D, 1e4, "cuda")
    pos = torch.randint(0, T + 3, (T,), generator=gen, device="cuda", dtype=torch.int32)
    g = rand(T, (n_q + n_k + n_v) * D).to(dtype)
    out = qknorm_rope(qkv, qw, kw, cos, sin, pos, n_q, n_k, D)
    out.backward(g)
    x = qkv.detach().double().requires_grad_()
    h = x.view(T, -1, D)
    a = h[:, :n_q + n_k]
    if normed:
        w = torch.cat([qw.double().expand(n_q, D), kw.double().expand(n_k, D)])
        a = a * torch.rsqrt(a.pow(2).mean(-1, keepdim=True) + 1e-6) * w
    c, s = cos.double()[pos.long()][:, None], sin.double()[pos.long()][:, None]
    lo, hi = a[..., :D // 2], a[..., D // 2:]
    ref = torch.cat([torch.cat([lo * c - hi * s, hi * c + lo * s], -1), h[:, n_q + n_k:]], 1).reshape(T, -1)
    ref.backward(g.double())
    # forward: both members of a pair are rounded twice before they are turned, the result once; backward: once
    mag = torch.cat([(lo.abs() + hi.abs()).repeat(1, 1, 2), h[:, n_q + n_k:].abs()], 1).reshape(T, -1).detach()
    assert ((out.double() - ref).abs() <= 3.01 * UNIT[dtype] * mag + 1e-6).all()
    err, dx = (qkv.grad.double() - x.grad).abs(), x.grad.abs()
    assert (err <= 1.01 * UNIT[dtype] * dx + 2.0 ** -18 * dx.amax(-1, keepdim=True) + 1e-7).all()   # 2^-18: sums of 128 in fp32
    if n_v:
        assert torch.equal(out[:, (n_q + n_k) * D:], qkv[:, (n_q + n_k) * D:]) and torch.equal(qkv.grad[:, (n_q + n_k) * D:], g[:, (n_q + n_k) * D:])


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols,kind,res,dtype,wtype", [
    (3, 8, "rms", False, torch.bfloat16, torch.bfloat16),          # one vector
    (5, 2048, "rms", True, torch.bfloat16, torch.bfloat16),        # 256 vectors, one per thread
    (5, 2056, "layer", True, torch.bfloat16, torch.float32),       # two per thread, the second with a remainder
    (7, 5120, "rms", True, torch.float16, torch.float16),
    (2, 8192, "layer", False, torch.bfloat16, torch.bfloat16),     # the widest row
    (2, 8200, "rms", True, torch.bfloat16, torch.bfloat16),        # wider: the forward alone takes it
    (4, 4096, "rms", True, torch.float32, torch.float32),
])
def test_row_norms(rows, cols, kind, res, dtype, wtype):
    gen = torch.Generator(device="cuda").manual_seed(cols)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x = rand(rows, cols).to(dtype).requires_grad_()
    r = rand(rows, cols).to(dtype).requires_grad_() if res else None
    w, b = (1 + 0.2 * rand(cols)).to(wtype), (0.2 * rand(cols)).to(wtype) if kind == "layer" else None
    backward = cols * x.element_size() <= 16 * 1024
    gy, gh = rand(rows, cols).to(dtype), rand(rows, cols).to(dtype)
    y, h = rms_norm(x, w, 1e-6, r) if kind == "rms" else layer_norm(x, w, b, 1e-6, r)
    hd = (x.detach() + r.detach() if res else x.detach()).double().requires_grad_()
    m = hd.mean(-1, keepdim=True) if kind == "layer" else 0.0
    ref = (hd - m) * torch.rsqrt((hd - m).pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    if b is not None:
        ref = ref + b.double()
    if res:
        assert torch.equal(h, (x + r).detach())
    tol = lambda v: 1.01 * UNIT[dtype] * v.abs() + 2.0 ** -18 * v.abs().amax(-1, keepdim=True)   # the rounding, and sums of `cols` in fp32
    assert ((y.double() - ref).abs() <= tol(ref.detach())).all()
    if backward:
        (y * gy).sum().backward() if not res else torch.autograd.backward([y, h], [gy, gh])
        want = torch.autograd.grad(ref, hd, gy.double())[0]
        if res:
            want = want + gh.double()
        assert ((x.grad.double() - want).abs() <= tol(want)).all()
        if res:
            assert torch.equal(x.grad, r.grad)
