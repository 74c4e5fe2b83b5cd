"""Decode products over 4-bit integer codes for at most 16 tokens: units of four chunks dealt to the warps, slices of k in clusters."""
import ctypes

import pytest
import torch

from llm_in_practise_b200.ops import _native as nv
from llm_in_practise_b200.ops.w4 import w4_gemv


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,group,zeros,bias,dtype,split", [
    (1, 8, 128, 128, True, False, torch.bfloat16, {1}),        # less than a tile, one chunk
    (8, 40, 640, 128, True, True, torch.bfloat16, {1, 2}),     # five chunks: a whole unit and one of a single chunk; scales not in fours
    (9, 16 * 149, 1152, 384, False, False, torch.float16, {1, 2, 4}),  # more tiles than CTAs; a scale over three chunks
    (16, 2000, 4224, 128, True, True, torch.float16, {1, 2, 4}),
    (5, 4096, 12288, 128, True, False, torch.bfloat16, {2, 4}),   # slices of k in a cluster
    (13, 1000, 17408, 256, True, True, torch.bfloat16, {4}),   # 68 units over four slices
    (16, 5120, 17408, 128, False, False, torch.bfloat16, {4}),
    (8, 40, 65536, 128, True, False, torch.bfloat16, {0}),     # no slice of the activations fits: the kernel for any size
    (17, 64, 1024, 128, True, False, torch.bfloat16, {0}),     # more tokens than this one takes
])
def test_integer_codes(M, N, K, group, zeros, bias, dtype, split):
    plan = nv.proto("b200_w4_units_split", [ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_int])
    assert plan(M, N, K, group, nv.dtype_code(dtype)) in split
    gen = torch.Generator(device="cuda").manual_seed(N + K + M)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x = rand(M, K).to(dtype)
    packed = torch.randint(0, 256, (N, K // 2), generator=gen, device="cuda", dtype=torch.uint8)
    scale = (rand(N, K // group).abs() + 0.1) * K ** -0.5 / 8
    zs = scale * (8 + rand(N, K // group)) if zeros else None
    b = rand(N).to(dtype) if bias else None
    lut = torch.arange(16, dtype=torch.float32, device="cuda")
    y = w4_gemv(x, packed.reshape(-1), scale.reshape(-1), None if zs is None else zs.reshape(-1), N, K, group, lut, b)
    codes = torch.stack((packed >> 4, packed & 15), -1).view(N, K).double()
    w = codes * scale.double().repeat_interleave(group, 1)
    if zs is not None:
        w = w - zs.double().repeat_interleave(group, 1)
    ref = x.double() @ w.T
    # fp32 sums of (offset + code) x, offset 128 (bf16) or 1024 (fp16), 128 terms to a sum whose partial ones are rounded eight times,
    # then at most K / 128 of them one after the other; and the rounding of the result
    off = 1024 if dtype == torch.float16 else 128
    mag = x.double().abs() @ (scale.double().repeat_interleave(group, 1) * (off + 16)).T
    if b is not None:
        ref = ref + b.double()
    bound = mag * (8 + K / 128 / 8) * 2.0 ** -24 + ref.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10)
    assert ((y.double() - ref).abs() <= bound + 1e-6).all()
    again = w4_gemv(x, packed.reshape(-1), scale.reshape(-1), None if zs is None else zs.reshape(-1), N, K, group, lut, b)
    assert torch.equal(y, again)
