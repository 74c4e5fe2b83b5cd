"""Products of 17 to 64 tokens with 4-bit integer codes on tcgen05: tiles, units and clusters at their edges."""
import ctypes

import pytest
import torch

from llm_in_practise_b200.ops import _native as nv
from llm_in_practise_b200.ops.w4 import w4_gemv, w4_tc


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,zeros,bias,dtype,split", [
    (17, 1, 512, True, False, torch.bfloat16, {1}),               # one row, one unit
    (32, 124, 1024, True, True, torch.bfloat16, {1, 2}),
    (33, 125 * 148, 512, False, True, torch.float16, {1}),        # a second tile with a row or none in each CTA
    (64, 124 * 148 + 1, 1024, True, False, torch.bfloat16, {1, 2}),
    (40, 2387, 4096, True, True, torch.bfloat16, {2, 4}),         # slices of k in a cluster
    (64, 1000, 17408, False, False, torch.float16, {4}),          # 34 units over four slices
    (50, 10000, 3584, True, True, torch.float16, {1, 2}),         # seven units, several tiles
    (16, 4096, 4096, True, False, torch.bfloat16, {0}),           # fewer tokens, a K of less than whole units: the other kernels
    (20, 256, 640, True, False, torch.bfloat16, {0}),
])
def test_integer_codes(M, N, K, zeros, bias, dtype, split):
    plan = nv.proto("b200_w4_tc_split", [ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_int])
    assert plan(M, N, K, 128) in split
    gen = torch.Generator(device="cuda").manual_seed(N + K + M)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x = rand(M, K).to(dtype)
    packed = torch.randint(0, 256, (N, K // 2), generator=gen, device="cuda", dtype=torch.uint8)
    scale = (rand(N, K // 128).abs() + 0.1) * K ** -0.5 / 8
    zs = scale * (8 + rand(N, K // 128)) if zeros else None
    b = rand(N).to(dtype) if bias else None
    y = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
    z = None if zs is None else zs.reshape(-1)
    took = w4_tc(x, packed.reshape(-1), scale.reshape(-1), z, N, K, 128, (1.0, 0.0), b, y)
    assert took == (split != {0})
    if not took:
        return
    wide = scale.double().repeat_interleave(128, 1)
    w = torch.stack((packed >> 4, packed & 15), -1).view(N, K).double() * wide
    if zs is not None:
        w = w - zs.double().repeat_interleave(128, 1)
    ref = x.double() @ w.T
    # a group's sums of (offset + code) x and of offset x (offset 128 or 1024) are rounded eight times each, their factors and products twice;
    # the sum over the groups is rounded twice a group; and the rounding of the result
    off = 1024 if dtype == torch.float16 else 128
    mag = x.double().abs() @ (wide * (off + 16)).T
    sums = x.double().abs() @ w.abs().T
    if b is not None:
        ref = ref + b.double()
    bound = (mag * 20 + sums * (2 * K / 128)) * 2.0 ** -24 + ref.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10)
    assert ((y.double() - ref).abs() <= bound + 1e-6).all()
    again = torch.empty_like(y)
    assert w4_tc(x, packed.reshape(-1), scale.reshape(-1), z, N, K, 128, (1.0, 0.0), b, again)
    assert torch.equal(y, again)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,lin,mean", [
    (17, 1000, 4096, (1.0, 0.0), 2.0),                            # activations whose mean is far from zero, unsigned codes with a zero
    (64, 4100, 2048, (1.0, 8.0), 2.0),                            # symmetric codes
    (33, 600, 5120, (0.5, 8.0), 0.0),
    (40, 2387, 1024, (1.0, -3.0), -1.0),
    (64, 333, 17408, (-2.0, 64.0), 0.5),
])
def test_forms_and_error(M, N, K, lin, mean, dtype):
    """Every factor and offset of the codes' map, rows of wider matrices, and no more error than sums of 16 + code (64 + code in fp16) have."""
    gen = torch.Generator(device="cuda").manual_seed(N + K + M)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    wide_x = (rand(M, K + 24) + mean).to(dtype)
    x = wide_x[:, 16:16 + K]
    packed = torch.randint(0, 256, (N, K // 2), generator=gen, device="cuda", dtype=torch.uint8)
    scale = (rand(N, K // 128).abs() + 0.1) * K ** -0.5 / 8
    zs = scale * (8 + rand(N, K // 128)) if lin == (1.0, 0.0) else None
    wide_y = torch.full((M, N + 13), 7.0, dtype=dtype, device="cuda")
    y = wide_y[:, 5:5 + N]
    assert w4_tc(x, packed.reshape(-1), scale.reshape(-1), None if zs is None else zs.reshape(-1), N, K, 128, lin, None, y)
    assert (wide_y[:, :5] == 7).all() and (wide_y[:, 5 + N:] == 7).all()
    up = lambda t: t.double().repeat_interleave(128, 1)
    code = torch.stack((packed >> 4, packed & 15), -1).view(N, K).double()
    a = up(scale) * lin[0]
    minus = a * lin[1] + (0 if zs is None else up(zs))
    w = a * code - minus
    ref = x.double() @ w.T
    # a group's sums of (base + code) x and of base x are truncated eight times each, their factors and products rounded twice; the sum over
    # the groups is rounded twice a group; the result by half a unit in its last place of 8 or 11 bits
    base = 16 if dtype == torch.bfloat16 else 64
    mag = x.double().abs() @ ((base + 15) * a.abs() + (base * a + minus).abs()).T
    sums = x.double().abs() @ w.abs().T
    bound = (mag * 20 + sums * (2 * K / 128)) * 2.0 ** -24
    half = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    err = (y.double() - ref).abs()
    assert (err <= bound + half * (ref.abs() + bound) + 2.0 ** -25).all()
    # and as a norm the sums' own error is less than a seventh of the result's rounding
    assert err.norm() <= 1.01 * (ref.to(dtype).double() - ref).norm()


@pytest.mark.gpu
def test_large_products_go_there():
    M, N, K = 33, 4096, 4096
    x = torch.randn(M, K, device="cuda").bfloat16()
    packed = torch.randint(0, 256, (N * K // 2,), device="cuda", dtype=torch.uint8)
    scale = torch.rand(N * K // 128, device="cuda")
    before = nv.launch_count
    y = w4_gemv(x, packed, scale, scale * 8, N, K, 128, torch.arange(16, dtype=torch.float32, device="cuda"))
    assert nv.launch_count == before + 2                          # the tokens' order, the product
    z = torch.empty_like(y)
    assert w4_tc(x, packed, scale, scale * 8, N, K, 128, (1.0, 0.0), None, z) and torch.equal(y, z)
    graph = torch.cuda.CUDAGraph()                                # the two launches overlap; so they do in a replay
    z.zero_()
    with torch.cuda.graph(graph):
        assert w4_tc(x, packed, scale, scale * 8, N, K, 128, (1.0, 0.0), None, z)
    graph.replay()
    assert torch.equal(y, z)
