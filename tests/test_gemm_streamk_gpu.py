"""GEMMs of few tiles: tiles cut into parts whose fp32 partials their owner sums, and what such sums may be off by."""
import ctypes

import pytest
import torch

from llm_in_practise_b200.ops import _native as nv
from llm_in_practise_b200.ops.gemm import gemm


# M, N, K, fp32 result, beta: tiles of one CTA and of a pair in two to eight parts, whole tiles beside parts (2345 rows), ragged last rows and
# columns, a result that is added to. All are cut.
@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,f32,beta", [
    (64, 4096, 4096, False, 0.0), (100, 4100, 12288, False, 0.0), (37, 5128, 2112, True, 0.5), (1, 2048, 8192, True, 0.0),
    (300, 4096, 16384, True, 1.0), (549, 2048, 2048, True, 0.0), (549, 2040, 4096, False, 0.5), (490, 4096, 12288, False, 0.0),
    (700, 1528, 8192, True, 0.0), (1024, 72, 4096, False, 0.0), (2345, 2048, 4096, True, 0.0)])
def test_parts_of_tiles_against_fp64(m, n, k, f32, beta):
    assert plan(m, n, k)[2] == 1
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    b = torch.randn(n, k, device="cuda", generator=g).bfloat16()
    d = torch.randn(m, n, device="cuda", generator=g).to(torch.float32 if f32 else torch.bfloat16)
    ref = a.double() @ b.double().t() + beta * d.double()
    # any order of k + 1 fp32 additions, rounded or truncated: k * 2^-23 of the sum of magnitudes; then the result's rounding
    bound = k * 2.0 ** -23 * (a.abs().double() @ b.abs().double().t() + d.abs().double())
    if not f32:
        bound = bound + 2.0 ** -8 * ref.abs()
    for _ in range(2):                                       # the second launch meets the first one's flags
        out = d.clone()
        gemm(a, b, out=out, beta=beta)
        assert bool(((out.double() - ref).abs() <= bound).all())


def plan(m, n, k):
    """(CTAs of a tile, its columns, whether k is cut into parts, k-blocks of the longest chain) on a B200."""
    out = (ctypes.c_int * 4)()
    fn = nv.proto("b200_gemm_plan", [ctypes.c_int] * 7 + [ctypes.c_void_p])
    assert fn(m, n, k, 1, 0, nv.DT_BF16, 148, ctypes.addressof(out)) == 0
    return tuple(out)


# What a chain of additions on the tensor cores may be off by, as a norm: a k-block is four steps, each truncates the sum so far by 2^-24 of
# it in the mean, and a sum of n random steps has grown to 2 / 3 of its last size in the mean; then a rounding for each part of a tile, for
# beta's product and for its sum.
def norm_bound(k, chain):
    return (8 / 3 * chain + -(-k // 64) / chain + 3) * 2.0 ** -24


# the shapes above that are cut, two that are not, and one whose result is a row
CUT = [(64, 4096, 4096), (37, 5128, 2112), (1, 2048, 8192), (300, 4096, 16384), (549, 2048, 2048), (490, 4096, 4096), (700, 1528, 8192), (2345, 2048, 4096)]
WHOLE = [(200, 16384, 512), (4096, 2048, 1024)]


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", CUT + WHOLE)
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_error_of_fp32_results(m, n, k, beta):
    _, _, parts, chain = plan(m, n, k)
    assert parts == ((m, n, k) in CUT)
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    b = torch.randn(n, k, device="cuda", generator=g).bfloat16()
    d = torch.randn(m, n, device="cuda", generator=g)
    ref = a.double() @ b.double().t() + beta * d.double()
    out = gemm(a, b, out=d.clone(), beta=beta)
    assert float((out.double() - ref).norm() / ref.norm()) <= norm_bound(k, chain)
