"""GEMMs of few tiles: one wave of narrow tiles, and tiles cut into parts whose fp32 partials their owner sums."""
import pytest
import torch

from llm_in_practise_b200.ops.gemm import gemm

pytestmark = pytest.mark.gpu


# M, N, K, fp32 result, beta: parts of one tile in two and three units, a pair's tiles, ragged last rows and columns,
# a result that is added to, and the sizes on either side of the choice between a wave of tiles and parts
@pytest.mark.parametrize("m,n,k,f32,beta", [
    (64, 4096, 4096, False, 0.0), (100, 4100, 12288, False, 0.0), (37, 5128, 2112, True, 0.5), (1, 2048, 8192, True, 0.0),
    (300, 4096, 16384, True, 1.0), (549, 2048, 2048, True, 0.0), (549, 2040, 4096, False, 0.5), (490, 4096, 12288, False, 0.0),
    (700, 1528, 8192, True, 0.0), (1024, 72, 4096, False, 0.0), (2345, 2048, 4096, True, 0.0)])
def test_parts_of_tiles_against_fp64(m, n, k, f32, beta):
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
