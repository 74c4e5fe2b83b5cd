"""4-bit weights expanded beside and ahead of their GEMMs: the kernel at the edges of its runs, the buffers under any order of requests."""
import random

import pytest
import torch

from llm_in_practise_b200.ops import w4 as W
from llm_in_practise_b200.ops.dequant_pipeline import DequantPipeline
from llm_in_practise_b200.ops.gemm import gemm

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


@pytest.mark.parametrize("N,K,group,dtype,stride,shards,zeros", [
    (1, 32, 32, torch.bfloat16, 0, 1, False),          # one word column, one row
    (7, 1024, 64, torch.float16, 0, 1, True),          # exactly one run
    (5, 1056, 32, torch.bfloat16, 8, 1, True),         # a run and one group of the next, strided rows
    (64, 4000, 160, torch.float16, 64, 2, True),       # groups that no shift gives and that cross runs, two shards
    (3600, 1984, 64, torch.bfloat16, 0, 4, False),     # more runs than warps
    (40, 6144, 2048, torch.bfloat16, 0, 1, True),      # groups longer than a run
])
def test_expansion(N, K, group, dtype, stride, shards, zeros):
    g = torch.Generator().manual_seed(N * K)
    packed = torch.randint(0, 256, (N * K // 2,), dtype=torch.uint8, generator=g).cuda()
    scale = torch.rand(N * K // group, generator=g).cuda()
    zs = torch.rand(N * K // group, generator=g).cuda() if zeros else None
    out = torch.full((N, K + stride), 7.0, dtype=dtype, device="cuda")
    rows = N // shards
    ptrs = [(packed.data_ptr() + s * rows * K // 2, scale.data_ptr() + s * rows * K // group * 4,
             zs.data_ptr() + s * rows * K // group * 4 if zeros else 0) for s in range(shards)]
    W.w4_dequant(packed, scale, zs, N, K, group, None, dtype, out[:, :K], shards=ptrs, rows_per_shard=rows)
    exact = W._w4_dequant_ref(packed, scale, zs, N, K, group, None, torch.float32)
    # one rounding of lut * scale - zero to the type (the difference is one fp32 operation, of magnitude 2 at most)
    eps = torch.finfo(dtype).eps / 2
    assert ((out[:, :K].float() - exact).abs() <= eps * exact.abs() + 2 ** -22).all()
    assert (out[:, K:] == 7.0).all()


def test_any_order_of_requests():
    """Every request gets its weight, whatever was predicted, with GEMMs that read the buffers in between."""
    rng = random.Random(3)
    qs = []
    for n, k in ((256, 128), (1024, 512), (128, 2048), (512, 512), (2048, 256)):
        qs.append(W.NF4Weight.quantize(torch.randn(n, k, device="cuda").bfloat16() * 0.1, double_quant=False))
    dense = [q.dequantize(torch.bfloat16).clone() for q in qs]
    pipe = DequantPipeline(torch.device("cuda", 0))
    step = [(i, False) for i in range(5)] + [(i, True) for i in reversed(range(5))]
    mixed = [(rng.randrange(5), rng.random() < 0.5) for _ in range(60)]
    checks = []
    for at, (i, back) in enumerate(step * 3 + mixed + step):
        if at == 2 * len(step):
            learned = pipe.misses
        elif at == 3 * len(step):
            assert pipe.misses == learned                 # the order is known by the third step
        q = qs[i]
        w = pipe.get(q, torch.bfloat16, back)
        assert tuple(w.shape) == (q.N, q.K)
        x = torch.randn(64, q.N if back else q.K, device="cuda").bfloat16()
        checks.append((gemm(x, w, b_mn=back), gemm(x, dense[i], b_mn=back)))
        if rng.random() < 0.7:
            pipe.done()
    for a, b in checks:
        assert torch.equal(a, b)
