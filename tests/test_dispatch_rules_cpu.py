"""Rules that pick a kernel by sizes, where the choice itself needs no GPU."""
import ctypes

import pytest

from llm_in_practise_b200.inference.ragged import make_pieces
from llm_in_practise_b200.ops import _native as nv
from llm_in_practise_b200.ops.linear_scan import _chunks_pay

library = pytest.mark.skipif(not nv.lib_path().exists(), reason="no kernel library here")


@pytest.mark.parametrize("lens,H,G,D,chunks", [
    ([1] * 64, 16, 4, 128, False),                        # a decode batch
    ([150] * 3, 16, 4, 128, False),                       # short runs beside one another: 74 us in chunks, 56 token by token
    ([2048], 16, 4, 128, True),                           # 225 against 502
    ([2048, 513], 16, 4, 128, True),                      # 285 against 586
])
def test_delta_rule_in_chunks(lens, H, G, D, chunks):
    """With the runs known on the host, and without them, where they count as equally long."""
    pieces = make_pieces([(sum(lens[:i]), n, 0, i) for i, n in enumerate(lens)], "cpu")
    assert _chunks_pay(sum(lens), len(lens), pieces, H, G, D, D) == chunks
    if len(set(lens)) == 1:
        assert _chunks_pay(sum(lens), len(lens), None, H, G, D, D) == chunks


@library
@pytest.mark.parametrize("m,n,k,chain", [
    (20, 4096, 2048, 6), (64, 4096, 4096, 11), (128, 8192, 2048, 10), (64, 5120, 17408, 37), (200, 2048, 2048, 5), (200, 6144, 4096, 21),
    (490, 4096, 2048, 14), (490, 6144, 4096, 42), (549, 2048, 2048, 11), (549, 4096, 4096, 43), (1024, 2048, 4096, 29), (1500, 2048, 4096, 43),
    (2048, 768, 3072, 16), (2345, 768, 3072, 20), (2345, 2048, 2048, 32)])
def test_chains_of_few_tiles_stay_short(m, n, k, chain):
    """Products of fewer tiles than SMs are cut along k. A rule that takes one wave of narrow tiles instead is faster and adds up two to six
    times as many k-blocks (of 64 here) in one chain, with an error that grows as the chain does."""
    out = (ctypes.c_int * 4)()
    assert nv.proto("b200_gemm_plan", [ctypes.c_int] * 7 + [ctypes.c_void_p])(m, n, k, 1, 0, nv.DT_BF16, 148, ctypes.addressof(out)) == 0
    assert out[3] <= chain
