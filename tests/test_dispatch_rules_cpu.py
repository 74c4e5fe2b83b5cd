"""Rules that pick a kernel by sizes, where the choice itself needs no GPU."""
import ctypes

import pytest

from llm_in_practise_b200.inference.ragged import make_pieces
from llm_in_practise_b200.ops import _native as nv
from llm_in_practise_b200.ops.linear_scan import _chunks_pay

library = pytest.mark.skipif(not nv.lib_path().exists(), reason="no kernel library here")


@pytest.mark.parametrize("lens,H,G,D,chunks", [
    ([1] * 64, 16, 4, 128, False),                        # a decode batch
    ([150] * 3, 16, 4, 128, False),                       # short runs beside one another: 71 us in chunks, 59 token by token
    ([2048], 16, 4, 128, True),                           # 153 against 506
    ([2048, 513], 16, 4, 128, True),                      # 198 against 590
    ([512] * 4, 16, 16, 64, True),                        # a q/k head for each head: 85 against 131
    ([1000], 32, 32, 128, True),                          # 181 against 293
    ([200] * 16, 32, 32, 128, False),                     # 759 against 561
])
def test_delta_rule_in_chunks(lens, H, G, D, chunks):
    """With the runs known on the host, and without them, where they count as equally long."""
    pieces = make_pieces([(sum(lens[:i]), n, 0, i) for i, n in enumerate(lens)], "cpu")
    assert _chunks_pay(sum(lens), len(lens), pieces, H, G, D, D) == chunks
    if len(set(lens)) == 1:
        assert _chunks_pay(sum(lens), len(lens), None, H, G, D, D) == chunks


@library
@pytest.mark.parametrize("H", [1, 16, 32, 40])
def test_workspace_of_the_delta_rule_is_bounded(H):
    """At most 4.3 MB per head, however long the step and however many q/k heads it has; at least a chunk's matrices (7872 words per head, 20480 per
    q/k head for keys of 128); and asked for as it always was, without the q/k heads."""
    fn = nv.lib().b200_delta_chunk_workspace
    fn.restype, fn.argtypes = ctypes.c_longlong, [ctypes.c_int] * 3
    for tokens, runs in [(1, 1), (64, 1), (500, 3), (2368, 1), (8192, 1), (1 << 20, 64), ((1 << 31) - 1, 1)]:
        words = fn(tokens, runs, H)
        assert H * (7872 + 20480) <= words <= H * 128 * 8320
        if tokens // 64 + runs <= 37:
            assert words == (tokens // 64 + runs) * H * (7872 + 20480)


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


@library
@pytest.mark.parametrize("sms", [148, 132, 7])
@pytest.mark.parametrize("m,n,k", [(20, 4096, 2048), (64, 4096, 4096), (64, 5120, 17408), (300, 4096, 16384), (490, 6144, 4096), (549, 2048, 2048),
                                   (1024, 72, 4096), (2048, 5120, 5120), (2048, 5120, 17408), (2345, 2048, 2048)])
def test_parts_wait_only_for_what_started_before_them(m, n, k, sms):
    """A tile's owner sums the parts of other units. Units that start in order, each kept on the GPU until what it waits for is there, all finish
    whatever the number that fits at once, one included; they do not if one waits for a unit that starts after it."""
    fn = nv.proto("b200_gemm_streamk_waits", [ctypes.c_int] * 7 + [ctypes.c_void_p, ctypes.c_int])
    out = (ctypes.c_int * 4000)()
    count = fn(m, n, k, 1, 0, nv.DT_BF16, sms, ctypes.addressof(out), 2000)
    plan = (ctypes.c_int * 4)()
    assert nv.proto("b200_gemm_plan", [ctypes.c_int] * 7 + [ctypes.c_void_p])(m, n, k, 1, 0, nv.DT_BF16, sms, ctypes.addressof(plan)) == 0
    assert 0 <= count <= 2000 and (count > 0) == bool(plan[2])
    waits = [(out[2 * i], out[2 * i + 1]) for i in range(count)]
    assert all(0 <= other < unit < sms // plan[0] for unit, other in waits)


@library
@pytest.mark.parametrize("m,n,k,b_mn", [
    (4096, 1536, 512, 0), (2345, 1536, 512, 0), (2345, 2048, 512, 0), (4096, 1000, 640, 0), (1024, 768, 768, 0), (1024, 3072, 768, 0), (300, 768, 768, 0),
    (549, 1024, 1024, 0), (300, 5120, 2048, 0), (512, 768, 768, 1), (549, 16, 2048, 0), (8192, 8192, 8192, 0)])
def test_whole_tiles(m, n, k, b_mn):
    """Products that are not cut take tiles of whole 32 columns, unless the matrix is narrower: half of them cost more than the columns saved."""
    out = (ctypes.c_int * 4)()
    assert nv.proto("b200_gemm_plan", [ctypes.c_int] * 7 + [ctypes.c_void_p])(m, n, k, 1, b_mn, nv.DT_BF16, 148, ctypes.addressof(out)) == 0
    assert not out[2] and (out[1] % 32 == 0 or out[1] >= n)


@library
@pytest.mark.parametrize("m,n,k", [(2345, 5120, 17408), (4096, 4096, 12288), (300, 24576, 4096)])
def test_more_than_a_wave_is_not_cut(m, n, k):
    """Parts of 17408 values in more than one wave read all of A and B from memory again: 488 us for the first, 314 by whole tiles."""
    out = (ctypes.c_int * 4)()
    assert nv.proto("b200_gemm_plan", [ctypes.c_int] * 7 + [ctypes.c_void_p])(m, n, k, 1, 0, nv.DT_BF16, 148, ctypes.addressof(out)) == 0
    assert out[2] == 0


@library
@pytest.mark.parametrize("B,S,H,Hkv,D", [(16, 4096, 32, 32, 128), (2, 8192, 32, 8, 128), (64, 1024, 12, 12, 128), (1, 1 << 20, 8, 2, 128), (3, 70000, 5, 5, 128), (1, 16 << 20, 8, 2, 64)])
def test_keys_of_a_group_of_heads_fit_the_cache(B, S, H, Hkv, D):
    """The forward's tiles of heads of 128 go out by groups of heads whose keys and values stay in L2 (126 MB) while the group's tiles read them."""
    group = nv.proto("b200_flash_tc_group", [ctypes.c_longlong] + [ctypes.c_int] * 5)(B * S, B, S, H, Hkv, D)
    rep, kv = H // Hkv, S * D * 4
    if B * Hkv * kv <= 126 << 20:
        assert group == H * B
    else:
        assert group % rep == 0 and (group == rep or group // rep * kv <= 48 << 20)
        assert group == rep or 3 * group * kv >= rep * (48 << 20)                   # and no fewer than need be


@library
def test_small_batches_are_one_group():
    call = nv.proto("b200_flash_tc_group", [ctypes.c_longlong] + [ctypes.c_int] * 5)
    assert call(4 * 512, 4, 512, 40, 8, 128) == 160 and call(4096, 1, 4096, 32, 8, 128) == 32
    assert call(64 * 1024, 64, 1024, 12, 12, 64) == 768                    # heads of 64 do not wait for memory
    assert call(64, 2, 65535 * 128 + 1, 4, 2, 64) == 8                     # more tiles than a grid's second dimension
    assert call(64, 2, 512, 4, 3, 64) == 0
