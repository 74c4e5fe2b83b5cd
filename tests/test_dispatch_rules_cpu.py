"""Rules that pick a kernel by sizes, where the choice itself needs no GPU."""
import pytest

from llm_in_practise_b200.inference.ragged import make_pieces
from llm_in_practise_b200.ops.linear_scan import _chunks_pay


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
