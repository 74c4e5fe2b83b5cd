"""What the kernels' sources have to keep to and no run would show."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "csrc"
# a wait in which every lane polls for itself; what one lane polls for, or what ends with all of them together
ALONE = re.compile(r"\bmbar_wait(_spin|_sleep)?\(|ld\.acquire\.gpu")
TOGETHER = re.compile(r"__syncwarp\(\)|\b(mbar_wait_warp|bw_wait_warp|wt_wait)\(|bar\.sync|__syncthreads\(\)")
# instructions of a whole warp: elect.sync with what it picks the lane for, and tcgen05's loads
WHOLE = re.compile(r"\b(issue_qk|issue_sdp|umma_f16_w|umma_f16_ts_w|umma_row_ss|umma_row_ts|umma_commit_w|umma_kblock|umma_kstep|umma_commit_elected|"
                   r"tma_load_4d_elected|mbar_expect_tx_elected|wt_group|wt_commit|tmem_ld_32x32|tmem_ld_32x16)\b\s*[(<]")


@pytest.mark.parametrize("name", ["flash_tc.cu", "flash_bwd_tc.cu", "gemm_tcgen05.cu", "w4_tc.cu"])
def test_lanes_meet_before_instructions_of_a_warp(name):
    """Lanes that have each looked at a barrier for themselves may have seen it at different times. Read line by line: after such a wait a
    warp comes together before the next instruction that is one of all 32 lanes."""
    apart, bad, seen = 0, [], 0
    for at, line in enumerate((CSRC / name).read_text().splitlines(), 1):
        code = line.split("//")[0]
        if re.search(r"__device__|else if \(.*warp|^  if \(.*warp|= \[&\]", code):      # another function, role or lambda
            apart = 0
        if "lane == 0" in code or "threadIdx.x & 31" in code:
            code = ALONE.sub("", code)
        alone, meet, whole = ALONE.search(code), TOGETHER.search(code), WHOLE.search(code)
        if whole and not code.lstrip().startswith("auto"):
            seen += 1
            if apart:
                bad.append((apart, at, line.strip()))
        if alone:
            apart = at
        if meet:
            apart = 0
    assert seen > 3 and not bad
