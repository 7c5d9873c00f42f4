"""What gemm_tc.cu does when one of its waits runs out, read from its source (no GPU: nothing here makes a wait run out)."""

from __future__ import annotations

import re
from pathlib import Path

SOURCE = (Path(__file__).resolve().parent.parent / "mini_gpt_inference_b200" / "csrc" / "gemm_tc.cu").read_text()


def test_an_incomplete_accumulator_is_not_handed_to_the_epilogue():
    issue = SOURCE[SOURCE.index("} else if (issues) {"): SOURCE.index("} else if (warp < EPI_WARPS) {")]
    commits = [line for line in issue.splitlines() if "umma_commit" in line and "acc_full" in line]
    assert commits and all(re.match(r"\s*if \(ok\) umma_commit", line) for line in commits)


def test_every_wait_that_runs_out_is_recorded_and_marks_its_own_cta():
    body = SOURCE[SOURCE.index("gemm_tc_kernel("): SOURCE.index("// ---- host side")]
    assert len(re.findall(r"mbar_wait\(", body)) == 4
    # the loads', the products' (both waits) and the epilogue's: a code for the host, and `failed`, behind which the CTA waits for
    # copies in flight before it returns
    for code in (1, 2, 3):
        record = body.index(f"atomicExch(g.status, {code});")
        assert "ctl->failed = 1;" in body[record: record + 80]
