"""What gemm_tc.cu and gemm_split.cu do when one of their waits runs out, read from the source (no GPU: nothing here makes a
wait run out)."""

from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "mini_gpt_inference_b200" / "csrc"
SOURCE = (CSRC / "gemm_tc.cu").read_text()
SPLIT = (CSRC / "gemm_split.cu").read_text()


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


def test_split_tiles_every_worker_comes_to_every_barrier():
    """The sixteen workers meet in named barriers, which have no limit: a worker whose wait ran out while others got theirs must
    not leave the way to one.  So nothing in front of a tile's barriers returns or breaks on what a wait said."""
    workers = SPLIT[SPLIT.index("// ---- loads, splitting, and the slices' sums ----"): SPLIT.index("// a wait ran out")]
    add_up = workers[workers.index("auto add_up = "): workers.index("int tile = blockIdx.x, slice = 0")]
    steps = workers[workers.index("for (long long i = 0; i < steps; ++i)"):]
    assert "break;" not in steps and "return" not in steps and "continue" not in steps
    barriers = [m.start() for m in re.finditer(r'asm volatile\("(bar|barrier)\.', add_up)]
    assert barriers and not re.search(r'"(bar|barrier)\.', workers.replace(add_up, ""))
    leaving = re.findall(r"[^\n]*\b(?:return|break|continue)\b[^\n]*", add_up[: barriers[-1]])
    assert [line.strip() for line in leaving] == ["if (slice + 1 < slices) return;"]          # (the same in all workers)
    for at in barriers:                                        # ... and none of them stands in a branch on what a wait said
        assert "if (ok" not in add_up[add_up.rindex("\n", 0, at): at]
    # the wait is asked once a worker, and the status word tells of it
    assert len(re.findall(r"warp_wait\(", add_up)) == 1 and "if (ok) ok = warp_wait(" in add_up
    assert "atomicExch(g.status, 81);" in steps and "ctl.failed = 1;" in steps
