"""Properties of the kernel sources that no run can show, because the case that breaks them would hang a GPU."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "cosmos_rl_b200" / "csrc"


def test_decode_softmax_warps_leave_their_loops_together():
    """The four softmax warps of the decode attention meet at a named barrier, which has no time limit. Their waits do have
    one, and may run out in some of the warps only. So a warp may leave a loop only on a value that the barrier returned to
    all four: every ``break`` follows an assignment from ``softmax_bar``, and no loop condition reads the abort flag."""
    src = (CSRC / "paged_decode_tc.cu").read_text()
    role = src[src.index("softmax / epilogue (warps 2..5)"):]
    role = role[:role.index("__syncthreads()")]
    lines = [re.sub(r"//.*", "", line).strip() for line in role.splitlines()[1:]]
    lines = [line for line in lines if line and not line.startswith("#")]
    leaving = [i for i, line in enumerate(lines) if re.search(r"\b(break|goto)\b", line)]
    assert leaving
    for i in leaving:
        assert lines[i] == "if (!ok) break;" and lines[i - 1].startswith("ok = softmax_bar("), lines[i - 1:i + 1]
    for line in lines:
        if line.startswith(("for (", "while (")):
            assert "abort_flag" not in line, line
