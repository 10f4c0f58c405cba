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


def test_local_arrays_read_as_vectors_are_aligned():
    """An array of 2-byte values that is read as one 16-byte vector says so in its declaration: as long as it lives in
    registers nothing depends on it, but in local memory the load would be misaligned."""
    for path in sorted(CSRC.glob("*.cu*")):
        src = path.read_text()
        for name in set(re.findall(r"\*reinterpret_cast<(?:const )?uint4\*>\((\w+)\)", src)):
            for decl in re.findall(r"^.*\b__nv_bfloat16 %s\[\d+\];" % re.escape(name), src, flags=re.M):
                assert "alignas(16)" in decl, (path.name, decl.strip())
