"""What can be checked of the kernels by reading their sources, without a GPU."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "koboldcpp_b200" / "csrc"


def body(source, head):
    """Text of the block that the first `{` behind `head` opens."""
    at = source.index("{", source.index(head))
    depth = 0
    for i in range(at, len(source)):
        depth += {"{": 1, "}": -1}.get(source[i], 0)
        if depth == 0:
            return source[at:i + 1]
    raise AssertionError(head)


def test_delta_scan_roles_meet_at_a_named_barrier():
    """__syncthreads() is defined only where all threads of the CTA reach the same one; the scan's two roles meet from two branches."""
    kernel = body((CSRC / "recur.cu").read_text(), "delta_rule_scan_kernel(const b200_delta_rule_args a)")
    code = re.sub(r"//[^\n]*", "", kernel)
    assert "__syncthreads" not in code
    assert code.count("dr_meet()") == 2
