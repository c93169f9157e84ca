"""Rules of the kernels' sources that no run can be relied on to show broken."""
import re
from pathlib import Path

import sharedtensor_b200

CUDA = Path(sharedtensor_b200.__file__).parent / "csrc" / "cuda"


def _code(name):
    """The file without comments and line breaks."""
    return re.sub(r"\s+", " ", re.sub(r"//[^\n]*", "", (CUDA / name).read_text()))


def _body(code, function):
    """What stands between the braces of the function."""
    start = code.index("{", code.index(f" {function}("))
    depth = 0
    for i in range(start, len(code)):
        depth += (code[i] == "{") - (code[i] == "}")
        if depth == 0:
            return code[start:i]


def _conditions(code):
    """What stands between the parentheses of each if and while."""
    for m in re.finditer(r"\b(?:if|while) \(", code):
        depth, i = 1, m.end()
        while depth:
            depth += (code[i] == "(") - (code[i] == ")")
            i += 1
        yield code[m.end():i - 1]


def test_the_service_warp_takes_no_branch_on_what_each_lane_has_read_for_itself():
    """Compute warps and neighbours change these words at any time.  Lanes that saw different values would part, and meet
    different warp-wide calls."""
    reads = re.compile(r"volatile|ld_shared_acquire|ld_relaxed_sys|ld_acquire_sys|ld_cg_u32|mbar_test|mbar_wait_bounded|atomic")
    found = [c for c in _conditions(_body(_code("round.cu"), "service_warp"))]
    assert len(found) > 20
    for c in found:
        assert not reads.search(c) or "lane == 0" in c, c


def test_what_one_lane_knows_to_be_there_is_ordered_for_the_warp_that_reads_it():
    """Table magnitudes: lane 0 counts a chunk and learns that it was the last one, then all lanes read what other CTAs have
    written.  A shuffle orders no memory: lane 0's fence behind the count and a warp barrier behind the shuffle do."""
    body = _body(_code("table.cu"), "table_sums_kernel")
    count, told, read = body.index("atomicAdd(counters"), body.index("__shfl_sync(0xffffffffu, last, 0)"), body.index("__ldcg(partials")
    assert count < told < read
    assert "__threadfence()" in body[count:told] and "__syncwarp()" in body[told:read]
