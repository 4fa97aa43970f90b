"""The resident kernel's warp loop, read as text: a lane that leaves it alone
would leave the others waiting in a full-mask warp operation, a fault that no
run may show on a GPU.  So every exit of the loop is taken on a warp vote."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "drawlab_gb300", "csrc")


def body_after(src, start):
    """The brace-enclosed text that follows `start`."""
    i = src.index("{", src.index(start))
    depth = 0
    for j in range(i, len(src)):
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        if depth == 0:
            return src[i:j + 1]
    raise AssertionError("unbalanced braces after %s" % start)


def test_warps_leave_the_resident_loop_as_one():
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "resident.cu")).read())
    kernel = body_after(src, "k_resident(RenderParams P, int slots, unsigned tail)")
    loop = body_after(kernel, "for (;;)")
    exits = re.findall(r"[^;{}]*\bbreak;", loop)
    assert len(exits) == 2 and "return" not in loop
    for e in exits:
        assert re.search(r"if \(__(any|all)_sync\(0xffffffffu,", e), e
