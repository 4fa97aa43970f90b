"""The resident kernel, read as text for what no run may show on a GPU: a lane
that left the warp's loop alone would leave the others waiting in a full-mask
warp operation, and an index from a queue outside its array would fault."""
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


def code():
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "resident.cu")).read())


def test_warps_leave_the_resident_loop_as_one():
    kernel = body_after(code(), "k_resident(RenderParams P, int slots, unsigned tail)")
    loop = body_after(kernel, "for (;;)")
    exits = re.findall(r"[^;{}]*\bbreak;", loop)
    assert len(exits) == 2 and "return" not in loop
    for e in exits:
        assert re.search(r"if \(__(any|all)_sync\(0xffffffffu,", e), e


def test_the_checked_build_checks_what_the_queues_hold():
    src = code()
    # entries name slots of the block
    assert "< Sm::kBlockSlots, &P.cnt->err)" in body_after(src, "uint32_t ring_take(")
    # a hit names its queue
    done = body_after(src, "void ray_done(")
    assert src.count("hit[slot] >> 27") == 1
    assert done.index("hit[slot] >> 27") < done.index("DL_IN_BOUNDS(q >= 0 && q <= kEndedQueue") < done.index("sm.queue[q]")
    # the wavefront's last paths lie in its queue
    assert "DL_IN_BOUNDS(pid < (unsigned)P.capacity, &P.cnt->err) ? P.ext_q[0][pid]" in src
    assert src.count("P.ext_q[") == 1
