"""The hand-over from one token to the next inside a launch, read from the source: no run can show a missing fence.

Blocks leave rows of the cache, then a flag; 32 lanes poll the flags with relaxed loads; lane 0 issues the copies that read the rows. So every lane needs a
fence after its polls, the lanes a barrier that orders memory (shuffles do not), and lane 0 a proxy fence after that."""
import os
import re

CORE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm.metal_b200", "csrc", "decode_token_core.cuh")


def body(name):
    with open(CORE) as f:
        s = re.sub(r"//[^\n]*", "", f.read())
    at = s.index("{", s.index(" " + name + "("))
    depth, end = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(s[end], 0)
        end += 1
        if depth == 0:
            return s[at:end]


def test_readers_fence_in_every_lane():
    b = body("next_token")
    polls, lane0 = b.index("fl_poll<"), b.index("if (lane == 0)")
    fence, joined, proxy = b.index("__threadfence();", polls), b.index("__syncwarp();", polls), b.index("fence.proxy.async", lane0)
    assert polls < fence < joined < lane0 < proxy


def test_writers_fence_before_the_flag():
    b = body("run_matvec")
    flag = b.index("fl_store<false>(p.d_am")
    assert 0 < b.rindex("named_barrier(1, TK_NC)", 0, flag) < b.rindex("else if (p.n_tokens > 1) __threadfence();", 0, flag) < flag
