"""How the tensor-core kernels may wait, checked in their source text (no GPU).

`mbar_wait` answers lane by lane; `mbar_wait_warp` makes one answer for the warp. Tensor-memory instructions, votes and
elections are warp-aligned: a lane that gave up alone (or came back late) ahead of one leaves the others at it. So a lane's own
wait may stand only
  * in a region that one lane runs, after which its warp meets a __syncwarp before the role's next warp-aligned operation, or
  * in a function whose calls all stand in such a region or inside a warp vote.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dark-forest_b200", "csrc")
ONE_LANE = re.compile(r"\b(lane|threadIdx\.x)\s*==\s*0\b")
ALIGNED = re.compile(r"tmem_(ld|st|wait)|tcgen05\.(ld|st|wait)|__(any|all|shfl|reduce)\w*_sync|elect_one|commit_elected|_warp\(|__syncwarp")



def _blocks(src):
    """(start, end, header) of every brace block, outermost first; the header is the text since the statement before it."""
    out, stack, since = [], [], 0
    for m in re.finditer(r"[{};]", src):
        i, ch = m.start(), m.group()
        if ch == "{":
            stack.append((i, src[since:i]))
        elif ch == "}":
            start, header = stack.pop()
            out.append((start, i, header))
        since = i + 1
    assert not stack
    return sorted(out)


def lone_waits(src):
    """Line numbers of the lane-by-lane waits that break the rule above."""
    src = re.sub(r"/\*.*?\*/|//[^\n]*", lambda m: re.sub(r"[^\n]", " ", m.group()), src, flags=re.S)
    blocks = _blocks(src)
    bad = []

    def allowed(pos, end, depth=0):
        around = [b for b in blocks if b[0] < pos < b[1]]
        kernel = max((n for n, b in enumerate(around) if "__global__" in b[2]), default=None)
        if kernel is None:
            return True  # not in a kernel: the definition of the wait itself
        inner = around[kernel + 1:]
        role_end = inner[0][1] if inner else around[kernel][1]
        statement = src[max(src.rfind(c, 0, pos) for c in ";{}") + 1:pos]
        if re.search(r"__(all|shfl)_sync\(0xffffffffu,\s*$", statement):
            return True
        region_end = None
        if ONE_LANE.search(statement):
            region_end = end
        for b in inner:  # the outermost one-lane region, if any
            if ONE_LANE.search(b[2]):
                region_end = b[1]
                break
        if region_end is not None:
            after = ALIGNED.search(src, region_end, role_end)
            return after is None or after.group() == "__syncwarp"
        for b in reversed(inner):  # a lambda: every call of it has to stand where the wait could
            name = re.search(r"auto\s+(\w+)\s*=\s*\[&\]", b[2])
            if name and depth < 3:
                calls = [m for m in re.finditer(r"\b%s\(" % name.group(1), src) if around[kernel][0] < m.start() < around[kernel][1]]
                return all(allowed(m.start(), m.end(), depth + 1) for m in calls)
        return False

    for m in re.finditer(r"\bmbar_wait\(", src):
        if not allowed(m.start(), src.find(";", m.start())):
            bad.append(src.count("\n", 0, m.start()) + 1)
    return bad


def test_the_rule_sees_what_it_is_about():
    def kernel(body):
        return "__global__ void k() { auto take = [&](int n) { return mbar_wait(b, n, f); }; if (warp == 0) { %s } }" % body

    assert lone_waits(kernel("if (lane == 0) { mbar_wait(b, 0, f); take(1); }")) == []
    assert lone_waits(kernel("if (!mbar_wait_warp(b, 0, f)) return; tmem_ld32(a, r);")) == []
    assert lone_waits(kernel("__all_sync(0xffffffffu, take(1)); tmem_ld32(a, r);")) == []
    assert lone_waits(kernel("if (lane == 0 && mbar_wait(b, 0, f)) go(); __syncwarp(); tmem_ld32(a, r);")) == []
    assert lone_waits(kernel("for (;;) { if (!mbar_wait(b, 0, f)) break; tmem_ld32(a, r); }")) == [1]
    assert lone_waits(kernel("if (threadIdx.x == 0 && mbar_wait(b, 0, f)) go(); tmem_ld32(a, r);")) == [1]
    assert lone_waits(kernel("if (take(1)) tmem_ld32(a, r);")) == [1]


@pytest.mark.parametrize("name", ["attn_fwd_sm100.cu", "attn_fwd_row2_sm100.cu", "attn_bwd_sm100.cu", "attn_bwd_bf16_sm100.cu", "linear_sm100.cu"])
def test_whole_warps_wait_as_warps(name):
    with open(os.path.join(CSRC, name)) as f:
        src = f.read()
    assert "mbar_wait" in src and "tmem_ld32" in src
    assert lone_waits(src) == []


def test_the_cluster_barrier_brings_its_warps_together():
    """Its instructions are warp-aligned, and kernels come to it out of one-lane regions (set-up, producers)."""
    with open(os.path.join(CSRC, "sm100_ptx.cuh")) as f:
        body = re.search(r"void cluster_sync\(\) \{(.*?)\n\}", f.read(), re.S).group(1)
    assert body.index("__syncwarp();") < body.index("barrier.cluster.arrive.release.aligned")
