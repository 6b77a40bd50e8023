"""The waits of the tensor-core kernels' warp roles, read from their source.

A bounded wait can run out in one lane of a warp and not in another, and a
shared-memory load of one lane can be in flight when another lane's value has
arrived.  So a role that a whole warp plays leaves its loop by a vote, a stage
is given back by an arrival that depends on all lanes' loads, and a wait that
ran out raises the error flag whichever lane saw it.  None of these can be
provoked in a test on the GPU without a race or a hang."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "image360_b200", "csrc", "learned.cu")


def _source():
    with open(SRC) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _enclosing(src, at):
    """The text that heads each block open at `at`, innermost last."""
    heads, start = [], 0
    for m in re.finditer(r"[{};]", src[:at]):
        c = m.group()
        if c == "{":
            heads.append(src[start:m.start()].strip())
        elif c == "}":
            heads.pop()
        start = m.end()
    return heads


def test_warps_leave_their_loops_by_a_vote():
    src = _source()
    waits = [m.start() for m in re.finditer(r"tc::mbar_wait\(", src)]
    assert len(waits) >= 7
    for at in waits:
        if any(h.endswith("if (lane == 0)") for h in _enclosing(src, at)):
            continue  # one thread's role
        stmt = src[max(src.rfind(c, 0, at) for c in ";{}") + 1:]
        m = re.match(r"\s*(?:const )?bool (\w+) = tc::mbar_wait", stmt)
        assert m, "a warp's wait is not held for a vote: " + stmt[:120]
        after = stmt[stmt.index(";") + 1:]
        assert re.match(r"\s*(if \(!__all_sync\(0xffffffffu, %s\)\)|%s = __all_sync\(0xffffffffu, %s\);)"
                        % ((m.group(1),) * 3), after), after[:120]


def test_a_stage_is_released_behind_every_lanes_loads():
    src = _source()
    calls = list(re.finditer(r"tc::mbar_arrive_after\(&\w+\[\w+\], (\w+), \w+\)", src))
    assert calls
    for m in calls:
        before = src[:m.start()]
        before = before[:before.rindex(";") + 1]
        assert re.search(r"%s = __reduce_or_sync\(0xffffffffu, %s\);\s*$" % ((m.group(1),) * 2), before)


def test_every_lane_raises_the_error_flag():
    src = _source()
    flags = re.findall(r"if \(([^\n]*)\) atomicOr\((?:a\.)?error, 1\)", src)
    assert len(flags) >= 2 and all(f == "!ok" for f in flags), flags
