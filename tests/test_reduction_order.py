"""The memory order of the grid reductions, read from their source.

A reduction's last block reads what other blocks' threads wrote, having learned
of it from an atomic counter.  In the PTX memory model that takes an acquire
pattern -- the atomic and then a fence -- in ONE thread, before the block's barrier
passes the knowledge on; fences that other threads execute behind the barrier do
not make one.  No run can show the difference reliably, so the order is checked here.
"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "alien_b200" / "csrc"


def _code(name: str) -> str:
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def _body(src: str, start: int) -> str:
    """The brace block that opens first after `start`."""
    i = src.index("{", start)
    depth = 0
    for j in range(i, len(src)):
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        if depth == 0:
            return src[i:j + 1]
    raise AssertionError("unbalanced braces")


def test_every_arrival_is_released_and_acquired_by_the_thread_that_makes_it():
    src = _code("reduce.cuh")
    arrivals = [m.start() for m in re.finditer(r"atomicAdd\(", src)]
    assert arrivals
    for at in arrivals:
        before, after = src[:at], src[at:]
        # released: nothing but the start of the statement between a fence and the atomic
        assert re.search(r"fence_gpu\(\);\s*[\w\s]*=?\s*$", before), src[at - 120:at + 40]
        # acquired: a fence before the thread reaches a barrier or leaves the function
        fence, barrier = after.find("fence_gpu()"), after.find("__syncthreads")
        leave = after.find("\n}")
        assert 0 <= fence < min(x for x in (barrier, leave) if x >= 0), src[at - 120:at + 200]


def test_reductions_read_partials_behind_one_arrival():
    src = _code("reduce.cuh")
    for name in ("grid_reduce", "grid_reduce_v", "grid_reduce_r"):
        body = _body(src, re.search(rf"\b{name}\(", src).start())
        arrive, read = body.find("last_arrival("), body.find("sum_partials<")
        assert 0 <= arrive < read, name
        assert "__syncthreads" in body[arrive:read], name
