"""Which lanes' copies are ordered after a flag that other lanes of the warp
read: k_wave's loader (lanes 0 and 1 watch the completion words, every lane
copies) and k_jacobi_flow's thirteenth warp (lanes 0-8 watch the neighbours'
flags, lane 0 copies).  A vote makes the lanes agree on a value but orders no
memory; a warp barrier orders what each lane has observed before what every
lane does next.  The model keeps, for each lane, the set of stores that happen
before its next action."""
import pytest

LANES = range(32)


def observe(watchers, barrier):
    """The stores each lane's next copy is ordered after, when each watcher
    acquires the flag of a publisher of its own."""
    seen = [{("publisher", l)} if l in watchers else set() for l in LANES]
    # The vote: every lane learns that all flags are set, nothing more.
    if barrier:
        every = set().union(*seen)
        seen = [set(every) for _ in LANES]
    return seen


@pytest.mark.parametrize("watchers,copiers", [((0, 1), LANES), (range(9), (0,))])
def test_copies_follow_every_watched_publisher(watchers, copiers):
    need = {("publisher", l) for l in watchers}
    seen = observe(watchers, True)
    assert all(need <= seen[l] for l in copiers)
    seen = observe(watchers, False)  # a vote alone does not order them
    assert not all(need <= seen[l] for l in copiers)


def test_lanes_that_wait_agree_before_they_go_on():
    """A lane's own test of a barrier, or its own reading of the timer, may
    differ from the next lane's: every branch that leads to a shuffle, a vote
    or a block barrier is taken by the whole warp or not at all."""
    code = body("k_pressure.cu", "auto claim = [&]", "if (fail && lane == 0) {\n    atomicExch")
    assert "mbar_test(" not in code.replace("warp_test(", "")
    waits = [x for x in code.splitlines() if "mbar_wait_bounded(" in x or "MBAR_WAIT_NS" in x]
    assert len(waits) == 2 and all("_sync(0xffffffffu" in x for x in waits)


def body(path, start, end):
    import os

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    text = open(os.path.join(root, "fluid_gb300", "csrc", path)).read()
    at = text.index(start)
    return text[at:text.index(end, at)]


@pytest.mark.parametrize("path,start,end", [
    ("k_lexsor.cu", "auto ready = [&](int c)", "auto publish"),
    ("k_pressure.cu", "bool flow_ready_warp(", "constexpr int FW"),
])
def test_a_warp_barrier_follows_the_vote(path, start, end):
    code = body(path, start, end)
    assert code.index("__all_sync") < code.index("__syncwarp()")
