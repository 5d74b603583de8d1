"""A bounded wait that runs out must leave the lanes of a warp together.

Each lane of a warp polls an mbarrier by itself and looks at the clock and at the CTA's abort flag
only every 64 polls, so when a phase completes around the time limit some lanes of one warp may
return true and others false.  Lanes that go on then reach instructions that take the whole warp
(tensor-memory loads, votes, shuffles) while the others wait in the kernel's closing barrier, and the
bounded wait has become an endless one.  `run_warp` restates that; the last test reads the kernels'
sources for the rule that prevents it: either the lanes vote on the result of a wait, or the result
decides nothing and the abort flag is voted on before anything is stored.
"""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ring_attention_b200", "csrc")
LANES, POLLS_PER_LOOK = 32, 64


def _wait(lane, done_at, limit):
    """mbar_wait of one lane: `lane` polls behind the others; true once the phase (complete at
    `done_at`) is seen, false when a look at the clock finds the time limit passed."""
    for it in range(1, 10 * (done_at + limit + LANES)):
        now = it + lane
        if now >= done_at:
            return True
        if it % POLLS_PER_LOOK == 0 and now > limit:
            return False
    raise AssertionError("unbounded")


def run_warp(done_at, limit, lag, vote):
    """Whether the warp gets to the closing barrier: the lanes that went on after the wait execute a
    warp-wide instruction, which completes only with all lanes."""
    results = [_wait(lag[i], done_at, limit) for i in range(LANES)]
    if vote:
        results = [all(results)] * LANES
    return all(results) or not any(results)


@pytest.mark.parametrize("vote", [True, False])
def test_lanes_leave_a_wait_together(vote):
    rng = random.Random(1)
    stuck = 0
    for _ in range(400):
        limit = rng.randrange(100, 400)
        done_at = limit + rng.randrange(-40, 120)  # the phase completes around the limit
        stuck += not run_warp(done_at, limit, [rng.randrange(0, 40) for _ in range(LANES)], vote)
    assert stuck == 0 if vote else stuck > 20


@pytest.mark.parametrize("name", ["fwd_sm100.cu", "bwd_sm100.cu"])
def test_no_lane_acts_on_its_own_wait(name):
    text = re.sub(r"//[^\n]*", lambda m: " " * len(m.group()), open(os.path.join(CSRC, name)).read())
    waits = [m.start() for m in re.finditer(r"\bmbar_wait\(", text)]
    alone, discarded = [], False
    for at in waits:
        statement = text[max(text.rfind(c, 0, at) for c in ";{}") + 1 : text.find(";", at)].strip()
        if "kStFwdProducer" in statement:  # the forward's TMA producer runs in lane 0 alone
            continue
        if statement.startswith("mbar_wait("):
            discarded = True
        elif "__all_sync(0xffffffffu, mbar_wait(" not in statement:
            alone.append(text.count("\n", 0, at) + 1)
    assert len(waits) > 5
    assert not alone, f"{name}: lanes act on their own wait in lines {alone}"
    if discarded:
        assert re.search(r"__all_sync\(0xffffffffu, mbar_wait\([^;]*\*abort_flag == 0\)", text), name
