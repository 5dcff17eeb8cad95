"""The time limit of a search's waiting blocks beside a block that stays busy
over rounds (oracle/lock_model.py busy_rounds_model), every interleaving."""
import pytest

from oracle import lock_model as lm


@pytest.mark.parametrize("waiters,rounds", [(1, 4), (2, 3), (3, 2)])
def test_no_time_out_beside_a_block_that_works(waiters, rounds):
    init, actors, final = lm.busy_rounds_model(waiters=waiters, rounds=rounds)
    res = lm.explore(init, actors, final, progress=True)
    assert res.finals >= 1 and not res.deadlocks and not res.stuck


def test_looking_at_busy_alone_times_out():
    init, actors, final = lm.busy_rounds_model(stamps=False)
    with pytest.raises(lm.Violation, match="beside a block that works"):
        lm.explore(init, actors, final)


@pytest.mark.parametrize("waiters", [1, 2])
def test_a_block_that_stops_is_noticed_by_every_waiter(waiters):
    init, actors, _ = lm.busy_rounds_model(waiters=waiters, hangs=True)
    ends = []
    res = lm.explore(init, actors, lambda g, trace: ends.append(g))
    # only the stopped block is left: every run ends with all waiters timed out
    assert res.deadlocks and not ends
    for t in res.deadlocks:
        assert sum(step.endswith("times out") for step in t) == waiters
