"""Protocols of the bulk operations and the searches' exchange, every
interleaving (oracle/lock_model.py): the last node given back, the end of a
bulk delete, the locks of the next level, the heap build; and the served
loop's lock."""
import pytest

from oracle import lock_model as lm


def finishes(model):
    init, actors, final = model
    res = lm.explore(init, actors, final, progress=True)
    assert res.finals >= 1 and not res.deadlocks and not res.stuck, (res.deadlocks[:1], res.stuck[:1])


@pytest.mark.parametrize("refuse", [True, False])
@pytest.mark.parametrize("as_found", [True, False])
def test_last_node_given_back(refuse, as_found):
    finishes(lm.exchange_giveback_model(refuse=refuse, back_as_found=as_found))


def test_last_node_written_and_given_back_as_found_is_caught():
    init, actors, final = lm.exchange_giveback_model(unchanged=False)
    with pytest.raises(lm.Violation, match="stale copy"):
        lm.explore(init, actors, final)


@pytest.mark.parametrize("blocks,items", [(2, 0), (3, 0), (3, 2), (4, 2), (2, 4)])
def test_bulk_delete_ends_for_every_block(blocks, items):
    finishes(lm.delete_stop_model(blocks=blocks, items=items))


def test_a_ticket_given_up_hangs_blocks_that_do_not_look():
    init, actors, final = lm.delete_stop_model(blocks=4, items=0, lookers=1)
    assert lm.explore(init, actors, final).deadlocks


@pytest.mark.parametrize("levels,sifts,inserts", [(3, 1, 1), (4, 2, 1), (4, 1, 2), (3, 2, 2)])
def test_next_level_locked_before_the_last_is_released(levels, sifts, inserts):
    finishes(lm.next_level_model(levels=levels, sifts=sifts, inserts=inserts))


def test_waiting_for_the_parent_there_deadlocks():
    init, actors, final = lm.next_level_model(try_once=False)
    assert lm.explore(init, actors, final).deadlocks


@pytest.mark.parametrize("nodes,blocks", [(1, 2), (3, 1), (6, 2), (7, 2), (7, 3), (12, 2)])
def test_heap_build_finishes(nodes, blocks):
    finishes(lm.build_model(nodes=nodes, blocks=blocks))


def test_heap_build_in_ascending_order_deadlocks():
    init, actors, final = lm.build_model(nodes=7, blocks=2, descending=False)
    assert lm.explore(init, actors, final).deadlocks


@pytest.mark.parametrize("pollers", [1, 2, 3])
def test_a_completion_gets_the_served_loops_lock(pollers):
    finishes(lm.serve_lock_model(pollers=pollers))


@pytest.mark.parametrize("mistake", [dict(keep_off=False), dict(raise_only=False)])
def test_admissions_that_pass_a_waiting_completion_are_caught(mistake):
    init, actors, final = lm.serve_lock_model(**mistake)
    with pytest.raises(lm.Violation, match="past a waiting completion"):
        lm.explore(init, actors, final)
