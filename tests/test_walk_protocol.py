"""CPU model of a walk group's phases (walk_pair in rfd_engine.cu): the members read the pair's state,
sweep together (barriers in the sweep) or take a result that is at hand, the first member writes the
next phase, all meet.  Every interleaving of two members has to lead both through the same phases,
with no barrier of one phase met in another."""
import pytest

VE_AT_HAND = {"dfd": False, "vefd": True, "search": False}
NEXT = {"dfd": "vefd", "vefd": "search", "search": "done"}


def member(rank, barrier_at_hand):
    """Steps of one member: ("read",), ("write", phase) or ("barrier", where)."""
    while True:
        phase = yield ("read",)
        if phase == "done":
            return
        if not VE_AT_HAND[phase]:
            yield ("barrier", phase + " sweep")
        elif barrier_at_hand:
            yield ("barrier", phase + " at hand")
        if rank == 0:
            yield ("write", NEXT[phase])
        yield ("barrier", phase + " end")


def explore(barrier_at_hand):
    """Outcomes of all interleavings: a set of True (together throughout) and False."""
    outcomes = set()

    def replay(trace):
        ms = [member(r, barrier_at_hand) for r in range(2)]
        state, step, at = "dfd", [next(m) for m in ms], [None, None]
        for r in trace:
            kind = step[r][0]
            sent = None
            if kind == "read":
                sent = state
            elif kind == "write":
                state = step[r][1]
            else:  # arrive; the second to arrive releases both
                at[r] = step[r][1]
                if at[1 - r] is None:
                    continue
                if at[0] != at[1]:
                    return "apart"
                for q in (0, 1):
                    at[q] = None
                    step[q] = advance(ms[q], None)
                continue
            step[r] = advance(ms[r], sent)
        return [r for r in (0, 1) if step[r] is not None and at[r] is None], step, at

    def advance(m, sent):
        try:
            return m.send(sent)
        except StopIteration:
            return None

    todo = [[]]
    while todo:
        trace = todo.pop()
        got = replay(trace)
        if got == "apart":
            outcomes.add(False)
            continue
        ready, step, at = got
        if not ready:  # both left, or one waits for a member that has left
            outcomes.add(step == [None, None])
            continue
        todo += [trace + [r] for r in ready]
    return outcomes


@pytest.mark.parametrize("barrier_at_hand,want", [(True, {True}), (False, {True, False})])
def test_members_go_through_the_phases_together(barrier_at_hand, want):
    """With the barrier before a result at hand is taken all interleavings agree; without it some
    do not (the model sees the fault that the barrier is there for)."""
    assert explore(barrier_at_hand) == want
