"""When idle warps may leave: the enumeration kernel's busy count and ready
ring, restated step by step and explored over every interleaving of a few warps.
A task that one warp publishes must be solved before the last warp leaves.

Every step below is one access to a shared word.  The ring's count of filled
cells is a word of its own, and nothing orders its add before the same warp's
later steps on other words: it may become visible at any later time.
"""
from __future__ import annotations

import pytest

# A warp's state is (step, value); a task's value is how often it still hops: its
# taker publishes one task of one hop less, then ends.
IDLE, POLL, LOOK, TAKE, UNDO, FREE, WORK, PUSH, END, LEFT, START = range(11)


def explore(start_hops, blocks, protocol, late_start=None):
    """All reachable states; returns those in which every warp has left.  Warp 0
    holds an item; the others have found no more of them, but for the last one
    if it starts late, which still claims an item of late_start hops."""
    warps = [(WORK, start_hops) if i == 0 else (IDLE, 0) for i in range(len(blocks))]
    if late_start is not None:
        warps[-1] = (START, late_start)
    warps = tuple(warps)
    # busy count, visible ring count, ring adds not yet visible, tasks in the ring, poll tokens, warps
    first = (1, 0, 0, (), (0,) * (max(blocks) + 1), warps)
    seen, todo, finals = {first}, [first], []
    while todo:
        state = todo.pop()
        if all(w[0] == LEFT for w in state[5]):
            finals.append(state)
        busy, count, late, ring, tokens, ws = state
        after = [(busy, count + 1, late - 1, ring, tokens, ws)] if late else []
        for i, w in enumerate(ws):
            after += protocol(state, i, blocks[i], w)
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return finals


def moved(state, i, w, busy=None, count=None, late=None, ring=None, token=None, block=0):
    b, c, l, r, t, ws = state
    if token is not None:
        t = t[:block] + (token,) + t[block + 1:]
    return (b if busy is None else busy, c if count is None else count, l if late is None else late,
            r if ring is None else ring, t, ws[:i] + (w,) + ws[i + 1:])


def tasks_counted(state, i, block, w):
    """As in the kernel: the busy count holds warps and unfinished tasks."""
    busy, count, late, ring, tokens, _ = state
    step, val = w
    if step == START:  # counted before the first claim
        return [moved(state, i, (WORK, val), busy=busy + 1)]
    if step == IDLE:
        if tokens[block] == 2:  # the block's last poller saw nobody busy
            return [moved(state, i, (LEFT, 0))] if busy == 0 else [moved(state, i, (IDLE, 0), token=0, block=block)]
        return [moved(state, i, (POLL, 0), token=1, block=block)] if tokens[block] == 0 else []
    if step == POLL:
        return [moved(state, i, (FREE, "leave") if busy == 0 else (LOOK, 0))]
    if step == LOOK:
        return [moved(state, i, (TAKE, 0) if count > 0 else (FREE, "stay"))]
    if step == TAKE:
        if count <= 0:
            return [moved(state, i, (UNDO, 0), count=count - 1)]
        return [moved(state, i, (FREE, ring[0]), count=count - 1, ring=ring[1:])]
    if step == UNDO:
        return [moved(state, i, (FREE, "stay"), count=count + 1)]
    if step == FREE:
        if val == "leave":
            return [moved(state, i, (LEFT, 0), token=2, block=block)]
        return [moved(state, i, (IDLE, 0) if val == "stay" else (WORK, val), token=0, block=block)]
    if step == WORK:
        return [moved(state, i, (PUSH, val), busy=busy + 1) if val else moved(state, i, (END, 0))]
    if step == PUSH:
        return [moved(state, i, (END, 0), ring=ring + (val - 1,), late=late + 1)]
    if step == END:
        return [moved(state, i, (IDLE, 0), busy=busy - 1)]
    return []


def warps_counted(state, i, block, w):
    """A busy count of warps alone: "nobody busy, queue empty, nobody busy",
    twice, and the block leaves with its poller."""
    busy, count, late, ring, tokens, _ = state
    step, val = w
    if step == IDLE:
        if tokens[block] == 2:
            return [moved(state, i, (LEFT, 0))]
        return [moved(state, i, (POLL, val), token=1, block=block)] if tokens[block] == 0 else []
    if step == POLL:
        return [moved(state, i, (LOOK, (val, busy)))]
    if step == LOOK:
        quiet, before = val
        if count > 0:
            return [moved(state, i, (TAKE, 0), busy=busy + 1)]
        return [moved(state, i, (UNDO, ("again", quiet, before)))]
    if step == TAKE:
        if count <= 0:
            return [moved(state, i, (UNDO, ("count",)), count=count - 1)]
        return [moved(state, i, (FREE, ("work", ring[0])), count=count - 1, ring=ring[1:])]
    if step == UNDO:
        if val[0] == "count":
            return [moved(state, i, (UNDO, ("busy",)), count=count + 1)]
        if val[0] == "busy":
            return [moved(state, i, (FREE, ("stay", 0)), busy=busy - 1)]
        quiet = val[1] + 1 if val[2] == 0 and busy == 0 else 0
        return [moved(state, i, (FREE, ("leave", 0) if quiet >= 2 else ("stay", quiet)))]
    if step == FREE:
        what, v = val
        if what == "leave":
            return [moved(state, i, (LEFT, 0), token=2, block=block)]
        return [moved(state, i, (IDLE, v) if what == "stay" else (WORK, v), token=0, block=block)]
    if step == WORK:
        return [moved(state, i, (PUSH, val) if val else (END, 0))]
    if step == PUSH:
        return [moved(state, i, (END, 0), ring=ring + (val - 1,), late=late + 1)]
    if step == END:
        return [moved(state, i, (IDLE, 0), busy=busy - 1)]
    return []


@pytest.mark.parametrize("late_start", [None, 0, 2])
@pytest.mark.parametrize("blocks,hops", [((0, 0), 3), ((0, 1), 3), ((0, 0, 1), 2), ((0, 1, 0), 2), ((0, 1, 1), 2),
                                         ((0, 1, 2), 2)])
def test_no_task_is_left_behind(blocks, hops, late_start):
    finals = explore(hops, blocks, tasks_counted, late_start)
    assert finals
    assert all(s[0] == 0 and s[1] + s[2] == 0 and s[3] == () for s in finals)


def test_counting_warps_alone_can_leave_a_task():
    """The exploration sees the fault: with the ring's count late, both blocks
    leave while a task is in the ring."""
    finals = explore(1, (0, 1), warps_counted)
    assert any(s[3] for s in finals) and any(not s[3] for s in finals)
