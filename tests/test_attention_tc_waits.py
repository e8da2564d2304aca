"""The waits of the tcgen05 attention kernel, walked through on the CPU in every order that the hardware allows.

``locus_attn_tc_wait`` says which barrier and which parity each role waits for before each of its steps (the kernel takes them
from the same functions).  Here the roles' steps, the arrival of loads and the completion of products are taken in every
possible order, the barriers counted as mbarriers count; a wait must never pass before what it waits for has happened, and no order may
leave the roles waiting for each other."""
import ctypes
from functools import lru_cache

import pytest

from locus_b200.csrc import build

WAITS = ("k_place", "v_place", "k_there", "s_place", "v_there", "p_there", "s_there", "summed", "v_clear", "done")
SCORES = 3   # places of the scores


class Waits:
    def __init__(self, rot):
        build.ensure(["attention_tc"])
        fn = build.load("attention_tc").locus_attn_tc_wait
        fn.argtypes, fn.restype = [ctypes.c_int] * 3, ctypes.c_int
        self.places = 2 if rot else 3   # of K and of V
        self.end = lambda last: [self.done(last)]
        for i, name in enumerate(WAITS):
            setattr(self, name, lru_cache(None)(lambda j, i=i: (lambda v: None if v < 0 else (v >> 1, v & 1))(fn(int(rot), i, j))))


def walk(w, n):
    """Every order of the steps of a block of ``n`` key tiles."""
    D, last = w.places, n - 1
    # the loader's order: the first places' K, then V and K in turn
    loads = [("K", j) for j in range(min(D, n))]
    for j in range(n):
        loads.append(("V", j))
        if j + D < n:
            loads.append(("K", j + D))
    # state: loads issued, loads under way, score products issued / done, sums issued / done, per group of warps (tile, step);
    # step 0: before the scores, 1: scores read, 2: rescales the sum, 3: reference handed on, 4 (last tile): V's dead rows are cleared, 5: the whole sum read
    start = (0, frozenset(), 0, 0, 0, 0, ((0, 0), (1, 0)))
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()
        issued, flying, s_out, s_done, v_out, v_done, groups = state
        there = lambda kind, j: (kind, j) in loads[:issued] and (kind, j) not in flying
        ready = lambda j: groups[j & 1][0] > j             # the weights of tile j are written
        handed = lambda j: ready(j) or groups[j & 1] in ((j, 3), (j, 4))

        def turns(bar):   # ends of a turn so far: every arrival ends one
            count = sum(1 for kind, j in loads[:issued] if there(kind, j) and (w.k_there if kind == "K" else w.v_there)(j)[0] == bar)
            count += sum((w.k_place(j)[0] == bar) + (w.s_there(j)[0] == bar) for j in range(s_done))
            count += sum(bar in {w.v_place(j)[0], w.s_place(j)[0]} for j in range(v_done))
            count += v_done == n and w.done(last)[0] == bar
            return count + sum(w.p_there(j)[0] == bar for j in range(n) if ready(j))

        def passes(wait, truth, what):
            if wait is None:
                return True
            bar, parity = wait
            if (turns(bar) & 1) == parity:
                return False
            assert truth, f"{what} in {state}"
            return True

        after = []
        if issued < len(loads):
            kind, j = loads[issued]
            free = j < D or (s_done > j - D if kind == "K" else v_done > j - D)
            if passes((w.k_place if kind == "K" else w.v_place)(j), free, f"{kind}{j} into a place in use"):
                after.append((issued + 1, flying | {(kind, j)}, s_out, s_done, v_out, v_done, groups))
        for load in flying:
            after.append((issued, flying - {load}, s_out, s_done, v_out, v_done, groups))
        if s_out < n and passes(w.k_there(s_out), there("K", s_out), f"scores {s_out} without K") \
                and passes(w.s_place(s_out), s_out < SCORES or v_done > s_out - SCORES, f"scores {s_out} into a place in use"):
            after.append((issued, flying, s_out + 1, s_done, v_out, v_done, groups))
        if s_done < s_out:
            after.append((issued, flying, s_out, s_done + 1, v_out, v_done, groups))
        if v_out < n and passes(w.v_there(v_out), there("V", v_out), f"sum {v_out} without V") \
                and passes(w.p_there(v_out), ready(v_out), f"sum {v_out} without weights"):
            after.append((issued, flying, s_out, s_done, v_out + 1, v_done, groups))
        if v_done < v_out:
            after.append((issued, flying, s_out, s_done, v_out, v_done + 1, groups))
        for x in (0, 1):
            j, step = groups[x]

            def to(tile, nxt):
                after.append((issued, flying, s_out, s_done, v_out, v_done, tuple((tile, nxt) if y == x else groups[y] for y in (0, 1))))

            if j > last:
                if step == 0 and all(passes(wait, v_done == n, "the whole sum read too early") for wait in w.end(last)):
                    to(j, 5)
                continue
            if step == 0 and passes(w.s_there(j), s_done > j, f"scores {j} read too early"):
                to(j, 1)
            elif step == 1 and (j == 0 or handed(j - 1)):
                to(j, 3)
                if j > 0:
                    to(j, 2)
            elif step == 2 and passes(w.summed(j - 1), v_done >= j, f"the sum before tile {j} rescaled too early"):
                to(j, 3)
            elif step == 3 and j < last:
                to(j + 2, 0)
            elif step == 3 and passes(w.v_clear(j), j < D or v_done > j - D, f"V of tile {j} cleared while tile {j - D} uses its place"):
                to(j, 4)
            elif step == 4 and passes(w.v_there(j), there("V", j), f"V of tile {j} cleared before it is there"):
                to(j + 2, 0)
        if not after:
            assert v_done == n and issued == len(loads) and not flying and groups[0][1] == groups[1][1] == 5, f"stuck: {state}"
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return len(seen)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("rot", [False, True])
def test_no_order_of_steps_is_stuck_or_early(rot, n):
    assert walk(Waits(rot), n) >= n


def test_the_walk_finds_a_scores_place_that_shares_the_barrier_of_vs_place():
    """Two places of V, three of the scores: the sum of the tile after next in V's place may end the turn behind."""
    w = Waits(True)
    w.s_place = lambda j: (w.v_place(0)[0] + (j - SCORES) % 2, ((j - SCORES) // 2) & 1) if j >= SCORES else (w.v_place(0)[0], 1)
    with pytest.raises(AssertionError, match="stuck"):
        walk(w, 6)


def test_the_walk_finds_rows_of_v_cleared_too_early():
    """Two places of V: before the sum of the tile before in V's place, a wait for V passes with that tile's turn still to come."""
    w = Waits(True)
    w.v_clear = lambda j: None
    with pytest.raises(AssertionError, match="cleared before it is there"):
        walk(w, 3)


@pytest.mark.parametrize("rot", [False, True])
def test_the_walk_finds_a_last_sum_waited_for_at_vs_place(rot):
    """The place of V turns twice for the last tile and the one before in its place: a warp that asks for the first turn behind the second
    is stuck, one that asks for the second alone may pass before the first."""
    w = Waits(rot)
    D = w.places
    w.end = lambda last: [w.summed(last)] if last < D else [w.summed(last - D)]
    with pytest.raises(AssertionError, match="stuck|too early"):
        walk(w, D + 1)
    w.end = lambda last: [w.summed(last)]
    with pytest.raises(AssertionError, match="too early"):
        walk(w, 2 * D + 1)
