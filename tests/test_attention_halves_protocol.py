"""Model check of how two groups of softmax warps share the rows of a tile in the tcgen05 attention pipeline
(zipage_b200/csrc/zp_attn_tc.cuh, two groups) on the CPU.

The issuer of products, the tensor pipe and the two warps of a row (one per half of the keys) of both tiles run as coroutines under random
schedules.  Both hand over two units of weights a step, and a product waits for both.  The warps exchange an item's sums through one place in
shared memory and meet there; scores without a cap a step's maxima too (capped ones have a fixed reference: their warps do not meet
in a step, and never rescale).  Checked: no deadlock; what a warp reads there is the other's number of the same step or item; products read
the weights of their step; a rescaled accumulator is the step before's and is whole before the next product (also without the meeting that follows
a rescale); an item's output is its own.  Without a cap, one meeting instead of two at an item's end lets the next step's maximum overwrite a sum that
is still to be read.  A product that waits for one group alone reads weights that are not there yet.  A product has to be reported before the next scores
are, as in the form of one group.  A warp that gives up arrives once more on its way out; without that its partner waits for good.
"""
import random
from collections import deque

import pytest

from test_slot_protocol import Bar, Violation


class Meeting:                          # barrier.cta.sync / .arrive of two warps
    def __init__(self):
        self.n, self.phase = 0, 0

    def arrive(self):
        self.n += 1
        if self.n == 2:
            self.n, self.phase = 0, self.phase + 1


def run(seed, capped=False, meetings=2, rescale_meets=True, waits_for_both=True, done_before_scores=True, fail_at=None, arrives_on_exit=True, n_items=25):
    rnd = random.Random(seed)
    items = [(rnd.randint(0, 3), rnd.randint(0, 3)) for _ in range(n_items)]
    sfull, pvdone = [Bar(1), Bar(1)], [Bar(1), Bar(1)]
    pfull = [[Bar(2 if waits_for_both else 1) for _ in range(2)] for _ in range(2)]
    pipe, over, abort = deque(), [False], [False]
    scores, weights, out = [None, None], [[[None] * 2, [None] * 2] for _ in range(2)], [None, None]
    meeting, place = [Meeting(), Meeting()], [[None, None], [None, None]]

    class Abort(Exception):
        pass

    def wait(bar, parity):
        for _ in range(3000):            # (a wait that runs out raises the flag)
            if bar.done(parity):
                return
            if abort[0]:
                raise Abort
            yield
        abort[0] = True
        raise Abort

    def issuer():
        cnt = [0, 0]
        for w, n in enumerate(items):
            for t in range(2):
                if n[t]:
                    pipe.append(("scores", t, (w, 0)))
                    pipe.append(("commit", sfull[t]))
            for j in range(max(n)):
                for t in range(2):
                    if j >= n[t]:
                        continue
                    for u in range(2):
                        yield from wait(pfull[t][u], cnt[t] & 1)
                        pipe.append(("product", t, (w, j), u))
                        yield
                    cnt[t] += 1
                    if done_before_scores:
                        pipe.append(("commit", pvdone[t]))
                    if j + 1 < n[t]:
                        pipe.append(("scores", t, (w, j + 1)))
                        pipe.append(("commit", sfull[t]))
                    if not done_before_scores:
                        for _ in range(rnd.choice([0, 0, 200])):
                            yield
                        pipe.append(("commit", pvdone[t]))
                    yield

    def tensor_pipe():
        while not over[0] or pipe:
            for _ in range(rnd.randint(0, 2)):
                yield
            if not pipe:
                yield
                continue
            op = pipe.popleft()
            if op[0] == "commit":
                op[1].arrive()
            elif op[0] == "scores":
                scores[op[1]] = op[2]
            else:
                _, t, step, u = op
                if weights[t][u] != [step, step]:
                    raise Violation("a product reads another step's weights")
                if step[1] == 0 and u == 0:
                    out[t] = [step[0], 0, {0, 1}]
                elif out[t][0] != step[0] or out[t][2] != {0, 1}:
                    raise Violation("a product into another item's or a half rescaled accumulator")
                out[t][1] = step[1]

    def warp(t, half):
        cnt = 0

        def meet():
            m = meeting[t]
            phase = m.phase
            m.arrive()
            while m.phase == phase:
                yield
            if abort[0]:
                raise Abort

        def swap(mine):
            place[t][half] = mine
            yield from meet()
            for _ in range(rnd.choice([0, 0, 30])):
                yield
            if place[t][1 - half] != mine:
                raise Violation("another number of the partner's")

        try:
            for w, n in enumerate(items):
                for j in range(n[t]):
                    if fail_at == (t, half, w, j):
                        abort[0] = True
                        raise Abort
                    yield from wait(sfull[t], cnt & 1)
                    if scores[t] != (w, j):
                        raise Violation("scores of another step")
                    if not capped:
                        yield from swap(("max", w, j))
                    if not capped and j > 0 and (w + j) % 3 == 0:        # the reference moves
                        yield from wait(pvdone[t], (cnt & 1) ^ 1)
                        if out[t][:2] != [w, j - 1]:
                            raise Violation("another step's accumulator is rescaled")
                        if out[t][2] == {0, 1}:
                            out[t][2] = set()
                        out[t][2].add(half)
                        if rescale_meets:
                            yield from meet()
                    for u in range(2):
                        for _ in range(rnd.randint(0, 3)):
                            yield
                        weights[t][u][half] = (w, j)
                        if waits_for_both or half == 0:
                            pfull[t][u].arrive()
                    cnt += 1
                if n[t]:
                    yield from wait(pvdone[t], (cnt & 1) ^ 1)
                    yield from swap(("sum", w))
                    if meetings == 2:
                        yield from meet()
                    for _ in range(rnd.choice([0, 2, 60])):
                        if out[t][:2] != [w, n[t] - 1]:
                            raise Violation("an item's output is read from another accumulator")
                        yield
        except Abort:
            if arrives_on_exit:
                meeting[t].arrive()

    def role(g):
        try:
            yield from g
        except Abort:
            pass
        over[0] = over[0] or g is first

    first = issuer()
    procs = [role(first), tensor_pipe()] + [warp(t, h) for t in range(2) for h in range(2)]
    alive, steps = [True] * len(procs), 0
    while any(alive):
        i = rnd.randrange(len(procs))
        if alive[i]:
            try:
                next(procs[i])
            except StopIteration:
                alive[i] = False
        steps += 1
        if steps > 400000:
            raise Violation("deadlock")
    if fail_at is None and abort[0]:
        raise Violation("a wait ran out")


def broken(seeds, fail_item=None, **how):
    """What the checks say of a broken form; at least one schedule has to show it.  `fail_item`: a warp gives up in one of so many items."""
    said = []
    for seed in range(seeds):
        try:
            run(seed, fail_at=(0, 0, seed % fail_item, 0) if fail_item else None, **how)
        except Violation as e:
            said.append(str(e))
    assert said
    return said


@pytest.mark.parametrize("capped", [False, True])
@pytest.mark.parametrize("seed", range(20))
def test_the_halves_of_a_row_agree(seed, capped):
    run(seed, capped)


@pytest.mark.parametrize("seed", range(10))
def test_nothing_hangs_on_the_meeting_after_a_rescale(seed):
    run(seed, rescale_meets=False)


def test_one_meeting_at_the_end_of_an_item_is_unsafe():
    assert all("partner" in s for s in broken(10, meetings=1))


@pytest.mark.parametrize("capped", [False, True])
def test_a_product_that_waits_for_one_group_is_unsafe(capped):
    assert all("weights" in s for s in broken(10, capped=capped, waits_for_both=False))


@pytest.mark.parametrize("capped", [False, True])
def test_reporting_a_product_after_the_next_scores_is_unsafe(capped):
    broken(10, capped=capped, done_before_scores=False)


@pytest.mark.parametrize("capped", [False, True])
@pytest.mark.parametrize("seed", range(10))
def test_a_warp_that_gives_up_holds_nobody_up(seed, capped):
    for t in range(2):
        for half in range(2):
            run(seed, capped, fail_at=(t, half, seed % 5, 0))


def test_leaving_without_an_arrival_is_unsafe():
    assert all("deadlock" in s for s in broken(6, fail_item=3, arrives_on_exit=False))
