"""Model check of the hand-over of accumulators in the shared tcgen05 attention pipeline (zipage_b200/csrc/zp_attn_tc.cuh) on the CPU: one
group of softmax warps a tile (two groups: test_attention_halves_protocol.py).

The issuer of products, the tensor pipe (which works the issued products and commits off in order) and the softmax warps of both
tiles are replayed as coroutines over models of the mbarriers, under random schedules and random numbers of key tiles per item.  Checked:
no deadlock; a softmax warp reads the scores of its own step; the product reads the weights of its own step; and the output of
an item is read from that item's accumulator, although the next item's first product overwrites all of it.  A wait for a product
compares the parity of its barrier, so that the product before has to be reported before the next scores are: the other order takes the one
for the other.
"""
import random
from collections import deque

import pytest

from test_slot_protocol import Bar, Violation

WARPS = 4


def run(seed, done_before_scores=True, n_items=25):
    rnd = random.Random(seed)
    items = [(rnd.randint(0, 3), rnd.randint(0, 3)) for _ in range(n_items)]      # key tiles of the two query tiles
    sfull, pvdone = [Bar(1), Bar(1)], [Bar(1), Bar(1)]
    pfull = [[Bar(WARPS), Bar(WARPS)] for _ in range(2)]
    pipe, over = deque(), [False]      # what was issued; the issuer is done
    scores, weights, out = [None, None], [[None] * 2 for _ in range(2)], [None, None]

    def wait(bar, parity):
        while not bar.done(parity):
            yield

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
                        for _ in range(rnd.choice([0, 0, 200])):      # (an instruction that has to be fetched)
                            yield
                        pipe.append(("commit", pvdone[t]))
                    yield
        over[0] = True

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
                if weights[t][u] != step:
                    raise Violation("a product reads another step's weights")
                if step[1] == 0 and u == 0:
                    out[t] = (step[0], 0)                     # overwrites all columns
                elif out[t][0] != step[0]:
                    raise Violation("products of two items in one accumulator")
                out[t] = (step[0], step[1])

    def softmax_warp(t):
        cnt = 0
        for w, n in enumerate(items):
            for j in range(n[t]):
                yield from wait(sfull[t], cnt & 1)
                if scores[t] != (w, j):
                    raise Violation("scores of another step")
                if j > 0 and (w + j) % 3 == 0:        # the reference moves, and the accumulator with it
                    yield from wait(pvdone[t], (cnt & 1) ^ 1)
                    if out[t] != (w, j - 1):
                        raise Violation("another step's accumulator is rescaled")
                for u in range(2):
                    for _ in range(rnd.randint(0, 3)):
                        yield
                    weights[t][u] = (w, j)
                    pfull[t][u].arrive()
                cnt += 1
            if n[t]:
                yield from wait(pvdone[t], (cnt & 1) ^ 1)
                for _ in range(rnd.choice([0, 2, 60])):       # (loads of the gate, stores held up)
                    if out[t] != (w, n[t] - 1):
                        raise Violation("an item's output is read from another accumulator")
                    yield

    procs = [issuer(), tensor_pipe()] + [softmax_warp(t) for t in range(2) for _ in range(WARPS)]
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


@pytest.mark.parametrize("seed", range(20))
def test_an_items_output_is_its_own(seed):
    run(seed)


def test_reporting_a_product_after_the_next_scores_is_unsafe():
    failures = 0
    for seed in range(10):
        try:
            run(seed, done_before_scores=False)
        except Violation:
            failures += 1
    assert failures > 0
