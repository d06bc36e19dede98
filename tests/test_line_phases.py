"""The mbarrier protocol of the line kernel (sdg_tend_line.cuh) as a model: a
parity wait passes while the barrier's current phase has the other parity, so a
wait for a phase that may already be two phases back never passes.  Every
interleaving of the producer and the consumers must come to its end, and the
producer's waits in the source must be the model's."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "scale-dg-kernel-extraction_b200", "csrc", "sdg_tend_line.cuh")
# The producer's waits of iteration `it`, in order, as the source spells them.
PRODUCER_WAITS = [("eu", "(it - 1) & 1"), ("done", "(it - 1) & 1")]
TILES = 7


def producer(waits_first=()):
    for it in range(TILES):
        for bar, parity in waits_first:
            if it >= 2:
                yield "wait", bar, eval(parity, {"it": it})
        yield "arrive", "fq%d" % (it & 1), 0
        if it > 0:
            yield "wait", "eu", (it - 1) & 1
        yield "arrive", "fu", 0
        if it > 0:
            yield "wait", "done", (it - 1) & 1
        yield "arrive", "fv", 0
        yield "arrive", "fw", 0


def consumer(late):
    yield "wait", "fq0", 0
    for it in range(TILES):
        yield "wait", "fq%d" % (it & 1), (it >> 1) & 1
        yield "wait", "fu", it & 1
        if it > 0:
            yield "wait", "done", (it - 1) & 1
        yield "wait", "fv", it & 1
        yield "arrive", "eu", 0
        yield "wait", "fw", it & 1
        if not late:
            yield "arrive", "done", 0
        if it + 1 < TILES:
            yield "wait", "fq%d" % ((it + 1) & 1), ((it + 1) >> 1) & 1
        if late:
            yield "arrive", "done", 0


def stuck_states(prod, cons):
    """Reachable states in which neither side can go on and one has not ended."""
    bars = sorted({op[1] for op in prod + cons})
    start = (0, 0, (0,) * len(bars))
    seen, todo, stuck = {start}, [start], []
    while todo:
        pc = todo.pop()
        nexts = []
        for side, prog in ((0, prod), (1, cons)):
            if pc[side] == len(prog):
                continue
            op, bar, parity = prog[pc[side]]
            phase = list(pc[2])
            b = bars.index(bar)
            if op == "wait" and (phase[b] & 1) == parity:
                continue
            if op == "arrive":
                phase[b] += 1
            at = [pc[0], pc[1]]
            at[side] += 1
            nexts.append((at[0], at[1], tuple(phase)))
        if not nexts and (pc[0] < len(prod) or pc[1] < len(cons)):
            stuck.append(pc)
        for n in nexts:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return stuck


@pytest.mark.parametrize("late", [False, True])
def test_every_interleaving_ends(late):
    assert not stuck_states(list(producer()), list(consumer(late)))


def test_the_model_sees_a_wait_for_a_phase_twice_back():
    twice = list(producer([("done", "it & 1")]))
    assert stuck_states(twice, list(consumer(False)))


def test_source_has_the_models_waits():
    text = open(SRC).read()
    text = text[text.index("// ---- Producer"):text.index("// ---- Consumers")]
    text = re.sub(r"//[^\n]*", "", text)
    assert re.findall(r"mbar_wait_bounded\((\w+), ([^,]*), spins\)", text) == PRODUCER_WAITS
