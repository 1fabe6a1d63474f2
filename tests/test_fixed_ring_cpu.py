"""The rings of the fixed-point product, modelled on the CPU: several groups of converting warps take the steps of one ring in turn, and a
wait by parity only tells a barrier's phase from the one before it.  Loads that land late and out of order must never let a group read a
stage that its step's load has not filled."""

import heapq
import random
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "pyre_b200" / "csrc" / "gemm_fixed.cu").read_text()
WIDTHS = (8, 16, 32, 48, 64)


def constant(name: str, tn: int) -> int:
    """The value of an integer constant of the kernel's source for tiles of ``tn`` tokens (a literal or a chain of ``a ? b : c``)."""
    expr = re.search(rf"\b{name} = ([^,;]+)[,;]", SOURCE).group(1)
    while "?" in expr:
        condition, rest = expr.split("?", 1)
        yes, no = rest.split(":", 1)
        expr = yes if eval(condition, {}, {"TN": tn}) else no
    return int(expr)


class Barrier:
    """The completed phases of an mbarrier; ``passes`` is what a wait for a parity sees."""

    def __init__(self, count: int):
        self.count, self.left, self.phase = count, count, 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1

    def passes(self, parity: int) -> bool:
        return (self.phase - 1) & 1 == parity


def run_ring(w_stages: int, a_stages: int, groups: int, steps: int, rng: random.Random, late: "dict[int, int]") -> "list[int]":
    """Steps whose group read a stage before that step's load had filled it.  ``late``: cycles that a step's load takes beyond the usual."""
    w_full, w_empty = [Barrier(1) for _ in range(w_stages)], [Barrier(1) for _ in range(w_stages)]
    a_full, a_empty = [Barrier(1) for _ in range(a_stages)], [Barrier(1) for _ in range(a_stages)]
    holds = [-1] * w_stages      # the step whose weights a stage holds
    wrong, events = [], []
    order = iter(range(1 << 60))

    def at(time, fn, *args):
        heapq.heappush(events, (time, next(order), fn, args))

    def wait(time, barrier, parity, then):      # polls every few cycles
        def poll(now):
            if barrier.passes(parity):
                then(now)
            else:
                at(now + 7, poll, now + 7)
        poll(time)

    def produce(now, step):
        if step == steps:
            return
        s = step % w_stages

        def issue(t):
            def land(t2):
                holds[s] = step
                w_full[s].arrive()
            t2 = t + 700 + rng.randrange(60) + late.get(step, 0)
            at(t2, land, t2)
            at(t + 10, produce, t + 10, step + 1)
        wait(now, w_empty[s], (step // w_stages & 1) ^ 1, issue)

    def convert(now, step):
        if step >= steps:
            return
        s, sa = step % w_stages, step % a_stages

        def read(t):
            if holds[s] != step:
                wrong.append(step)
            t2 = t + 120 + rng.randrange(20)

            def done(t3):
                w_empty[s].arrive()

                def store(t4):
                    a_full[sa].arrive()
                    at(t4 + 40, convert, t4 + 40, step + groups)
                wait(t3, a_empty[sa], (step // a_stages & 1) ^ 1, store)
            at(t2, done, t2)
        wait(now, w_full[s], step // w_stages & 1, read)

    def multiply(now, step):
        if step == steps:
            return
        sa = step % a_stages

        def go(t):
            t2 = t + 64
            at(t2, a_empty[sa].arrive)
            at(t2, multiply, t2, step + 1)
        wait(now, a_full[sa], step // a_stages & 1, go)

    at(0, produce, 0, 0)
    for g in range(groups):
        at(0, convert, 0, g)
    at(0, multiply, 0, 0)
    n = 0
    while events and n < 400 * steps:      # a ring whose phases went wrong may never come to its end
        time, _, fn, args = heapq.heappop(events)
        fn(*args)
        n += 1
    return wrong


@pytest.mark.parametrize("tn", WIDTHS)
def test_no_group_reads_a_stage_ahead_of_its_load(tn):
    w, a, groups = constant("W_STAGES", tn), constant("A_STAGES", tn), constant("GROUPS", tn)
    rng = random.Random(tn)
    for _ in range(60):
        late = {rng.randrange(60): rng.choice([300, 1500, 6000]) for _ in range(rng.randint(1, 4))}
        assert run_ring(w, a, groups, 64, rng, late) == [], late


def test_the_model_finds_a_ring_that_groups_share():
    """Nine stages for four groups: a group waits for a phase whose predecessor another group waited for."""
    rng = random.Random(9)
    assert any(run_ring(9, 6, 4, 64, rng, {step: 1500}) for step in range(40))
