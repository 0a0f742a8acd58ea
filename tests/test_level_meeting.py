"""The cluster sweep's meeting between levels, as a model on the CPU.

Between two levels every CTA arrives at a barrier of every CTA and waits at its
own until all have arrived.  Arrivals carry no sender and remote ones reach
different CTAs in any order.  The model walks through all orders of delivery
for three CTAs and looks for one in which a CTA leaves a level before
everybody's arrival for that level has reached it.  The number of barriers the
levels take in turn is read from the kernel's source.
"""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "monolish_b200", "csrc", "mlsh_sweep_cluster.cuh")


def leaves_early(barriers, ctas=3, levels=4):
    """Whether some order lets a CTA leave a level before all arrivals for it
    are there.  State: each CTA's level, each CTA's barriers as (arrivals of
    the phase, phases completed), and the arrivals under way."""
    everyone = range(ctas)

    def sent(level, cta):
        return frozenset((level, cta, to) for to in everyone)

    start = ((0,) * ctas, ((((0, 0),) * barriers),) * ctas,
             frozenset().union(*(sent(0, c) for c in everyone)))
    seen, todo = {start}, [start]
    while todo:
        at, bars, under_way = todo.pop()
        steps = []
        for m in under_way:  # an arrival reaches its CTA
            level, _, to = m
            b = level % barriers
            n, done = bars[to][b]
            n, done = (0, done + 1) if n + 1 == ctas else (n + 1, done)
            mine = bars[to][:b] + ((n, done),) + bars[to][b + 1:]
            steps.append((at, bars[:to] + (mine,) + bars[to + 1:], under_way - {m}))
        for c in everyone:  # a CTA finds its barrier's phase completed and goes on
            level = at[c]
            if level == levels:
                continue
            _, done = bars[c][level % barriers]
            if (done & 1) == ((level // barriers) & 1):
                continue  # the awaited phase is the current one
            if any(m[0] == level and m[2] == c for m in under_way):
                return True
            on = under_way | (sent(level + 1, c) if level + 1 < levels else frozenset())
            steps.append((at[:c] + (level + 1,) + at[c + 1:], bars, on))
        for s in steps:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return False


def kernel_barriers():
    with open(SOURCE) as f:
        m = re.search(r"uint64_t level_bar(?:\[(\d+)\])?;", f.read())
    return int(m.group(1) or 1)


@pytest.mark.parametrize("levels", [2, 3, 4])
def test_nobody_leaves_early(levels):
    assert not leaves_early(kernel_barriers(), levels=levels)


def test_one_barrier_would_not_do():
    """An arrival for the next level takes the place of a late one."""
    assert leaves_early(1)
