"""The barriers of a team of CTAs (csrc/fit_kernel.cuh) when a bulk-copy wait gives
up in some of its CTAs, as a model: each CTA is a generator that yields at
every cluster barrier, and the team hangs as soon as one CTA waits at a
barrier that another does not reach.  After a lost copy a CTA's chi^2, and so
its decisions, may be its own.  With the flag told to all CTAs before the
barrier that ends the sweep, they leave the fit together before its next
iteration, its result is marked and the team takes no further item; left to
the CTA that met it, the team can hang."""
import random

import pytest

ITEMS, MAX_ITER = 6, 8


class Team:
    def __init__(self, size, told, seed, p_lost):
        self.rng = random.Random(seed)
        self.size, self.told, self.p_lost = size, told, p_lost
        self.flag = [False] * size      # each CTA's C_TIMEOUT
        self.lost = set()               # items in which some CTA lost a copy
        self.marked, self.finished = set(), set()
        self.next_item = 0

    def decision(self, rank, what):
        """Alike in all CTAs while none of them lost a copy."""
        common = random.Random(repr(what)).random()
        return random.Random(repr((what, rank))).random() if self.flag[rank] else common

    def sweep(self, rank, item):
        if self.rng.random() < self.p_lost:
            self.lost.add(item)
            for r in range(self.size) if self.told else [rank]:
                self.flag[r] = True

    def cta(self, rank):
        while True:
            yield "slab free"
            if rank == 0:
                # told: the first CTA's flag is the team's; untold: the flags are
                # gathered here, between items
                stop = self.flag[0] if self.told else any(self.flag)
                self.item = ITEMS if stop else self.next_item
                self.next_item += 1
            yield "item handed on"
            item = self.item
            yield "item read"
            if item >= ITEMS:
                return
            moved = first = True
            for it in range(MAX_ITER):
                if self.told and self.flag[rank]:
                    break
                if moved:
                    for k in range(3 if first else 1):  # set-up of an evaluation; after a trial its own
                        yield "evaluation set-up"
                    first = False
                    self.sweep(rank, item)
                    yield "rows swept"
                    yield "curve sums"
                    yield "normal matrix"
                for k in range(3):
                    yield "trial set-up"
                yield "trial swept"
                moved = self.decision(rank, (item, it, "accept")) < 0.5
                if self.decision(rank, (item, it, "done")) < 0.1:
                    break
            if rank == 0:
                self.finished.add(item)
                if self.flag[0]:
                    self.marked.add(item)

    def run(self):
        """True if every CTA ends; False if some wait where others do not come."""
        ctas = [self.cta(r) for r in range(self.size)]
        while True:
            at = [next(c, None) for c in ctas]
            if all(a is None for a in at):
                return True
            if len(set(at)) > 1:
                return False


@pytest.mark.parametrize("size", [2, 4, 8])
def test_team_leaves_a_fit_together(size):
    for seed in range(400):
        t = Team(size, True, seed, 0.02)
        assert t.run()
        assert t.marked == t.lost and len(t.lost) <= 1
        assert t.finished == set(range(max(t.finished) + 1))


def test_model_shows_the_hang_and_the_unmarked_fit():
    runs = [(t, t.run()) for t in (Team(4, False, seed, 0.02) for seed in range(400))]
    assert any(not ended for _, ended in runs)
    assert any(t.lost - t.marked for t, _ in runs)
