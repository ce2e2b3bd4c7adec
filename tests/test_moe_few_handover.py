"""The hand-over of table blocks and values inside the expert kernels for a handful of pairs (csrc/moe_few.cuh, few_sums), as a model
on the CPU: barriers that are waited for by phase parity, warps scheduled at random, table blocks that land late and out of order.
Every row's sum must be made of every block's values once, in order, and every wait must end."""
import random
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "ojasx-vector-24x96_b200" / "csrc" / "moe_few.cuh").read_text()
SLOTS = int(re.search(r"constexpr int kFewSlots = (\d+);", SOURCE)[1])
WARPS = int(re.search(r"constexpr int kFewThreads = (\d+);", SOURCE)[1]) // 32


def gatherers(nrb):
    return min(WARPS - nrb, SLOTS * 2 * nrb)


class Barrier:
    def __init__(self, count):
        self.count, self.left, self.phases = count, count, 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phases = self.count, self.phases + 1

    def done(self, parity):
        return (self.phases & 1) != parity


def hand_over(rng, nrb, blocks, nblk, ng, slot_first=True):
    """False: a wrong value, or warps that wait for one another for ever.  blocks = 0: the table lies there whole."""
    upb = 2 * nrb
    full, empty = [Barrier(1) for _ in range(blocks)], [Barrier(upb) for _ in range(blocks)]
    vfull, vempty = [Barrier(upb) for _ in range(SLOTS)], [Barrier(nrb) for _ in range(SLOTS)]
    table, slots, flying = [None] * blocks, [[None] * upb for _ in range(SLOTS)], []
    wrong = []

    def bring():
        for b in range(nblk):
            if b >= blocks:
                while not empty[b % blocks].done((b // blocks - 1) & 1):
                    yield False
            flying.append(b)
            yield True

    def land():
        while True:
            if flying:
                b = flying.pop(rng.randrange(len(flying)))
                table[b % blocks] = b
                full[b % blocks].arrive()
                yield True
            else:
                yield False

    def gather(w):
        for u in range(w, nblk * upb, ng):
            b, r = divmod(u, upb)
            for what in ("slot", "table") if slot_first else ("table", "slot"):
                if what == "slot" and b >= SLOTS:
                    while not vempty[b % SLOTS].done((b // SLOTS - 1) & 1):
                        yield False
                if what == "table" and blocks:
                    while not full[b % blocks].done((b // blocks) & 1):
                        yield False
            yield True
            if blocks and table[b % blocks] != b:
                wrong.append(("table", b))
            slots[b % SLOTS][r] = b
            yield True
            if blocks:
                empty[b % blocks].arrive()
            vfull[b % SLOTS].arrive()
            yield True

    def add(rb):
        for b in range(nblk):
            while not vfull[b % SLOTS].done((b // SLOTS) & 1):
                yield False
            yield True
            if slots[b % SLOTS][2 * rb:2 * rb + 2] != [b, b]:
                wrong.append(("slot", b))
            vempty[b % SLOTS].arrive()
            yield True

    live = [add(rb) for rb in range(nrb)] + [gather(w) for w in range(ng)] + ([bring()] if blocks else [])
    landing = land() if blocks else None
    speed = {id(g): rng.choice((1, 1, 1, 20)) for g in live}      # some warps fall far behind
    idle = 0
    while live and not wrong and idle < 200:     # 200 rounds without a step: 1 in 20 warps is asked in a round at the least
        idle += 1
        for g in rng.sample(live, len(live)):
            if rng.randrange(speed[id(g)]):
                continue
            try:
                if next(g):
                    idle = 0
            except StopIteration:
                live.remove(g)
                idle = 0
        if landing and rng.random() < 0.5 and next(landing):
            idle = 0
    return not live and not wrong


@pytest.mark.parametrize("nrb", range(1, 9))
def test_every_wait_is_one_phase_behind_at_most(nrb):
    rng = random.Random(nrb)
    for blocks in (0, 4, 5, 7, 12):
        for nblk in (1, 4, 5, 9, 20, 33):
            for _ in range(4 if nrb > 2 else 12):
                assert hand_over(rng, nrb, min(blocks, nblk), nblk, gatherers(nrb)), (nrb, blocks, nblk)


def test_the_model_sees_waits_that_are_two_phases_behind():
    rng = random.Random(0)
    assert not all(hand_over(rng, 1, 12, 20, WARPS - 1) for _ in range(40))      # fifteen warps for one block of rows


def test_the_kernel_has_the_bound():
    body = re.search(r"constexpr int few_gatherers\(int nrb\) \{\s*return (.*?);", SOURCE)[1]
    for nrb in range(1, 9):
        text = body.replace("kFewThreads", str(32 * WARPS)).replace("kFewSlots", str(SLOTS)).replace("nrb", str(nrb)).replace("/", "//")
        cond, a, b = re.match(r"(.*?) \? (.*?) : (.*)", text).groups()
        assert (eval(a) if eval(cond) else eval(b)) == gatherers(nrb)
