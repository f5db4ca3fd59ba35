"""Host-side model of the shared-memory ring of grouped_down_kernel (csrc/grouped.cu), with the kernel's own constants.

Warp w takes the items w, w + warps, ...; a ring stage holds `sub` consecutive items, and one loader refills the slots in
turn. A wait names only the parity of a barrier's phase, so it also returns while the barrier is a whole phase behind the
awaited one. The model runs the ring under many orders of copies and warps (copies that land as late as they can among them)
and checks that a warp only ever computes on the stage that it waited for, and that the ring never gets stuck."""
import random
import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "turbo_fieldfare_b200" / "csrc" / "grouped.cu"


def _kernel_ring():
    """(warps, items per stage, slots, whether a warp waits for its slot's previous release) as the source has them."""
    text = SOURCE.read_text()
    numbers = [int(re.search(rf"constexpr int {name} = (\d+);", text).group(1)) for name in ("kDownWarps", "kDownSub", "kDownStages")]
    consumer = text[text.index("grouped_down_kernel(const GroupedArgs args)"):].split("// loader:")[0]
    return (*numbers, "mbar_wait_both(bar_empty(st), (use - 1) & 1, bar_full(st), use & 1)" in consumer)


class _Barrier:
    """Phases completed so far; wait(parity) returns true when the phase before the current one has that parity."""

    def __init__(self, count):
        self.count, self.arrived, self.phases = count, 0, 0

    def arrive(self):
        self.arrived += 1
        if self.arrived == self.count:
            self.arrived, self.phases = 0, self.phases + 1

    def passes(self, parity):
        return (self.phases - 1) & 1 == parity


class _Ring:
    def __init__(self, warps, sub, slots, after_release, stages):
        self.warps, self.sub, self.slots, self.after_release, self.stages = warps, sub, slots, after_release, stages
        self.full = [_Barrier(1) for _ in range(slots)]
        self.empty = [_Barrier(sub) for _ in range(slots)]
        self.issued, self.landed = 0, set()
        self.next_item = list(range(warps))
        self.released = [not after_release] * warps         # the first of a warp's two waits for its item has returned
        self.wrong = []                         # (warp, stage) computed on other bytes than the stage's

    def load(self):
        slot, use = self.issued % self.slots, self.issued // self.slots
        if self.issued == self.stages or (use > 0 and not self.empty[slot].passes((use - 1) & 1)):
            return False
        self.issued += 1
        return True

    def land(self, stage):
        if stage >= self.issued or stage in self.landed:
            return False
        self.landed.add(stage)
        self.full[stage % self.slots].arrive()
        return True

    def work(self, warp):
        item = self.next_item[warp]
        stage = item // self.sub
        if stage >= self.stages:
            return False
        slot, use = stage % self.slots, stage // self.slots
        if not self.released[warp]:
            self.released[warp] = self.empty[slot].passes((use - 1) & 1)
            return self.released[warp]
        if not self.full[slot].passes(use & 1):
            return False
        if stage not in self.landed:
            self.wrong.append((warp, stage))
        self.next_item[warp] += self.warps
        self.released[warp] = not self.after_release
        self.empty[slot].arrive()
        return True

    def done(self):
        return all(item // self.sub >= self.stages for item in self.next_item)


def _run(ring, rng, late):
    """Random interleaving; the copies of `late` stages land only when nothing else can move."""
    while not ring.done() and not ring.wrong:
        moves = [ring.load] + [lambda w=w: ring.work(w) for w in range(ring.warps)]
        moves += [lambda s=s: ring.land(s) for s in range(max(0, ring.issued - 2 * ring.slots), ring.issued) if s not in late]
        rng.shuffle(moves)
        if not any(move() for move in moves) and not any(ring.land(s) for s in sorted(late)):
            return False                        # stuck
    return not ring.wrong


def _holds(warps, sub, slots, after_release):
    stages = 4 * warps * slots // sub
    for seed in range(8):
        rng = random.Random(seed)
        lates = [set(), set(rng.sample(range(stages), stages // 5))] + [{s} for s in range(0, stages, 1 + seed)]
        if not all(_run(_Ring(warps, sub, slots, after_release, stages), rng, late) for late in lates):
            return False
    return True


def test_down_ring_computes_on_the_stage_that_it_waited_for():
    assert _holds(*_kernel_ring())


@pytest.mark.parametrize("warps,slots,after_release,sound", [(11, 7, False, False), (11, 9, False, False), (12, 7, False, False),
                                                             (12, 9, False, True), (11, 7, True, True), (11, 3, True, True)])
def test_the_model_tells_sound_rings_from_others(warps, slots, after_release, sound):
    """Four items a stage. Sound are rings in which the same warps see every use of a slot (slots a multiple of warps / 4), and
    those whose warps wait for the release of the slot's previous use first."""
    assert _holds(warps, 4, slots, after_release) is sound
