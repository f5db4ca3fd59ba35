"""Host-side model of the two MMA issuers of qmm_tcgen05_kernel (csrc/qmm_tcgen05.cu, one CTA per tile) and its epilogue.

The stages of a CTA's tiles go to the issuers in turn. Each issuer accumulates its stages of a tile in an accumulator of its own
(two buffers, used in turn), commits it to the epilogue after its last one, and waits for the epilogue's release of the
buffer's previous tile before the first. A wait names only the parity of a barrier's phase. The model runs the roles under many
orders (an issuer that stands still while anything else can move among them) and checks that an issuer never multiplies
into a buffer that the epilogue has not emptied, that the epilogue reads only finished accumulators, and that nothing gets stuck."""
import random
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "turbo_fieldfare_b200" / "csrc" / "qmm_tcgen05.cu"


def _waits_only_with_a_stage():
    """Whether the source's issuers skip the wait for the accumulator of a tile that they have no stage of."""
    text = SOURCE.read_text()
    issuers = text[text.index("// ===================== MMA issuers"):text.index("// ===================== dequantisers")]
    return ("const bool takes_part = !kTwoIssuers || ksteps > 1 || (count & 1) == who;" in issuers and
            "if (takes_part && uacc > 0 && !q_mbar_wait(bar_acc_empty(buf)" in issuers)


class _Barrier:
    """Phases completed so far (one arrival each); passes(parity) as mbarrier.try_wait.parity."""

    def __init__(self):
        self.phases = 0

    def passes(self, parity):
        return (self.phases - 1) & 1 == parity


class _Cta:
    def __init__(self, ksteps, tiles, only_with_a_stage):
        self.ksteps, self.tiles, self.only_with_a_stage = ksteps, tiles, only_with_a_stage
        self.full = [[_Barrier(), _Barrier()] for _ in range(2)]           # [issuer][buffer]
        self.empty = [_Barrier(), _Barrier()]
        self.tile, self.waited = [0, 0], [False, False]
        self.read = 0                                                       # tiles that the epilogue has emptied
        self.wrong = False

    def stages(self, tile, who):
        return [c for c in range(tile * self.ksteps, (tile + 1) * self.ksteps) if c % 2 == who]

    def issue(self, who):
        tile = self.tile[who]
        if tile == self.tiles:
            return False
        buf, use, mine = tile % 2, tile // 2, self.stages(tile, who)
        if not self.waited[who]:
            skip = use == 0 or (self.only_with_a_stage and not mine)
            self.waited[who] = skip or self.empty[buf].passes((use - 1) & 1)
            return self.waited[who]
        if mine:
            self.wrong |= self.read < tile - 1                              # the buffer's previous tile is still being read
            self.full[who][buf].phases += 1
        self.tile[who], self.waited[who] = tile + 1, False
        return True

    def epilogue(self):
        tile = self.read
        if tile == self.tiles:
            return False
        buf, use = tile % 2, tile // 2
        who = [w for w in range(2) if self.stages(tile, w)]
        if not all(self.full[w][buf].passes(use & 1) for w in who):
            return False
        self.wrong |= any(self.tile[w] <= tile for w in who)
        self.empty[buf].phases += 1
        self.read += 1
        return True


def _runs(ksteps, tiles, only_with_a_stage, rng, slow):
    """Random interleaving; the roles in `slow` move only when nothing else can."""
    cta = _Cta(ksteps, tiles, only_with_a_stage)
    roles = [lambda: cta.issue(0), lambda: cta.issue(1), cta.epilogue]
    while cta.read < tiles:
        quick = [r for i, r in enumerate(roles) if i not in slow]
        rng.shuffle(quick)
        if not any(r() for r in quick) and not any(roles[i]() for i in slow):
            return False
        if cta.wrong:
            return False
    return True


def _holds(ksteps, only_with_a_stage):
    return all(_runs(ksteps, 12, only_with_a_stage, random.Random(seed), slow)
               for seed in range(40) for slow in ((), (0,), (1,), (2,), (0, 2), (1, 2)))


@pytest.mark.parametrize("ksteps", [1, 2, 3, 4, 11])
def test_issuers_keep_up_with_the_accumulators(ksteps):
    assert _holds(ksteps, _waits_only_with_a_stage())


@pytest.mark.parametrize("ksteps,only_with_a_stage,sound", [(1, False, False), (1, True, True), (2, False, True), (3, False, True)])
def test_the_model_tells_sound_issuers_from_others(ksteps, only_with_a_stage, sound):
    """With one stage per tile an idle issuer that waits all the same may miss a phase: the buffer is used again without it."""
    assert _holds(ksteps, only_with_a_stage) is sound
