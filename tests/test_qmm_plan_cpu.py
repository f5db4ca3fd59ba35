"""How qmm_tcgen05_kernel (csrc/qmm_tcgen05.cu) divides its shared memory, for every width, form and tile size that a launch can take.

The arithmetic of qmm_plan, qmm_most_wide and the kernel's own split of the activation ring, with the constants of the source: every
ring has the slots that its roles rely on, nothing overlaps, and slots start on the 1024 bytes that the swizzle needs."""
import re
from pathlib import Path

import pytest

TEXT = (Path(__file__).resolve().parent.parent / "turbo_fieldfare_b200" / "csrc" / "qmm_tcgen05.cu").read_text()


def _const(name):
    return int(re.search(rf"constexpr (?:int|uint32_t) {name} = (\d+)", TEXT).group(1))


ROWS, BOX, STAGE_K, MAX_K, RAW_MAX = (_const(n) for n in ("kQmmRows", "kQmmBoxMax", "kQmmStageK", "kQmmMaxK", "kQmmRawMax"))
STAGING, TABLE, BARRIERS = _const("kQmmStageBytes"), 256 * 16, 1024
RAW, ROW = ROWS * STAGE_K // 2, STAGE_K * 2


def _plan(k, nmat):
    budget, groups = 227 * 1024 - 1024, k // 64
    plane = (ROWS // nmat * groups * 2 + 15) & ~15
    planes = nmat * 2 * plane
    for bufs in ((4,) if 4 * planes <= 48 * 1024 else (2,)) + (1,):
        fixed = bufs * planes + STAGING + TABLE + BARRIERS
        raws = [r for r in range(RAW_MAX, 1, -2) if fixed + r * RAW + 2 * BOX * ROW <= budget]
        if raws:
            return raws[0], (budget - fixed - raws[0] * RAW) & ~2047, bufs * planes
    return None


def test_the_source_computes_what_this_file_does():
    for line in ("const uint32_t raw_stages = !PAIR && plan.b_bytes < (kTwoIssuers ? 4 : 3) * b_slot ? 2u : plan.raw_stages;",
                 "const uint32_t b_fit = kTwoIssuers ? b_bytes / b_slot & ~1u : b_bytes / b_slot;",
                 "const uint32_t b_slot = n_top / kCtas * kQmmRowBytes;",
                 "const uint32_t fit = (p.off_b + p.b_bytes - 2 * kQmmRawBytes) / (2 * kQmmRowBytes) & ~15u;",
                 "p->total = p->off_bars + 1024u + 1024u;"):
        assert line in TEXT


@pytest.mark.parametrize("nmat", [1, 2])
def test_rings_of_every_form_fit(nmat):
    for k in range(64, MAX_K + 1, 64):
        raw, b_bytes, planes = _plan(k, nmat)
        assert raw * RAW + b_bytes + planes + STAGING + TABLE + 2048 <= 227 * 1024
        most_wide = min(128, (raw * RAW + b_bytes - 2 * RAW) // (2 * ROW) & ~15)
        forms = [("few", n) for n in range(16, BOX + 1, 16)] + [("pair", n) for n in range(32, 2 * BOX + 1, 32)]
        forms += [("wide", n) for n in range(BOX + 16, most_wide + 1, 16)]
        for form, n in forms:                           # n: the launch's largest tile
            slot = n // (2 if form == "pair" else 1) * ROW
            stages = 2 if form != "pair" and b_bytes < {"few": 4, "wide": 3}[form] * slot else raw
            ring = raw * RAW + b_bytes - stages * RAW
            slots = ring // slot & (~1 if form == "few" else ~0)
            assert slots >= 2 and stages >= 2 and stages % 2 == 0
            assert slot % 1024 == 0 and stages * RAW % 1024 == 0
            assert stages * RAW + slots * slot <= raw * RAW + b_bytes
