"""Slots of shared memory that a copy refills: a consumer must hand one back only when what it has loaded from it is in its registers.

A plain arrival on the slot's barrier waits for no load, so it has to come behind instructions that used the values and cannot be moved (stores of
sums), or take values that depend on the loads (mbar_arrive_after). Read off the sources: a race of this kind shows on no GPU at will."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "turbo_fieldfare_b200" / "csrc"


def _arrivals(text, barrier):
    """The arrivals on a barrier by name: (function, arguments after the barrier)."""
    return re.findall(rf"\b(q_mbar_arrive|mbar_arrive|mbar_arrive_after)\({barrier}\([^()]*(?:\([^()]*\))?[^()]*\)(?:, ([^;]*))?\);", text)


# (source, part of it from, to, barrier, loaded registers that the arrivals must name)
RELEASES = [
    ("qmm_tcgen05.cu", "// ===================== dequantisers", "// ===================== epilogue", "bar_empty_raw", ["c[0]", "c[1]", "c[2]", "c[3]"]),
    ("grouped.cu", "// =========================== reducer warp q", "grouped_down_kernel", "bar_red_free", ["acc[0]", "acc[NMAT - 1]"]),
    ("grouped.cu", "grouped_down_kernel(const GroupedArgs args)", "// loader: lane 0 moves", "bar_empty", ["y[0]", "y[2]"]),
]


@pytest.mark.parametrize("source,begin,end,barrier,values", RELEASES)
def test_slots_are_released_after_the_loaded_values(source, begin, end, barrier, values):
    text = (CSRC / source).read_text()
    part = text[text.index(begin):]
    part = part[:part.index(end)]
    found = _arrivals(part, barrier)
    assert found and all(name == "mbar_arrive_after" for name, _ in found)
    for v in values:
        assert any(v in args for _, args in found)


# (source, from, barrier): plain arrivals right behind the stores of sums that need every load
@pytest.mark.parametrize("source,begin,end,barrier,store", [
    ("grouped.cu", "if constexpr (NT == 1) {\n            // All codes", "// the reducer's buffer is claimed first", "bar_empty", "sts_f32x2("),
    ("grouped.cu", "// the reducer's buffer is claimed first", "// =========================== loader warp", "bar_empty", "sts_f32x2("),
    ("decode_step.cu", "__device__ __forceinline__ void run_items(", "// B fragments and group sums", "ds_bar_empty", "partial[it * 16 + g] = acc0"),
])
def test_plain_arrivals_follow_the_stores_of_the_sums(source, begin, end, barrier, store):
    text = (CSRC / source).read_text()
    part = text[text.index(begin):]
    part = part[:part.index(end)]
    at = [m.start() for m in re.finditer(rf"\bmbar_arrive\({barrier}\(", part)]
    assert len(at) == 1 and 0 < part.index(store) < at[0]
    assert "__syncwarp();" in part[part.rindex(store, 0, at[0]):at[0]]


def test_a_dependent_arrival_takes_its_values():
    body = (CSRC / "async_copy.cuh").read_text()
    body = body[body.index("void mbar_arrive_after(uint32_t addr, uint32_t v) {"):]
    body = body[:body.index("\n}")]
    assert 'asm("mov.u32 %0, %%ctaid.z;" : "=r"(zero));' in body and "mbar_arrive(addr | (v & zero));" in body
    # the zero: launches of these kernels have one layer in z
    for source in ("grouped.cu", "qmm_tcgen05.cu"):
        text = (CSRC / source).read_text()
        for grid in re.findall(r"launch_pdl(?:_cluster)?\([^;]*?dim3\(((?:[^()]|\([^()]*\))*)\)", text):
            assert re.sub(r"\([^()]*\)", "", grid).count(",") <= 1


def test_one_token_kernels_wait_again_for_copies_in_flight():
    """A wait for a landing copy that runs out is recorded, and the copies under way get one more bounded wait before the block, and with it
    their destination, goes away."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "one_token.cu").read_text())
    first = [m for m in re.finditer(r"(?:!mbar_wait\(|= mbar_wait\()(bars? ?\+?[^,]*|bar), ", text) if "slots + slot" not in m.group(1)]
    assert len(first) == 4                            # front: tiles, router's codes; gate/up: tiles; down: both phases
    for m in first:
        after = text[m.end():]
        after = after[:after.index("__syncthreads();") if "__syncthreads();" in after else None]
        again = re.search(r"(?<![!= ]) mbar_wait\(|\n\s*mbar_wait\(|\) mbar_wait\(", after)
        assert again, text[m.start():m.start() + 80]
