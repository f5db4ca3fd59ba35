"""What the down launches of csrc/grouped.cu and csrc/qmm_tcgen05.cu may read before their own wait for the previous launch.

They start while the gate/up launch of the same call still runs. A launch that has not waited is promised nothing about cached lines
of memory that earlier launches wrote, so the tables that it reads must come through EarlyTable (loads at GPU scope), and the
gate/up launch must let it start only after its own wait. Both are read off the sources: a race of this kind shows on no GPU
at will."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "turbo_fieldfare_b200" / "csrc"
KERNELS = [("grouped.cu", "GroupedArgs", {"sorted_pairs", "groups", "chunk_group", "chunk_start", "counters"}),
           ("qmm_tcgen05.cu", "QmmArgs", {"groups", "totals"})]


@pytest.mark.parametrize("source,struct,tables", KERNELS)
def test_tables_of_an_early_launch_are_read_past_the_l1_cache(source, struct, tables):
    text = (CSRC / source).read_text()
    members = re.search(rf"struct {struct} {{(.*?)\n}};", text, re.S).group(1)
    early = set(re.findall(r"EarlyTable<\w+> (\w+);", members))
    assert early == tables
    raw = set(re.findall(r"\* (\w+)(?:\[\d+\])?;", members))
    assert not raw & tables


def test_early_tables_are_loaded_at_gpu_scope_only():
    body = re.search(r"struct EarlyTable {(.*?)\n};", (CSRC / "tf_common.cuh").read_text(), re.S).group(1)
    loads = re.findall(r'asm volatile\("(\S+)', body)
    assert loads and all(op.startswith("ld.relaxed.gpu.global") for op in loads)


@pytest.mark.parametrize("source,struct,tables", KERNELS)
def test_down_launches_read_every_table_as_before_the_wait(source, struct, tables):
    text = (CSRC / source).read_text()
    reads = list(re.finditer(rf"\bargs\.(?:{'|'.join(tables)})\b\.(?:at|field)<([^>]*)>", text))
    assert len(reads) == len(re.findall(rf"\bargs\.(?:{'|'.join(tables)})\b", text))
    for r in reads:
        if r.group(1) == "false":                   # allowed in the warps of the down kernel that have waited, and nowhere else
            kernel = text[text.rindex("__global__", 0, r.start()):r.start()]
            assert "grouped_down_kernel" in kernel and "if (early) pdl_wait();           // the activations" in kernel
            assert "// loader:" not in kernel
        else:
            assert r.group(1) in ("NMAT == 1", "EARLY", "true")
    if source == "grouped.cu":
        assert "template <int NMAT, bool DENSE, int NT, bool EARLY = NMAT == 1>" in text
        loader = text[text.index("// loader: lane 0 moves a stage's codes"):]
        assert "std::false_type" not in loader[:loader.index("atomicCAS")]


@pytest.mark.parametrize("source,before,after", [
    ("grouped.cu", "if (NMAT == 2 && !DENSE) {", "} else {"),
    ("qmm_tcgen05.cu", "if (!early) pdl_wait();", "const uint32_t ngroups"),
])
def test_the_routed_gate_up_launch_waits_before_it_lets_the_down_launch_start(source, before, after):
    text = (CSRC / source).read_text()
    part = text[text.index(before):]
    part = part[:part.index(after)]
    assert 0 <= part.index("pdl_wait();") < part.index("pdl_launch_dependents();")
