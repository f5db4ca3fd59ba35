"""Loads of what earlier kernels write, in kernels that wait for those kernels themselves (griddepcontrol.wait, or a flag of a peer).

A load through a `const __restrict__` parameter of a kernel, and an `__ldg`, count as invariant: the compiler may move them ahead of the wait. So only
weights, scales and other planes that no such kernel writes may be spelled so. Read off the sources: the order that a compiler happens to choose
shows in no result until it changes."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "turbo_fieldfare_b200" / "csrc"
# Parameters that no kernel of a chain writes: packed codes, scales, biases, norm weights, a router's scales and biases.
STATIC = {"W", "S", "B", "w", "eff", "per_expert_scale", "logit_bias"}
# What an __ldg may be given: those, and pointers taken from them.
STATIC_LOADS = {"w", "gs", "gb", "a.norm_w", "a.eff", "eff", "per_expert_scale", "S", "B", "Wrow", "s_row", "b_row", "wl", "sr", "br", "sp"}
FILES = sorted(p for p in list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")))


def _kernels():
    for path in FILES:
        text = re.sub(r"//[^\n]*", "", path.read_text())
        starts = [m.start() for m in re.finditer(r"__global__ ", text)]
        for begin, end in zip(starts, starts[1:] + [len(text)]):
            part = text[begin:end]
            end_of_body = re.search(r"\n}", part).end()
            name = re.search(r"(\w+_kernel)\(", part).group(1)
            yield path.name, name, part[:end_of_body]


WAITING = [(f, n, body) for f, n, body in _kernels() if "pdl_wait()" in body or "peer_wait_in_block(" in body]


def test_the_waiting_kernels_are_found():
    names = {n for _, n, _ in WAITING}
    assert {"router_approx_kernel", "router_approx_few_kernel", "router_recheck_kernel", "router_split_kernel", "router_rows_kernel", "grouped_ksplit_kernel",
            "grouped_down_kernel", "ep_pack_kernel", "ep_combine_kernel", "qmm_prepare_kernel", "combine_rows_pipelined_kernel", "gemv_stream_kernel",
            "one_token_front_kernel"} <= names


@pytest.mark.parametrize("source,name,body", WAITING, ids=[n for _, n, _ in WAITING])
def test_parameters_that_are_read_behind_a_wait_are_plain_pointers(source, name, body):
    params = body[:body.index(") {")]
    invariant = set(re.findall(r"const \w+\*(?: const\*)? __restrict__ (\w+)", params))
    assert invariant <= STATIC, f"{source}: {name}"
    # read and written in place: also through a plain pointer
    for kind, p in re.findall(r"[(,]\s*((?:\w+ )*\w+)\* __restrict__ (\w+)", params):
        if not kind.startswith("const "):
            assert not re.search(rf"\*reinterpret_cast<const \w+\*>\({p}\b|= {p}\[|= \*{p};", body), f"{source}: {name} reads {p}"


def test_invariant_loads_are_of_static_planes():
    for path in FILES:
        if path.name in ("decode_step.cu", "rowdot.cuh"):        # no such waits: grid barriers (its hidden row comes by __ldcg), whole launches
            continue
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__ldg\((?:reinterpret_cast<const \w+\*>\()?\(?([\w.]+)", text):
            assert m.group(1) in STATIC_LOADS, f"{path.name}: __ldg({m.group(1)}"
