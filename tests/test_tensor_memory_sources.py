"""A tensor-memory load writes its registers asynchronously: they may not be read, copied or spilled before the wait.  The kernels
state that to the compiler by handing every register in flight to the wait."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gevva_b200", "csrc")
LOAD = r"\b(?:tmem_load_\d+x\d+|wp_load_16x32)\("
SOURCES = sorted(p for pattern in ("*.cu", "*.cuh") for p in glob.glob(os.path.join(CSRC, pattern)) if re.search(LOAD + "|tcgen05.ld", open(p).read()))


def code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)


def arguments(text, start):
    """Of the call whose opening bracket ends at `start`."""
    depth, at, parts = 1, start, [""]
    while depth:
        c = text[at]
        depth += (c in "([{") - (c in ")]}")
        if c == "," and depth == 1:
            parts.append("")
        elif depth:
            parts[-1] += c
        at += 1
    return [p.strip() for p in parts]


def calls(text):
    """(position, 'load' or 'wait', register arrays) of the calls, definitions left out."""
    for m in re.finditer(LOAD + r"|\btmem_load_wait\(", text):
        if text[: m.start()].endswith("void "):
            continue
        wait = m[0].startswith("tmem_load_wait")
        args = arguments(text, m.end())
        yield m.start(), "wait" if wait else "load", [re.sub(r"\[\w\]$", "", a) for a in (args if wait else args[-1:])]


def test_sources_are_found():
    assert {"gv_common.cuh", "grouped_gemm_w13_pair.cu", "experts_stream.cu", "router_project.cu"} <= {os.path.basename(p) for p in SOURCES}


@pytest.mark.parametrize("source", [os.path.basename(p) for p in SOURCES])
def test_waits_take_the_registers_in_flight(source):
    in_flight = set()
    for _, kind, arrays in calls(code(os.path.join(CSRC, source))):
        if kind == "load":
            in_flight |= set(arrays)
        else:
            assert set(arrays) - {""} and in_flight <= set(arrays), (in_flight, arrays)
            in_flight = set()
    assert not in_flight


def test_the_wait_names_its_registers():
    text = code(os.path.join(CSRC, "gv_common.cuh"))
    bodies = re.findall(r"void tmem_load_wait\(([^{]*)\) \{(.*?)\n?\}\n", text, flags=re.S)
    assert len(bodies) >= 4
    for parameters, body in bodies:
        names = re.findall(r"\(&(\w+)\)", parameters)
        assert names and all(re.search(rf"GV_LOADED\d+\({name}\b", body) for name in names)
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        assert len(re.findall(r"tcgen05\.wait::ld", code(path))) == (os.path.basename(path) == "gv_common.cuh")


@pytest.mark.parametrize("source", [os.path.basename(p) for p in SOURCES])
def test_no_branch_between_a_load_and_its_wait(source):
    """A load that is branched over, with its wait behind the branch, would let the compiler merge old and new registers in between."""
    text = code(os.path.join(CSRC, source))
    assert not re.findall(r"\bif\s*(?:constexpr\s*)?\([^;{}]*\)\s*(?:load|tmem_load_\d+x\d+|wp_load_16x32)\(", text)


@pytest.mark.parametrize("source", [os.path.basename(p) for p in SOURCES if p.endswith(".cu")])
def test_warps_agree_before_they_load(source):
    """The loads are made by whole warps.  A wait that runs out may run out for some of its lanes: the warp votes, and goes on or leaves
    together."""
    text = code(os.path.join(CSRC, source))
    waits = [m.start() for m in re.finditer(r"wait_or_abort\(&smem->acc_full", text)]
    assert waits and all(text[:at].endswith("__all_sync(0xffffffffu, ") for at in waits)
