"""The streaming kernel's items are shared out so that a running CTA never waits for one that has not started, as
happens when another stream holds a part of the SMs (host form of csrc/gv_stream_schedule.h)."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    binary = str(tmp_path_factory.mktemp("schedule") / "probe")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-o", binary,
                    os.path.join(ROOT, "tests", "stream_schedule_probe.cpp")], check=True)
    return binary


@pytest.mark.parametrize("chunks", [1, 8, 27, 128, 148, 160, 256])
@pytest.mark.parametrize("ctas,running", [(148, 148), (148, 147), (148, 74), (148, 1), (132, 16), (1, 1)])
def test_no_wait_on_a_cta_that_is_not_running(probe, chunks, ctas, running):
    for seed in range(3):
        result = subprocess.run([probe, str(chunks), str(ctas), str(running), str(seed)], capture_output=True, text=True)
        assert result.stdout.strip() == "ok", (chunks, ctas, running, seed, result.stdout)


def test_claim_warp_gives_up_only_what_is_not_there(tmp_path):
    """A claim warp that gave up would leave w2 items out, which nobody waits for: it looks again before it does, and reports it."""
    binary = str(tmp_path / "probe")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-o", binary, os.path.join(ROOT, "tests", "stream_wait_probe.cpp")], check=True)
    assert subprocess.run([binary], capture_output=True, text=True).stdout.strip() == "ok"
    with open(os.path.join(ROOT, "gevva_b200", "csrc", "experts_stream.cu")) as f:
        text = f.read()
    claims = text[text.index("---------------- claims") : text.index("---------------- publisher")]
    assert "kWaitLimitCycles" not in claims  # its waits are that one


def test_counts_have_arrived_when_a_cta_ends():
    """The CTA that finishes last puts the counters back to zero, so whatever another one adds has to have arrived before that one ends: every
    addition is one whose answer is waited for, none is sent off without (`red`, or an atomic whose result nothing uses)."""
    with open(os.path.join(ROOT, "gevva_b200", "csrc", "experts_stream.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    assert not re.search(r"\bred\.", text)
    for line in text.splitlines():
        if re.search(r"atomic(Add|Exch)\((sync|p\.plan)", line):
            assert re.search(r"[=?+] *atomic", line), line


@pytest.mark.parametrize("ctas", [1, 2, 16, 115, 126, 132, 148, 256])
def test_shares_and_pool_hold_every_item_once(tmp_path, ctas):
    """Every number of chunks: both sides of the shortest share that gives items to the pool, and of the shares that begin with extra items."""
    binary = str(tmp_path / "probe")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-o", binary, os.path.join(ROOT, "tests", "stream_pool_probe.cpp")], check=True)
    for chunks in range(1, 257):
        result = subprocess.run([binary, str(chunks), str(ctas)], capture_output=True, text=True)
        assert result.stdout.strip() == "ok", (chunks, ctas, result.stdout)
