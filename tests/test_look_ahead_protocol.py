"""Host checks of what the walker of the look-ahead sweep (csrc/sweep_ahead.cu) shares with the warps
beside it.

The walker publishes an entry per attempt; the look-ahead warp follows the entries of a block and clears
them once it has read the last one, at a time of its own.  So nothing that the walker decides may depend
on an entry it has published.  No GPU is involved."""
from __future__ import annotations

import itertools
import re
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
SOURCE = (ROOT / "replica_exchange_wang_landau_b200" / "csrc" / "sweep_ahead.cu").read_text()


def _walker_loop() -> str:
    return SOURCE[SOURCE.index("auto run = [&](auto it_tag"):SOURCE.index("auto run_stage")]


def _interleavings(a: list, b: list):
    """Every order of the steps of two warps, each in its own order."""
    for places in itertools.combinations(range(len(a) + len(b)), len(a)):
        ia, ib = iter(a), iter(b)
        yield [next(ia) if k in places else next(ib) for k in range(len(a) + len(b))]


def _opened(reads_entry: bool, accepted: bool, stays: bool) -> set:
    """Bins counted by the first attempt of an epoch that starts in an unvisited bin and whose attempt is
    the block's last: all answers over the orders of the walker's and the look-ahead's steps."""
    answers = set()
    for order in _interleavings(["publish", "count"], ["follow", "clear"]):
        if order.index("follow") < order.index("publish"):
            continue  # it waits for the entry
        entry, counted = 0, 0
        for step in order:
            if step == "publish":
                entry = 1 | (0x40000000 if accepted else 0)
                counted = 1 if accepted else 0  # an accepted flip finds its bin unvisited and counts it
            elif step == "clear":
                entry = 0
            elif step == "count":
                rejected = not entry & 0x40000000 if reads_entry else stays and counted == 0
                counted += 1 if rejected else 0
        answers.add(counted)
    return answers


def test_the_count_of_the_starting_bin_does_not_depend_on_the_other_warp():
    for accepted, stays in ((False, True), (True, True), (True, False)):
        assert _opened(False, accepted, stays) == {1}
    # the model is not vacuous: the cleared entry of an accepted attempt reads as one of a rejected attempt
    assert _opened(True, True, False) == {1, 2}


def test_the_walker_reads_no_entry_it_has_published():
    body = re.sub(r"//[^\n]*", "", _walker_loop())
    assert "opened_by_staying(" in body
    assert re.findall(r"\be_(?:mark|p)\s*\[|\*\s*e_(?:mark|p)\b", body) == []


def test_opened_by_staying(tmp_path):
    exe = tmp_path / "opened_bin_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-I/usr/local/cuda/include",
                    str(ROOT / "tests" / "native" / "opened_bin_check.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.startswith("ok"), res.stdout
