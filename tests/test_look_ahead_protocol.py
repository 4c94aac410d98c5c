"""Host checks of what the walker of the look-ahead sweep (csrc/sweep_ahead.cu) shares with the warps
beside it.

The walker publishes an entry per attempt; the look-ahead warp follows the entries of a block and clears
them once it has read the last one, at a time of its own.  So nothing that the walker decides may depend
on an entry it has published.

At an epoch's end the look-ahead warp publishes one word that says whether the roles go on.  Every wait for it
is bounded, and a role that goes on meets the others at barriers: so all roles have to take the same word,
also when one of them gives up waiting while the look-ahead warp is about to publish.  No GPU is involved."""
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


def test_visits_of_a_launch_fit_their_counter(tmp_path):
    exe = tmp_path / "shared_epochs_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I/usr/local/cuda/include",
                    str(ROOT / "tests" / "native" / "shared_epochs_check.cpp"), "-o", str(exe), "-L/usr/local/cuda/lib64",
                    "-lcudart"], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, env={"LD_LIBRARY_PATH": "/usr/local/cuda/lib64"})
    assert res.returncode == 0 and res.stdout == "ok\n", res.stdout
    engine = (ROOT / "replica_exchange_wang_landau_b200" / "csrc" / "engine.cpp").read_text()
    launch = engine[engine.index("void Engine::launch_epochs("):engine.index("void Engine::maybe_checkpoint(")]
    assert "std::min(count, most_shared_epochs(p_.exchange_interval))" in launch


def _epoch_end(replaces: bool, waiting: int = 2):
    """All outcomes of an epoch's end: `waiting` roles that look at the word at any time and give up at any
    later one, against the look-ahead warp that publishes "go on" at any time.  The word is 0 until then;
    with `replaces` it is replaced by compare-and-swap, else stored, and a role that gives up just leaves."""
    seen = set()

    def step(word, roles, ahead):
        if all(r in ("on", "left") for r in roles) and ahead in ("on", "left"):
            seen.add(tuple(sorted({*roles, ahead})))
            return
        if ahead == "before":
            if not replaces:
                step("on", roles, "on")
            else:
                step(word or "on", roles, "left" if word == "left" else "on")
        for i, r in enumerate(roles):
            if r != "waits":
                continue
            to = lambda x: roles[:i] + (x,) + roles[i + 1:]
            if word:
                step(word, to("on" if word == "on" else "left"), ahead)
            elif replaces:  # gives up: its word for all
                step("left", to("left"), ahead)
            else:
                step(word, to("left"), ahead)

    step("", ("waits",) * waiting, "before")
    return seen


def test_all_roles_take_the_same_word_at_an_epochs_end():
    assert _epoch_end(True) == {("on",), ("left",)}
    # the model is not vacuous: with a plain store one role leaves and the others wait for it at a barrier
    assert ("left", "on") in _epoch_end(False)


def test_the_word_is_replaced_by_compare_and_swap():
    body = re.sub(r"//[^\n]*", "", SOURCE)
    assert len(re.findall(r"atomicCAS\(word \+ kGo,", body)) == 2
    assert re.findall(r"st_(?:release|relaxed)\(word \+ kGo,", body) == []


def test_the_epochs_end_waits_for_the_walker():
    """A look-ahead warp that gives up is ahead of the walker: what the walker leaves for the epoch's end is
    initialised before the roles part, and read after the walker has said that it is complete."""
    body = SOURCE[SOURCE.index("__noinline__ uint32_t end_epoch("):SOURCE.index("template <int kPrec, bool kPow2, bool kAlone")]
    ended = body.index("wait_at_least(word + kEnded, epochs, nullptr)")
    assert ended < min(m.start() for m in re.finditer(r"io->", body))
    staging = SOURCE[SOURCE.index("// ---- stage the walker"):SOURCE.index("// ---- the walker ---")]
    assert "EpochIo first{};" in staging
    walker = SOURCE[SOURCE.index("// ---- the walker ---"):SOURCE.index("// ---- draws ---")]
    end = walker[walker.index("io->energy = E;"):]
    assert end.index("io->batch = batch;") < end.index("st_release(word + kEnded, epochs)") < end.index("kEntStop")


def _books_read(waits: str, ahead_delay: int, blocks: int = 12, per_block: int = 3) -> list:
    """Walker, look-ahead warp and books over `blocks` blocks of `per_block` entries in two buffers, the
    look-ahead warp `ahead_delay` steps behind in every block (its fields come late): the blocks whose entries
    the books have read for each block.  The walker ends its batch with the last block's last draw and then
    says that it has stopped.  `waits`: the books enter a block after the look-ahead warp has ("always"), or
    so unless the walker has stopped ("until stop"), or at once ("")."""
    entry = [[None] * per_block, [None] * per_block]
    walker = {"b": 0, "e": 0}
    ahead = {"b": 0, "late": ahead_delay}
    books = {"b": 0, "e": 0}
    handed, booked, read, stopped = 0, 0, [], False
    for _ in range(10000):
        if walker["b"] < blocks:
            if walker["e"] < per_block:
                entry[walker["b"] & 1][walker["e"]] = walker["b"]
                walker["e"] += 1
                stopped = walker == {"b": blocks - 1, "e": per_block}
            elif handed > walker["b"]:
                walker = {"b": walker["b"] + 1, "e": 0}
        if not waits or ahead["b"] >= books["b"] or (waits == "until stop" and stopped):
            x = entry[books["b"] & 1][books["e"]]
            if x is not None:
                read.append((books["b"], x))
                books["e"] += 1
                if books["e"] == per_block:
                    books = {"b": books["b"] + 1, "e": 0}
                    booked = books["b"]
            elif books["b"] == blocks and stopped:
                break  # the batch ended with the last block
        if ahead["b"] < blocks and entry[ahead["b"] & 1][-1] == ahead["b"]:
            if ahead["late"]:
                ahead["late"] -= 1
            elif ahead["b"] == 0 or booked >= ahead["b"]:
                if ahead["b"]:
                    entry[(ahead["b"] + 1) & 1] = [None] * per_block
                handed = ahead["b"] + 1
                ahead = {"b": ahead["b"] + 1, "late": ahead_delay}
    return read


def test_the_books_read_the_entries_of_their_own_block():
    for delay in range(12):
        read = _books_read("always", delay)
        assert len(read) == 36 and all(b == x for b, x in read), delay
    # the model is not vacuous: books that do not wait read the entries of two blocks before, and so do, at the
    # end of a batch that ends with a block, books that wait no longer once the walker has stopped
    assert any(b != x for b, x in _books_read("", 8))
    assert min(b for b, x in _books_read("until stop", 8) if b != x) == 12


def test_the_books_wait_for_the_look_ahead_warp():
    books = SOURCE[SOURCE.index("// ---- the books: pilot statistics"):]
    loop = books[books.index("for (uint32_t b = 0;;) {"):]
    assert loop.index("wait_at_least(word + kAheadIn, b, nullptr)") < loop.index("block->entry[e].x")
