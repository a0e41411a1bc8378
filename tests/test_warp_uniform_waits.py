"""Waits of the kernels, read from their text: what goes wrong around them cannot be shown by running it.

A barrier's phase may complete between the probes of two lanes, and another warp may raise a block's abort flag between two lanes'
reads.  A branch on such a probe may therefore split the warp, and a vote, a shuffle, an MMA or a tensor-memory load behind it waits for
all lanes without a limit.  So a condition that probes a barrier or reads the flag goes through a vote (warp_wait, __all_sync,
__any_sync) wherever what it guards, or what it chooses instead, is warp-wide work, unless a single lane runs it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cut_b200", "csrc")
VOTES = re.compile(r"\b(__all_sync|__any_sync|warp_wait)\s*\(")
PER_LANE = re.compile(r"\bmbar_(test|try_wait|wait_\w+|spin_\w+)\s*\(|\baborted\(\)")
WARP_WIDE = re.compile(r"_sync\(\s*0x|\b__syncwarp\b|\bwarp_wait\b|sync\.aligned|\btmem_(ld|st)|\bgr_mma\b|\b(break|return|continue)\b")
ONE_LANE = re.compile(r"\blane == 0\b|\bleader\b|\btid == 0\b")


def _match(text, at, left, right):
    """Index behind the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == left) - (text[i] == right)
        if depth == 0:
            return i + 1
    raise ValueError("unbalanced")


def _without_comments(text):
    text = re.sub(r"/\*.*?\*/", " ", text, flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _statement(text, at):
    """End of the statement that starts at or behind `at`."""
    at += len(text[at:]) - len(text[at:].lstrip())
    if text[at] == "{":
        return _match(text, at, "{", "}")
    m = re.match(r"(if|for|while)\s*(constexpr\s*)?\(", text[at:])
    if m:
        end = _statement(text, _match(text, at + m.end() - 1, "(", ")"))
        other = re.match(r"\s*else\b", text[end:])
        return _statement(text, end + other.end()) if m.group(1) == "if" and other else end
    return text.index(";", at) + 1


def _ifs(text):
    for m in re.finditer(r"\bif\s*\(", text):
        end = _match(text, m.end() - 1, "(", ")")
        yield text[m.end(): end - 1], end, _statement(text, m.start())  # (with its else)


def _unvoted(cond):
    while m := VOTES.search(cond):
        cond = cond[: m.start()] + cond[_match(cond, m.end() - 1, "(", ")"):]
    return cond


def split_warps(text):
    """Conditions that lanes decide for themselves in front of warp-wide work."""
    text, found = _without_comments(text), []
    every = list(_ifs(text))
    for cond, start, end in every:
        if not PER_LANE.search(_unvoted(cond)):
            continue
        alone = any(ONE_LANE.search(c) for c, s, e in every if s <= start and end <= e)
        if not alone and WARP_WIDE.search(text[start: end]):
            found.append(cond)
    return found


KERNELS = sorted(p for p in glob.glob(os.path.join(CSRC, "*.cu*")) if os.path.basename(p) != "common.cuh")  # (which defines the waits)


@pytest.mark.parametrize("path", KERNELS, ids=os.path.basename)
def test_no_lane_waits_alone_before_warp_wide_work(path):
    with open(path) as f:
        assert split_warps(f.read()) == []


def split_loads(text):
    """Loops that some lanes go round ahead of the others, into a tensor-memory load that wants the whole warp."""
    text, found = _without_comments(text), []
    for m in re.finditer(r"\bfor\s*\(", text):
        start = _match(text, m.end() - 1, "(", ")")
        body = text[start: _statement(text, start)]
        load = re.search(r"\btmem_ld\w*\(", body)
        inner = any(re.search(r"\btmem_ld\w*\(", body[f.end():]) for f in re.finditer(r"\bfor\s*\(", body[: load.start()])) if load else False
        if load and not inner and re.search(r"\bcontinue;", body[load.end():]) and "__syncwarp()" not in body[: load.start()]:
            found.append(text[m.start(): start])
    return found


@pytest.mark.parametrize("path", KERNELS, ids=os.path.basename)
def test_a_warp_meets_before_it_loads_tensor_memory(path):
    with open(path) as f:
        assert split_loads(f.read()) == []


@pytest.mark.parametrize("path", KERNELS, ids=os.path.basename)
def test_copies_in_flight_are_waited_for_whoever_gives_up_and_when(path):
    """A copy warp that has issued everything may end before another warp gives up: its wait for copies does not hang on the flag."""
    with open(path) as f:
        text = _without_comments(f.read())
    assert [c for c, start, end in _ifs(text) if "aborted()" in c and ("mbar_drain" in text[start: end] or "mbar_wait_bounded" in text[start: end]) and "tmem_ld" not in text[start: end]] == []


def test_the_reading_finds_what_it_is_for():
    assert split_warps("if (!mbar_test(b, p)) { if (!__all_sync(0xffffffffu, mbar_wait_bounded(b, p))) dead = true; }")
    assert split_warps("if (!dead && !mbar_wait_probe_first(b, p)) break;")
    assert split_warps("if (dead || aborted()) { dead = true; break; }")
    assert split_warps("if (!mbar_wait_bounded(b, 0)) { give_up(); } else { tmem_ld32(t, v); }")
    assert not split_warps("if (!__all_sync(0xffffffffu, !aborted() && mbar_wait_bounded(b, 0))) give_up(); else tmem_ld32(t, v);")
    assert not split_warps("if (!dead && !warp_wait(b, p)) { dead = true; break; }")
    assert not split_warps("if (lane == 0) { if (!mbar_spin_bounded(b, p)) break; }")
    assert not split_warps("if (!dead && !mbar_spin_bounded(b, p)) { give_up(); dead = true; }")


def test_shuffles_name_their_lanes():
    """The lanes of a shuffle or a vote are stated: which of them happen to be together is the compiler's choice."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            assert "__activemask" not in _without_comments(f.read()), path
