"""Rules of the kernels that are checked on their sources, since what breaks them (a full-mask vote or an ``.aligned``
instruction that some lanes of a warp do not execute, a read that races with the kernel before) cannot be provoked safely
or surely on a GPU."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "csrc"
SOURCES = sorted(list((CSRC / "kernels").rglob("*.cu")) + list((CSRC / "kernels").rglob("*.cuh")))
# every wait on an mbarrier whose answer is a lane's own
LANE_WAIT = re.compile(r"\b(\w*mbar_try\w*|mbar_wait_bounded|mbar_wait_quick|mbar_wait_g)\s*\(")
WARP_WIDE = re.compile(r"\b__(all|any|ballot|shfl\w*|match\w*|reduce\w*)_sync\s*\(|\b__syncwarp\s*\(|\.aligned")


def _code(path):
    """The source without comments, positions kept."""
    blank = lambda m: re.sub(r"[^\n]", " ", m.group(0))
    return re.sub(r"//[^\n]*|/\*.*?\*/", blank, path.read_text(), flags=re.S)


def _close(s, i, pair):
    """Position after the bracket that closes the one at s[i]."""
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == pair[0]) - (s[j] == pair[1])
        if depth == 0:
            return j + 1
    raise AssertionError("unbalanced")


def _branches(s):
    """(condition, body, line) of every if / while / for."""
    for m in re.finditer(r"\b(if|while|for)\s*\(", s):
        end = _close(s, m.end() - 1, "()")
        b = re.compile(r"\s*").match(s, end).end()
        body = s[b:_close(s, b, "{}")] if s[b] == "{" else s[b:s.index(";", b) + 1]
        yield s[m.end():end - 1], body, s.count("\n", 0, m.start()) + 1


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_warp_wide_instruction_under_a_lanes_own_wait(path):
    """A branch on a lane's own wait, taken by some lanes and not by others, holds nothing that all lanes have to execute."""
    bad = [(line, cond.strip()) for cond, body, line in _branches(_code(path))
           if LANE_WAIT.search(re.sub(r"__all_sync\s*\([^;]*", "", cond)) and WARP_WIDE.search(body)]
    assert not bad, bad


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_waits_of_whole_warps_are_voted(path):
    """Lanes may leave a wait at different tries, so outside the wait helpers a wait is either voted or run by one lane:
    the mma and tcgen05 instructions behind it are .aligned."""
    s = _code(path)
    alone = [(s.index(body), s.index(body) + len(body)) for cond, body, _ in _branches(s) if "lane == 0" in cond]
    helpers = [(m.start(), _close(s, m.end() - 1, "{}")) for m in re.finditer(r"\bbool\s+\w*(mbar|pf)_\w+\([^)]*\)\s*\{", s)]
    bad = [s.count("\n", 0, m.start()) + 1 for m in LANE_WAIT.finditer(s) if not any(a <= m.start() < b for a, b in alone + helpers)]
    assert not bad, bad


@pytest.mark.parametrize("path", [p for p in SOURCES if "barrier.cluster" in p.read_text()], ids=lambda p: p.name)
def test_cluster_barriers_are_reached_by_whole_warps(path):
    """barrier.cluster...aligned is executed by helpers that bring the warp together first."""
    s = _code(path)
    for m in re.finditer(r"barrier\.cluster\.arrive[\w.]*\.aligned", s):
        assert "__syncwarp" in s[s.rindex("__device__", 0, m.start()):m.start()]


def _loops(s):
    """(body, line) of every for loop."""
    for m in re.finditer(r"\bfor\s*\(", s):
        b = re.compile(r"\s*").match(s, _close(s, m.end() - 1, "()")).end()
        if s[b] == "{":
            yield s[b:_close(s, b, "{}")], s.count("\n", 0, m.start()) + 1


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_loops_over_tensor_memory_bring_the_warp_together(path):
    """A loop that reads TMEM (tcgen05.ld is .aligned) and writes results with the lanes on their own also has a
    __syncwarp, so that every turn starts with the whole warp."""
    s = _code(path)
    readers = re.findall(r"\bvoid\s+(\w+)\(.*\{\s*asm volatile\(\s*\"tcgen05\.ld", s)
    assert bool(readers) == ("tcgen05.ld" in s)
    bad = [line for body, line in _loops(s)
           if any(re.search(r"\b%s\s*\(" % r, body) for r in readers) and re.search(r"\bif\b", body) and "__syncwarp" not in body]
    assert not bad, bad


@pytest.mark.parametrize("path", [p for p in SOURCES if p.name.startswith("wq_") and "pdl_wait()" in p.read_text()], ids=lambda p: p.name)
def test_only_packed_weights_are_read_before_the_dependency_wait(path):
    """Everything else a launch reads (activations, norm weights, statistics, residuals) may come from the kernel before."""
    s = _code(path)
    for m in re.finditer(r"__global__[^;{]*\{", s):
        body = s[m.end() - 1:_close(s, m.end() - 1, "{}")]
        before = body[:body.find("pdl_wait()")] if "pdl_wait()" in body else ""
        assert not re.search(r"\b(a\.)?(norm_w|ss_in|resid|scratch|x)\s*(\[|\+\s*[a-z(])", before)
