"""Rules for kernels that start while their predecessor still runs, held against the sources."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "ksa_b200" / "csrc"


def _functions(text):
    """(header, body) of every device function and kernel."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"(?:__global__|__device__)[^;{}()]*(?:\([^(){};]*\)[^;{}()]*)*?\b\w+\s*\(([^{};]*?)\)\s*\{", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(0), text[m.end():at]


SOURCES = [(f.name, *fn) for f in sorted(CSRC.glob("*.cu")) for fn in _functions(f.read_text())]
WAITS_FOR_PEERS = re.compile(r"flag_wait_ge\(")


def test_what_waits_for_other_gpus_lets_no_successor_start():
    """Its successors, always launched dependently, would hold SMs for as long as the peers take."""
    checked = 0
    for name, header, body in SOURCES:
        if not WAITS_FOR_PEERS.search(body):
            continue
        checked += 1
        for line in body.split("\n"):
            if re.search(r"grid_dependency_(enter|launch)\(", line):
                assert re.search(r"\bif \(", line), (name, header[-120:], line)
    assert checked >= 4


def test_kernels_that_start_early_promise_nothing_about_their_memory():
    """``const __restrict__`` lets loads move ahead of the wait or hit lines that an SM kept from before."""
    kernels = [(n, h) for n, h, body in SOURCES if "__global__" in h and "grid_dependency_" in body]
    assert len(kernels) >= 25
    assert not [(n, h) for n, h in kernels if "__restrict__" in h]


def test_kernels_that_run_beside_another_read_nothing_that_an_sm_kept_from_before():
    """They have not waited when they read, so the fences that stand in for the wait come before anything else they do with memory."""
    common = [body for header, body in _functions((CSRC / "common.cuh").read_text()) if "grid_dependency_enter(int beside)" in header]
    assert len(common) == 1 and re.match(r"\s*if \(beside\) grid_dependency_observe\(\);\s*else grid_dependency_wait\(\);", common[0])
    checked = 0
    for name, header, body in SOURCES:
        if "grid_dependency_leave(" not in body:
            continue
        checked += 1
        at = re.search(r"grid_dependency_observe\(\)|grid_dependency_enter\([^)]+\)", body)
        assert at, (name, header[-120:])
        reads = re.finditer(r"\bload_w(?:eights)?\(|\bload_acts\(|tma_load_2d(?:_pair)?\(|const uint4\*>\((?:A |key_row)", body)
        reads = [m.start() for m in reads]
        assert reads and min(reads) > at.start(), (name, header[-120:])
    assert checked >= 6
