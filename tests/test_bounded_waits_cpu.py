"""Kernels with bounded waits: after one that ran out no warp is left at a barrier that another does not come to, and warps stay together.

Read from the sources: such a wait runs out only when something else is broken, which no test brings about on a GPU."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "deepseek-v4-sm80_b200" / "ops" / "csrc"
SOURCES = [p for p in sorted(CSRC.glob("*.cu")) if "mbar_wait" in p.read_text()]


def _source(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def _closing(src, at, pair):
    depth = 0
    for i in range(at, len(src)):
        depth += (src[i] == pair[0]) - (src[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError("no closing " + pair[1])


def _loops(src):
    """(header, first and last character of the body) of each loop with a body in braces."""
    for m in re.finditer(r"\b(?:for|while)\s*\(", src):
        end = _closing(src, m.end() - 1, "()")
        body = end + 1 + len(src[end + 1:]) - len(src[end + 1:].lstrip())
        if src[body] == "{":
            yield src[m.end():end], body, _closing(src, body, "{}")


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_no_barrier_in_a_loop_that_some_warps_leave(path):
    """Where a loop has a barrier over several warps, a warp whose wait ran out goes on to the barrier, and round by round to the end."""
    src = _source(path)
    for bar in re.finditer(r"\bbar(?:rier)?(?:\.cta)?\.sync\b", src):
        for header, first, last in _loops(src):
            if not first < bar.start() < last or "mbar_wait" not in src[first:last]:
                continue
            where = f"{path.name}: barrier within for ({header.strip()})"
            assert not re.search(r"\bok\b", header), where
            assert not re.search(r"\b(?:break|return)\b", src[first:last]), where
            assert not re.search(r"(?:!\s*ok|mbar_wait)\b[^;{}]*\)\s*\{?\s*continue\b", src[first:bar.start()]), where


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_lanes_without_a_row_come_to_the_next_load(path):
    """Loads from tensor memory take a warp as a whole: where a loop issues them, no lane goes on to the next round ahead of the others."""
    src = _source(path)
    for header, first, last in _loops(src):
        body = src[first:last]
        if "tmem_ld_32x" in body and not any(first < f < last and "tmem_ld_32x" in src[f:e] for _, f, e in _loops(src)):
            assert not re.search(r"\bcontinue\b", body[body.index("tmem_ld_32x"):]), f"{path.name}: for ({header.strip()})"


@pytest.mark.parametrize("path", [p for p in SOURCES if "tmem_dealloc" in p.read_text()], ids=lambda p: p.stem)
def test_tensor_memory_is_freed_behind_what_is_in_flight(path):
    """After a wait that ran out, MMAs and copies may still be under way: they are waited for, with a limit, before tensor memory is freed."""
    src = _source(path)
    for free in re.finditer(r"tmem_dealloc\(", src):
        assert re.search(r"if \(\*abort_flag\) drain_after_abort\([^;]*;\s*$", src[:free.start()]), path.name
