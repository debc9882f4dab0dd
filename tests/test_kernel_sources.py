"""Ordering rules of the kernels that no run shows reliably, checked in their sources (CPU)."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "fastisostasy.jl_b200" / "csrc"
SOURCES = sorted(p for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh"))


def _code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_block_copies_are_followed_by_a_barrier(path):
    """copy_words(&x, ...) spreads the words of a shared object over the block's threads: nothing
    touches x between the copy and the next block barrier."""
    src = _code(path)
    for c in re.finditer(r"copy_words\(&([\w.]+), [^;]*;", src):
        rest = src[c.end():]
        end = rest.find("__syncthreads()")
        assert end >= 0, (path.name, c.group(0))
        use = re.search(r"(?<![\w.])" + re.escape(c.group(1)) + r"\b", rest[:end])
        assert not use, f"{path.name}: {c.group(1)} is used before a barrier: {rest[use.start() - 40:use.end() + 40]!r}"
