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


@pytest.mark.parametrize("name", ["fno.cu", "fno_gemm.cuh"])
def test_failure_words_are_read_behind_their_barrier(name):
    """A block leaves a loop on the shared word that thread 0 sets when a wait gives up: read anywhere
    but directly behind a block barrier, one warp could see the next wait's answer and leave one barrier
    before the others."""
    src = _code(CSRC / name)
    reads = [m.start() for m in re.finditer(r"if \(s_fail\)", src)]
    assert reads
    for i in reads:
        before = src[:i].rstrip()
        assert before.endswith("__syncthreads();"), (name, before[-120:])
