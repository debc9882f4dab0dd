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


def test_programmatic_launches_read_coherently():
    """A kernel launched while the one before it still runs reads what that one writes: its parameters
    promise nothing that would let the compiler take the non-coherent path, whose data must not change
    while the kernel lives (the loads would not be ordered behind the wait either)."""
    src = _code(CSRC / "fno.cu") + _code(CSRC / "fno_gemm.cuh")
    names = set(re.findall(r"launch_dep\(\(?(k_\w+)", src)) | {"k_pix", "k_dft2"}
    assert {"k_adam", "k_pack_spec", "k_loss", "k_reduce_map", "k_gemm_tc"} <= names
    for name in sorted(names):
        sig = re.search(r"__global__ void[^;{]*?\b" + name + r"\((.*?)\)\s*\{", src, flags=re.S)
        assert sig, name
        assert "__restrict__" not in sig.group(1), (name, sig.group(1))


@pytest.mark.parametrize("name", ["k_pix", "k_wgrad"])
def test_late_launch_waits_for_the_whole_block(name):
    """One thread's launch_dependents counts for its block: in kernels whose warps have different jobs,
    some threads none, the late one stands behind the block's last barrier."""
    src = _code(CSRC / "fno.cu")
    body = src[re.search(r"__global__ void[^;{]*?\b" + name + r"\(", src).end():]
    body = body[:body.index("\n}\n")]
    late = body.index("if (!dep_early()) dep_launch();")
    assert body.count("dep_launch();") == 2
    assert body[:late].rstrip().endswith("__syncthreads();")
    assert "__syncthreads" not in body[late:]


def test_plain_form_allocates_what_it_uses():
    """Every buffer of the plain FP64 form's struct has a use besides its allocation (a plane is 8 bytes
    a cell in every handle)."""
    src = _code(CSRC / "fi_api.cu")
    struct = re.search(r"struct PlainBufs \{(.*?)\n\};", src, flags=re.S)
    names = re.findall(r"\*\s*(\w+)", struct.group(1))
    names += re.findall(r", (\w+)(?=[,;\[])", struct.group(1))
    assert {"fscratch", "rhs", "Mxy"} <= set(names)
    rest = src[:struct.start()] + src[struct.end():]
    rest = re.sub(r"double\*\* bufs\[\] = \{.*?\};", "", rest, flags=re.S)
    rest = re.sub(r"RET\(dalloc\([^;]*;", "", rest)
    unused = [n for n in names if not re.search(r"\bp\." + n + r"\b", rest)]
    assert not unused, unused
