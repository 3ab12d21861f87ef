"""Rules that the kernels' memory ordering rests on, read off their sources: what breaks them is a race that no run on a
GPU shows reliably."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bitladder_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def _code(path):
    """The file's lines without their comments."""
    return [re.sub(r"//.*", "", line) for line in open(path)]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_an_arrival_is_counted_in_behind_a_fence(path):
    """What a CTA or warp has read or written has to be ordered before the count that lets the last one go on."""
    lines = _code(path)
    for i, line in enumerate(lines):
        if "atomicAdd(" in line:
            assert "__threadfence" in "".join(lines[max(0, i - 4):i]), f"line {i + 1}"


def test_a_rolling_cta_reads_its_lengths_once():
    """The last CTA of a sequence overwrites the lengths: one thread of each CTA reads them, in front of its fence."""
    code = "".join(_code(os.path.join(CSRC, "bd_pack.cu")))
    for name in ("roll_res_lens", "roll_cache_seqlens"):
        reads = [m.start() for m in re.finditer(rf"(?<!\w)p\.{name}\[ib\](?! = )", code)]
        assert len(reads) == 1
        opened = code.rindex("if (tid == 0) {", 0, reads[0])
        assert "}" not in code[opened:reads[0]] and reads[0] < code.index("atomicAdd(")


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_nothing_is_read_as_constant_memory(path):
    """A kernel that is staged early is resident while the kernel in front still writes what it will read, so no load may
    be non-coherent: those promise memory that nobody writes for the kernel's whole life, and may be moved across the
    wait."""
    code = "".join(_code(path))
    assert "__ldg(" not in code and "global.nc" not in code


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_a_wait_of_its_own_comes_before_what_earlier_kernels_wrote(path):
    """Only a kernel's own griddepcontrol.wait makes earlier kernels' writes visible to it (that the kernel in front has
    waited, and let this one start afterwards, does not), so the lengths and the table of a ragged batch are read behind
    one.  Whether a kernel waits there may hang on nothing but that there is such a table."""
    code = "".join(_code(path))
    for cond in re.findall(r"if (?:constexpr )?\(((?:[^()]|\([^()]*\))*)\)\s*\{?\s*asm volatile\(\"griddepcontrol.wait", code):
        assert "p." not in re.sub(r"p\.part\.table|\browid\b.*|\bn(rows|parts)\b.*", "", cond), cond
    for body in code.split("__global__")[1:]:
        if "griddepcontrol.wait" not in body:
            continue
        body = re.sub(r"\{[^{}]*griddepcontrol\.wait[^{}]*return;\s*\}", "", body)          # a warp that leaves
        read = re.search(r"ragged_entry\(|part_range\(|(cache_seqlens|res_lens)\[", body)
        assert not read or body.index("griddepcontrol.wait") < read.start()


def test_the_short_kernel_gives_up_as_one():
    """What a wait that runs out leads to (nothing of it can be provoked on a GPU at will): the lanes of a warp agree, a
    warp sets a flag that nobody but itself initialises, and copies in flight are given
    time to land before a full tail is packed through the tiles they arrive in."""
    code = "".join(_code(os.path.join(CSRC, "bd_decode_short.cu")))
    assert re.findall(r"(\w+)\([^;]*mbar_wait_bounded\(", code) == ["__all_sync"]
    assert set(re.findall(r"gave_up\[(\w+)\] = ", code)) == {"warp"} and "abort_flag" not in code
    assert code.index("__nanosleep(") < code.index("pack_k_part<")
