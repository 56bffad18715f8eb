"""Rules that the tensor-pipe kernels keep on paths no test may take on a GPU (a wait that gives up, a circular wait),
checked on their sources."""
import glob
import os
import re

import numpy as np
import pytest

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "nerva_b200", "csrc")


def _kernels():
    """name -> body of every kernel that allocates tensor memory."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = open(path).read()
        for m in re.finditer(r"__global__[^;{]*?(\w+_kernel)\([^{]*\)\s*\{", text):
            end = text.index("\n}\n", m.end())
            body = text[m.end():end]
            if "tcgen05.alloc" in body:
                out[m.group(1)] = body
    return out


KERNELS = _kernels()


def test_all_tensor_memory_kernels_are_looked_at():
    assert set(KERNELS) == {"gemm_tc_kernel", "gemm_wide_kernel", "moe_block_gemm_kernel", "prefill_attention_kernel"}


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_a_block_that_gave_up_drains_before_it_frees_tensor_memory(name):
    body = KERNELS[name]
    teardown = body[body.rindex("sh.abort != 0u"):body.index("tcgen05.dealloc")]
    rings = set(re.findall(r"mbar_arrive_expect_tx\(&sh\.(\w*full)", body))  # named directly ...
    rings |= {r for r in ("k_full", "v_full") if f"&sh.{r}[st]" in body}     # ... or through a choice of two
    assert rings
    for ring in rings:
        assert f"drain_copies(sh.{ring}," in teardown, ring
    assert "drain_mmas(&sh.drained)" in teardown or "mbar_wait_bounded(&sh.drained, 0)" in teardown
    assert teardown.count("__syncthreads();") == 1  # the drains end before the memory is freed


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_waits_in_front_of_warp_wide_accesses_are_taken_by_the_whole_warp(name):
    """Between a wait that a single lane may leave early and the role's end there is no tensor-memory access of the warp."""
    body = KERNELS[name]
    for wait in re.finditer(r"\babortable_wait\(", body):
        role = body[wait.end():]
        ends = [role.find(end) for end in ("} else if (warp", "} else {\n    // ------", "} else {\n    const uint32_t quarter",
                                           "// ---- teardown") if end in role]
        assert not re.search(r"tmem_(load|store)\w*\(|tcgen05\.(ld|st)", role[:min(ends)]), role[:80]


def test_blocks_that_fit_on_an_sm_together_never_ask_for_more_tensor_memory_than_there_is(built_lib):
    """An allocation that does not fit waits for another block to leave, and that block may be of a dependent launch that
    waits for this one: so no set of blocks whose shared memory fits an SM may exceed its 512 columns."""
    smem, columns = np.zeros(256, np.uint32), np.zeros(256, np.uint32)
    n = built_lib.nerva_b200_tensor_memory_launches(smem.ctypes.data, columns.ctypes.data, 256)
    shapes = sorted({(int(s), int(c)) for s, c in zip(smem[:n], columns[:n])})
    assert 4 <= n <= 256 and all(c in (128, 256, 512) and 0 < s <= 227 * 1024 for s, c in shapes)
    per_sm, reserved = 228 * 1024, 1024  # shared memory of an SM; what the system takes of it per block

    def most_columns(room):
        return max((c + most_columns(room - s - reserved) for s, c in shapes if s + reserved <= room), default=0)

    assert most_columns(per_sm) <= 512


def test_rings_that_issue_through_an_elected_lane_give_up_as_a_warp():
    """elect.sync waits for all lanes: a ring whose copies are issued behind it may not be given up by some lanes only."""
    rings = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = open(path).read()
        if "elected()" not in text:
            continue
        for wait in re.findall(r"if \(!(?:\w+\.)?dead && !(\w+)\(", text):
            assert wait == "warp_wait_bounded", os.path.basename(path)
            rings += 1
    assert rings == 2  # row_stream.cuh, moe.cu
    common = open(os.path.join(CSRC, "common.cuh")).read()
    assert re.search(r"bool warp_wait_bounded\([^)]*\) \{\s*return __all_sync\(0xffffffffu, mbar_wait_bounded\(bar, parity\)\);", common)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_no_lane_leaves_a_loop_of_warp_wide_loads_on_its_own(name):
    body = KERNELS[name]
    for load in re.finditer(r"tmem_load\d+\(", body):
        depth, at = 0, load.end()
        while depth >= 0:  # to the end of the block that holds the load
            depth += {"{": 1, "}": -1}.get(body[at], 0)
            at += 1
        assert "continue;" not in body[load.end():at], body[load.start():at]


def test_shared_arrays_that_are_accessed_in_wider_pieces_are_aligned():
    """reinterpret_cast<float2 / float4 / uint2 / uint4 *> of a __shared__ array needs an alignment of its own."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = open(path).read()
        for kernel in re.split(r"(?=__global__)", text):
            arrays = {name: "__align__" in line
                      for line in re.findall(r"__shared__[^;]*;", kernel) for name in re.findall(r"(\w+)\[", line)}
            for name in re.findall(r"reinterpret_cast<(?:const )?(?:float|uint)[24] \*>\((\w+)", kernel):
                assert arrays.get(name, True), (os.path.basename(path), name)


def test_static_scratch_error_word_is_trusted_only_behind_a_call_that_ended_well():
    """A launch that fails between the kernel that sets the word and the one that reports it leaves it set: whatever way a call
    ends but the last one, the next call clears the word."""
    text = open(os.path.join(CSRC, "attention_static_scratch.cu")).read()
    call = text[text.index("int nerva_b200_gqa_decode_attention_static_scratch("):]
    taken, launched = call.index("clean.exchange(false)"), call.index("launch_attention(")
    assert taken < launched and "cudaMemsetAsync(error_word, 0" in call[taken:launched]
    assert text.count("clean = true") == 1 and call.index("clean = true") > call.rindex("return -1;")
