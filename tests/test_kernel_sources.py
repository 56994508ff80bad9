"""What no run shows, read in the kernels' sources (no GPU)."""
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "metallix_b200", "csrc", "kernels")


@pytest.mark.parametrize("name", ["gemm_tcgen05.cu", "gemm_tcgen05_rows.cu", "gemm_float_split.cu", "attention_prefill_tcgen05.cu"])
def test_warps_that_use_tensor_memory_wait_and_give_up_as_a_whole(name):
    """A warp takes loads and stores of tensor memory, elections and votes as one: no lane may end a wait, or see that its
    block has given up, by itself."""
    with open(os.path.join(KERNELS, name)) as handle:
        text = re.sub(r"//[^\n]*", "", handle.read())
    assert not re.findall(r"\bbarrier_wait\(", text)
    reads = [line.strip() for line in text.split("\n") if re.search(r"\bfailed\b", line)
             and not re.search(r"given_up\(failed\)|failed = |failed_slot|if \(failed && threadIdx\.x == 0\)", line)]
    assert reads == []


def test_warps_that_exchange_values_wait_as_a_whole():
    """The delta rule's walkers exchange sums by shuffles of the whole warp; only its fetching lane waits alone."""
    with open(os.path.join(KERNELS, "delta_prompt.cu")) as handle:
        text = handle.read()
    assert text.count("= barrier_wait(&empty[stage]") == 1 and len(re.findall(r"\bbarrier_wait\(", text)) == 1


def test_lanes_without_rows_are_back_before_tensor_memory_is_loaded():
    """Lanes whose row does not exist store nothing and are ahead of the others: the warp meets before the next load."""
    with open(os.path.join(KERNELS, "tc_epilogue.cuh")) as handle:
        epilogue = handle.read()
    assert re.search(r"__syncwarp\(\);[^\n]*\n\s*tc_load\(taddr, acc\);", epilogue)
    with open(os.path.join(KERNELS, "gemm_float_split.cu")) as handle:
        adders = handle.read().split("// ---- adders")[1].split("// ---- splitters")[0]
    assert "continue;" not in adders.split("again_any")[0] and re.search(r"__syncwarp\(\);[^\n]*\n *}\n", adders)


def test_every_exported_function_is_reached():
    """What the shared library exports, the Python side binds, or a C program links against."""
    from metallix_b200 import ops
    exported = set()
    for name in os.listdir(KERNELS):
        if name.endswith(".cu"):
            with open(os.path.join(KERNELS, name)) as handle:
                exported |= set(re.findall(r"MXB_API\s+[\w ]+?\b(mxb_\w+)\(", handle.read()))
    with open(ops.__file__) as handle:
        by_hand = set(re.findall(r"\.(mxb_\w+)", handle.read()))
    with open(os.path.join(KERNELS, "attention_decode_noalloc.h")) as handle:
        linked = set(re.findall(r"\b(mxb_\w+)\(", handle.read()))
    assert len(exported) > 60 and exported - set(ops._SIGNATURES) - by_hand - linked == set()
