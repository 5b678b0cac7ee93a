"""What the blocks of a cluster wait for, read from the kernels' text (a missing order shows on no run that one could count on)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pulsar_b200", "csrc")


def _text(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_waits_for_other_blocks_are_ordered_for_the_whole_cluster():
    """Peers arrive at ``part_full`` and ``part_empty``: what they wrote or read before has to be ordered before what follows the wait."""
    waits = re.findall(r"(mbar_wait\w*)\((part_\w+)", _text("gemm_tcgen05_stream.cu"))
    assert sorted({bar for _, bar in waits}) == ["part_empty", "part_full"]
    assert {call for call, _ in waits} == {"mbar_wait_cluster"}


def test_tensor_memory_is_freed_behind_the_work_in_flight():
    """A block that gave up a wait lets its copies and products land before it frees the tensor memory that they write."""
    for name in ("gemm_tcgen05.cu", "gemm_tcgen05_stream.cu", "attention_prefill_tcgen05.cu", "attention_prefill_tcgen05_dual.cu"):
        order = re.findall(r"__nanosleep|tcgen05\.dealloc", _text(name))
        assert order and order == ["__nanosleep", "tcgen05.dealloc"] * (len(order) // 2), name
