"""The ring of the pipelined kernels, on the CPU: what the lanes of a producer warp share between two stages."""
import os
import re

from tests.helpers import ROOT

SOURCE = os.path.join(ROOT, "slora_b200", "csrc", "lora_pipelined.cuh")


def _body(source, head):
    """Text of the function that starts with `head`, braces matched."""
    at = source.index("{", source.index(head))
    depth = 0
    for i in range(at, len(source)):
        depth += {"{": 1, "}": -1}.get(source[i], 0)
        if depth == 0:
            return re.sub(r"//[^\n]*", "", source[at:i + 1])
    raise AssertionError(head)


def test_lanes_of_a_producer_share_nothing_through_memory_between_stages():
    """Every lane allocates every stage for itself, and nothing but the loop of ring_alloc keeps the lanes together: what
    it reads of earlier stages may not be a word that one lane has stored, and all lanes must leave a wait with the same
    outcome."""
    with open(SOURCE) as f:
        source = f.read()
    body = _body(source, "uint32_t ring_alloc(")
    assert set(re.findall(r"\bc\.(\w+)", body)) <= {"empty", "full"}     # barriers only
    assert len(re.findall(r"mbar_wait_timed\(", body)) == len(re.findall(r"__all_sync\(FULL_MASK, mbar_wait_timed\(", body)) > 0
