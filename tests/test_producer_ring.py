"""The ring of the pipelined kernels, on the CPU: what the lanes of a producer warp share between two stages, and which
items may be in flight together."""
import os
import re
import shutil
import subprocess

import pytest

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


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
def test_no_two_open_items_share_a_reduction_buffer(tmp_path):
    """The kernels' own allocation rules, replayed on the host over hidden sizes, rows and tokens (tests/ring_model.cu)."""
    exe = str(tmp_path / "ring_model")
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", os.path.dirname(SOURCE), "-I",
                    os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "ring_model.cu"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout[:2000]
