"""Big same-adapter groups of a planned batch (tensor-core kernels) whose tokens lie together, apart or in between others:
tiles of consecutive tokens are moved whole, the others token by token; a tile's last rows may belong to other tokens, whose
outputs must not change.  Checked against the CPU oracle.  Needs a B200."""
import numpy as np
import pytest
import torch

import slora_b200 as sl
from slora_b200.workloads import build_workload
from tests.helpers import assert_parity, orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ids(case):
    if case == "runs":              # whole prompts, lengths that leave partial tiles, decode tokens behind them
        return [0] * 128 + [1] * 200 + [2] * 131 + [3, 4, 5, 3, 6]
    if case == "apart":             # a prompt in two runs with another one between, and decode tokens of its adapter
        return [0] * 140 + [1] * 129 + [0] * 70 + [2, 0, 3, 0, 1, 4]
    if case == "interleaved":       # no two neighbours of one adapter
        return [i % 2 for i in range(300)] + [2, 3]
    return [i % 70 for i in range(70 * 128)]   # more big groups than the plan keeps in order


@pytest.mark.parametrize("case", ["runs", "apart", "interleaved", "many"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_big_groups(case, dtype):
    ids = _ids(case)
    many = case == "many"
    wl = build_workload(3, dtype=dtype, pool_rows=8192 if many else 4096, n_adapters=70 if many else 8,
                        decode_tokens=len(ids), prefill=None, hidden=512 if many else 1024,
                        rank_choices=(8, 16) if many else (8, 32, 64))
    wl.ids = torch.tensor(ids)
    w = wl.to(DEV)
    ops = sl.LoraBatchOps(w.a_start, w.a_len, w.a_loc, w.a_scaling, w.pools_a, w.pools_b, wl.max_rank)
    ops.prepare(w.ids)
    g = torch.Generator().manual_seed(3)
    base = [torch.randn((wl.T, ho), generator=g).to(dtype) for _, ho in wl.proj_dims()]
    outs = [b.to(DEV) for b in base]
    ops.lora_get_qkv(0, w.x_qkv[0], *outs[:3])
    ops.lora_get_o(0, w.x_o[0], outs[3])
    torch.cuda.synchronize()
    ops.plan.check()
    for p in range(4):
        x = wl.x_o[0] if p == 3 else wl.x_qkv[0]
        ref = orc.lora_delta_grouped(base[p].float().numpy(), x, wl.pools_a[0], wl.pools_b[0], wl.a_start, wl.a_len, wl.a_loc,
                                     wl.ids, p, wl.a_scaling)
        assert_parity(outs[p], ref, dtype, what=f"{case} proj {p}")
