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


def _bits(t):
    return t.view(torch.int16)


def _foreign_batch(dtype):
    """Prompts whose last tile is not full, with rows behind it that belong to other tokens, to ids without an adapter and
    to nobody: [(id, tokens)], outputs that hold -0.0 in every second column."""
    parts = [(0, 140), (-1, 9), (1, 200), (5, 3), (99, 4), (2, 129), (3, 2), (6, 1), (-1, 30), (4, 1), (0, 5)]
    ids = [a for a, n in parts for _ in range(n)]
    wl = build_workload(3, dtype=dtype, pool_rows=4096, n_adapters=8, decode_tokens=len(ids), prefill=None, hidden=1024,
                        rank_choices=(8, 32, 64))
    wl.ids = torch.tensor(ids)
    g = torch.Generator().manual_seed(11)
    base = [torch.randn((wl.T, ho), generator=g).to(dtype) for _, ho in wl.proj_dims()]
    for b in base:
        b[:, ::2] = -0.0
    return wl, parts, base


@pytest.mark.parametrize("use_pdl", [True, False])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_rows_of_other_tokens_keep_their_bits(use_pdl, dtype):
    wl, _, base = _foreign_batch(dtype)
    w = wl.to(DEV)

    def layer(**kw):
        ops = sl.LoraBatchOps(w.a_start, w.a_len, w.a_loc, w.a_scaling, w.pools_a, w.pools_b, wl.max_rank, use_pdl)
        ops.prepare(w.ids, **kw)
        outs = [b.to(DEV) for b in base]
        ops.lora_get_qkv(0, w.x_qkv[0], *outs[:3])
        ops.lora_get_o(0, w.x_o[0], outs[3])
        torch.cuda.synchronize()
        return [o.cpu() for o in outs]

    nobody = (wl.ids < 0) | (wl.ids >= 8)
    small = (wl.ids >= 3) & (wl.ids < 8)
    tiles = layer(big_groups=False)           # every group on the tile kernels: each row is written by its own token only
    for _ in range(20):
        outs = layer()
        for p in range(4):
            assert torch.equal(_bits(outs[p][nobody]), _bits(base[p][nobody]))
            assert torch.equal(_bits(outs[p][small]), _bits(tiles[p][small]))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_segment_calls_leave_rows_outside_their_segments(dtype):
    wl, parts, base = _foreign_batch(dtype)
    w = wl.to(DEV)
    segs, at = [], 0
    for a, n in parts:
        if 0 <= a < 8:
            segs.append((at, n, a))
        at += n
    start = torch.tensor([s[0] for s in segs], dtype=torch.int32, device=DEV)
    length = torch.tensor([s[1] for s in segs], dtype=torch.int32, device=DEV)
    adapter = torch.tensor([s[2] for s in segs], dtype=torch.int64, device=DEV)
    nobody = (wl.ids < 0) | (wl.ids >= 8)
    for p, (h_in, h_out) in enumerate(wl.proj_dims()):
        x = w.x_o[0] if p == 3 else w.x_qkv[0]
        delta = torch.zeros((wl.T, wl.max_rank), dtype=dtype, device=DEV)
        y = base[p].to(DEV)
        sl.lora_get_qkvo_fwd_shrink(x, w.pools_a[0], delta, w.a_loc, w.a_start, w.a_len, start, length, adapter, h_in, p,
                                    wl.max_rank, 200)
        sl.lora_get_qkvo_fwd_expand(delta, w.pools_b[0], y, w.a_scaling, w.a_loc, w.a_start, w.a_len, start, length, adapter,
                                    h_out, p, wl.max_rank, 200)
        torch.cuda.synchronize()
        assert torch.equal(_bits(y.cpu()[nobody]), _bits(base[p][nobody]))
        ids = wl.ids.clone()
        ids[nobody] = 0
        ref = orc.lora_delta_grouped(base[p].float().numpy(), x.cpu(), wl.pools_a[0], wl.pools_b[0], wl.a_start, wl.a_len,
                                     wl.a_loc, ids, p, wl.a_scaling)
        assert_parity(y.cpu()[~nobody], ref[~nobody.numpy()], dtype, what=f"proj {p}")
