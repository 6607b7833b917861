"""Sizes at which the pipelined kernels' fragments, stages and work items change: tokens per tile (1 to 8, and more than a
tile), ranks (row blocks of 4, 8 and 16; ranks that fill none of them), hidden sizes whose rows end inside a K unit, pool
rows that an expand chunk straddles.  Checked against the CPU oracle, and planned against per-token calls, which must agree
bit for bit: an output's bits depend on its own row and token only.  Needs a B200."""
import numpy as np
import pytest
import torch

import slora_b200 as sl
from slora_b200.batch_infer import shrink_multi
from slora_b200.workloads import build_workload
from tests.helpers import assert_parity, orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(wl, **kw):
    w = wl.to(DEV)
    ops = sl.LoraBatchOps(w.a_start, w.a_len, w.a_loc, w.a_scaling, w.pools_a, w.pools_b, wl.max_rank)
    ops.prepare(w.ids, **kw)
    outs = [torch.zeros((wl.T, ho), dtype=wl.dtype, device=DEV) for _, ho in wl.proj_dims()]
    ops.lora_get_qkv(0, w.x_qkv[0], *outs[:3])
    ops.lora_get_o(0, w.x_o[0], outs[3])
    torch.cuda.synchronize()
    if ops.plan is not None:
        ops.plan.check()
    return outs


def _oracle(wl):
    refs = []
    for p, (_, ho) in enumerate(wl.proj_dims()):
        x = wl.x_o[0] if p == 3 else wl.x_qkv[0]
        refs.append(orc.lora_delta_grouped(np.zeros((wl.T, ho), np.float32), x, wl.pools_a[0], wl.pools_b[0], wl.a_start,
                                           wl.a_len, wl.a_loc, wl.ids, p, wl.a_scaling))
    return refs


@pytest.mark.parametrize("tokens", [1, 2, 3, 4, 5, 7, 8, 9, 13])
@pytest.mark.parametrize("rank", [8, 16, 32, 64, 128])
def test_tokens_per_tile(tokens, rank):
    wl = build_workload(5, pool_rows=4096, n_adapters=3, decode_tokens=3 * tokens, hidden=4096, h_kv=512,
                        rank_choices=(rank,))
    wl.ids = torch.arange(3 * tokens) % 3      # every adapter has `tokens` tokens
    ref, planned, single = _oracle(wl), _layer(wl), _layer(wl, use_plan=False)
    for p in range(4):
        assert_parity(planned[p], ref[p], what=f"n={tokens} r={rank} proj {p}")
        assert torch.equal(planned[p], single[p])


@pytest.mark.parametrize("hidden", [520, 1032, 4104, 5128, 6152])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_rows_that_end_inside_a_unit(hidden, dtype):
    wl = build_workload(5, dtype=dtype, pool_rows=8192, n_adapters=9, decode_tokens=40, hidden=hidden, h_kv=hidden,
                        rank_choices=(8, 16, 64))
    ref, planned, single = _oracle(wl), _layer(wl, mixed_ranks=True), _layer(wl, use_plan=False)
    for p in range(4):
        assert_parity(planned[p], ref[p], dtype, what=f"H={hidden} proj {p}")
        assert torch.equal(planned[p], single[p])


def _few_at_a_time(wl, n=48):
    """Per-token calls of `n` tokens: too few items for more than four rows each."""
    w = wl.to(DEV)
    ops = sl.LoraBatchOps(w.a_start, w.a_len, w.a_loc, w.a_scaling, w.pools_a, w.pools_b, wl.max_rank)
    outs = [torch.zeros((wl.T, ho), dtype=wl.dtype, device=DEV) for _, ho in wl.proj_dims()]
    for at in range(0, wl.T, n):
        part = slice(at, at + n)
        ops.prepare(w.ids[part], use_plan=False)
        ops.lora_get_qkv(0, w.x_qkv[0][part], *(o[part] for o in outs[:3]))
        ops.lora_get_o(0, w.x_o[0][part], outs[3][part])
    torch.cuda.synchronize()
    return outs


@pytest.mark.parametrize("rows_case", ["16 rows", "8 rows", "8 rows, exact items"])
def test_taller_items(rows_case):
    """Batches large enough for items of sixteen and of eight rows, against calls of 48 tokens, whose items have four."""
    if rows_case == "16 rows":      # 61 tokens an adapter: tiles of eight
        wl = build_workload(5, pool_rows=8192 + 512, n_adapters=33, decode_tokens=33 * 61, hidden=1032, h_kv=1032,
                            rank_choices=(64,))
        wl.ids = torch.arange(33 * 61) % 33
    else:
        wl = build_workload(5, pool_rows=65536, n_adapters=250, decode_tokens=300, hidden=1032, h_kv=1032,
                            rank_choices=(64,) if rows_case == "8 rows" else (8, 16, 32, 64))
    ref = _oracle(wl)
    planned = _layer(wl, mixed_ranks=rows_case.endswith("items"), big_groups=False)
    single = _few_at_a_time(wl)
    for p in range(4):
        assert_parity(planned[p], ref[p], what=f"{rows_case} proj {p}")
        assert torch.equal(planned[p], single[p])


def test_ranks_that_fill_no_block():
    """The shrink takes any rank: 3, 12 and 24 rows against the oracle's intermediate."""
    wl = build_workload(5, pool_rows=4096, n_adapters=8, decode_tokens=21, hidden=2048, h_kv=2048, rank_choices=(3, 12, 24))
    w = wl.to(DEV)
    delta = torch.zeros((wl.T, wl.max_rank), dtype=wl.dtype, device=DEV)
    for p in range(4):
        x = w.x_qkv[0]
        sl.dispatch_bgmv(delta, x, w.pools_a[0].view(-1, 16, 128), w.a_start, w.a_len, w.a_loc, w.ids, p, w.a_scaling)
        ref = orc.lora_shrink_ref(wl.x_qkv[0], wl.pools_a[0], wl.a_start, wl.a_len, wl.a_loc, wl.ids, p,
                                  out_width=wl.max_rank)
        got = delta.float().cpu().numpy()
        for t, a in enumerate(wl.ids.tolist()):
            r = wl.ranks[a]
            np.testing.assert_allclose(got[t, :r], ref[t, :r], rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("hidden", [640, 1280, 1536, 2048])
def test_partly_filled_items_of_sixteen_rows(hidden, exact):
    """Ranks of 8 and 64 in items of sixteen rows, tiles of one token and of many: at these hidden sizes a short item is one
    stage and a long one several, and the launch has two reduction buffers (tests/ring_model.cu)."""
    wl = build_workload(5, pool_rows=200 * 4 * 64, n_adapters=200, decode_tokens=2048, hidden=hidden, h_kv=hidden,
                        rank_choices=(8, 64))
    # half of the adapters have one token, the others share the rest
    wl.ids = torch.cat([torch.arange(100), 100 + torch.arange(1948) % 100])
    single, ref = _few_at_a_time(wl), _oracle(wl)
    for turn in range(3):
        planned = _layer(wl, mixed_ranks=exact, big_groups=False)
        for p in range(4):
            assert torch.equal(planned[p], single[p]), (turn, p)
    for p in range(4):
        assert_parity(planned[p], ref[p], what=f"H={hidden} proj {p}")


@pytest.mark.parametrize("hidden", [5120, 8192])
def test_sums_are_as_exact_as_fma_sums(hidden):
    """Share of fp16 intermediates that are not the nearest value to the 64-bit sum.  FP32 sums by fused multiply-adds (256
    partial sums of a row, added as a tree) leave 0.9 of a thousand at these sizes, sums that an mma truncates over a whole
    row 1.3 and 1.6: the bound is the former plus four standard deviations of the count (172 +- 13 of 196608)."""
    T, n, rank = 1024, 200, 64
    g, gc = torch.Generator(device=DEV).manual_seed(hidden), torch.Generator().manual_seed(hidden)
    pool = torch.empty((n * 4 * rank, hidden), dtype=torch.float16, device=DEV).normal_(0, hidden ** -0.5, generator=g)
    x = torch.empty((T, hidden), dtype=torch.float16, device=DEV).normal_(0, 1, generator=g)
    loc = torch.randperm(n * 4 * rank, generator=gc).to(DEV)
    ids = torch.randint(0, n, (T,), generator=gc).to(DEV)
    lens = torch.full((n,), 4 * rank, dtype=torch.int64, device=DEV)
    start = lens.cumsum(0) - lens
    plan = sl.BatchPlan(ids, start, lens, loc.numel())
    deltas = [torch.zeros((T, rank), dtype=torch.float16, device=DEV) for _ in range(3)]
    shrink_multi(plan, ids, [0, 1, 2], deltas, x, pool, start, lens, loc)
    wrong = 0
    for p in range(3):
        for at in range(0, T, 64):
            tok = ids[at:at + 64]
            rows = loc[(start[tok] + rank * p)[:, None] + torch.arange(rank, device=DEV)]
            exact = torch.einsum("tk,trk->tr", x[at:at + 64].double(), pool[rows].double())
            wrong += int((deltas[p][at:at + 64] != exact.float().half()).sum())
    assert wrong <= 224, wrong
