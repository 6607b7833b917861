"""What the performance of this library is measured on: the LoRA deltas of transformer layers, called the way a serving
program calls them.

Every case is a batch of tokens with an adapter each, adapter tables over a pool whose rows are scattered by a random
page permutation, and base outputs that the calls add their deltas to.  Values: x ~ N(0, 1), A ~ N(0, 1 / hidden),
B ~ N(0, 0.02^2), scale = 16 / rank, base outputs ~ N(0, 0.1^2).  ``via`` says which entry points a pass goes through:

* ``step``      what a server does for every batch it forms, call by call: ``LoraBatchOps.prepare`` and then
                ``lora_get_qkv`` + ``lora_get_o`` of every layer.
* ``layers``    the layers of a batch that has been prepared (``prepare`` is once per batch, the layers many times).
* ``graph``     the same layers as one CUDA graph, as a server replays a decode step.
* ``rope``      as ``graph``: ``lora_get_qkv`` with rotary embedding and KV-pool scatter, then ``lora_get_o``.
* ``dispatch``  ``dispatch_bgmv`` per projection and direction (eight calls a layer), without a plan.
* ``segments``  ``lora_get_qkvo_fwd_shrink`` / ``_expand`` per projection over prefill requests.
"""
import torch

import slora_b200 as sl

ALPHA = 16.0
KV_ROWS = 4096      # rows of a KV pool that the rope cases scatter into
HEAD_DIM = 128


def _case(via, hidden, kv, layers, adapters, ranks, decode, zipf, prefill, dtype, name=None):
    """prefill: texts like "8x512" (sequences of one length) or "8:8-512" (count, lengths uniform in a range)."""
    c = {"via": via, "hidden": hidden, "kv": kv, "layers": layers, "adapters": adapters, "ranks": ranks,
         "decode": decode, "zipf": zipf, "prefill": prefill, "dtype": dtype}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a server with next to no load: one request, its batch formed and two layers run; launches and host time count
        _case("step", 4096, 4096, 2, 16, "16", 1, 0.0, "", "fp16", "step_one_token"),
        # the drop-in entry point on the smallest configuration: 32 decode tokens over 4 adapters of rank 8
        _case("dispatch", 4096, 4096, 1, 4, "8", 32, 0.0, "", "fp16", "dispatch_32_tokens"),
        # the decode step of a 7B-shaped model, 1000 adapters of one rank, popularity Zipf(1)
        _case("graph", 4096, 4096, 8, 1000, "8", 256, 1.0, "", "fp16", "decode_7b_rank8"),
        # the same batch with what follows the q/k/v delta in a layer: rotary embedding, new k and v into the KV pool
        _case("rope", 4096, 4096, 4, 1000, "8", 256, 1.0, "", "fp16", "decode_7b_rope"),
        # an odd number of requests in bf16 over adapters of every rank
        _case("graph", 4096, 4096, 4, 500, "8,16,32,64", 77, 1.0, "", "bf16", "decode_7b_ragged_bf16"),
        # the headline: 13B-shaped, 512 tokens of which 51 prefill, 2000 adapters, ranks 16 to 64
        _case("layers", 5120, 5120, 1, 2000, "16,32,64", 461, 0.8, "1:51-51", "fp16", "mixed_13b"),
        # decode beside long prefill requests: some adapters have hundreds of tokens, most have one
        _case("layers", 4096, 4096, 1, 500, "8,16,32,64", 248, 1.0, "8:8-512", "fp16", "mixed_7b_prefill"),
        # the 70B shape: wide, k and v narrow (grouped heads), about five tokens an adapter, rank 64
        _case("layers", 8192, 1024, 1, 200, "64", 1024, 0.0, "", "fp16", "decode_70b_gqa"),
        # the same shape in bf16 with few adapters: tiles of eight tokens
        _case("layers", 8192, 1024, 1, 40, "32", 333, 0.0, "", "bf16", "decode_70b_few_adapters_bf16"),
        # a batch of prompts and nothing else
        _case("layers", 4096, 4096, 1, 64, "8,16,32,64", 0, 1.0, "8x512", "fp16", "prefill_8x512"),
        # the reference's prefill entry points, requests of any length
        _case("segments", 4096, 4096, 1, 64, "8,16,32,64", 0, 1.0, "8:8-512", "fp16", "segments_ragged"),
        # a whole step as an eager server runs it: the batch formed, then eight layers
        _case("step", 4096, 4096, 8, 1000, "8", 256, 1.0, "", "fp16", "step_7b_eager"),
    ]


def _spread(rng, lo, hi):
    """Uniform over the logarithm, odd sizes included."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    via = rng.choice(["step", "layers", "graph", "rope", "dispatch", "segments", "layers", "graph"])
    dtype = rng.choice(["fp16", "fp16", "bf16"])
    hidden, kv = rng.choice([(4096, 4096), (5120, 5120), (8192, 1024)])
    ranks = rng.choice(["8", "16", "32", "64", "8,16,32,64", "16,32,64"])
    zipf = rng.choice([0.0, 0.8, 1.0])
    adapters = _spread(rng, 4, 500)
    decode, prefill, layers = 0, "", 1
    if via == "dispatch":
        decode = _spread(rng, 1, 128)
    elif via == "segments":
        hidden = kv = 4096
        prefill = "%d:%d-%d" % (_spread(rng, 1, 8), _spread(rng, 8, 64), _spread(rng, 64, 512))
    elif via == "layers":
        decode = _spread(rng, 16, 768)
        if rng.random() < 0.4:
            prefill = "%d:%d-%d" % (_spread(rng, 1, 6), _spread(rng, 8, 64), _spread(rng, 64, 384))
    else:
        decode = _spread(rng, 1, 256)
        layers = rng.choice([1, 2, 3])
    return _case(via, hidden, kv, layers, adapters, ranks, decode, zipf, prefill, dtype)


# ---- what a program has in hand before the call -------------------------------------------------------------------
def _dtype(case):
    return torch.float16 if case["dtype"] == "fp16" else torch.bfloat16


def _batch(case, seed):
    """Ranks per adapter, adapter of every token, and the prefill requests (start, length, adapter)."""
    g = torch.Generator().manual_seed(7919 * seed + 11)
    choices = [int(r) for r in case["ranks"].split(",")]
    n = case["adapters"]
    ranks = [choices[i] for i in torch.randint(0, len(choices), (n,), generator=g).tolist()]
    p = torch.arange(1, n + 1, dtype=torch.float64) ** (-case["zipf"])

    def adapters(count):
        return torch.multinomial(p / p.sum(), count, replacement=True, generator=g).tolist() if count else []

    lens = []
    if "x" in case["prefill"]:
        count, length = case["prefill"].split("x")
        lens = [int(length)] * int(count)
    elif case["prefill"]:
        count, span = case["prefill"].split(":")
        lo, hi = (int(v) for v in span.split("-"))
        # the lengths belong to the case (a batch keeps its size from seed to seed), their adapters to the seed
        shape = torch.Generator().manual_seed(int(count) * 1000003 + lo * 1009 + hi)
        lens = torch.randint(lo, hi + 1, (int(count),), generator=shape).tolist()
    ids, requests = [], []
    for length, a in zip(lens, adapters(len(lens))):
        requests.append((len(ids), length, a))
        ids += [a] * length
    return ranks, ids + adapters(case["decode"]), requests


def prepare(case, seed):
    dev, dt, H, K, L = "cuda", _dtype(case), case["hidden"], case["kv"], case["layers"]
    ranks, ids, requests = _batch(case, seed)
    T = len(ids)
    gc = torch.Generator().manual_seed(seed)
    gd = torch.Generator(device=dev).manual_seed(seed)
    lens = torch.tensor([4 * r for r in ranks], dtype=torch.int64)
    rows = int(lens.sum())
    pool_rows = rows + rows // 8 + 64          # some rows belong to nobody
    s = {"case": case, "ids": torch.tensor(ids, dtype=torch.int64).to(dev), "start": (lens.cumsum(0) - lens).to(dev),
         "len": lens.to(dev), "loc": torch.randperm(pool_rows, generator=gc)[:rows].to(dev),
         "scale": torch.tensor([ALPHA / r for r in ranks], dtype=dt).to(dev), "max_rank": max(ranks)}

    def normal(shape, std):
        return torch.empty(shape, dtype=dt, device=dev).normal_(0.0, std, generator=gd)

    s["A"] = [normal((pool_rows, H), H ** -0.5) for _ in range(L)]
    s["B"] = [normal((pool_rows, H), 0.02) for _ in range(L)]
    s["x"] = [normal((T, H), 1.0) for _ in range(L)]       # the layer's input
    s["xo"] = [normal((T, H), 1.0) for _ in range(L)]      # the attention's output
    s["y"] = [[normal((T, K if p in (1, 2) else H), 0.1) for p in range(4)] for _ in range(L)]
    via = case["via"]
    if via in ("rope", "rope_inputs"):
        angle = torch.rand((T, HEAD_DIM // 2), generator=gd, device=dev) * 6.28
        s["cos"], s["sin"] = torch.cos(angle).to(dt), torch.sin(angle).to(dt)
        s["kv_rows"] = torch.randperm(KV_ROWS, generator=gc)[:T].to(dev)
        s["kv"] = [[torch.zeros((KV_ROWS, K), dtype=dt, device=dev) for _ in range(2)] for _ in range(L)]
    if via in ("dispatch", "segments"):
        s["delta"] = [torch.zeros((T, s["max_rank"]), dtype=dt, device=dev) for _ in range(4)]
        s["A3"] = [a.view(pool_rows, H // HEAD_DIM, HEAD_DIM) for a in s["A"]]
        # dispatch_bgmv reads B with the output width as its row stride
        s["B3"] = [b.view(pool_rows, H // HEAD_DIM, HEAD_DIM) for b in s["B"]]
        s["seg_start"] = torch.tensor([r[0] for r in requests], dtype=torch.int32).to(dev)
        s["seg_len"] = torch.tensor([r[1] for r in requests], dtype=torch.int32).to(dev)
        s["seg_adapter"] = torch.tensor([r[2] for r in requests], dtype=torch.int64).to(dev)
        s["longest"] = max([r[1] for r in requests], default=1)
    elif via in ("step", "layers", "graph", "rope"):
        s["ops"] = sl.LoraBatchOps(s["start"], s["len"], s["loc"], s["scale"], s["A"], s["B"], s["max_rank"])
        s["ops"].prepare(s["ids"])
    if via in ("graph", "rope"):
        base = [[t.clone() for t in ys] for ys in s["y"]]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _layers(s)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"], stream=side):
            _layers(s)
        for ys, bs in zip(s["y"], base):       # what the first run of the layers added is taken out again
            for y, b in zip(ys, bs):
                y.copy_(b)
    return s


def _layers(s):
    ops = s["ops"]
    for layer in range(s["case"]["layers"]):
        q, k, v, o = s["y"][layer]
        if s["case"]["via"] == "rope":
            ops.lora_get_qkv(layer, s["x"][layer], q, k, v, rope=(s["cos"], s["sin"]),
                             kv_dest=(s["kv_rows"], s["kv"][layer][0], s["kv"][layer][1]))
        else:
            ops.lora_get_qkv(layer, s["x"][layer], q, k, v)
        ops.lora_get_o(layer, s["xo"][layer], o)


def run(s):
    """One pass.  The deltas are added to the base outputs in place, so a second pass adds them again."""
    case = s["case"]
    via = case["via"]
    if via == "step":
        s["ops"].prepare(s["ids"])
        _layers(s)
    elif via == "layers":
        _layers(s)
    elif via in ("graph", "rope"):
        s["graph"].replay()
        if via == "rope":
            return {"q_o": [[ys[0], ys[3]] for ys in s["y"]], "kv": s["kv"]}
    elif via == "dispatch":
        for layer in range(case["layers"]):
            for p in range(4):
                x, y, d = s["xo" if p == 3 else "x"][layer], s["y"][layer][p], s["delta"][p]
                sl.dispatch_bgmv(d, x, s["A3"][layer], s["start"], s["len"], s["loc"], s["ids"], p, s["scale"])
                sl.dispatch_bgmv(y, d, s["B3"][layer], s["start"], s["len"], s["loc"], s["ids"], p, s["scale"])
        return {"y": s["y"], "delta": s["delta"]}
    else:
        for layer in range(case["layers"]):
            for p in range(4):
                x, y, d = s["xo" if p == 3 else "x"][layer], s["y"][layer][p], s["delta"][p]
                sl.lora_get_qkvo_fwd_shrink(x, s["A"][layer], d, s["loc"], s["start"], s["len"], s["seg_start"],
                                            s["seg_len"], s["seg_adapter"], case["hidden"], p, s["max_rank"],
                                            s["longest"])
                sl.lora_get_qkvo_fwd_expand(d, s["B"][layer], y, s["scale"], s["loc"], s["start"], s["len"],
                                            s["seg_start"], s["seg_len"], s["seg_adapter"], y.size(1), p,
                                            s["max_rank"], s["longest"])
        return {"y": s["y"], "delta": s["delta"]}
    return {"y": s["y"]}


def work(case):
    """Each distinct adapter's rows, x (once for q, k, v and once for o) and the base outputs read once, the outputs
    written once.  The batch is a typical one: adapters differ from seed to seed."""
    ranks, ids, _ = _batch(case, 1)
    H, K, T = case["hidden"], case["kv"], len(ids)
    dims = [(H, H), (H, K), (H, K), (H, H)]
    rows = sum(ranks[a] * (hi + ho) * 2 for a in set(ids) for hi, ho in dims)
    acts = T * 2 * H * 2 + T * sum(2 * ho * 2 for _, ho in dims)
    flops = sum(2 * ranks[a] * (hi + ho) for a in ids for hi, ho in dims)
    return {"bytes": float((rows + acts) * case["layers"]), "flops": float(flops * case["layers"])}


def tolerance(case):
    # 16-bit results: the intermediate and the output are rounded once each (2^-11 resp. 2^-8 of a value at most); where
    # scale * sum is rounded before it is added, a third time
    return {"rel": 1.5e-3} if case["dtype"] == "fp16" else {"rel": 1.2e-2}


def exact(case, seed):
    """What the first pass on these inputs leaves, in 64 bits and without any rounding between the steps."""
    s = _plain(case, seed)
    H, K, T, R = case["hidden"], case["kv"], s["ids"].numel(), s["max_rank"]
    ids = s["ids"].tolist()
    start, lens, loc = s["start"].tolist(), s["len"].tolist(), s["loc"]
    order = {}
    for t, a in enumerate(ids):
        order.setdefault(a, []).append(t)
    index = {a: torch.tensor(ts, device=loc.device) for a, ts in order.items()}
    ys, deltas = [], []
    for layer in range(case["layers"]):
        outs, deltas = [], []
        for p in range(4):
            x = s["xo" if p == 3 else "x"][layer].double()
            y = s["y"][layer][p].double()
            width = y.size(1)
            delta = torch.zeros((T, R), dtype=torch.float64, device=loc.device)
            for a, ts in index.items():
                r = lens[a] // 4
                rows = loc[start[a] + r * p: start[a] + r * (p + 1)]
                d = x[ts] @ s["A"][layer][rows].double().t()
                b = s["B"][layer][rows].reshape(-1)[: width * r].view(width, r).double()
                delta[ts, :r] = d
                y[ts] += float(s["scale"][a]) * (d @ b.t())
            outs.append(y)
            deltas.append(delta)
        ys.append(outs)
    if case["via"] in ("dispatch", "segments"):
        return {"y": ys, "delta": deltas}
    if case["via"] == "rope":
        kv = []
        for layer in range(case["layers"]):
            q, k, v, _ = ys[layer]
            ys[layer][0] = _rotate(q, s["cos"], s["sin"])
            pair = [torch.zeros((KV_ROWS, K), dtype=torch.float64, device=loc.device) for _ in range(2)]
            pair[0][s["kv_rows"]] = _rotate(k, s["cos"], s["sin"])
            pair[1][s["kv_rows"]] = v
            kv.append(pair)
        return {"q_o": [[y[0], y[3]] for y in ys], "kv": kv}
    return {"y": ys}


def _plain(case, seed):
    """The inputs of ``prepare`` with none of the library's objects made or run."""
    return prepare(dict(case, via="rope_inputs" if case["via"] == "rope" else "inputs"), seed)


def _rotate(t, cos, sin):
    half = HEAD_DIM // 2
    h = t.view(t.size(0), -1, HEAD_DIM)
    c, s = cos.double()[:, None, :], sin.double()[:, None, :]
    lo, hi = h[..., :half], h[..., half:]
    return torch.cat([lo * c - hi * s, lo * s + hi * c], -1).reshape(t.shape)
