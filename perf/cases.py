"""What a user of this package has it do, as cases that can be timed: the selected-attention operator (training and
prefill), the whole FlashSparseAttention layer (training and prefill) and the decode step (eager and from a CUDA graph).

Sizes are those of the package's benchmark configurations and tests, or lie between them; ``draw`` spreads over the same
ranges.  Sequence lengths are texts ("300,212") so that a case is a dict of plain values.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "flash-sparse-attention_b200"))

from fsa.module.fsa import FlashSparseAttention, RopeConfig  # noqa: E402
from fsa.ops import FSA_topk_sparse_attention  # noqa: E402
from fsa_preview.module import FlashSparseAttentionDecode, FlashSparseAttentionDecodeKernel, GraphedStep  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
# NSA settings of the benchmark's layer and decode configurations
NSA = dict(kernel_size=32, kernel_stride=16, block_size=64, topk=16, init_blocks=1, local_blocks=2, window_size=512)
GROW = 1024      # tokens a decode cache has room for beyond the lengths that it starts with


def _sel(name, seqlens, Hk, G, d, bs, T, dtype, train):
    return dict(name=name, kind="sel", seqlens=seqlens, Hk=Hk, G=G, d=d, bs=bs, T=T, dtype=dtype, train=train)


def _layer(name, seqlens, hidden, Hq, Hk, d, train):
    return dict(name=name, kind="layer", seqlens=seqlens, hidden=hidden, Hq=Hq, Hk=Hk, d=d, train=train)


def _decode(name, seqlens, hidden, Hq, Hk, d, proj, graph):
    return dict(name=name, kind="decode", seqlens=seqlens, hidden=hidden, Hq=Hq, Hk=Hk, d=d, proj=proj, graph=graph)


def listed():
    return [
        # the operator alone, forward + backward: two short packed sequences, as in a fine-tuning micro-batch or a test
        _sel("sel_train_300_212", "300,212", 2, 2, 128, 64, 8, "bf16", True),
        # the headline configuration: 64K tokens in four sequences
        _sel("sel_train_4x16384", "16384,16384,16384,16384", 4, 2, 128, 64, 16, "bf16", True),
        # the other block size that is used (128 keys, top-8), no grouping of heads, ragged lengths
        _sel("sel_train_bk128_ragged", "9001,4100,7777,130", 4, 1, 128, 128, 8, "bf16", True),
        # the wide heads of the group-size sweep
        _sel("sel_train_d256", "16384", 4, 2, 256, 64, 16, "bf16", True),
        # forward only, as in prefill with an own layer around it: many ragged sequences, one of a single token, fp16
        _sel("sel_prefill_ragged_fp16", "7001,1,333,4097,2500,64,1999", 8, 4, 128, 64, 16, "fp16", False),
        # a training step of the layer at the benchmark's size
        _layer("layer_train_2x32768", "32768,32768", 4096, 32, 8, 128, True),
        # a training step on a short ragged batch, heads split over two GPUs (this is one GPU's share)
        _layer("layer_train_ragged", "3001,777,2049,1365", 4096, 16, 4, 128, True),
        # prefill of one short prompt: the time to the first token of an interactive request
        _layer("layer_prefill_517", "517", 4096, 32, 8, 128, False),
        # prefill of a batch of long prompts
        _layer("layer_prefill_long", "20011,12345", 4096, 32, 8, 128, False),
        # one interactive request being decoded, launched kernel by kernel
        _decode("decode_1x8191_eager", "8191", 4096, 32, 8, 128, True, False),
        # a small batch of requests of mixed lengths, attention without the projections, from a CUDA graph
        _decode("decode_8_ragged_graph", "40003,517,12000,3333,28672,90,7001,16385", 4096, 32, 8, 128, False, True),
        # the benchmark's decode configuration: a full batch with long caches
        _decode("decode_64x131072_graph", ",".join(["131072"] * 64), 4096, 32, 8, 128, False, True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _split(rng, total, parts):
    """``total`` tokens in ``parts`` ragged pieces of at least one token."""
    parts = min(parts, total)
    cuts = sorted(rng.sample(range(1, total), parts - 1)) if parts > 1 else []
    return ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]))


def draw(rng):
    kind = rng.choice(["sel", "sel", "layer", "decode"])
    if kind == "sel":
        train = rng.random() < 0.6
        d = rng.choice([128, 128, 128, 64, 256])
        bs, T = rng.choice([(64, 16), (64, 16), (128, 8), (32, 16), (64, 8)])
        Hk, G = rng.choice([1, 2, 4, 8]), rng.choice([1, 2, 4, 8, 16])
        most = 65536 * 8 * 128 // (Hk * G * d)                     # the headline configuration's tokens x heads x head size
        seqlens = _split(rng, _log_int(rng, 256, min(most, 65536)), rng.choice([1, 1, 2, 4, 8]))
        c = _sel("", seqlens, Hk, G, d, bs, T, rng.choice(["bf16", "bf16", "fp16"]), train)
    elif kind == "layer":
        hidden, Hq, Hk, d = rng.choice([(4096, 32, 8, 128), (4096, 16, 4, 128), (4096, 8, 2, 128), (2048, 16, 4, 128), (1024, 16, 4, 64)])
        seqlens = _split(rng, _log_int(rng, 400, 40000), rng.choice([1, 1, 2, 4]))
        c = _layer("", seqlens, hidden, Hq, Hk, d, rng.random() < 0.5)
    else:
        batch = _log_int(rng, 1, 64)
        longest = _log_int(rng, 600, 65536)
        lens = [longest] + [_log_int(rng, max(40, longest // 20), longest) for _ in range(batch - 1)]
        hidden, Hq, Hk, d = rng.choice([(4096, 32, 8, 128), (4096, 32, 8, 128), (4096, 16, 4, 128), (1024, 16, 4, 64)])
        proj = rng.random() < 0.5
        c = _decode("", ",".join(str(n) for n in lens), hidden, Hq, Hk, d, proj, not proj and rng.random() < 0.7)
    del c["name"]
    return c


def _lens(case):
    return [int(n) for n in case["seqlens"].split(",")]


def _cu(lens, dev):
    return torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=dev)


def _block_ids(lens, Hk, T, bs, g, dev):
    """Causal block ids as the block selection gives them: block 0, the token's own block and earlier blocks (here a
    uniform sample without replacement), ascending, padded with -1."""
    out = []
    for L in lens:
        nb = -(-L // bs)
        ids = torch.arange(nb, device=dev)
        for a in range(0, L, 4096):
            own = (torch.arange(a, min(L, a + 4096), device=dev) // bs)[:, None]
            key = torch.rand(Hk, own.shape[0], nb, device=dev, generator=g)
            key.masked_fill_((ids > own), -1.0)
            key.masked_fill_((ids == own) | (ids == 0), 2.0)
            val, pick = key.topk(min(T, nb), dim=-1)
            pick = pick.masked_fill(val < 0, 1 << 30).sort(dim=-1).values
            pick = pick.masked_fill(pick == 1 << 30, -1).to(torch.int32)
            out.append(torch.nn.functional.pad(pick, (0, T - pick.shape[-1]), value=-1))
    return torch.cat(out, 1).contiguous()


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(int(seed))
    lens = _lens(case)
    N = sum(lens)

    def normal(*shape, std=1.0, dtype=torch.bfloat16):
        return torch.empty(shape, dtype=dtype, device=dev).normal_(0, std, generator=g)

    if case["kind"] == "sel":
        dt, Hk, d = DTYPES[case["dtype"]], case["Hk"], case["d"]
        Hq = Hk * case["G"]
        s = dict(q=normal(N, Hq, d, dtype=dt), k=normal(N, Hk, d, dtype=dt), v=normal(N, Hk, d, dtype=dt), cu=_cu(lens, dev),
                 idx=_block_ids(lens, Hk, case["T"], case["bs"], g, dev))
        if case["train"]:
            s["do"] = normal(N, Hq, d, dtype=dt)
    else:
        hidden, Hq, Hk, d = case["hidden"], case["Hq"], case["Hk"], case["d"]
        rope = RopeConfig(max_position_embeddings=131072, head_dim=d, rope_theta=500000.0)
        with torch.device("meta"):      # no host initialisation: the weights are drawn on the GPU below
            if case["kind"] == "layer":
                mod = FlashSparseAttention(hidden, Hq, Hk, d, *NSA.values(), rope_config=rope)
            elif case["proj"]:
                mod = FlashSparseAttentionDecode(hidden, Hq, Hk, d, *NSA.values(), rope_config=rope)
            else:
                mod = FlashSparseAttentionDecodeKernel(Hq * d, Hq, Hk, d, *NSA.values())
        mod = mod.to_empty(device=dev).to(torch.bfloat16)
        if hasattr(mod, "rope"):
            mod.rope = type(mod.rope)(rope)
        with torch.no_grad():
            for p in mod.parameters():
                torch.nn.init.xavier_uniform_(p, generator=g)       # as the layer initialises itself
        s = dict(mod=mod)
        if case["kind"] == "layer":
            s.update(x=normal(N, hidden), cu=_cu(lens, dev), lens=lens)
            if case["train"]:
                s["dy"] = normal(N, hidden)
        else:
            B = len(lens)
            cache = mod.new_cache(B, max(lens) + GROW, device=dev)
            for t in (cache.k, cache.v, cache.cmp_k, cache.cmp_v, cache.k_tail, cache.v_tail):
                t.normal_(0, 1, generator=g)
            cache.host_len = list(lens)
            cache.seq_len.copy_(torch.tensor(lens, dtype=torch.int32))
            new = [normal(B, hidden)] if case["proj"] else [normal(B, Hq, d), normal(B, Hk, d), normal(B, Hk, d)]
            s.update(cache=cache, lens=lens, start=cache.seq_len.clone(), new=new)
            s["graph"] = GraphedStep(mod.step, cache, new) if case["graph"] else None
    s["case"] = case
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "sel":
        if not case["train"]:
            return FSA_topk_sparse_attention(s["q"], s["k"], s["v"], s["idx"], case["bs"], s["cu"])
        q, k, v = (s[n].detach().requires_grad_(True) for n in "qkv")
        o = FSA_topk_sparse_attention(q, k, v, s["idx"], case["bs"], s["cu"])
        o.backward(s["do"])
        return o.detach(), q.grad, k.grad, v.grad
    if case["kind"] == "layer":
        mod = s["mod"]
        if not case["train"]:
            with torch.no_grad():
                return mod(s["x"], s["cu"], s["lens"])
        x = s["x"].detach().requires_grad_(True)
        mod.zero_grad(set_to_none=True)
        y = mod(x, s["cu"], s["lens"])
        y.backward(s["dy"])
        return {"y": y.detach(), "dx": x.grad, **{n: p.grad for n, p in mod.named_parameters()}}
    cache = s["cache"]
    if max(cache.host_len) >= cache.max_len:        # the cache is full: its slots go to requests of the first lengths again
        cache.host_len = list(s["lens"])
        cache.seq_len.copy_(s["start"])
    y = s["graph"](*s["new"]) if s["graph"] is not None else s["mod"].step(*s["new"], cache)
    # the updated state too; the last row of every cache buffer is a spare one that takes writes meant for nobody
    new = {n: getattr(cache, n)[:-1] for n in ("k_tail", "v_tail", "cmp_k", "cmp_v")}
    return {"y": y, "seq_len": cache.seq_len, **new}


def _sel_pairs(lens, bs, T):
    """(token, key) pairs of one head that the selection attends: full earlier blocks and the own block up to the token."""
    total = 0
    for L in lens:
        for b in range(-(-L // bs)):
            n = min(bs, L - b * bs)
            total += n * (min(T, b + 1) - 1) * bs + n * (n + 1) // 2
    return total


def _num_cmp(L):
    return (L - NSA["kernel_size"]) // NSA["kernel_stride"] + 1 if L >= NSA["kernel_size"] else 0


def work(case):
    lens, Hk, d = _lens(case), case["Hk"], case["d"]
    N = sum(lens)
    if case["kind"] == "sel":
        Hq = Hk * case["G"]
        P = Hq * _sel_pairs(lens, case["bs"], case["T"])
        io = 2 * d * (2 * N * Hq + 2 * N * Hk) + 4 * Hk * N * case["T"]            # q, o, k, v and the ids
        if not case["train"]:
            return {"bytes": io, "flops": 4 * d * P}
        return {"bytes": io + 2 * d * (2 * N * Hq + 2 * N * Hk), "flops": 14 * d * P}     # and dO, dq, dk, dv
    hidden, Hq = case["hidden"], case["Hq"]
    ks, st, W = NSA["kernel_size"], NSA["kernel_stride"], NSA["window_size"]
    weights = hidden * (Hq * d + 2 * Hk * d) + Hq * d * hidden + 3 * hidden
    comp = 2 * Hk * ks * d * d                                                     # both compression weights
    if case["kind"] == "layer":
        cmp_pairs = sum(sum(range(1, _num_cmp(L) + 1)) * st - (st - 1 - (L - ks) % st) * _num_cmp(L) for L in lens if L >= ks)
        win_pairs = sum(L * (W + 1) - W * (W + 1) // 2 if L > W else L * (L + 1) // 2 for L in lens)
        P = Hq * (cmp_pairs + win_pairs + _sel_pairs(lens, NSA["block_size"], NSA["topk"]))
        proj = 2 * N * weights + 2 * sum(_num_cmp(L) for L in lens) * comp
        if not case["train"]:
            return {"bytes": 2 * (weights + comp + 2 * N * hidden), "flops": proj + 4 * d * P}
        return {"bytes": 2 * (2 * (weights + comp) + 4 * N * hidden), "flops": 3 * proj + 14 * d * P}
    # decode: the visible compressed rows, the selected blocks and the part of the window that they do not cover, of K and V
    keys = 0
    for L in lens:
        sel = min(NSA["topk"] * NSA["block_size"], L + 1)
        keys += _num_cmp(L + 1) + min(L + 1, sel + max(0, W + 1 - NSA["local_blocks"] * NSA["block_size"]))
    B = len(lens)
    weights = weights if case["proj"] else 3 * Hq * d
    return {"bytes": 2 * (2 * keys * Hk * d + weights + B * (2 * hidden + 2 * Hk * d)), "flops": 4 * d * Hq * keys + 2 * B * weights}


def tolerance(case):
    # bf16 / fp16 results of bf16 / fp16 inputs with 32-bit sums; a layer's gradients pass several such roundings, and a near
    # tie in its block selection moves single rows
    if case["kind"] == "layer":
        return {"rel": 2e-2, "max": 0.9} if case["train"] else {"rel": 1e-2, "max": 0.6}
    return {"rel": 1e-2, "max": 0.5}
