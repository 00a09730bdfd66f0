"""The layer's native function where its kernels take the paths of ordinary sizes: more blocks than the selection takes, more output
rows than the merges of a warp per row serve, an index of several launches and cut K/V stretches (tests/test_nsa_layer_gpu.py
is too short for any of these)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from fsa.module.fsa import FlashSparseAttention, RopeConfig
from fsa.module.rope import compute_inv_freq
from fsa.synthetic import make_cu_seqlens

DEV = "cuda:0"
CFG = dict(hidden_size=512, num_q_heads=16, num_kv_heads=4, head_dim=128, kernel_size=32, kernel_stride=16, block_size=64, topk=16,
           init_blocks=1, local_blocks=2, window_size=512)


def _layer(seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    layer = FlashSparseAttention(**CFG, rope_config=RopeConfig(head_dim=CFG["head_dim"])).to(DEV).to(torch.bfloat16)
    with torch.no_grad():
        for p in layer.parameters():
            torch.nn.init.xavier_uniform_(p, generator=g)
        # one element a head: the bias of the compressed keys is then a row of the weight, whatever the order of its sum
        layer.intra_block_pe.zero_()
        layer.intra_block_pe[:, 3, 5] = 1.0
    return layer, g


def _pass(layer, x, cu, seqlens, dy):
    xl = x.clone().requires_grad_(True)
    layer.zero_grad(set_to_none=True)
    y = layer(xl, cu, seqlens)
    y.backward(dy)
    return {"y": y.detach(), "ids": layer.last_topk_idx, "dx": xl.grad, **{n: p.grad for n, p in layer.named_parameters()}}


class _Round(torch.autograd.Function):
    """Rounds to bf16 where the layer keeps a tensor of that type; its gradient passes unrounded."""

    @staticmethod
    def forward(ctx, t):
        return t.to(torch.bfloat16).float()

    @staticmethod
    def backward(ctx, g):
        return g


def _reference(layer, x, seqlens, ids, dy):
    """The layer in fp32 with the ids fed in: dense attention per sequence under the three branches' masks, and autograd."""
    Hq, Hk, d, ks, st, bs, W = (CFG[n] for n in ("num_q_heads", "num_kv_heads", "head_dim", "kernel_size", "kernel_stride", "block_size", "window_size"))
    rd = _Round.apply
    P = {n: p.detach().float().requires_grad_(True) for n, p in layer.named_parameters()}
    xf = x.float().requires_grad_(True)
    freq = compute_inv_freq(RopeConfig(head_dim=d)).to(DEV)
    q, k, v = (rd(xf @ P[f"proj_{n}.weight"].t()).view(x.shape[0], -1, d) for n in "qkv")
    gate = rd(torch.sigmoid(rd(xf @ P["gate.0.weight"].t())))
    bias = rd(torch.einsum("hkd,hkde->he", P["intra_block_pe"], P["compress_key"].view(Hk, ks, d, d)))

    def rope(t, step):
        a = (torch.arange(t.shape[0], device=DEV) * step).float()[:, None] * freq
        c, s = (f(a).to(torch.bfloat16).float()[:, None, :] for f in (torch.cos, torch.sin))
        t1, t2 = t.chunk(2, -1)
        return rd(torch.cat([t1 * c - t2 * s, t1 * s + t2 * c], -1))

    def attend(q, k, v, seen):
        k, v = (t.repeat_interleave(Hq // Hk, 1) for t in (k, v))
        s = torch.einsum("thd,chd->htc", q, k) * d ** -0.5
        p = torch.softmax(s.masked_fill(~seen, float("-inf")), -1).masked_fill(~seen, 0.0)
        return rd(torch.einsum("htc,chd->thd", p, v))

    out, a = [], 0
    for L in seqlens:
        qs, kk, vs = q[a : a + L], k[a : a + L], v[a : a + L]
        win = lambda t: (t.unfold(0, ks, st) if L >= ks else t.new_zeros(0, Hk, d, ks)).transpose(2, 3)  # noqa: E731  [windows, Hk, ks, d]
        ck, cv = (rd(torch.einsum("chkd,hkde->che", win(t), P[w].view(Hk, ks, d, d))) for t, w in ((kk, "compress_key"), (vs, "compress_value")))
        ck = rope(rd(ck + bias), st)
        qs, kr = rope(qs, 1), rope(kk, 1)
        t = torch.arange(L, device=DEV)
        c = torch.arange(ck.shape[0], device=DEV)
        picked = torch.zeros(Hk, L, -(-L // bs) + 1, dtype=torch.bool, device=DEV)
        picked.scatter_(2, ids[:, a : a + L].long() % picked.shape[2], True)                  # (-1: the spare column)
        causal = t[:, None] >= t
        o_cmp = attend(qs, ck, cv, (t[:, None] >= c * st + ks - 1)[None])
        o_sel = attend(qs, kr, vs, (picked[:, :, :-1].repeat_interleave(bs, 2)[:, :, :L] & causal).repeat_interleave(Hq // Hk, 0))
        o_win = attend(qs, kr, vs, (causal & (t[:, None] - t <= W))[None])
        gs = gate[a : a + L, :, None, None]
        out.append(rd(gs[:, 0] * o_cmp + gs[:, 1] * o_sel + gs[:, 2] * o_win))
        a += L
    y = torch.cat(out).flatten(1) @ P["proj_o.weight"].t()
    y.backward(dy.float())
    return {"y": y.detach(), "dx": xf.grad, **{n: p.grad for n, p in P.items()}}


@pytest.mark.parametrize("seqlens", [[1100, 2900, 1365], [2049, 20, 1531]])
def test_native_layer_where_it_selects(seqlens):
    layer, g = _layer(sum(seqlens))
    N = sum(seqlens)
    assert N * CFG["num_q_heads"] >= 24000 and max(seqlens) > 16 * CFG["block_size"]
    x, dy = (torch.randn(N, CFG["hidden_size"], device=DEV, generator=g).to(torch.bfloat16) for _ in range(2))
    cu = make_cu_seqlens(seqlens).to(DEV)
    got = _pass(layer, x, cu, seqlens, dy)
    again = _pass(layer, x, cu, seqlens, dy)
    for n in got:
        assert torch.equal(got[n], again[n]), f"{n}: two passes differ"
    # the same kernels called one by one (a hook on the gate keeps the native function away): the same forward bits
    hook = layer.gate.register_forward_hook(lambda m, i, o: None)
    parts = _pass(layer, x, cu, seqlens, dy)
    hook.remove()
    assert torch.equal(got["ids"], parts["ids"]) and torch.equal(got["y"], parts["y"])
    want = _reference(layer, x, seqlens, got["ids"], dy)
    # A rounding to bf16 is off by up to 2^-9 of a value, about 1.1e-3 in the root mean square, and y, the gradients and their inputs
    # pass up to a dozen: 4e-3 in all, three times that allowed.  A row (a token, or an output of a weight) that lost a K/V tile
    # somewhere is off by about its own size.
    for n, w in want.items():
        err = (got[n].float() - w).norm(dim=-1)
        rel, row = float(err.norm() / w.norm()), float(err.max() / w.norm(dim=-1).square().mean().sqrt())
        assert rel <= 1.2e-2 and row <= 0.25, f"{n}: relative L2 {rel:.2e}, worst row {row:.2e}"


@pytest.mark.parametrize("seqlens", [[1024], [1024, 1, 31, 700], [64, 65, 128, 1023], [72], [517] * 3])
def test_native_layer_of_whole_sequences(seqlens):
    """Sequences of at most topk blocks, where the selection is causal attention and no block is looked for: the ids are those that
    the selection gives, every tensor is near the fp32 layer, and near the same layer with the selection run (a hook keeps the
    native function away)."""
    layer, g = _layer(sum(seqlens) + len(seqlens))
    N = sum(seqlens)
    assert max(seqlens) <= CFG["topk"] * CFG["block_size"]
    x, dy = (torch.randn(N, CFG["hidden_size"], device=DEV, generator=g).to(torch.bfloat16) for _ in range(2))
    cu = make_cu_seqlens(seqlens).to(DEV)
    got, again = _pass(layer, x, cu, seqlens, dy), _pass(layer, x, cu, seqlens, dy)
    with torch.no_grad():
        assert torch.equal(layer(x, cu, seqlens), got["y"])
    hook = layer.gate.register_forward_hook(lambda m, i, o: None)
    parts = _pass(layer, x, cu, seqlens, dy)
    hook.remove()
    assert torch.equal(got["ids"], parts["ids"])
    want = _reference(layer, x, seqlens, got["ids"], dy)
    # (bounds of the test above; a row beside the root mean square of the rows: short sequences have rows of few large gradients)
    for n, w in want.items():
        assert torch.equal(got[n], again[n]), f"{n}: two passes differ"
        err, other = ((t[n].float() - w).norm() / w.norm() for t in (got, parts))
        assert float(err) <= 1.2e-2 and float(err) <= 1.1 * float(other) + 1e-4, f"{n}: relative L2 {float(err):.2e}, with the selection run {float(other):.2e}"
