"""Calls that the native functions do not serve run as their parts: weights in another memory order give the results of ordinary ones,
and what no path takes raises."""
import copy

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from fsa.module.fsa import FlashSparseAttention, RopeConfig
from fsa_preview.module import FlashSparseAttentionDecode, FlashSparseAttentionDecodeKernel
from fsa_preview.ops.decode import nsa_decode_mixed

DEV = "cuda:0"


def _reordered(p):
    """The same values in another memory order."""
    return torch.nn.Parameter(p.detach().transpose(0, -1).contiguous().transpose(0, -1))


def _layer():
    torch.manual_seed(7)
    layer = FlashSparseAttention(256, 4, 2, 128, 32, 16, 64, 6, 1, 2, 128, rope_config=RopeConfig(head_dim=128)).to(DEV).to(torch.bfloat16)
    with torch.no_grad():       # (the bias of the compressed keys is one row of the weight, whatever the order of its sum)
        layer.intra_block_pe.zero_()
        layer.intra_block_pe[:, 0, 0] = 1.0
    x = torch.randn(700, 256, device=DEV).to(torch.bfloat16)
    return layer, x, torch.tensor([0, 500, 700], dtype=torch.int32, device=DEV)


def _holder(layer, name):
    owner, _, leaf = name.rpartition(".")
    return layer.get_submodule(owner), leaf


NAMES = ["proj_q.weight", "proj_k.weight", "proj_v.weight", "gate.0.weight", "compress_key", "compress_value", "intra_block_pe"]


@pytest.mark.parametrize("name", NAMES)
def test_layer_takes_a_weight_in_another_memory_order(name):
    layer, x, cu = _layer()
    y = layer(x, cu, [500, 200])
    ids = layer.last_topk_idx
    owner, leaf = _holder(layer, name)
    setattr(owner, leaf, _reordered(getattr(owner, leaf)))
    assert not getattr(owner, leaf).is_contiguous()
    y2 = layer(x, cu, [500, 200])
    assert torch.equal(ids, layer.last_topk_idx)
    # (a library GEMM may sum another order of a weight otherwise: 2^-8 of the largest output)
    assert float((y2 - y).abs().max()) <= 2.0 ** -8 * float(y.abs().max())
    y2.float().square().sum().backward()
    assert getattr(owner, leaf).grad is not None


@pytest.mark.parametrize("name", NAMES)
def test_layer_refuses_a_weight_of_another_type(name):
    layer, x, cu = _layer()
    owner, leaf = _holder(layer, name)
    setattr(owner, leaf, torch.nn.Parameter(getattr(owner, leaf).detach().float()))
    with pytest.raises((RuntimeError, AssertionError)):
        layer(x, cu, [500, 200])


@pytest.mark.parametrize("name", ["compress_key", "compress_value", "intra_block_pe"])
def test_layer_refuses_a_weight_of_another_shape(name):
    layer, x, cu = _layer()
    owner, leaf = _holder(layer, name)
    setattr(owner, leaf, torch.nn.Parameter(getattr(owner, leaf).detach()[:, :-8].contiguous()))
    with pytest.raises((ValueError, RuntimeError, AssertionError)):
        layer(x, cu, [500, 200])


def test_layer_keeps_a_scaled_or_hooked_rotation():
    layer, x, cu = _layer()
    y = layer(x, cu, [500, 200])
    scaled = copy.deepcopy(layer)
    scaled.rope.attention_scaling = 0.5
    calls = []
    layer.rope.register_forward_hook(lambda m, i, o: calls.append(1))
    assert torch.equal(layer(x, cu, [500, 200]), y) and len(calls) == 3
    assert not torch.equal(scaled(x, cu, [500, 200]), y)


@pytest.mark.parametrize("kind", ["list", "tuple", "array", "tensor", "none"])
@pytest.mark.parametrize("lens", [[500, 200], [300, 0, 400], [0, 31, 669, 0]])
def test_layer_takes_lengths_of_any_kind(kind, lens):
    layer, x, _ = _layer()
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
    given = dict(list=lens, tuple=tuple(lens), array=np.asarray(lens), tensor=torch.tensor(lens), none=None)[kind]

    def grads():
        xl = x.clone().requires_grad_(True)
        layer.zero_grad(set_to_none=True)
        y = layer(xl, cu, given)
        y.backward(x.flip(0) if y.shape == x.shape else torch.ones_like(y))
        return [y.detach(), layer.last_topk_idx, xl.grad] + [p.grad for p in layer.parameters()]

    got = grads()
    hook = layer.gate.register_forward_hook(lambda m, i, o: None)
    want = grads()
    hook.remove()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    for a, b in zip(got[2:], want[2:]):       # (sums of the branches' gradients rounded once here, at every sum there)
        assert float((a.float() - b.float()).norm()) <= 1e-2 * float(b.float().norm())


NSA = dict(kernel_size=32, kernel_stride=16, block_size=64, topk=8, init_blocks=1, local_blocks=2, window_size=100)


def _decode(hidden, Hq, Hk, D, lens, max_len, **over):
    torch.manual_seed(8)
    cfg = {**NSA, **over}
    mod = (FlashSparseAttentionDecode(hidden, Hq, Hk, D, rope_config=RopeConfig(head_dim=D), **cfg) if hidden
           else FlashSparseAttentionDecodeKernel(Hq * D, Hq, Hk, D, **cfg)).to(DEV).to(torch.bfloat16)
    with torch.no_grad():
        for p in mod.parameters():
            p.normal_(0, 0.05)

    def cache(dtype=torch.bfloat16):
        torch.manual_seed(9)
        c = mod.new_cache(len(lens), max_len, dtype=dtype, device=DEV)
        for t in c.buffers()[:6]:
            t.normal_()
        c.host_len = list(lens)
        c.seq_len.copy_(torch.tensor(lens, dtype=torch.int32))
        return c

    def new():
        B = len(lens)
        shapes = [(B, hidden)] if hidden else [(B, Hq, D), (B, Hk, D), (B, Hk, D)]
        return [torch.randn(s, device=DEV).to(torch.bfloat16) for s in shapes]

    return mod, cache, new


@pytest.mark.parametrize("hidden,Hq,Hk,D,lens,max_len,over", [
    (0, 2, 1, 64, [30, 63], 200, dict(kernel_size=4, kernel_stride=4, block_size=32)),     # a window that is not a multiple of 8
    (0, 2, 1, 64, [200, 143], 400, dict(kernel_size=144, kernel_stride=16)),               # one above 128
    (260, 2, 2, 64, [70, 90, 31], 200, {}),                                                # a gate input that is not a multiple of 8
    (0, 16, 1, 64, [700, 652000], 652800, {}),                                             # more merge weights than shared memory holds
])
def test_decode_sizes_outside_the_native_step_run_as_parts(hidden, Hq, Hk, D, lens, max_len, over):
    mod, cache, new = _decode(hidden, Hq, Hk, D, lens, max_len, **over)
    a, b = cache(), cache()
    for _ in range(3):
        ins = new()
        y, ids = mod.step(*ins, a), mod.last_topk_idx
        hook = mod.gate.register_forward_hook(lambda *x: None)
        ref = mod.step(*ins, b)
        hook.remove()
        assert torch.equal(y, ref) and torch.equal(ids, mod.last_topk_idx) and bool(torch.isfinite(y).all())
    assert a.host_len == b.host_len == [n + 3 for n in lens]
    for x, z in zip(a.buffers(), b.buffers()):
        assert torch.equal(x, z)


@pytest.mark.parametrize("name", ["proj_q.weight", "proj_v.weight", "proj_o.weight", "gate.0.weight", "compress_key", "compress_value", "intra_block_pe"])
def test_decode_takes_a_weight_in_another_memory_order_as_parts(name):
    mod, cache, new = _decode(256, 4, 2, 128, [95, 130], 300)
    owner, leaf = _holder(mod, name)
    setattr(owner, leaf, _reordered(getattr(owner, leaf)))
    a, b, ins = cache(), cache(), new()
    y = mod.step(*ins, a)
    hook = mod.gate.register_forward_hook(lambda *x: None)
    assert torch.equal(mod.step(*ins, b), y)
    hook.remove()
    assert a.host_len == b.host_len == [96, 131]


def test_decode_mixed_keeps_its_options_as_parts():
    mod, cache, new = _decode(0, 4, 2, 128, [95, 130], 300)
    c, (q, _, _) = cache(), new()
    gate = torch.rand(2, 3, device=DEV).to(torch.bfloat16)
    args = (q, c.k, c.v, c.cmp_k, c.cmp_v, c.seq_len, c.seq_row0, c.cmp_row0, gate)
    y, ids = nsa_decode_mixed(*args, max_len=300, **NSA)
    y2, ids2 = nsa_decode_mixed(*args, max_len=300, cmp_chunk=64, shard=None, ops=None, **NSA)
    assert torch.equal(ids, ids2) and float((y - y2).abs().max()) <= 2.0 ** -6 * float(y.abs().max())


@pytest.mark.parametrize("hidden", [256, 0])
def test_decode_refuses_what_does_not_fit_the_cache_and_leaves_it_alone(hidden):
    mod, cache, new = _decode(hidden, 4, 2, 128, [95, 130, 64], 300)
    c = cache()
    before = [t.clone() for t in c.buffers()]
    ins = new()
    short, wide = [t[:2] for t in ins], [torch.cat([t, t]) for t in ins]
    other = [t[..., :-64].contiguous() for t in ins]
    for bad in (short, wide, other):
        with pytest.raises(ValueError):
            mod.step(*bad, c)
    half = cache(torch.float16)
    with pytest.raises((RuntimeError, ValueError, AssertionError)):
        mod.step(*ins, half)
    assert c.host_len == half.host_len == [95, 130, 64]
    for x, z in zip(c.buffers(), before):
        assert torch.equal(x, z)
    assert torch.equal(half.seq_len, before[6])


def test_decode_under_autocast_runs_as_parts():
    """Weights of 32 bits under autocast: the parts' products take 16-bit operands."""
    mod, cache, new = _decode(256, 4, 2, 128, [95, 130], 300)
    wide = copy.deepcopy(mod).float()
    a, b, ins = cache(), cache(), new()
    y = mod.step(*ins, a)
    with torch.autocast("cuda", torch.bfloat16):
        y2 = wide.step(*ins, b)
    assert float((y2 - y).abs().max()) <= 2.0 ** -6 * float(y.abs().max()) and b.host_len == [96, 131]
