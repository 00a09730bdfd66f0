"""Calls that the native functions do not serve run as their parts: weights in another memory order give the results of ordinary ones,
and what no path takes raises."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu

from fsa.module.fsa import FlashSparseAttention, RopeConfig

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
