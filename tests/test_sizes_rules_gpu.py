"""Sizes at which the size rules of the launches change: short and mid-sized tile lists of the selected-attention kernels
(the scheduling runs of the backward get shorter with the list), and long rows of K/V tiles of range attention."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from fsa.ops.FSA_topk_sparse_attention import sel_attn_bwd, sel_attn_fwd
from fsa.ops.range_attention import compressed_attention_core
from fsa.synthetic import make_cu_seqlens, make_qkv, make_topk_idx
from oracle.sel_attn_oracle import sel_attn_forward_backward

DEV = "cuda:0"


def _close(got, ref, name):
    err = (got.float().cpu() - ref).abs()
    scale = max(1.0, float(ref.abs().max()) / 2.0)
    assert float(err.max()) <= 2e-2 * scale, f"{name}: max-abs {float(err.max()):.3e}"
    assert float(err.mean()) <= 1e-3 * scale, f"{name}: mean-abs {float(err.mean()):.3e}"


@pytest.mark.parametrize("seqlens,Hk,G,T,d,bs", [([1], 1, 1, 2, 128, 64), ([1100], 1, 2, 16, 128, 64), ([2371, 200], 2, 2, 16, 128, 64),
                                                 ([1500, 33], 2, 8, 16, 128, 64), ([2371, 200, 65], 2, 2, 8, 128, 128),
                                                 ([1100, 129], 2, 4, 16, 64, 64), ([900, 257], 1, 4, 4, 64, 256)])
def test_scheduling_runs_of_short_lists(seqlens, Hk, G, T, d, bs):
    N = sum(seqlens)
    q, k, v, do = make_qkv(N, Hk * G, Hk, d, 300 + N)
    idx, cu = make_topk_idx(seqlens, Hk, T, bs, 301 + N), make_cu_seqlens(seqlens)
    ref = sel_attn_forward_backward(q, k, v, do, idx, bs, cu, d ** -0.5)
    qc, kc, vc, dc, ic, cc = (x.to(DEV) for x in (q, k, v, do, idx, cu))
    o, lse, ws = sel_attn_fwd(qc, kc, vc, ic, bs, cc, d ** -0.5, check_status=True)
    grads = sel_attn_bwd(qc, kc, vc, o, lse, dc, ic, bs, cc, d ** -0.5, ws, check_status=True)
    for name, got, want in zip(("o", "dq", "dk", "dv"), (o, *grads), (ref[0], *ref[2:])):
        _close(got, want, name)


def test_long_rows_are_the_same_every_time():
    """Row warps run up to two P V products ahead of the tensor core: the last products must be waited for all the same."""
    N, ks, st = 20011, 32, 16
    C = (N - ks) // st + 1
    g = torch.Generator(device=DEV).manual_seed(1)
    q, k, v = (torch.randn(n, h, 128, device=DEV, generator=g).to(torch.bfloat16) for n, h in ((N, 32), (C, 8), (C, 8)))
    cu_q, cu_k = (torch.tensor([0, n], dtype=torch.int32, device=DEV) for n in (N, C))
    o0, lse0 = compressed_attention_core(q, k, v, ks, st, cu_q, cu_k, C)
    for _ in range(4):
        o, lse = compressed_attention_core(q, k, v, ks, st, cu_q, cu_k, C)
        assert torch.equal(o, o0) and torch.equal(lse, lse0)


@pytest.mark.parametrize("d,bs,T,dtype", [(64, 32, 8, torch.float16), (128, 64, 16, torch.bfloat16), (128, 256, 2, torch.bfloat16), (256, 128, 3, torch.bfloat16)])
def test_row_strides_beyond_32_bit_offsets(d, bs, T, dtype):
    """q and dO whose rows lie more than 2^34 elements apart in all: the pipelined kernels address rows by 32-bit offsets in units of 8
    elements and leave these to the unpipelined ones (34 GB are reserved for them, of which only the rows are touched)."""
    seqlens, Hk, G = [333, 80], 2, 2
    N, Hq = sum(seqlens), Hk * G
    q, k, v, do = (t.to(dtype) for t in make_qkv(N, Hq, Hk, d, 77 + d))
    idx, cu = make_topk_idx(seqlens, Hk, T, bs, 78 + d), make_cu_seqlens(seqlens)
    step = (2 ** 34 // N + 8) // 8 * 8
    assert step * N >= 2 ** 34
    try:
        room = torch.empty(N * step, dtype=dtype, device=DEV)
    except torch.OutOfMemoryError:
        pytest.skip("less than 34 GB free")
    far = []
    for i, t in enumerate((q, do)):
        far.append(room.as_strided((N, Hq, d), (step, d, 1), i * Hq * d))
        far[-1].copy_(t)
    ref = sel_attn_forward_backward(q, k, v, do, idx, bs, cu, d ** -0.5)
    kc, vc, ic, cc = (x.to(DEV) for x in (k, v, idx, cu))
    o, lse, ws = sel_attn_fwd(far[0], kc, vc, ic, bs, cc, d ** -0.5, check_status=True)
    # q far away alone, dO alone, and both
    for qx, dx in ((far[0], do.to(DEV)), (q.to(DEV), far[1]), tuple(far)):
        grads = sel_attn_bwd(qx, kc, vc, o, lse, dx, ic, bs, cc, d ** -0.5, ws, check_status=True)
        for name, got, want in zip(("o", "dq", "dk", "dv"), (o, *grads), (ref[0], *ref[2:])):
            _close(got, want, name)
