"""The merges on resident warps (many rows) against the ones of a warp per row (few rows): the sequences of a batch together and
one by one give the same o, lse and dQ bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from fsa.ops.FSA_topk_sparse_attention import sel_attn_bwd, sel_attn_fwd
from fsa.synthetic import make_cu_seqlens, make_qkv, make_topk_idx

DEV = "cuda:0"


@pytest.mark.parametrize("seqlens,Hk,G,T,d,bs,dtype", [([1499, 1000, 502], 2, 4, 16, 128, 64, "bf16"), ([2999, 1, 70], 1, 8, 9, 64, 32, "fp16"),
                                                       ([1300, 1333], 3, 4, 8, 128, 128, "bf16"), ([1100, 900], 2, 7, 4, 128, 256, "bf16"),
                                                       ([1700, 1350], 8, 1, 3, 128, 64, "fp16"), ([2701, 2600], 1, 5, 16, 64, 64, "bf16"),
                                                       ([1999, 1001, 1], 3, 3, 7, 64, 128, "fp16")])
def test_resident_merge(seqlens, Hk, G, T, d, bs, dtype):
    N = sum(seqlens)
    assert N * Hk * G >= 24000 > max(seqlens) * Hk * G
    dt = torch.bfloat16 if dtype == "bf16" else torch.float16
    q, k, v, do = (x.to(dt).to(DEV) for x in make_qkv(N, Hk * G, Hk, d, 5))
    idx = make_topk_idx(seqlens, Hk, T, bs, 6).to(DEV)

    def run(a, b):
        cu = make_cu_seqlens(seqlens if b - a == N else [b - a]).to(DEV)
        i = idx[:, a:b].contiguous()
        o, lse, ws = sel_attn_fwd(q[a:b], k[a:b], v[a:b], i, bs, cu, d ** -0.5, check_status=True)
        dq, _, _ = sel_attn_bwd(q[a:b], k[a:b], v[a:b], o, lse, do[a:b], i, bs, cu, d ** -0.5, ws, check_status=True)
        return o, lse, dq

    o, lse, dq = run(0, N)
    a = 0
    for n in seqlens:
        o1, lse1, dq1 = run(a, a + n)
        assert torch.equal(o[a : a + n], o1) and torch.equal(lse[:, a : a + n], lse1) and torch.equal(dq[a : a + n], dq1)
        a += n


@pytest.mark.parametrize("seqlens,Hk,G,T,d", [([1500, 1503], 2, 4, 12, 128), ([1500, 1503], 2, 4, 13, 128), ([2000, 1100], 8, 1, 15, 64),
                                              ([1999, 1300], 1, 8, 1, 64), ([2701, 1400], 2, 3, 14, 64)])
def test_resident_merge_row_counts(seqlens, Hk, G, T, d):
    """Counts of partial rows around the one from which all 16 are taken without a test, and tokens that have fewer than that."""
    test_resident_merge(seqlens, Hk, G, T, d, 64, "bf16")
