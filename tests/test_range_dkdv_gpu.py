"""dK / dV of range attention (key-tile-major kernel): stretches cut into several items, K/V tiles that nobody sees, rows past
G * tokens of a tile, ranges that are not monotone, K/V rows past the last sequence -- against fp32 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from fsa.ops.range_attention import range_attention
from fsa.synthetic import make_cu_seqlens

DEV = "cuda:0"


@pytest.mark.parametrize("seqlens,klens,spare,Hk,G,mode", [
    ([1], [1], 0, 1, 1, "all"),
    ([130, 1, 257], [127, 1, 129], 70, 2, 3, "all"),            # 40 tokens x 3 heads: eight rows of a tile are never loaded
    ([2100], [300], 0, 1, 32, "all"),                           # 525 row tiles of four tokens, cut into stretches
    ([900, 500], [640, 200], 5, 1, 16, "gap"),                  # nobody sees the rows in the middle
    ([1500, 40], [700, 256], 0, 2, 4, "random"),
])
def test_dk_dv(seqlens, klens, spare, Hk, G, mode):
    N, Nk, d = sum(seqlens), sum(klens) + spare, 128
    g = torch.Generator().manual_seed(N + G)
    q, do = (torch.randn(N, Hk * G, d, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    k, v = (torch.randn(Nk, Hk, d, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    lo, hi, t0, k0 = torch.zeros(N, dtype=torch.int32), torch.zeros(N, dtype=torch.int32), 0, 0
    for n, m in zip(seqlens, klens):
        a, b = torch.zeros(n, dtype=torch.int64), torch.full((n,), m - 1)
        if mode == "gap":
            b[: n // 2] = 100
            a[n // 2 :] = m - 60
        elif mode == "random":
            a, b = torch.randint(0, m, (n,), generator=g), torch.randint(0, m, (n,), generator=g)      # empty where a > b
        lo[t0 : t0 + n], hi[t0 : t0 + n] = a + k0, b + k0
        t0, k0 = t0 + n, k0 + m
    lo, hi = lo.to(DEV), hi.to(DEV)
    cu_q, cu_k = make_cu_seqlens(seqlens).to(DEV), make_cu_seqlens(klens).to(DEV)

    got = []
    for _ in range(2):
        ts = [t.clone().requires_grad_(True) for t in (q, k, v)]
        o, _lse = range_attention(*ts, cu_q, cu_k, lo, hi, (max(klens) + 63) // 64 + 1)
        o.backward(do)
        got.append([o.detach()] + [t.grad for t in ts])
    for a, b in zip(*got):
        assert torch.equal(a, b)

    fs = [t.float().requires_grad_(True) for t in (q, k, v)]
    rows = torch.arange(Nk, device=DEV)
    mask = (rows >= lo[:, None]) & (rows <= hi[:, None])
    s = torch.einsum("nhd,mhd->hnm", fs[0], fs[1].repeat_interleave(G, 1)) * d ** -0.5
    p = s.masked_fill(~mask, -1e30).softmax(-1) * mask          # (a row that sees nothing: 0)
    ref = torch.einsum("hnm,mhd->nhd", p, fs[2].repeat_interleave(G, 1))
    ref.backward(do.float())
    for a, b, name in zip(got[0], [ref.detach()] + [t.grad for t in fs], ("o", "dq", "dk", "dv")):
        scale = max(1.0, float(b.abs().max()) / 2.0)
        err = (a.float() - b).abs()
        assert float(err.max()) <= 2e-2 * scale and float(err.mean()) <= 1e-3 * scale, (name, float(err.max()), float(err.mean()), scale)
