"""The native decode step against the same step composed of the separate operators (a hook on the gate makes the modules take
that path), at the sizes where its kernels change shape: rows of x around one and two MMA tiles, more sequences than one turn
of the compressor takes, both head sizes, groups up to 16; and the split reduction of the prefill compressor."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from fsa.module.rope import RopeConfig  # noqa: E402
from fsa.ops.linear_compress import linear_compress  # noqa: E402
from fsa_preview.module import FlashSparseAttentionDecode, FlashSparseAttentionDecodeKernel  # noqa: E402

DEV = "cuda:0"


def _close(got, ref, what):
    got, ref = got.float(), ref.float()
    scale = max(1.0, float(ref.abs().max()) / 2)
    err = (got - ref).abs()
    assert float(err.max()) <= 2e-2 * scale and float(err.mean()) <= 1e-3 * scale, f"{what}: {float(err.max()):.3e} {float(err.mean()):.3e}"


@pytest.mark.parametrize("B,Hk,G,D,hidden,proj,dtype", [(1, 2, 4, 128, 256, True, torch.bfloat16), (9, 2, 1, 64, 512, True, torch.float16),
                                                        (17, 1, 16, 128, 256, True, torch.bfloat16), (11, 2, 3, 128, 264, True, torch.bfloat16),
                                                        (33, 2, 2, 128, 0, False, torch.bfloat16)])
def test_native_step_matches_the_composed_step(B, Hk, G, D, hidden, proj, dtype):
    torch.manual_seed(B * 100 + G)
    cfg = dict(kernel_size=32, kernel_stride=16, block_size=64, topk=8, init_blocks=1, local_blocks=2, window_size=100)
    Hq = Hk * G
    if proj:
        mod = FlashSparseAttentionDecode(hidden, Hq, Hk, D, rope_config=RopeConfig(head_dim=D), **cfg)
    else:
        mod = FlashSparseAttentionDecodeKernel(Hq * D, Hq, Hk, D, **cfg)
    mod = mod.to(DEV).to(dtype)
    with torch.no_grad():
        for p in mod.parameters():
            p.normal_(0, 0.05)
    lens = [30 + 16 * (b % 40) + b % 3 for b in range(B)]      # many of them complete a window in the second step
    caches = []
    for _ in range(2):
        torch.manual_seed(1)
        c = mod.new_cache(B, 800, dtype=dtype, device=DEV)
        for t in (c.k, c.v, c.cmp_k, c.cmp_v, c.k_tail, c.v_tail):
            t.normal_()
        c.host_len = list(lens)
        c.seq_len.copy_(torch.tensor(lens, dtype=torch.int32))
        caches.append(c)
    for s in range(4):
        ins = [torch.randn(B, hidden, device=DEV).to(dtype)] if proj else [torch.randn(B, H, D, device=DEV).to(dtype) for H in (Hq, Hk, Hk)]
        y = mod.step(*ins, caches[0])
        ids = mod.last_topk_idx
        hook = mod.gate.register_forward_hook(lambda *a: None)
        ref = mod.step(*ins, caches[1])
        hook.remove()
        same = (ids == mod.last_topk_idx).all(-1).all(-1)       # a near tie may fall the other way: those sequences apart
        assert float(same.float().mean()) >= 0.8
        _close(y[same], ref[same], f"step {s}")
    assert torch.equal(caches[0].seq_len, caches[1].seq_len) and caches[0].host_len == caches[1].host_len
    for n in ("k", "v", "cmp_k", "cmp_v", "k_tail", "v_tail"):
        _close(getattr(caches[0], n)[:-1], getattr(caches[1], n)[:-1], n)


@pytest.mark.parametrize("seqlens,H,D,ks,st", [([47], 2, 128, 32, 16), ([517], 8, 128, 32, 16), ([31, 3000, 32, 1], 3, 64, 32, 16),
                                               ([100 + 7 * i for i in range(14)], 1, 128, 16, 16), ([9000, 900], 8, 128, 32, 16)])
def test_compressor_reductions(seqlens, H, D, ks, st):
    """One to eight CTAs per tile, more sequences than a launch takes, a bias."""
    torch.manual_seed(len(seqlens))
    N = sum(seqlens)
    x = torch.randn(N, H, D, device=DEV).to(torch.bfloat16)
    w = (torch.randn(H, ks * D, D, device=DEV) * 0.02).to(torch.bfloat16)
    pe = torch.randn(H, ks, D, device=DEV).to(torch.bfloat16)
    cu = torch.tensor([sum(seqlens[:i]) for i in range(len(seqlens) + 1)], dtype=torch.int32, device=DEV)
    y, ycu = linear_compress(x, w, cu, ks, st, pe, seqlens)
    at = 0
    for i, L in enumerate(seqlens):
        n = (L - ks) // st + 1 if L >= ks else 0
        if n:
            win = x[int(cu[i]) : int(cu[i]) + L].double().unfold(0, ks, st).permute(1, 0, 3, 2).reshape(H, n, ks * D)
            ref = torch.bmm(win, w.double()).transpose(0, 1) + (pe.double().reshape(H, -1, 1) * w.double()).sum(1)
            # two roundings (the product, then the sum with the bias)
            assert float((y[at : at + n].double() - ref).norm() / ref.norm()) <= 5e-3, f"sequence {i}"
        at += n
    assert at == y.shape[0] == int(ycu[-1])


@pytest.mark.parametrize("B,Hk,G,D,hidden", [(1, 8, 4, 128, 4096), (12, 2, 4, 64, 1024), (20, 4, 4, 128, 2048)])
def test_steps_in_a_row_match_steps_one_by_one(B, Hk, G, D, hidden):
    """The kernels of a step start while the one before them ends: steps without a wait between them, each fed with the output of the
    one before, against the same steps with a wait after each -- outputs and caches bit for bit."""
    torch.manual_seed(B)
    mod = FlashSparseAttentionDecode(hidden, Hk * G, Hk, D, 32, 16, 64, 8, 1, 2, 100, rope_config=RopeConfig(head_dim=D)).to(DEV).to(torch.bfloat16)
    with torch.no_grad():
        for p in mod.parameters():
            torch.nn.init.xavier_uniform_(p)
    lens = [600 + 37 * b for b in range(B)]
    x0 = torch.randn(B, hidden, device=DEV).to(torch.bfloat16)

    def run(wait):
        torch.manual_seed(1)
        c = mod.new_cache(B, 2048, dtype=torch.bfloat16, device=DEV)
        for t in (c.k, c.v, c.cmp_k, c.cmp_v, c.k_tail, c.v_tail):
            t.normal_()
        c.host_len = list(lens)
        c.seq_len.copy_(torch.tensor(lens, dtype=torch.int32))
        x, ys = x0, []
        for _ in range(40):
            x = (x + mod.step(x, c)).clamp(-4, 4)
            ys.append(x)
            if wait:
                torch.cuda.synchronize()
        return ys + [getattr(c, n)[:-1] for n in ("k", "v", "cmp_k", "cmp_v", "k_tail", "v_tail")] + [c.seq_len]

    with torch.no_grad():
        assert all(torch.equal(a, b) for a, b in zip(run(False), run(True)))


@pytest.mark.parametrize("B,D,ks,st,dtype", [(250, 64, 32, 16, torch.bfloat16), (3, 128, 64, 16, torch.float16), (17, 128, 40, 8, torch.bfloat16),
                                             (5, 64, 24, 8, torch.bfloat16), (16, 128, 32, 16, torch.bfloat16), (79, 128, 16, 8, torch.bfloat16)])
def test_compressor_turns_and_chunks(B, D, ks, st, dtype):
    """The incremental compressor against the prefill one on the window that ends with the new token: around the rows of an MMA tile,
    more sequences than a turn takes, reductions of one, two and one and a half chunks; rows of other sequences stay as they were."""
    torch.manual_seed(B + ks)
    Hk = 2
    mod = FlashSparseAttentionDecodeKernel(2 * Hk * D, 2 * Hk, Hk, D, ks, st, 64, 8, 1, 2, 100).to(DEV).to(dtype)
    with torch.no_grad():
        for p in mod.parameters():
            p.normal_(0, 0.05)
    lens = [ks - 1 + st * (b % 5) + (7 if b % 16 == 3 else 0) for b in range(B)]        # all but a few complete a window now
    cache = mod.new_cache(B, 400, dtype=dtype, device=DEV)
    for t in (cache.k, cache.v, cache.cmp_k, cache.cmp_v, cache.k_tail, cache.v_tail):
        t.normal_()
    cache.host_len = list(lens)
    cache.seq_len.copy_(torch.tensor(lens, dtype=torch.int32))
    before = cache.cmp_k.clone(), cache.cmp_v.clone()
    with torch.no_grad():
        mod.step(*(torch.randn(B, H, D, device=DEV).to(dtype) for H in (2 * Hk, Hk, Hk)), cache)
    for got, old, tail, w, pe in ((cache.cmp_k, before[0], cache.k_tail, mod.compress_key, mod.intra_block_pe), (cache.cmp_v, before[1], cache.v_tail, mod.compress_value, None)):
        want = old.clone()
        ring = tail[:-1].view(B, ks, Hk, D)
        for b, L in enumerate(lens):
            if (L + 1 - ks) % st == 0:
                x = torch.cat([ring[b, (L + 1) % ks :], ring[b, : (L + 1) % ks]]).double()
                y = torch.einsum("khd,hkde->he", x, w.double().view(Hk, ks, D, D)).to(dtype)
                if pe is not None:
                    y = y + torch.einsum("hkd,hkde->he", pe.double(), w.double().view(Hk, ks, D, D)).to(dtype)
                want[int(cache.cmp_row0[b]) + (L + 1 - ks) // st] = y
        changed = (want != old).any(-1).any(-1)
        assert torch.equal(got[~changed], old[~changed])
        # fp32 sums of exact products: the result is one rounding (keys: two and their sum's) from the 64-bit one
        assert float((got[changed].double() - want[changed].double()).norm() / want[changed].double().norm()) <= (6e-4 if dtype == torch.float16 else 4e-3)


def test_inputs_of_a_captured_step_are_copied_in_one_launch():
    """fsa_copy at sizes and alignments that end within a 16-byte unit; what is more than a copy of bytes is left to copy_."""
    from fsa._host import host

    torch.manual_seed(3)
    src = [torch.randn(s, device=DEV).to(torch.bfloat16) for s in ((3, 5), (1, 8, 128), (0, 4), (1,), (70000, 3))]
    src.append(torch.randn(257, device=DEV).to(torch.bfloat16)[1:])
    dst = [torch.zeros_like(t) for t in src]
    assert host().copy_inputs(dst, src) and all(torch.equal(a, b) for a, b in zip(src, dst))
    a, b = torch.zeros(4, 6, device=DEV), torch.randn(4, 6, device=DEV)
    for d, s in ((a, b.double()), (a, b.t().contiguous().t()), (a, b[:1]), (a, b.cpu()), (a[:2], a[1:3])):
        assert not host().copy_inputs([d], [s])
