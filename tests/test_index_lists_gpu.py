"""The block -> entries index at the edges of its launch rules: one launch or five, groups of 32 tokens with and without a block
that a list names twice, lists that are not kept in registers, tables of keys without room for the lane bits."""
from ctypes import byref, c_int, c_int64

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from fsa import _lib
from fsa.ops.FSA_topk_sparse_attention import sel_attn_fwd
from fsa.synthetic import make_cu_seqlens, make_qkv, make_topk_idx

DEV = "cuda:0"


@pytest.mark.parametrize("seqlens,Hk,T,bs,twice", [([33], 1, 4, 64, False), ([700, 31], 2, 16, 64, True), ([1025], 8, 8, 32, False),
                                                   ([1000], 1, 16, 64, True), ([1001], 2, 16, 64, True), ([517], 8, 9, 64, True), ([5000], 1, 6, 128, False),
                                                   ([1] * 3300, 1, 4, 32, False), ([2500], 1, 20, 64, False)])
def test_every_entry_once_in_order(seqlens, Hk, T, bs, twice):
    N, B, d = sum(seqlens), len(seqlens), 64
    cu, idx = make_cu_seqlens(seqlens), make_topk_idx(seqlens, Hk, T, bs, 9)
    if twice:
        idx[:, 5 :: 77, 3] = idx[:, 5 :: 77, 1]
    q, k, v = make_qkv(N, Hk, Hk, d, 1, with_do=False)
    L = _lib.lib()
    mt, tpt, nbmax = c_int64(0), c_int(0), c_int(0)
    assert L.fsa_sel_index_geometry(N, B, Hk, Hk, T, bs, byref(mt), byref(tpt), byref(nbmax)) == 0
    mt, tpt, nbmax = mt.value, tpt.value, nbmax.value
    _, _, ws = sel_attn_fwd(q.to(DEV), k.to(DEV), v.to(DEV), idx.to(DEV), bs, cu.to(DEV), d ** -0.5, check_status=True)
    rec, entries = np.zeros((mt, 4), np.int32), np.zeros(mt * tpt, np.uint32)
    key_tile, header = np.zeros(Hk * nbmax + 1, np.int32), np.zeros(64, np.int32)
    assert L.fsa_sel_index_dump(_lib.ptr(ws), N, B, Hk, Hk, T, bs, None, rec.ctypes.data, entries.ctypes.data, key_tile.ctypes.data,
                                header.ctypes.data) == 0
    nt = int(header[1])
    rec, entries = rec[:nt], entries[: nt * tpt].reshape(nt, tpt)
    ne = rec[:, 1] & 255
    used = np.arange(tpt)[None, :] < ne[:, None]
    assert ((entries != 0xFFFFFFFF) == used).all() and int(header[2]) == used.sum()
    key = np.repeat(rec[:, 2].astype(np.int64), ne)
    got = entries[used].astype(np.int64)
    assert (np.diff(rec[:, 2]) >= 0).all()
    same = key[1:] == key[:-1]
    assert (np.diff(got >> 11)[same] >= 0).all()                     # ascending groups of 32 tokens (6 bits of slot)
    cul = np.asarray(cu.tolist())
    seq = np.repeat(np.arange(B), seqlens)
    tok = np.arange(N)
    ids = idx.numpy().astype(np.int64)
    usable = (ids >= 0) & (ids <= ((tok - cul[seq]) // bs)[None, :, None])
    h, n, s = np.nonzero(usable)
    want = np.stack([h * nbmax + cul[seq[n]] // bs + seq[n] + ids[h, n, s], (n << 6) | s])
    order = lambda a: a[:, np.lexsort((a[1], a[0]))]  # noqa: E731
    assert np.array_equal(order(np.stack([key, got])), order(want))
