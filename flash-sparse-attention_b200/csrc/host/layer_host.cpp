// The layer between x and its output projection as one native autograd function: projections, compression, rotation, the three
// branches, block selection and the gate mix.  Seen as one function, the backward needs no pass over [N, hidden] or
// [N, heads, d] just to add gradients: the gate's backward starts dx and the GEMMs accumulate into it, the rotation's backward
// sums what the branches and the compressor give of dq, dk and dv, and the gate's backward delivers the
// sums of o dO that the attention backwards start from.
#include "host_common.h"

#include <cuda_runtime_api.h>

#include <optional>

namespace fsa_host {

struct LayerCfg {
    int Hq, Hk, D, ks, stride, bs, topk, init_blocks, local_blocks, window;
};
static LayerCfg layer_cfg(const std::vector<int64_t>& c) {
    TORCH_CHECK_VALUE(c.size() == 10, "layer settings");
    return {(int)c[0], (int)c[1], (int)c[2], (int)c[3], (int)c[4], (int)c[5], (int)c[6], (int)c[7], (int)c[8], (int)c[9]};
}

struct Lengths {
    std::vector<int32_t> tok;       // tokens of every sequence
    int64_t N = 0, Nc = 0;
    int B = 0, max_len = 0, max_cmp = 0;
    Lengths(const std::vector<int64_t>& seqlens, const LayerCfg& c) : tok(seqlens.begin(), seqlens.end()), B((int)seqlens.size()) {
        for (int L : tok) {
            const int n = L >= c.ks ? (L - c.ks) / c.stride + 1 : 0;
            N += L; Nc += n;
            max_len = std::max(max_len, L);
            max_cmp = std::max(max_cmp, n);
        }
    }
    int win_blocks(const LayerCfg& c) const { return (c.window + 1 + 63) / 64 + 1; }       // 64-row blocks that a token's range can touch
    int cmp_blocks() const { return (max_cmp + 63) / 64 + 1; }
    // Does every token select every block up to its own?  The selection then is causal attention over its whole sequence, for which
    // the query-tile-major kernels need no scores, no index and no partial rows.  32 / 8 heads, prefill of 517 tokens 202 -> 158 us, of 1024
    // 275 -> 195; 16 / 4 heads, training step on 8 x 1000 tokens 1909 -> 1640, on 64 x 200 2745 -> 2560.  From the first longer sequence on
    // the selection has to run for it.  (Head size 128: their backward; the block-major one that serves the others gains nothing.)
    bool every_block(const LayerCfg& c) const { return c.D == 128 && max_len <= (int64_t)c.topk * c.bs; }
    int own_blocks() const { return (max_len + 63) / 64 + 1; }
};

// What a forward leaves for the backward.
struct Kept {
    Tensor q, k_raw, k, v, ck, cv, cs, sn, cu_cmp, bounds, o_cmp, lse_cmp, topk, o_sel, lse_sel, ws, o_win, lse_win, gate;
};

// One of the dense branches: ranges of K/V rows in, o and lse out.
struct Range {
    const Tensor &k, &v, &cu_k;
    const int32_t *lo, *hi;
    Tensor &o, &lse;
    int32_t* status;
};
// Branches that do not wait for one another, in one launch (the longest first).
static void range_fwd(const Tensor& q, const Tensor& cu_q, std::initializer_list<Range> branches, float scale) {
    const int64_t N = q.size(0);
    fsa_range_problem a[3];
    int n = 0;
    for (const Range& r : branches) {
        r.o = fresh_like(q);
        r.lse = f32({q.size(1), N}, q);
        a[n++] = {ptr(q), ptr(r.k), ptr(r.v), iptr(cu_q), iptr(r.cu_k), r.lo, r.hi, N, r.k.size(0), q.stride(0), q.stride(1), r.k.stride(0), r.v.stride(0),
                  ptr(r.o), r.o.stride(0), r.o.stride(1), r.lse.data_ptr<float>(), r.status};
    }
    const Tensor& k = branches.begin()->k;
    check(fsa_range_attn_fwd_dense_several(n, a, (int)cu_q.size(0) - 1, (int)q.size(1), (int)k.size(1), (int)q.size(2), dtype_code(q), scale, stream_of(q)),
          "fsa_range_attn_fwd_dense");
}

static Tensor layer_fwd(const Tensor& x, const Tensor& wq, const Tensor& wk, const Tensor& wv, const Tensor& wg, const Tensor& w_key,
                        const Tensor& w_value, const Tensor& pe, const Tensor& inv_freq, const Tensor& cu, const Lengths& s, const LayerCfg& c,
                        Kept& t) {
    const int64_t N = s.N, hidden = x.size(1);
    const int dt = dtype_code(x);
    const float scale = (float)(1.0 / std::sqrt((double)c.D));
    void* st = stream_of(x);
    const Tensor word = checking_status() ? at::zeros({4}, x.options().dtype(at::kInt)) : Tensor();
    int32_t* status = word.defined() ? word.data_ptr<int32_t>() : nullptr;      // one for the two ranges and the selection
    t.cs = fresh({s.max_len, c.D / 2}, x);
    t.sn = fresh({s.max_len, c.D / 2}, x);
    t.cu_cmp = i32({s.B + 1}, x);
    check(fsa_layer_prep(iptr(cu), s.B, s.max_len, inv_freq.data_ptr<float>(), c.D, c.ks, c.stride, dt, ptr(t.cs), ptr(t.sn),
                         t.cu_cmp.data_ptr<int32_t>(), st),
          "fsa_layer_prep");
    t.k_raw = at::mm(x, wk.t()).view({N, c.Hk, c.D});
    t.v = at::mm(x, wv.t()).view({N, c.Hk, c.D});
    t.q = at::mm(x, wq.t()).view({N, c.Hq, c.D});
    t.ck = fresh({s.Nc, c.Hk, c.D}, x);
    t.cv = fresh_like(t.ck);
    {
        const Tensor scratch = bytes(fsa_compress_bias_scratch_bytes(c.Hk, c.D), x);
        check(fsa_compress_kv_fwd(ptr(t.k_raw), t.k_raw.stride(0), ptr(t.v), t.v.stride(0), ptr(w_key), ptr(w_value), ptr(pe), s.tok.data(), s.B, c.Hk,
                                  c.D, c.ks, c.stride, dt, ptr(t.ck), ptr(t.cv), (float*)ptr(scratch), st),
              "fsa_compress_kv_fwd");
        check_status((char*)ptr(scratch) + scratch.numel() - 16, x, "fsa_compress_kv_fwd status");
    }
    t.k = fresh_like(t.k_raw);
    t.bounds = i32({3, N}, x);
    int32_t* bd = t.bounds.data_ptr<int32_t>();
    check(fsa_layer_rope_fwd(ptr(t.q), t.q.stride(0), ptr(t.k_raw), t.k_raw.stride(0), ptr(t.ck), ptr(t.cs), ptr(t.sn), iptr(cu), iptr(t.cu_cmp), s.B,
                             N, s.Nc, c.Hq, c.Hk, c.D, c.ks, c.stride, c.window, dt, ptr(t.q), ptr(t.k), bd, bd + N, bd + 2 * N, st),
          "fsa_layer_rope_fwd");
    const Range cmp{t.ck, t.cv, t.cu_cmp, nullptr, bd, t.o_cmp, t.lse_cmp, status}, win{t.k, t.v, cu, bd + N, bd + 2 * N, t.o_win, t.lse_win, status};
    const int max_blocks = (s.max_len + c.bs - 1) / c.bs, t_out = std::min(c.topk, max_blocks);
    t.topk = i32({c.Hk, N, t_out}, x);
    if (s.every_block(c)) {
        check(fsa_layer_every_block(iptr(cu), s.B, N, c.Hk, t_out, c.bs, t.topk.data_ptr<int32_t>(), st), "fsa_layer_every_block");
        if (checking_status()) t.ws = at::zeros({4}, x.options().dtype(at::kInt));      // (the branch's own word, read as the operator's is)
        range_fwd(t.q, cu, {{t.k, t.v, cu, nullptr, bd + 2 * N, t.o_sel, t.lse_sel, t.ws.defined() ? t.ws.data_ptr<int32_t>() : nullptr}, win, cmp}, scale);
    } else {
        range_fwd(t.q, cu, {cmp, win}, scale);
        check(fsa_select_topk_fused(ptr(t.q), t.q.stride(0), ptr(t.ck), t.ck.stride(0), t.lse_cmp.data_ptr<float>(), iptr(cu), iptr(t.cu_cmp), N, s.Nc,
                                    s.B, c.Hq, c.Hk, c.D, dt, scale, c.ks, c.stride, c.bs, c.init_blocks, c.local_blocks, max_blocks, t_out,
                                    t.topk.data_ptr<int32_t>(), status, st),
              "fsa_select_topk_fused");
        std::tie(t.o_sel, t.lse_sel, t.ws) = sel_fwd(t.q, t.k, t.v, t.topk, c.bs, cu, scale);
    }
    t.gate = fresh({N, 3}, x);
    Tensor out = fresh({N, (int64_t)c.Hq * c.D}, x);
    check(fsa_gate_proj_mix_fwd(ptr(x), x.stride(0), ptr(wg), ptr(t.o_cmp), ptr(t.o_sel), ptr(t.o_win), N, (int)hidden, c.Hq * c.D, dt, ptr(out),
                                ptr(t.gate), st),
          "fsa_gate_proj_mix_fwd");
    if (t.ws.defined()) check_status(ptr(t.ws), x, "fsa_sel_fwd status");
    check_status(status, x, "range attention and block selection status");
    return out;
}

// dq, dk, dv of one of the dense branches
static std::tuple<Tensor, Tensor, Tensor> range_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& lse, const Tensor& dout,
                                                    const float* delta, const Tensor& cu_q, const Tensor& cu_k, const int32_t* lo, const int32_t* hi,
                                                    int max_blocks, float scale, const char* what = "fsa_range_attn_bwd_delta status") {
    const int64_t N = q.size(0), Nk = k.size(0);
    const int B = (int)cu_q.size(0) - 1, Hq = (int)q.size(1), Hk = (int)k.size(1), D = (int)q.size(2);
    int64_t ib = 0, fb = 0, bb = 0;
    check(fsa_range_attn_bytes(N, Nk, B, Hq, Hk, D, max_blocks, 64, &ib, &fb, &bb), "fsa_range_attn_bytes");
    const bool indexed = fsa_range_attn_bwd_indexed(D) != 0;
    const Tensor ws = bytes(indexed ? ib : 16, q), scratch = bytes(bb, q);
    if (indexed) check(fsa_range_attn_index(iptr(cu_q), iptr(cu_k), lo, hi, N, Nk, B, Hq, Hk, max_blocks, 64, ptr(ws), ws.numel(), stream_of(q)), "fsa_range_attn_index");
    Tensor dq = fresh_like(q), dk = fresh({Nk, Hk, D}, q), dv = fresh_like(dk);
    check(fsa_range_attn_bwd_delta(ptr(q), ptr(k), ptr(v), lse.data_ptr<float>(), ptr(dout), delta, iptr(cu_q), iptr(cu_k), lo, hi, N, Nk, B, Hq, Hk, D,
                                   max_blocks, 64, dtype_code(q), q.stride(0), q.stride(1), k.stride(0), v.stride(0), dout.stride(0), dout.stride(1),
                                   scale, ptr(dq), ptr(dk), ptr(dv), ptr(ws), ws.numel(), ptr(scratch), scratch.numel(), stream_of(q)),
          "fsa_range_attn_bwd_delta");
    check_status(ptr(ws), q, what);
    return {dq, dk, dv};
}

struct NsaLayer : torch::autograd::Function<NsaLayer> {
    static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const Tensor& wq, const Tensor& wk,
                                                  const Tensor& wv, const Tensor& wg, const Tensor& w_key, const Tensor& w_value, const Tensor& pe,
                                                  const Tensor& inv_freq, const Tensor& cu, const std::vector<int64_t>& seqlens,
                                                  const std::vector<int64_t>& cfg) {
        const LayerCfg c = layer_cfg(cfg);
        const Lengths s(seqlens, c);
        Kept t;
        Tensor out = layer_fwd(x, wq, wk, wv, wg, w_key, w_value, pe, inv_freq, cu, s, c, t);
        ctx->save_for_backward({x, wq, wk, wv, wg, w_key, w_value, pe, cu, t.q, t.k_raw, t.k, t.v, t.ck, t.cv, t.cs, t.sn, t.cu_cmp, t.bounds,
                                t.o_cmp, t.lse_cmp, t.topk, t.o_sel, t.lse_sel, t.ws, t.o_win, t.lse_win, t.gate});
        ctx->saved_data["seqlens"] = seqlens;
        ctx->saved_data["cfg"] = cfg;
        ctx->mark_non_differentiable({t.topk});
        ctx->set_materialize_grads(false);          // (no zeros for the ids)
        return {out, t.topk};
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
        const auto sv = ctx->get_saved_variables();
        const Tensor &x = sv[0], &wq = sv[1], &wk = sv[2], &wv = sv[3], &wg = sv[4], &w_key = sv[5], &w_value = sv[6], &pe = sv[7], &cu = sv[8],
                     &q = sv[9], &k_raw = sv[10], &k = sv[11], &v = sv[12], &ck = sv[13], &cv = sv[14], &cs = sv[15], &sn = sv[16], &cu_cmp = sv[17],
                     &bounds = sv[18], &o_cmp = sv[19], &lse_cmp = sv[20], &topk = sv[21], &o_sel = sv[22], &lse_sel = sv[23], &ws = sv[24],
                     &o_win = sv[25], &lse_win = sv[26], &gate = sv[27];
        if (!grads[0].defined()) return torch::autograd::variable_list(12);
        const LayerCfg c = layer_cfg(ctx->saved_data["cfg"].toIntVector());
        const Lengths s(ctx->saved_data["seqlens"].toIntVector(), c);
        c10::cuda::CUDAGuard guard(x.device());
        cudaSetDevice(x.get_device());      // (binds the context to the engine's thread: the first GEMM below wants one)
        const int64_t N = s.N, hidden = x.size(1);
        const int dt = dtype_code(x);
        const float scale = (float)(1.0 / std::sqrt((double)c.D));
        void* st = stream_of(x);
        const int32_t* bd = iptr(bounds);

        Tensor dx = fresh({N, hidden}, x), dwg = fresh_like(wg), delta = f32({3, c.Hq, N}, x);
        Tensor d_cmp = fresh_like(q), d_sel = fresh_like(q), d_win = fresh_like(q);
        {
            const Tensor dout = grads[0].contiguous();
            const Tensor scratch = bytes(fsa_gate_proj_mix_scratch_bytes(N, (int)hidden), x);
            check(fsa_gate_proj_mix_bwd_delta(ptr(x), x.stride(0), ptr(wg), ptr(gate), ptr(o_cmp), ptr(o_sel), ptr(o_win), ptr(dout), N, (int)hidden,
                                              c.Hq, c.D, dt, ptr(d_cmp), ptr(d_sel), ptr(d_win), ptr(dx), ptr(dwg), delta.data_ptr<float>(),
                                              (float*)ptr(scratch), scratch.numel(), st),
                  "fsa_gate_proj_mix_bwd_delta");
        }
        const float* dl = delta.data_ptr<float>();
        auto [dq0, dck, dcv] = range_bwd(q, ck, cv, lse_cmp, d_cmp, dl, cu, cu_cmp, nullptr, bd, s.cmp_blocks(), scale);
        d_cmp.reset();
        const float* dl_sel = dl + (int64_t)c.Hq * N;
        auto [dq1, dk, dv] = s.every_block(c) ? range_bwd(q, k, v, lse_sel, d_sel, dl_sel, cu, cu, nullptr, bd + 2 * N, s.own_blocks(), scale,
                                                          "fsa_sel_bwd_delta status")
                                              : sel_bwd_delta(q, k, v, lse_sel, d_sel, dl_sel, topk, c.bs, cu, scale, ws);
        if (!s.every_block(c)) check_status(ptr(ws), q, "fsa_sel_bwd_delta status");
        d_sel.reset();
        auto [dq2, dk2, dv2] = range_bwd(q, k, v, lse_win, d_win, dl + 2 * (int64_t)c.Hq * N, cu, cu, bd + N, bd + 2 * N, s.win_blocks(c), scale);
        d_win.reset();
        auto rope_bwd = [&](int64_t n, int64_t nc, const Tensor& dkc, const Tensor& dvc) {
            check(fsa_layer_rope_bwd(ptr(dq0), ptr(dq1), ptr(dq2), ptr(dk), ptr(dk2), ptr(dkc), ptr(dv), ptr(dv2), ptr(dvc), ptr(dck), ptr(cs), ptr(sn),
                                     iptr(cu), iptr(cu_cmp), s.B, n, nc, c.Hq, c.Hk, c.D, c.stride, dt, ptr(dq0), ptr(dk), ptr(dv), st),
                  "fsa_layer_rope_bwd");
        };
        rope_bwd(0, s.Nc, Tensor(), Tensor());
        Tensor dw_key = ctx->needs_input_grad(5) ? fresh_like(w_key) : Tensor(), dw_value = ctx->needs_input_grad(6) ? fresh_like(w_value) : Tensor(),
               dpe = ctx->needs_input_grad(7) ? fresh_like(pe) : Tensor();
        {
            const Tensor dkc = fresh_like(dk), dvc = fresh_like(dv), scratch = bytes(fsa_compress_kv_bwd_scratch_bytes(c.Hk, c.D), x);
            check(fsa_compress_kv_bwd(ptr(k_raw), k_raw.stride(0), ptr(v), v.stride(0), ptr(w_key), ptr(w_value), ptr(pe), ptr(dck), ptr(dcv), iptr(cu),
                                      s.tok.data(), s.B, c.Hk, c.D, c.ks, c.stride, dt, ptr(dkc), ptr(dvc), ptr(dw_key), ptr(dw_value), ptr(dpe),
                                      (float*)ptr(scratch), st),
                  "fsa_compress_kv_bwd");
            check_status((char*)ptr(scratch) + scratch.numel() - 16, x, "fsa_compress_kv_bwd status");
            rope_bwd(N, 0, dkc, dvc);
        }
        dq1.reset(); dq2.reset(); dk2.reset(); dv2.reset(); dck.reset(); dcv.reset();
        const Tensor gq = dq0.view({N, -1}), gk = dk.view({N, -1}), gv = dv.view({N, -1});
        Tensor dwq, dwk, dwv;
        if (ctx->needs_input_grad(1)) dwq = at::mm(gq.t(), x);
        if (ctx->needs_input_grad(2)) dwk = at::mm(gk.t(), x);
        if (ctx->needs_input_grad(3)) dwv = at::mm(gv.t(), x);
        if (ctx->needs_input_grad(0)) {
            at::addmm_out(dx, dx, gq, wq);
            at::addmm_out(dx, dx, gk, wk);
            at::addmm_out(dx, dx, gv, wv);
        } else {
            dx = Tensor();
        }
        return {dx, dwq, dwk, dwv, dwg, dw_key, dw_value, dpe, Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

// Nothing where a weight is of another type, device or memory order than the kernels read (the layer then runs as its parts).
std::optional<std::tuple<Tensor, Tensor>> nsa_layer(const Tensor& x_, const Tensor& wq, const Tensor& wk, const Tensor& wv, const Tensor& wg, const Tensor& w_key,
                                     const Tensor& w_value, const Tensor& pe, const Tensor& inv_freq, const Tensor& cu,
                                     const std::vector<int64_t>& seqlens, const std::vector<int64_t>& cfg) {
    c10::cuda::CUDAGuard guard(x_.device());
    for (auto* w : {&wq, &wk, &wv, &wg, &w_key, &w_value, &pe})
        if (w->scalar_type() != x_.scalar_type() || w->device() != x_.device() || !w->is_contiguous()) return std::nullopt;
    {
        // (raw pointers from here on; the lengths agree with x and cu: _native of fsa/module/fsa.py)
        const LayerCfg c = layer_cfg(cfg);
        const int64_t hidden = x_.size(1), q = (int64_t)c.Hq * c.D, kv = (int64_t)c.Hk * c.D;
        TORCH_CHECK_VALUE(wq.sizes() == at::IntArrayRef({q, hidden}) && wk.sizes() == at::IntArrayRef({kv, hidden}) &&
                              wv.sizes() == wk.sizes() && wg.sizes() == at::IntArrayRef({3, hidden}) &&
                              w_key.sizes() == at::IntArrayRef({c.Hk, (int64_t)c.ks * c.D, c.D}) && w_value.sizes() == w_key.sizes() &&
                              pe.sizes() == at::IntArrayRef({c.Hk, c.ks, c.D}) && inv_freq.numel() == c.D / 2,
                          "layer: a weight or the rotation has another shape than the layer's settings");
    }
    const Tensor x = x_.stride(1) == 1 && x_.stride(0) % 8 == 0 && ((uintptr_t)x_.data_ptr() & 15) == 0 ? x_ : x_.contiguous();
    if (wants_grad({&x, &wq, &wk, &wv, &wg, &w_key, &w_value, &pe})) {
        auto r = NsaLayer::apply(x, wq, wk, wv, wg, w_key, w_value, pe, inv_freq, cu, seqlens, cfg);
        return std::make_tuple(r[0], r[1]);
    }
    const LayerCfg c = layer_cfg(cfg);
    const Lengths s(seqlens, c);
    Kept t;
    Tensor out = layer_fwd(x, wq, wk, wv, wg, w_key, w_value, pe, inv_freq, cu, s, c, t);
    return std::make_tuple(out, t.topk);
}

void bind_layer(pybind11::module& m) { m.def("nsa_layer", &nsa_layer); }

}  // namespace fsa_host
