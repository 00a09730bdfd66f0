// Selected attention: workspaces, the two C-ABI calls and the autograd function around them, in native code.  A call of the
// operator on a short sequence is a dozen kernels of a few microseconds; prepared and launched from Python (ctypes argument
// conversion, autograd in the interpreter) the host took 200 us for what the GPU does in 60.
#include "host_common.h"

namespace fsa_host {

struct SelShapeArgs {
    int64_t N;
    int B, Hq, Hk, D, T, bs;
};

static SelShapeArgs shape_of(const Tensor& q, const Tensor& k, const Tensor& idx, const Tensor& cu, int64_t bs) {
    return {q.size(0), (int)cu.size(0) - 1, (int)q.size(1), (int)k.size(1), (int)q.size(2), (int)idx.size(-1), (int)bs};
}

// o, lse and the block -> entries index that the backward reuses
std::tuple<Tensor, Tensor, Tensor> sel_fwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& idx_, int64_t bs,
                                           const Tensor& cu_, double scale) {
    c10::cuda::CUDAGuard guard(q_.device());
    const Tensor q = rows(q_), k = rows(k_, true), v = rows(v_, true), idx = idx_.contiguous(), cu = cu_.contiguous();
    const SelShapeArgs s = shape_of(q, k, idx, cu, bs);
    int64_t nb = 0;
    check(fsa_sel_index_bytes(s.N, s.B, s.Hq, s.Hk, s.T, s.bs, &nb), "fsa_sel_index_bytes");
    Tensor ws = bytes(nb, q);
    check(fsa_sel_fwd_scratch_bytes(s.N, s.B, s.Hq, s.Hk, s.D, s.T, s.bs, &nb), "fsa_sel_fwd_scratch_bytes");
    const Tensor scratch = bytes(nb, q);
    Tensor o = fresh({s.N, s.Hq, s.D}, q), lse = f32({s.Hq, s.N}, q);
    check(fsa_sel_fwd(ptr(q), ptr(k), ptr(v), iptr(idx), iptr(cu), s.N, s.B, s.Hq, s.Hk, s.D, s.T, s.bs, dtype_code(q), q.stride(0),
                      q.stride(1), k.stride(0), v.stride(0), (float)scale, ptr(o), o.stride(0), o.stride(1), lse.data_ptr<float>(),
                      ptr(ws), ws.numel(), ptr(scratch), scratch.numel(), stream_of(q)),
          "fsa_sel_fwd");
    return {o, lse, ws};
}

std::tuple<Tensor, Tensor, Tensor> sel_bwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& o_, const Tensor& lse,
                                           const Tensor& do_, const Tensor& idx_, int64_t bs, const Tensor& cu_, double scale,
                                           const Tensor& ws) {
    c10::cuda::CUDAGuard guard(q_.device());
    const Tensor q = rows(q_), k = rows(k_, true), v = rows(v_, true), o = rows(o_), dout = rows(do_), idx = idx_.contiguous(),
                 cu = cu_.contiguous();
    const SelShapeArgs s = shape_of(q, k, idx, cu, bs);
    int64_t nb = 0;
    check(fsa_sel_bwd_scratch_bytes(s.N, s.B, s.Hq, s.Hk, s.D, s.T, s.bs, &nb), "fsa_sel_bwd_scratch_bytes");
    const Tensor scratch = bytes(nb, q);
    Tensor dq = fresh({s.N, s.Hq, s.D}, q), dk = fresh({s.N, s.Hk, s.D}, q), dv = fresh_like(dk);
    check(fsa_sel_bwd(ptr(q), ptr(k), ptr(v), ptr(o), lse.data_ptr<float>(), ptr(dout), iptr(idx), iptr(cu), s.N, s.B, s.Hq, s.Hk, s.D,
                      s.T, s.bs, dtype_code(q), q.stride(0), q.stride(1), k.stride(0), v.stride(0), o.stride(0), o.stride(1),
                      dout.stride(0), dout.stride(1), (float)scale, ptr(dq), ptr(dk), ptr(dv), ptr(ws), ws.numel(), ptr(scratch),
                      scratch.numel(), stream_of(q)),
          "fsa_sel_bwd");
    return {dq, dk, dv};
}

std::tuple<Tensor, Tensor, Tensor> sel_bwd_delta(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& lse, const Tensor& dout,
                                                 const float* delta, const Tensor& idx, int64_t bs, const Tensor& cu, double scale,
                                                 const Tensor& ws) {
    const SelShapeArgs s = shape_of(q, k, idx, cu, bs);
    int64_t nb = 0;
    check(fsa_sel_bwd_scratch_bytes(s.N, s.B, s.Hq, s.Hk, s.D, s.T, s.bs, &nb), "fsa_sel_bwd_scratch_bytes");
    const Tensor scratch = bytes(nb, q);
    Tensor dq = fresh_like(q), dk = fresh({s.N, s.Hk, s.D}, q), dv = fresh_like(dk);
    check(fsa_sel_bwd_delta(ptr(q), ptr(k), ptr(v), lse.data_ptr<float>(), ptr(dout), delta, iptr(idx), iptr(cu), s.N, s.B, s.Hq, s.Hk, s.D, s.T,
                            s.bs, dtype_code(q), q.stride(0), q.stride(1), k.stride(0), v.stride(0), dout.stride(0), dout.stride(1), (float)scale,
                            ptr(dq), ptr(dk), ptr(dv), ptr(ws), ws.numel(), ptr(scratch), scratch.numel(), stream_of(q)),
          "fsa_sel_bwd_delta");
    return {dq, dk, dv};
}

bool checking_status() {
    static const bool on = [] {
        const char* v = getenv("FSA_CHECK_STATUS");
        return v && v[0] == '1' && !v[1];
    }();
    return on;
}

void check_status(const void* word, const Tensor& like, const char* what) {
    if (!checking_status()) return;
    int st = 0;
    check(fsa_read_status(word, stream_of(like), &st), what);
}

struct SelAttention : torch::autograd::Function<SelAttention> {
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx,
                          const Tensor& cu, int64_t bs, double scale) {
        auto [o, lse, ws] = sel_fwd(q, k, v, idx, bs, cu, scale);
        check_status(ptr(ws), q, "fsa_sel_fwd status");
        ctx->save_for_backward({q, k, v, o, lse, idx, cu, ws});
        ctx->saved_data["bs"] = bs;
        ctx->saved_data["scale"] = scale;
        return o;
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list g) {
        const auto t = ctx->get_saved_variables();
        auto [dq, dk, dv] = sel_bwd(t[0], t[1], t[2], t[3], t[4], g[0], t[5], ctx->saved_data["bs"].toInt(), t[6],
                                    ctx->saved_data["scale"].toDouble(), t[7]);
        check_status(ptr(t[7]), t[0], "fsa_sel_bwd status");
        return {dq, dk, dv, Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

Tensor sel_attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, int64_t bs, const Tensor& cu, double scale) {
    if (wants_grad({&q, &k, &v})) return SelAttention::apply(q, k, v, idx, cu, bs, scale);
    auto [o, lse, ws] = sel_fwd(q, k, v, idx, bs, cu, scale);
    check_status(ptr(ws), q, "fsa_sel_fwd status");
    return o;
}

void bind_sel(pybind11::module& m) {
    m.def("sel_fwd", &sel_fwd);
    m.def("sel_bwd", &sel_bwd);
    m.def("sel_attention", &sel_attention);
}

}  // namespace fsa_host
