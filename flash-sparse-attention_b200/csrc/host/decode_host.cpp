// The one-GPU decode step in native code: scratch carved from one allocation, six to eight launches, no synchronisation (so
// that a CUDA graph can hold it).
#include "host_common.h"

#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>

#include <climits>
#include <optional>

namespace fsa_host {

struct DecodeCfg {
    int ks, stride, bs, topk, init_blocks, local_blocks, window;
    int64_t max_len;
    double scale;      // 0: 1 / sqrt(head_dim)
};

static DecodeCfg cfg_of(const std::vector<int64_t>& c, double scale) {
    TORCH_CHECK_VALUE(c.size() == 8, "decode settings");
    return {(int)c[0], (int)c[1], (int)c[2], (int)c[3], (int)c[4], (int)c[5], (int)c[6], c[7], scale};
}

static int64_t sms() {
    static const int64_t n = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
    return n;
}

// Chunks of the compressed rows.  Work per CTA of the two attention passes: as long as possible (few partials, a ring of loads that
// stays full) while about four CTAs per SM are left for each pass: a small batch is split finely, a full one takes 1024 rows /
// 16 blocks at a time.
struct Chunks {
    int rows, n;
    Chunks(const DecodeCfg& c, int64_t heads) {
        const int64_t max_cmp = std::max<int64_t>(c.max_len >= c.ks ? (c.max_len - c.ks) / c.stride + 1 : 0, 1);
        const int64_t ctas = 4 * sms(), per = (max_cmp * heads + ctas - 1) / ctas;
        rows = (int)std::min<int64_t>(1024, std::max<int64_t>(64, (per + 63) / 64 * 64));
        n = (int)((max_cmp + rows - 1) / rows);
    }
};

static int max_blocks(const DecodeCfg& c) { return (int)std::min<int64_t>((c.max_len + c.bs - 1) / c.bs, INT_MAX); }

// Do the kernels take these sizes?  (gate_dim: see fsa_decode_step_sizes)
static bool takes_sizes(int64_t B, int64_t Hq, int64_t Hk, int64_t D, const DecodeCfg& c, int64_t gate_dim) {
    return B > 0 && Hk > 0 && c.ks > 0 && c.stride > 0 && c.bs > 0 &&
           fsa_decode_step_sizes((int)Hq, (int)Hk, (int)D, c.ks, c.stride, c.bs, c.topk, max_blocks(c), Chunks(c, B * Hk).n, (int)gate_dim) == FSA_OK;
}

static bool packed_like(const Tensor& t, const Tensor& q, int64_t Hk) {
    return t.dim() == 3 && t.scalar_type() == q.scalar_type() && t.device() == q.device() && t.size(1) == Hk && t.size(2) == q.size(2) &&
           t.stride(2) == 1 && t.stride(1) == t.size(2) && t.stride(0) % 8 == 0 && ((uintptr_t)t.data_ptr() & 15) == 0;
}
static bool lengths_like(const Tensor& t, const Tensor& q, int64_t B) {
    return t.scalar_type() == at::kInt && t.device() == q.device() && t.numel() == B && t.is_contiguous();
}

// Three branches of one token per sequence and their gate mix; q [B, Hq, D] rotated, gate [B, 3].
static std::tuple<Tensor, Tensor> attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cmp_k, const Tensor& cmp_v,
                                            const Tensor& seq_len, const Tensor& seq_row0, const Tensor& cmp_row0, const Tensor& gate,
                                            const DecodeCfg& c) {
    const int B = (int)q.size(0), Hq = (int)q.size(1), D = (int)q.size(2), Hk = (int)k.size(1), dt = dtype_code(q);
    const float scale = (float)(c.scale > 0 ? c.scale : 1.0 / std::sqrt((double)D));
    void* st = stream_of(q);
    const Chunks chunks(c, (int64_t)B * Hk);
    const int chunk = chunks.rows, nchunk = chunks.n;
    const int npieces = (c.window + 1 + c.bs - 1) / c.bs, R = c.topk + npieces;
    int rpp = 16;
    while (rpp > 1 && (c.topk % rpp || (int64_t)B * Hk * ((R + rpp - 1) / rpp) < 2 * sms())) rpp /= 2;
    const int ns = c.topk / rpp, nw = (npieces + rpp - 1) / rpp, P2 = ns + nw;
    const int64_t ld = (int64_t)chunk * nchunk;
    auto al = [](int64_t n) { return (n + 255) / 256 * 256; };
    const int64_t rowsq = (int64_t)B * Hq;
    const int64_t b_o1 = al(rowsq * nchunk * D * 4), b_m1 = al(rowsq * nchunk * 8), b_sc = al((int64_t)B * Hk * ld * 4),
                  b_o2 = al(rowsq * P2 * D * 4), b_m2 = al(rowsq * P2 * 8), b_r = al((int64_t)B * Hk * R * 4), b_oc = al(rowsq * D * 2);
    const Tensor scratch = bytes(b_o1 + b_m1 + b_sc + b_o2 + b_m2 + 2 * b_r + b_oc, q);
    char* p = (char*)scratch.data_ptr();
    auto take = [&](int64_t n) { char* r = p; p += n; return r; };
    float* o1 = (float*)take(b_o1);
    float* m1 = (float*)take(b_m1);
    float* sc = (float*)take(b_sc);
    float* o2 = (float*)take(b_o2);
    float* m2 = (float*)take(b_m2);
    int32_t* lo = (int32_t*)take(b_r);
    int32_t* hi = (int32_t*)take(b_r);
    void* oc = take(b_oc);
    Tensor topk = i32({B, Hk, c.topk}, q), out = fresh_like(q);
    check(fsa_decode_cmp_partial(ptr(q), ptr(cmp_k), ptr(cmp_v), cmp_k.size(0), cmp_k.stride(0), iptr(seq_len), iptr(cmp_row0), B, Hq, Hk, D,
                                 c.ks, c.stride, chunk, nchunk, dt, scale, o1, m1, sc, ld, st),
          "fsa_decode_cmp_partial");
    check(fsa_decode_merge_select(o1, m1, nchunk, sc, ld, iptr(seq_len), iptr(seq_row0), B, Hq, Hk, D, c.ks, c.stride, c.bs, c.init_blocks,
                                  c.local_blocks, c.topk, max_blocks(c), c.window, npieces, dt, oc,
                                  topk.data_ptr<int32_t>(), lo, hi, st),
          "fsa_decode_merge_select");
    check(fsa_decode_attn_partial(ptr(q), ptr(k), ptr(v), k.size(0), k.stride(0), lo, hi, B, Hq, Hk, D, R, rpp, c.bs, 1, dt, scale, o2, m2,
                                  nullptr, 0, st),
          "fsa_decode_attn_partial");
    check(fsa_decode_finish(o2, m2, rowsq, ns, nw, P2, D, Hq, dt, oc, ptr(gate), ptr(out), st), "fsa_decode_finish");
    return {out, topk};
}

// What these functions return: the outputs, or nothing where the kernels do not take the call (before anything was launched).
using Outcome = std::optional<std::tuple<Tensor, Tensor>>;

Outcome decode_mixed(const Tensor& q_, const Tensor& k, const Tensor& v, const Tensor& cmp_k, const Tensor& cmp_v, const Tensor& seq_len,
                     const Tensor& seq_row0, const Tensor& cmp_row0, const Tensor& gate, const std::vector<int64_t>& cfg, double scale) {
    c10::cuda::CUDAGuard guard(q_.device());
    const DecodeCfg c = cfg_of(cfg, scale);
    const Tensor q = q_.contiguous();
    TORCH_CHECK_VALUE(q.dim() == 3 && k.dim() == 3 && gate.numel() == 3 * q.size(0), "decode: q [B, Hq, D], cache rows [rows, Hk, D], gate [B, 3]");
    const int64_t B = q.size(0), Hk = k.size(1);
    if (!takes_sizes(B, q.size(1), Hk, q.size(2), c, -1)) return std::nullopt;
    for (auto* t : {&k, &v, &cmp_k, &cmp_v})
        if (!packed_like(*t, q, Hk)) return std::nullopt;
    if (v.strides() != k.strides() || cmp_v.strides() != cmp_k.strides()) return std::nullopt;
    for (auto* t : {&seq_len, &seq_row0, &cmp_row0})
        if (!lengths_like(*t, q, B)) return std::nullopt;
    return attention(q, k, v, cmp_k, cmp_v, seq_len, seq_row0, cmp_row0, gate.to(q.scalar_type()).contiguous(), c);
}

// The buffers of a DecodeCache, in this order: k, v, cmp_k, cmp_v, k_tail, v_tail, seq_len, seq_row0, cmp_row0.
using Cache = std::vector<Tensor>;

static bool weight(const Tensor& w, const Tensor& x, at::IntArrayRef shape) {
    return w.scalar_type() == x.scalar_type() && w.device() == x.device() && w.is_contiguous() && w.sizes() == shape && ((uintptr_t)w.data_ptr() & 15) == 0;
}

// (under autocast the parts' library products take other types than their operands')
static bool native_call(const Tensor& x) { return x.is_cuda() && !at::autocast::is_autocast_enabled(at::kCUDA); }

// Does the native step take this call?  x stands for the type and the device of everything.
static bool served(const Cache& t, const Tensor& x, int64_t Hq, int64_t D, const Tensor& w_key, const Tensor& w_value, const Tensor& pe,
                   const DecodeCfg& c, int64_t gate_dim) {
    if (t.size() != 9 || t[0].dim() != 3) return false;
    const int64_t B = x.size(0), Hk = t[0].size(1), rows = t[0].size(0) - 1;        // (the last row of a buffer is a spare one)
    if (!takes_sizes(B, Hq, Hk, D, c, gate_dim) || rows <= 0 || rows % B || t[2].dim() != 3 || (t[2].size(0) - 1) % B) return false;
    const int64_t cmp_rows = t[2].size(0) - 1, ring = B * c.ks;
    const int64_t want[6] = {rows, rows, cmp_rows, cmp_rows, ring, ring};
    for (int i = 0; i < 6; ++i)
        if (!weight(t[i], x, {want[i] + 1, Hk, D})) return false;
    for (int i = 6; i < 9; ++i)
        if (!lengths_like(t[i], x, B)) return false;
    return weight(w_key, x, {Hk, c.ks * D, D}) && weight(w_value, x, {Hk, c.ks * D, D}) && weight(pe, x, {Hk, c.ks, D});
}

// Append (with the gate from logits z, or from gx and its weight), compressor, attention.
static std::tuple<Tensor, Tensor> step(const Tensor& q_in, const Tensor& k_new, const Tensor& v_new, Tensor q, const Tensor& inv_freq,
                                       const Tensor& z, const Tensor& gx, const Tensor& gw, const Cache& t, const Tensor& w_key,
                                       const Tensor& w_value, const Tensor& pe, bool compress, const DecodeCfg& c) {
    const int B = (int)k_new.size(0), Hk = (int)k_new.size(1), D = (int)k_new.size(2), Hq = (int)q.size(1), dt = dtype_code(k_new);
    const int cap = (int)((t[0].size(0) - 1) / B), cmp_cap = (int)((t[2].size(0) - 1) / B);
    const float* freq = inv_freq.defined() ? inv_freq.data_ptr<float>() : nullptr;
    void* st = stream_of(k_new);
    const Tensor gate = fresh({B, 3}, k_new);
    check(fsa_decode_append(ptr(q_in), ptr(k_new), ptr(v_new), ptr(q), ptr(t[0]), ptr(t[1]), ptr(t[4]), ptr(t[5]), freq,
                            t[6].data_ptr<int32_t>(), iptr(t[7]), B, cap, Hq, Hk, D, c.ks, ptr(z), ptr(gx), ptr(gw),
                            gx.defined() ? (int)gx.size(-1) : 0, ptr(gate), dt, st),
          "fsa_decode_append");
    if (compress)
        check(fsa_decode_compress(ptr(t[4]), ptr(t[5]), ptr(w_key), ptr(w_value), ptr(pe), freq, iptr(t[6]), iptr(t[8]), ptr(t[2]), ptr(t[3]), B,
                                  Hk, D, c.ks, c.stride, cmp_cap, dt, st),
              "fsa_decode_compress");
    return attention(q, t[0], t[1], t[2], t[3], t[6], t[7], t[8], gate, c);
}

// FlashSparseAttentionDecodeKernel.step: q, k_new, v_new in, [B, Hq * D] and the block ids out.
Outcome decode_kernel_step(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& gw, const Cache& t, const Tensor& w_key,
                           const Tensor& w_value, const Tensor& pe, bool compress, const std::vector<int64_t>& cfg, double scale) {
    if (!native_call(q_)) return std::nullopt;
    c10::cuda::CUDAGuard guard(q_.device());
    const DecodeCfg c = cfg_of(cfg, scale);
    const Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous();
    if (q.dim() != 3 || k.dim() != 3 || !weight(k, q, {q.size(0), k.size(1), q.size(2)}) || !weight(v, q, k.sizes()) || ((uintptr_t)q.data_ptr() & 15) ||
        t.size() != 9 || t[0].dim() != 3 || t[0].size(1) != k.size(1))
        return std::nullopt;
    const Tensor gx = q.view({q.size(0), -1});
    if (!weight(gw, q, {3, gx.size(1)}) || !served(t, q, q.size(1), q.size(2), w_key, w_value, pe, c, gx.size(1))) return std::nullopt;
    auto [y, ids] = step(q, k, v, q, Tensor(), Tensor(), gx, gw, t, w_key, w_value, pe, compress, c);
    return std::make_tuple(y.view({y.size(0), -1}), ids);
}

// Rows up to which the library's own skinny projection is used (one MMA tile of rows; above it a library GEMM's tiles are fuller).
constexpr int kProjRows = 16;

static void project(const Tensor& x, std::initializer_list<Tensor> ws, std::initializer_list<Tensor> ys) {
    const void* w[4];
    void* y[4];
    int rows[4];
    int64_t ystr[4];
    int n = 0;
    for (auto& t : ws) { w[n] = ptr(t); rows[n] = (int)t.size(0); ++n; }
    n = 0;
    for (auto& t : ys) { y[n] = ptr(t); ystr[n] = t.stride(0); ++n; }
    check(fsa_decode_proj(ptr(x), x.stride(0), (int)x.size(0), (int)x.size(1), n, w, rows, y, ystr, dtype_code(x), stream_of(x)), "fsa_decode_proj");
}

// FlashSparseAttentionDecode.step: x [B, hidden] in, [B, hidden] and the block ids out.
Outcome decode_layer_step(const Tensor& x_, const Tensor& wq, const Tensor& wk, const Tensor& wv, const Tensor& wo, const Tensor& gw,
                          const Tensor& inv_freq, int64_t D, const Cache& t, const Tensor& w_key, const Tensor& w_value, const Tensor& pe,
                          bool compress, const std::vector<int64_t>& cfg, double scale) {
    if (!native_call(x_)) return std::nullopt;
    c10::cuda::CUDAGuard guard(x_.device());
    const DecodeCfg c = cfg_of(cfg, scale);
    const Tensor flat = x_.contiguous(), x = flat.dim() == 2 ? flat : flat.view({flat.size(0), -1});
    const int64_t B = x.size(0), hidden = x.size(1), nq = wq.size(0), nk = wk.size(0);
    const bool skinny = B <= kProjRows && hidden % 256 == 0 && nq % 256 == 0;
    if (((uintptr_t)x.data_ptr() & 15) || t.size() != 9 || t[0].dim() != 3 || D <= 0 || nq % D || nk != t[0].size(1) * D ||
        inv_freq.scalar_type() != at::kFloat || inv_freq.device() != x.device() || inv_freq.numel() != D / 2 || !weight(wq, x, {nq, hidden}) ||
        !weight(wk, x, {nk, hidden}) || !weight(wv, x, {nk, hidden}) || !weight(wo, x, {wo.size(0), nq}) || !weight(gw, x, {3, hidden}) ||
        !served(t, x, nq / D, D, w_key, w_value, pe, c, skinny ? 0 : hidden))
        return std::nullopt;
    Tensor q, k, v, z;
    if (skinny) {
        q = fresh({B, nq}, x);
        k = fresh({B, nk}, x);
        v = fresh({B, nk}, x);
        z = fresh({B, 3}, x);
        project(x, {wq, wk, wv, gw}, {q, k, v, z});
    } else {
        q = at::linear(x, wq);
        k = at::linear(x, wk);
        v = at::linear(x, wv);
    }
    q = q.view({B, nq / D, D});
    auto [mixed, ids] = step(q, k.view({B, nk / D, D}), v.view({B, nk / D, D}), q, inv_freq, z, skinny ? Tensor() : x, gw, t, w_key, w_value, pe,
                             compress, c);
    const Tensor m = mixed.view({B, nq});
    if (!skinny) return std::make_tuple(at::linear(m, wo), ids);
    Tensor y = fresh({B, wo.size(0)}, x);
    project(m, {wo}, {y});
    return std::make_tuple(y, ids);
}

// dst[i].copy_(src[i]) of a captured step's inputs in one launch; false, and nothing done, where that is more than a copy of bytes.
static bool copy_inputs(const std::vector<Tensor>& dst, const std::vector<Tensor>& src) {
    const size_t n = dst.size();
    if (n != src.size() || n == 0 || n > 8) return false;
    const void* s[8];
    void* d[8];
    int64_t b[8];
    for (size_t i = 0; i < n; ++i) {
        if (!dst[i].is_cuda() || src[i].device() != dst[0].device() || dst[i].device() != dst[0].device() || src[i].scalar_type() != dst[i].scalar_type() ||
            src[i].sizes() != dst[i].sizes() || !src[i].is_contiguous() || !dst[i].is_contiguous() || src[i].is_conj() || src[i].is_neg() ||
            dst[i].is_conj() || dst[i].is_neg() || (dst[i].requires_grad() && at::GradMode::is_enabled()) || wants_grad({&src[i]}))
            return false;
        s[i] = src[i].data_ptr();
        d[i] = dst[i].data_ptr();
        b[i] = (int64_t)src[i].nbytes();
        for (size_t j = 0; j < n; ++j)      // (a source in another's destination: one after the other)
            if ((const char*)s[i] < (const char*)dst[j].data_ptr() + dst[j].nbytes() && (const char*)dst[j].data_ptr() < (const char*)s[i] + b[i]) return false;
    }
    c10::cuda::CUDAGuard guard(dst[0].device());
    check(fsa_copy((int)n, s, d, b, stream_of(dst[0])), "fsa_copy");
    return true;
}

void bind_decode(pybind11::module& m) {
    m.def("copy_inputs", &copy_inputs);
    m.def("decode_mixed", &decode_mixed);
    m.def("decode_kernel_step", &decode_kernel_step);
    m.def("decode_layer_step", &decode_layer_step);
}

}  // namespace fsa_host
