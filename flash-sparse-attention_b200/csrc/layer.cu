// Small kernels of the layer (fsa/module/fsa.py:71-171) around its GEMMs and attention kernels: rotation tables and compressed
// offsets, the rotations with the row ranges of the two dense branches, and the rotations' backward with the sums of the
// branches' gradients.  As torch glue these were 45 of the 79 launches of a forward and several passes over [N, heads, d].
#include "../../include/fsa_sm100.h"
#include "sel_common.cuh"

namespace fsa {

// cos / sin of position p (row p, [len, half], activation dtype, angle in fp32: nsa_ref/module/rope.py:113-124), and by the first
// CTA the compressed offsets cu_cmp[B + 1] (nsa_ref/ops/linear_compress.py:334-337).
template <typename ET>
__global__ void __launch_bounds__(256) layer_prep_kernel(const int* __restrict__ cu, int B, int64_t len, const float* __restrict__ inv_freq, int half,
                                                         int ks, int stride, ET* __restrict__ cs, ET* __restrict__ sn, int* __restrict__ cu_cmp) {
    const int64_t total = len * half;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t pos = i / half;
        const float a = (float)pos * __ldg(inv_freq + (i - pos * half));
        cs[i] = (ET)cosf(a);
        sn[i] = (ET)sinf(a);
    }
    if (blockIdx.x != 0) return;
    __shared__ int wsum[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int carry = 0;
    if (tid == 0) cu_cmp[0] = 0;
    for (int b0 = 0; b0 < B; b0 += 256) {
        const int b = b0 + tid;
        const int L = b < B ? __ldg(cu + b + 1) - __ldg(cu + b) : 0;
        int v = L >= ks ? (L - ks) / stride + 1 : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane == 31) wsum[warp] = v;
        __syncthreads();
        int base = carry;
        for (int w = 0; w < warp; ++w) base += wsum[w];
        if (b < B) cu_cmp[b + 1] = base + v;
        for (int w = 0; w < 8; ++w) carry += wsum[w];
        __syncthreads();
    }
}

// (x1, x2) = (x1 cos - x2 sin, x1 sin + x2 cos) on eight pairs
template <typename ET>
__device__ __forceinline__ void rotate8(float (&x1)[8], float (&x2)[8], const ET* cs, const ET* sn, float sign) {
    const uint4 co = __ldg(reinterpret_cast<const uint4*>(cs)), si = __ldg(reinterpret_cast<const uint4*>(sn));
    const uint32_t *pc = &co.x, *ps = &si.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 c = ElemTraits<ET>::unpack2(pc[i]);
        float2 s = ElemTraits<ET>::unpack2(ps[i]);
        s.x *= sign; s.y *= sign;
        const float a0 = x1[2 * i], b0 = x2[2 * i], a1 = x1[2 * i + 1], b1 = x2[2 * i + 1];
        x1[2 * i] = a0 * c.x - b0 * s.x;
        x2[2 * i] = a0 * s.x + b0 * c.x;
        x1[2 * i + 1] = a1 * c.y - b1 * s.y;
        x2[2 * i + 1] = a1 * s.y + b1 * c.y;
    }
}
template <typename ET>
__device__ __forceinline__ void add8(const uint4& v, float (&a)[8]) {
    const uint32_t* p = &v.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = ElemTraits<ET>::unpack2(p[i]);
        a[2 * i] += f.x;
        a[2 * i + 1] += f.y;
    }
}

// (read once; q may be rotated in place, so not through the read-only path)
__device__ __forceinline__ uint4 ld_stream(const uint4* p) { return __ldcs(p); }

struct LayerRopeParams {
    const int *cu, *cu_cmp;
    int B, Hq, Hk, D, ks, stride, window;
    int64_t N, Nc;
    const void *cs, *sn;
    // forward: q[0], k[0] in; backward: the gradients of the branches, summed before the rotation (q: 3, k: 2; k[2], that of the
    // unrotated keys, and all of v after it)
    const void* q[3];
    const void* k[3];
    const void* v[3];
    int64_t q_sn, k_sn;         // token strides of q[0], k[0] (forward; the gradients are contiguous)
    void *q_out, *k_out, *v_out;     // contiguous
    void* cmp;                  // [Nc, Hk, D] rotated in place: compressed keys or their gradient
    int *hi_cmp, *lo_win, *hi_win;   // [N] or null: row ranges of the dense branches (nsa_ref/ops/compressed_attention.py:77-80; the window)
};

// One thread = eight pairs of one row; rows of q, then of k, then of the compressed keys (whose position is their row times the
// stride, so the same tables serve them), then of v (backward: sums only).
template <bool BWD, typename ET>
__global__ void __launch_bounds__(256) layer_rope_kernel(const LayerRopeParams p) {
    const int half = p.D / 2, vec = half / 8;
    const int64_t nq = p.N * p.Hq * vec, nk = p.N * p.Hk * vec, nc = p.Nc * p.Hk * vec;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nq + nk + nc + (BWD ? nk : 0)) return;
    const int kind = i < nq ? 0 : i < nq + nk ? 1 : i < nq + nk + nc ? 2 : 3;
    i -= kind == 0 ? 0 : kind == 1 ? nq : kind == 2 ? nq + nk : nq + nk + nc;
    const int H = kind == 0 ? p.Hq : p.Hk;
    const uint32_t i32 = (uint32_t)i;                  // (N * Hq * D / 16 fits in 32 bits: checked on the host)
    const int v = (int)(i32 % (uint32_t)vec), h = (int)(i32 / (uint32_t)vec % (uint32_t)H), n = (int)(i32 / (uint32_t)(vec * H));
    const int64_t at = ((int64_t)n * H + h) * p.D + v * 8;       // contiguous element
    float x1[8], x2[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x1[j] = x2[j] = 0.f;
    // everything that does not depend on the position is loaded before the sequence is looked for
    uint4 a1[3], a2[3];
    auto load = [&](int j, const void* src, int64_t off) {
        a1[j] = ld_stream(reinterpret_cast<const uint4*>((const ET*)src + off));
        a2[j] = ld_stream(reinterpret_cast<const uint4*>((const ET*)src + off + half));
    };
    auto take = [&](int j) {
        add8<ET>(a1[j], x1);
        add8<ET>(a2[j], x2);
    };
    if (kind == 2) {
        load(0, p.cmp, at);
    } else if (!BWD) {
        load(0, kind == 0 ? p.q[0] : p.k[0], (int64_t)n * (kind == 0 ? p.q_sn : p.k_sn) + h * p.D + v * 8);
    } else {
#pragma unroll
        for (int j = 0; j < 3; ++j) load(j, kind == 0 ? p.q[j] : kind == 1 ? p.k[j] : p.v[j], at);
    }
    auto put = [&](void* dst, const float (&y1)[8], const float (&y2)[8]) {
        uint4 o1, o2;
        uint32_t *q1 = &o1.x, *q2 = &o2.x;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            q1[j] = ElemTraits<ET>::pack2(y1[2 * j], y1[2 * j + 1]);
            q2[j] = ElemTraits<ET>::pack2(y2[2 * j], y2[2 * j + 1]);
        }
        *reinterpret_cast<uint4*>((ET*)dst + at) = o1;
        *reinterpret_cast<uint4*>((ET*)dst + at + half) = o2;
    };
    if (BWD && kind == 3) {
        take(0); take(1); take(2);
        put(p.v_out, x1, x2);
        return;
    }
    const int* cu = kind == 2 ? p.cu_cmp : p.cu;
    const int b = find_seq(cu, p.B, n);
    const int pos = n - __ldg(cu + b);
    const int64_t trow = (int64_t)(kind == 2 ? pos * p.stride : pos) * half + v * 8;
    take(0);
    if (BWD && kind < 2) take(1);
    if (BWD && kind == 0) take(2);
    rotate8<ET>(x1, x2, (const ET*)p.cs + trow, (const ET*)p.sn + trow, BWD ? -1.f : 1.f);
    if (BWD && kind == 1) take(2);
    put(kind == 0 ? p.q_out : kind == 1 ? p.k_out : p.cmp, x1, x2);
    if (!BWD && kind == 1 && h == 0 && v == 0 && p.hi_cmp) {
        const int c0 = __ldg(p.cu_cmp + b), nb = __ldg(p.cu_cmp + b + 1) - c0;
        const int vis = pos >= p.ks - 1 ? min((pos - (p.ks - 1)) / p.stride + 1, nb) : 0;
        p.hi_cmp[n] = vis > 0 ? c0 + vis - 1 : -1;
        p.lo_win[n] = n - min(pos, p.window);
        p.hi_win[n] = n;
    }
}

// Partial column sums over contiguous shares of the rows, out[part, h, :] = sum of dy[row, h, :] (fp32, fixed order): the
// gradient of the compressor's bias, finished by its consumer (whose status word is cleared here).
template <int D, typename ET>
__global__ void __launch_bounds__(256) column_sum_kernel(const ET* __restrict__ dy, int64_t rows, int H, float* __restrict__ out, int* __restrict__ status) {
    constexpr int CG = D / 8, KL = 256 / CG;
    __shared__ float red[8][D];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cgi = tid % CG, kl = tid / CG, h = blockIdx.x;
    if (tid == 0 && h == 0 && blockIdx.y == 0) *status = kStatusOk;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const int64_t per = (rows + gridDim.y - 1) / gridDim.y, r1 = min(rows, per * (blockIdx.y + 1));
#pragma unroll 4
    for (int64_t r = per * blockIdx.y + kl; r < r1; r += KL) add8<ET>(__ldg(reinterpret_cast<const uint4*>(dy + (r * H + h) * D) + cgi), acc);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
        for (int o = CG; o < 32; o <<= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
        if (lane < CG) red[warp][cgi * 8 + j] = acc[j];
    }
    __syncthreads();
    if (tid < D) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += red[w][tid];
        out[((int64_t)blockIdx.y * H + h) * D + tid] = s;
    }
}

}  // namespace fsa

using namespace fsa;

extern "C" int fsa_layer_prep(const int32_t* cu_seqlens, int batch, int64_t max_len, const float* inv_freq, int head_dim, int kernel_size,
                              int kernel_stride, int dtype, void* cos_tab, void* sin_tab, int32_t* cu_cmp, void* stream) {
    if (!cu_seqlens || !inv_freq || !cos_tab || !sin_tab || !cu_cmp || batch < 0 || max_len < 0 || head_dim <= 0 || head_dim % 16 || kernel_stride <= 0)
        return FSA_ERR_BAD_ARG;
    if (dtype != FSA_DTYPE_BF16 && dtype != FSA_DTYPE_FP16) return FSA_ERR_BAD_ARG;
    (void)cudaGetLastError();
    const int64_t want = (max_len * (head_dim / 2) + 255) / 256, most = sm_count() * 8;
    const unsigned grid = (unsigned)(want < 1 ? 1 : want > most ? most : want);
    if (dtype == FSA_DTYPE_BF16)
        layer_prep_kernel<__nv_bfloat16><<<grid, 256, 0, (cudaStream_t)stream>>>(cu_seqlens, batch, max_len, inv_freq, head_dim / 2, kernel_size,
                                                                                kernel_stride, (__nv_bfloat16*)cos_tab, (__nv_bfloat16*)sin_tab, cu_cmp);
    else
        layer_prep_kernel<__half><<<grid, 256, 0, (cudaStream_t)stream>>>(cu_seqlens, batch, max_len, inv_freq, head_dim / 2, kernel_size, kernel_stride,
                                                                         (__half*)cos_tab, (__half*)sin_tab, cu_cmp);
    return cudaGetLastError() == cudaSuccess ? FSA_OK : FSA_ERR_CUDA;
}

template <bool BWD>
static int run_rope(const LayerRopeParams& p, int dtype, cudaStream_t stream) {
    if (dtype != FSA_DTYPE_BF16 && dtype != FSA_DTYPE_FP16) return FSA_ERR_BAD_ARG;
    if (p.D % 16) return FSA_ERR_BAD_ARG;
    const int64_t threads = (p.N * (p.Hq + (BWD ? 2 : 1) * p.Hk) + p.Nc * p.Hk) * (p.D / 16);
    if (threads >= ((int64_t)1 << 32)) return FSA_ERR_UNSUPPORTED;
    if (threads == 0) return FSA_OK;
    (void)cudaGetLastError();
    const unsigned grid = (unsigned)((threads + 255) / 256);
    if (prefer_l1(dtype == FSA_DTYPE_BF16 ? (const void*)layer_rope_kernel<BWD, __nv_bfloat16> : (const void*)layer_rope_kernel<BWD, __half>) != cudaSuccess)
        return FSA_ERR_CUDA;
    if (dtype == FSA_DTYPE_BF16) layer_rope_kernel<BWD, __nv_bfloat16><<<grid, 256, 0, stream>>>(p);
    else layer_rope_kernel<BWD, __half><<<grid, 256, 0, stream>>>(p);
    return cudaGetLastError() == cudaSuccess ? FSA_OK : FSA_ERR_CUDA;
}

extern "C" int fsa_layer_rope_fwd(const void* q, int64_t q_stride_n, const void* k, int64_t k_stride_n, void* cmp_k, const void* cos_tab,
                                  const void* sin_tab, const int32_t* cu_seqlens, const int32_t* cu_cmp, int batch, int64_t total, int64_t total_cmp,
                                  int num_q_heads, int num_kv_heads, int head_dim, int kernel_size, int kernel_stride, int window, int dtype,
                                  void* q_out, void* k_out, int32_t* hi_cmp, int32_t* lo_win, int32_t* hi_win, void* stream) {
    if (!q || !k || !cos_tab || !sin_tab || !cu_seqlens || !cu_cmp || !q_out || !k_out || (total_cmp > 0 && !cmp_k)) return FSA_ERR_BAD_ARG;
    if ((q_stride_n % 8) || (k_stride_n % 8) || (hi_cmp && (!lo_win || !hi_win))) return FSA_ERR_BAD_ARG;
    LayerRopeParams p = {};
    p.cu = cu_seqlens; p.cu_cmp = cu_cmp; p.B = batch; p.Hq = num_q_heads; p.Hk = num_kv_heads; p.D = head_dim; p.ks = kernel_size;
    p.stride = kernel_stride; p.window = window; p.N = total; p.Nc = total_cmp; p.cs = cos_tab; p.sn = sin_tab; p.q[0] = q; p.k[0] = k;
    p.q_sn = q_stride_n; p.k_sn = k_stride_n; p.q_out = q_out; p.k_out = k_out; p.cmp = cmp_k; p.hi_cmp = hi_cmp; p.lo_win = lo_win; p.hi_win = hi_win;
    return run_rope<false>(p, dtype, (cudaStream_t)stream);
}

extern "C" int fsa_layer_rope_bwd(const void* dq0, const void* dq1, const void* dq2, const void* dk0, const void* dk1, const void* dk2,
                                  const void* dv0, const void* dv1, const void* dv2, void* dcmp_k, const void* cos_tab, const void* sin_tab,
                                  const int32_t* cu_seqlens, const int32_t* cu_cmp, int batch, int64_t total, int64_t total_cmp, int num_q_heads,
                                  int num_kv_heads, int head_dim, int kernel_stride, int dtype, void* dq, void* dk, void* dv, void* stream) {
    if (total > 0 && (!dq0 || !dq1 || !dq2 || !dk0 || !dk1 || !dk2 || !dv0 || !dv1 || !dv2 || !dq || !dk || !dv)) return FSA_ERR_BAD_ARG;
    if (!cos_tab || !sin_tab || !cu_seqlens || !cu_cmp || (total_cmp > 0 && !dcmp_k)) return FSA_ERR_BAD_ARG;
    LayerRopeParams p = {};
    p.cu = cu_seqlens; p.cu_cmp = cu_cmp; p.B = batch; p.Hq = num_q_heads; p.Hk = num_kv_heads; p.D = head_dim; p.stride = kernel_stride;
    p.N = total; p.Nc = total_cmp; p.cs = cos_tab; p.sn = sin_tab; p.q[0] = dq0; p.q[1] = dq1; p.q[2] = dq2; p.k[0] = dk0; p.k[1] = dk1; p.k[2] = dk2;
    p.v[0] = dv0; p.v[1] = dv1; p.v[2] = dv2; p.q_out = dq; p.k_out = dk; p.v_out = dv; p.cmp = dcmp_k;
    return run_rope<true>(p, dtype, (cudaStream_t)stream);
}

namespace fsa {
__global__ void __launch_bounds__(256) layer_every_block_kernel(const int* __restrict__ cu, int B, int N, int Hk, int T, int BK, int* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;       // row (kv head, token), slot
    if (i >= (int64_t)Hk * N * T) return;
    const int64_t row = i / T;
    const int slot = (int)(i - row * T), n = (int)(row % N);
    out[i] = slot <= (n - __ldg(cu + find_seq(cu, B, n))) / BK ? slot : -1;
}
}  // namespace fsa

extern "C" int fsa_layer_every_block(const int32_t* cu_seqlens, int batch, int64_t total, int num_kv_heads, int topk, int block_size, int32_t* topk_idx,
                                     void* stream) {
    if (!cu_seqlens || batch < 0 || total < 0 || total >= kMaxTokens || num_kv_heads <= 0 || topk <= 0 || block_size <= 0 || (total > 0 && !topk_idx))
        return FSA_ERR_BAD_ARG;
    if (total == 0 || batch == 0) return FSA_OK;
    (void)cudaGetLastError();
    const int64_t n = total * num_kv_heads * topk;
    layer_every_block_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(cu_seqlens, batch, (int)total, num_kv_heads, topk, block_size, topk_idx);
    return cudaGetLastError() == cudaSuccess ? FSA_OK : FSA_ERR_CUDA;
}

// partial column sums [parts][H][D]; called by the compressor's backward
namespace fsa {
cudaError_t launch_column_sum(int dtype, int D, const void* dy, int64_t rows, int H, int parts, float* out, int* status, cudaStream_t stream) {
    const dim3 grid((unsigned)H, (unsigned)parts);
    if (dtype == FSA_DTYPE_BF16) {
        if (D == 128) column_sum_kernel<128, __nv_bfloat16><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)dy, rows, H, out, status);
        else column_sum_kernel<64, __nv_bfloat16><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)dy, rows, H, out, status);
    } else {
        if (D == 128) column_sum_kernel<128, __half><<<grid, 256, 0, stream>>>((const __half*)dy, rows, H, out, status);
        else column_sum_kernel<64, __half><<<grid, 256, 0, stream>>>((const __half*)dy, rows, H, out, status);
    }
    return cudaGetLastError();
}
}  // namespace fsa
