// The small kernels of a one-GPU decode step around decode_partial_tma (decode.cu): projections of a few rows, the append of
// the new token with its gate, the incremental compressor, and merge + top-k + row ranges.  A step moves megabytes through
// kernels of a few microseconds, so what bounds it is the number of launches and dependent steps: 63 launches (torch glue
// around the library's kernels) took 180 us of GPU time for eight requests whose bytes need 25.
//
// Every kernel of a step is launched as a dependent one (sm100_prims.cuh): its CTAs come up while the kernel before it ends, and the
// projections fetch their weights into L2 meanwhile (one request of 8191 tokens, 32 / 8 heads with projections: 58.0 -> 49.7 us a
// step, 33 MB of weights being on their way under the merge; from a graph, where launches cost less, 72.5 -> 71.0 for eight requests).
//
// Replaces the host-side glue of the reference's step (fsa_preview/module/fsa_decode.py:84-199: projections, torch.cat of
// the caches, the incremental compressor fsa_preview/ops/linear_compress_decode.py:14-76, gate).
#include "../../include/fsa_sm100.h"

#include <cooperative_groups.h>
#include <initializer_list>

#include "sm100_prims.cuh"

namespace fsa {

template <typename ET> __device__ __forceinline__ float round_et(float v) {
    return ElemTraits<ET>::unpack2(ElemTraits<ET>::pack2(v, 0.f)).x;
}

template <typename ET>
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (ElemTraits<ET>::kIsBF16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------------------------------------------ projections
// y_i[b, :] = x[b, :] W_i^T for up to four weight matrices [rows_i, K] and up to 16 rows of x, in one launch.  Bound by
// reading the weights once (K/V/Q projections of a 4096-wide layer: 50 MB, 8 us), so the layout serves the loads: a CTA =
// 16 weight rows, its 8 warps split K, every lane loads 16 bytes of two weight rows and of its x row and uses them as MMA
// fragments as they are (the k index inside a group of 32 is permuted alike in both operands, which a sum does not notice).
// The warp-level MMA only has to keep up with the loads.  One library GEMM per matrix took 44 us for the four of a layer at
// one request; above 16 rows the library's tiles are the better choice.
struct DecodeProjParams {
    const void* w[4];
    void* y[4];
    int64_t y_stride[4];
    int rows[4];
    int tile0[5];        // first 16-row tile of every matrix; tile0[n] = total
    int n;
    const void* x;
    int64_t x_stride;
    int B, K;
};

template <int NT, typename ET>
__global__ void __launch_bounds__(256) decode_proj_kernel(const DecodeProjParams p) {
    __shared__ float red[8][16][8 * NT + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
    int m = 0;
    while (m + 1 < p.n && (int)blockIdx.x >= p.tile0[m + 1]) ++m;
    const int row0 = ((int)blockIdx.x - p.tile0[m]) * 16, rows = p.rows[m];
    const int kw = p.K >> 3;                       // this warp's share of K (a multiple of 32)
    // rows past the end of the matrix (and of x) repeat its last row: their products are dropped below
    const ET* w0 = (const ET*)p.w[m] + (int64_t)min(row0 + gid, rows - 1) * p.K + warp * kw + tig * 8;
    const ET* w1 = (const ET*)p.w[m] + (int64_t)min(row0 + gid + 8, rows - 1) * p.K + warp * kw + tig * 8;
    const ET* xr[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) xr[t] = (const ET*)p.x + (int64_t)min(t * 8 + gid, p.B - 1) * p.x_stride + warp * kw + tig * 8;
    // the CTA's 16 rows of W are fetched while the kernel before this one ends (a hint: nothing is read yet)
    {
        const char* wb = reinterpret_cast<const char*>((const ET*)p.w[m] + (int64_t)row0 * p.K);
        const int lines = min(16, rows - row0) * (p.K / 64);            // of 128 bytes
        for (int i = tid; i < lines; i += 256) prefetch_l2(wb + (int64_t)i * 128);
    }
    follow();
    float c[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t) c[t][0] = c[t][1] = c[t][2] = c[t][3] = 0.f;
#pragma unroll 4
    for (int k = 0; k < kw; k += 32) {
        const uint4 a = __ldcs(reinterpret_cast<const uint4*>(w0 + k)), b = __ldcs(reinterpret_cast<const uint4*>(w1 + k));
        uint4 xv[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) xv[t] = __ldcg(reinterpret_cast<const uint4*>(xr[t] + k));
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            mma_16816<ET>(c[t], a.x, b.x, a.y, b.y, xv[t].x, xv[t].y);
            mma_16816<ET>(c[t], a.z, b.z, a.w, b.w, xv[t].z, xv[t].w);
        }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        red[warp][gid][t * 8 + tig * 2] = c[t][0];
        red[warp][gid][t * 8 + tig * 2 + 1] = c[t][1];
        red[warp][gid + 8][t * 8 + tig * 2] = c[t][2];
        red[warp][gid + 8][t * 8 + tig * 2 + 1] = c[t][3];
    }
    __syncthreads();
    for (int i = tid; i < 16 * 8 * NT; i += 256) {
        const int r = i & 15, b = i >> 4;
        if (b >= p.B || row0 + r >= rows) continue;
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += red[w][r][b];
        ((ET*)p.y[m])[(int64_t)b * p.y_stride[m] + row0 + r] = (ET)s;
    }
}

// ------------------------------------------------------------------------------------------------ copies
struct CopyParams {
    const char* src[8];
    char* dst[8];
    int64_t bytes[8], first[9];          // first: 16-byte units before a buffer's own
    int n;
};
__global__ void __launch_bounds__(256) copy_kernel(const CopyParams p) {
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < p.first[p.n]; i += (int64_t)gridDim.x * 256) {
        int m = 0;
        while (i >= p.first[m + 1]) ++m;
        const int64_t at = (i - p.first[m]) * 16;
        const char* s = p.src[m] + at;
        char* d = p.dst[m] + at;
        if ((((uintptr_t)s | (uintptr_t)d) & 15) == 0 && at + 16 <= p.bytes[m]) *reinterpret_cast<uint4*>(d) = *reinterpret_cast<const uint4*>(s);
        else
            for (int64_t j = 0; j < 16 && at + j < p.bytes[m]; ++j) d[j] = s[j];
    }
}

// ------------------------------------------------------------------------------------------------ append
// One CTA per sequence: rotates q and k of the new token at its position t = seq_len[b] (inv_freq null: they come rotated),
// writes k, v to row t of the cache and the raw k, v to the compressor's ring, gate = sigmoid(z) with z given or computed
// here (z = gx Wg^T), and advances seq_len.  Rounding points are those of the separate modules: cos / sin, z and the sigmoid
// in the activation dtype.
struct DecodeAppendParams {
    const void *q_in, *k_in, *v_in;      // [B, Hq, D], [B, Hk, D]
    void* q_out;                         // [B, Hq, D] rotated (may be q_in); unused without inv_freq
    void *k_cache, *v_cache;             // [B * cap + 1, Hk, D]; the last row takes what does not fit
    void *k_tail, *v_tail;               // [B * ks + 1, Hk, D]
    const float* inv_freq;               // [D / 2] or null
    int* seq_len;
    const int* seq_row0;
    int64_t spare_row;                   // B * cap
    int cap, ks;
    const void* z;                       // [B, 3] gate logits or null
    const void *gx, *gw;                 // [B, glen], [3, glen]
    int glen;
    void* gate;                          // [B, 3]
    int Hq, Hk, D;
};

template <typename ET>
__device__ __forceinline__ float sigmoid_et(float z) { return round_et<ET>(1.f / (1.f + __expf(-z))); }

template <typename ET>
__global__ void __launch_bounds__(256) decode_append_kernel(const DecodeAppendParams p) {
    __shared__ float s_cos[128], s_sin[128];
    __shared__ float s_z[3][8];
    const int b = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    follow();
    const int t = p.seq_len[b];
    const int half = p.D / 2;
    const bool rot = p.inv_freq != nullptr;
    if (rot && tid < half) {
        const float a = (float)t * p.inv_freq[tid];
        s_cos[tid] = round_et<ET>(cosf(a));
        s_sin[tid] = round_et<ET>(sinf(a));
    }
    if (!p.z) {
        const uint4* x = reinterpret_cast<const uint4*>((const ET*)p.gx + (int64_t)b * p.glen);
        const uint4* w = reinterpret_cast<const uint4*>((const ET*)p.gw);
        const int nv = p.glen / 8;
        float acc[3] = {0.f, 0.f, 0.f};
        for (int i = tid; i < nv; i += 256) {
            const uint4 xv = __ldcg(x + i);
            const uint32_t* px = &xv.x;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const uint4 wv = __ldcg(w + (int64_t)j * nv + i);
                const uint32_t* pw = &wv.x;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = ElemTraits<ET>::unpack2(px[e]), g = ElemTraits<ET>::unpack2(pw[e]);
                    acc[j] = fmaf(f.x, g.x, fmaf(f.y, g.y, acc[j]));
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
#pragma unroll
            for (int o = 16; o; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
            if (lane == 0) s_z[j][warp] = acc[j];
        }
    }
    __syncthreads();
    if (tid < 3) {
        float z = 0.f;
        if (p.z) z = (float)((const ET*)p.z)[b * 3 + tid];
        else {
#pragma unroll
            for (int w = 0; w < 8; ++w) z += s_z[tid][w];
            z = round_et<ET>(z);
        }
        ((ET*)p.gate)[b * 3 + tid] = (ET)sigmoid_et<ET>(z);
    }
    const int64_t row = t < p.cap ? (int64_t)p.seq_row0[b] + t : p.spare_row, ring = (int64_t)b * p.ks + t % p.ks;
    const int hv = half / 8;                         // 16-byte vectors per half row
    const int nq = rot ? p.Hq * hv : 0, nk = p.Hk * hv;
    for (int i = tid; i < nq + 2 * nk; i += 256) {
        const bool is_q = i < nq, is_k = !is_q && i < nq + nk;
        const int j = is_q ? i : is_k ? i - nq : i - nq - nk;
        const int h = j / hv, v = j - h * hv, H = is_q ? p.Hq : p.Hk;
        const ET* src = (const ET*)(is_q ? p.q_in : is_k ? p.k_in : p.v_in) + ((int64_t)b * H + h) * p.D + v * 8;
        const uint4 a = *reinterpret_cast<const uint4*>(src), c = *reinterpret_cast<const uint4*>(src + half);
        uint4 o1 = a, o2 = c;
        if (rot && (is_q || is_k)) {
            const uint32_t *pa = &a.x, *pc = &c.x;
            uint32_t *q1 = &o1.x, *q2 = &o2.x;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 x1 = ElemTraits<ET>::unpack2(pa[e]), x2 = ElemTraits<ET>::unpack2(pc[e]);
                const float cx = s_cos[v * 8 + 2 * e], cy = s_cos[v * 8 + 2 * e + 1], sx = s_sin[v * 8 + 2 * e], sy = s_sin[v * 8 + 2 * e + 1];
                q1[e] = ElemTraits<ET>::pack2(x1.x * cx - x2.x * sx, x1.y * cy - x2.y * sy);
                q2[e] = ElemTraits<ET>::pack2(x1.x * sx + x2.x * cx, x1.y * sy + x2.y * cy);
            }
        }
        ET* dst = is_q ? (ET*)p.q_out + ((int64_t)b * p.Hq + h) * p.D + v * 8
                       : (ET*)(is_k ? p.k_cache : p.v_cache) + (row * p.Hk + h) * p.D + v * 8;
        *reinterpret_cast<uint4*>(dst) = o1;
        *reinterpret_cast<uint4*>(dst + half) = o2;
        if (!is_q) {
            ET* tail = (ET*)(is_k ? p.k_tail : p.v_tail) + (ring * p.Hk + h) * p.D + v * 8;
            *reinterpret_cast<uint4*>(tail) = a;
            *reinterpret_cast<uint4*>(tail + half) = c;
        }
    }
    if (tid == 0) p.seq_len[b] = t + 1;              // (everybody read it before the barrier above)
}

// ------------------------------------------------------------------------------------------------ incremental compressor
// For every sequence whose length seq_len[b] (after the append) completes a window: y = ring rows (oldest first) W[h], rounded,
// plus the position-embedding bias pe W (keys), rotated at m * stride (keys, with inv_freq), to row m of the compressed
// cache.  A cluster of 8 CTAs per (kv head, K or V) splits the ks * D reduction; their partial sums meet in distributed
// shared memory.  When no sequence completes a window, which is most steps of a small batch, no weight is read and the launch
// ends at once (a batched library GEMM over all sequences read 17 MB every step: 35 us).
// Bound by reading W once (17 MB for 8 heads of 128): a CTA takes its 512 rows of it to shared memory, the ring rows of up to
// 79 sequences and pe beside them, and the warp-level MMA (fp32 sums) goes over both; a warp has D / 8 columns.  (As multiply-adds
// of a thread, eight sequences at a time and W read again for each eight, the average step of 64 sequences of one length took 460 us
// instead of 438, that of eight sequences 71.0 instead of 66.7.)
struct DecodeCompressParams {
    const void *k_tail, *v_tail;         // [B * ks + 1, Hk, D] rings
    const void *wk, *wv;                 // [Hk, ks * D, D]
    const void* pe;                      // [Hk, ks, D] or null
    const float* inv_freq;               // [D / 2] or null
    const int* seq_len;
    const int* cmp_row0;
    void *cmp_k, *cmp_v;                 // [rows, Hk, D]
    int B, Hk, ks, stride, cmp_cap;
};

// CTAs of a cluster; rows of a turn (sequences, and pe behind them); rows of W that are staged at a time; padding of a staged row
constexpr int kDcSplit = 8, kDcRows = 80, kDcChunk = 512, kDcPad = 8;
template <int D> constexpr int dc_smem() { return (kDcChunk * (D + kDcPad) + kDcRows * (kDcChunk + kDcPad)) * 2; }

__device__ __forceinline__ void ldsm_x2_trans(uint32_t addr, uint32_t& r0, uint32_t& r1) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr));
}

template <int D, typename ET>
__global__ void __launch_bounds__(256, 1) decode_compress_kernel(const DecodeCompressParams p) {
    namespace cg = cooperative_groups;
    constexpr int WP = D + kDcPad, AP = kDcChunk + kDcPad;      // pitches: 8 rows of a fragment lie in 8 different groups of banks
    constexpr int MT = kDcRows / 16, NT = D / 64;               // 16-row tiles of a turn; 8-column tiles of a warp
    constexpr int PAR = 256 / D;                                // rows that are finished at a time
    extern __shared__ __align__(128) unsigned char dcs[];
    ET* sw = reinterpret_cast<ET*>(dcs);                        // [kDcChunk][WP]
    ET* sa = sw + kDcChunk * WP;                                // [kDcRows][AP], later [kDcRows][D] sums
    float* part = reinterpret_cast<float*>(sa);
    __shared__ float s_y[PAR][D];
    __shared__ int s_act[kDcRows], s_len[kDcRows], s_n, s_next;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
    const int rank = blockIdx.x, h = blockIdx.y;
    const bool is_k = blockIdx.z == 0;
    const int KS = p.ks * D / kDcSplit;                         // a multiple of 64
    const ET* tail = (const ET*)(is_k ? p.k_tail : p.v_tail);
    const ET* w = (const ET*)(is_k ? p.wk : p.wv) + ((int64_t)h * p.ks * D + (int64_t)rank * KS) * D;
    const ET* pe = is_k && p.pe ? (const ET*)p.pe + (int64_t)h * p.ks * D + (int64_t)rank * KS : nullptr;
    follow();
    for (int next = 0;;) {
        if (warp == 0) {
            int n = 0, b0 = next;
            for (; b0 < p.B && n < kDcRows - 1; b0 += 32) {
                const int b = b0 + lane;
                const int len = b < p.B ? p.seq_len[b] : 0;
                unsigned m = __ballot_sync(0xffffffffu, len >= p.ks && (len - p.ks) % p.stride == 0);
                int last = 31;
                while (m && n < kDcRows - 1) {
                    last = __ffs(m) - 1;
                    if (lane == last) { s_act[n] = b; s_len[n] = len; }
                    ++n;
                    m &= m - 1;
                }
                if (n == kDcRows - 1) { b0 += last + 1; break; }
            }
            if (lane == 0) { s_n = n; s_next = b0; }
        }
        __syncthreads();
        const int n = s_n;
        if (n == 0) break;                             // (the same for every CTA of the cluster)
        const int mt = (n + (pe ? 1 : 0) + 15) / 16;
        float acc[MT][NT][4];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
        for (int k0 = 0; k0 < KS; k0 += kDcChunk) {
            const int kc = min(kDcChunk, KS - k0);
            if (k0) __syncthreads();                   // the chunk before has been read
            for (int i = tid; i < kc * (D / 8); i += 256) {
                const int e = i / (D / 8), c = i % (D / 8) * 8;
                cp_async16(smem_u32(sw + e * WP + c), w + (int64_t)(k0 + e) * D + c, true);
            }
            for (int i = tid; i < mt * 16 * (kc / 8); i += 256) {
                const int a = i / (kc / 8), e = i % (kc / 8) * 8;
                const ET* src = tail;                  // (rows behind the last one: zeros)
                if (a < n) {
                    const int kk = rank * KS + k0 + e, o = kk / D;
                    src = tail + (((int64_t)s_act[a] * p.ks + (s_len[a] + o) % p.ks) * p.Hk + h) * D + (kk - o * D);
                } else if (a == n && pe) {
                    src = pe + k0 + e;
                }
                cp_async16(smem_u32(sa + a * AP + e), src, a < n || (a == n && pe));
            }
            cp_async_commit();
            cp_async_wait<0>();
            __syncthreads();
            const uint32_t wb = smem_u32(sw + (lane & 15) * WP + warp * (D / 8) + (lane >> 4) * 8);
            const uint32_t ab = smem_u32(sa + (lane & 15) * AP + (lane >> 4) * 8);
#pragma unroll 2
            for (int k = 0; k < kc; k += 16) {
                uint32_t b[2 * NT];
                if constexpr (NT == 2)
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(wb + k * WP * 2));
                else ldsm_x2_trans(wb + k * WP * 2, b[0], b[1]);
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    if (i >= mt) break;
                    uint32_t a0, a1, a2, a3;
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3) : "r"(ab + (i * 16 * AP + k) * 2));
#pragma unroll
                    for (int j = 0; j < NT; ++j) mma_16816<ET>(acc[i][j], a0, a1, a2, a3, b[2 * j], b[2 * j + 1]);
                }
            }
        }
        __syncthreads();                               // the inputs have been read: the sums take their place
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            if (i >= mt) break;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                float* at = part + (i * 16 + gid) * D + warp * (D / 8) + j * 8 + tig * 2;
                *reinterpret_cast<float2*>(at) = make_float2(acc[i][j][0], acc[i][j][1]);
                *reinterpret_cast<float2*>(at + 8 * D) = make_float2(acc[i][j][2], acc[i][j][3]);
            }
        }
        cluster.sync();
        // row a is finished by CTA a % 8
        const int sub = tid / D, col = tid % D;
        for (int a0 = rank; a0 < n; a0 += kDcSplit * PAR) {
            const int a = a0 + kDcSplit * sub;
            const int m = a < n ? (s_len[a] - p.ks) / p.stride : 0;
            if (a < n) {
                float y = 0.f, bias = 0.f;
#pragma unroll
                for (int r = 0; r < kDcSplit; ++r) {
                    const float* other = cluster.map_shared_rank(part, r);
                    y += other[a * D + col];
                    if (pe) bias += other[n * D + col];
                }
                y = round_et<ET>(y);
                if (pe) y = round_et<ET>(y + round_et<ET>(bias));
                s_y[sub][col] = y;
            }
            __syncthreads();
            if (a < n && m < p.cmp_cap) {
                float y = s_y[sub][col];
                if (is_k && p.inv_freq) {
                    const int i = col % (D / 2);
                    const float ang = (float)(m * p.stride) * p.inv_freq[i];
                    const float c = round_et<ET>(cosf(ang)), s = round_et<ET>(sinf(ang));
                    const float x1 = s_y[sub][i], x2 = s_y[sub][i + D / 2];
                    y = col < D / 2 ? x1 * c - x2 * s : x1 * s + x2 * c;
                }
                ((ET*)(is_k ? p.cmp_k : p.cmp_v))[((int64_t)(p.cmp_row0[s_act[a]] + m) * p.Hk + h) * D + col] = (ET)y;
            }
            __syncthreads();
        }
        next = s_next;
        cluster.sync();                                // the partial sums have been read
    }
}

// ------------------------------------------------------------------------------------------------ merge, top-k, row ranges
// Between the two attention passes of a step, one CTA per (sequence, kv head): LSE merge of the compressed branch's partials
// of the G heads, the top-k blocks from the scores of the group's first head (the rule of decode_topk_kernel), and the cache
// rows of the selected blocks and of the sliding window (the rule of decode_ranges_kernel).  The top-k works on keys (bf16
// score, then the complement of the id, so that equal scores go to the lower id): every warp takes the best of its share with
// warp-wide maxima, then one warp takes the best of those -- two barriers instead of two per selected block (64 sequences of
// 2048 blocks: 34 us in the kernel with a CTA-wide maximum per selected block).
struct DecodeSelectParams {
    const float* o_part;     // [B, Hq, P, D]
    const float2* ml;        // [B, Hq, P]
    const float* scores;     // [B, Hk, ld]
    int64_t ld;
    const int *seq_len, *seq_row0;
    int B, Hk, G, D, P;
    int ks, stride, BK, init_blocks, local_blocks, T, nw, max_blocks, window, npieces;
    float w[16];
    void* o_cmp;             // [B, Hq, D]
    int32_t* topk;           // [B, Hk, T]
    int *rng_lo, *rng_hi;    // [B, Hk, T + npieces]
};

// The `want` <= 64 largest of the keys in[0 .. n), all different, none 0: to out[0 .. 64) in descending order, 0 behind them.
// One warp, keys in registers: a round is one warp maximum and a handful of instructions.  More than 192 keys go in turns, the
// best so far among the next ones.
__device__ __forceinline__ void warp_largest(const uint32_t* in, int n, int want, uint32_t* out, int lane) {
    constexpr int NR = 6;
    out[lane] = 0; out[lane + 32] = 0;
    __syncwarp();
    int i0 = 0;
    do {
        uint32_t key[NR + 2];
        key[0] = out[lane]; key[1] = out[lane + 32];
#pragma unroll
        for (int j = 0; j < NR; ++j) key[j + 2] = i0 + j * 32 + lane < n ? in[i0 + j * 32 + lane] : 0u;
        __syncwarp();
        for (int r = 0; r < want; ++r) {
            uint32_t mine = key[0];
#pragma unroll
            for (int j = 1; j < NR + 2; ++j) mine = max(mine, key[j]);
            const uint32_t m = __reduce_max_sync(0xffffffffu, mine);
            if (lane == 0) out[r] = m;
#pragma unroll
            for (int j = 0; j < NR + 2; ++j) key[j] = key[j] == m ? 0u : key[j];
        }
        __syncwarp();
        i0 += NR * 32;
    } while (i0 < n);
}

template <typename ET>
__global__ void __launch_bounds__(256) decode_select_kernel(const DecodeSelectParams p) {
    extern __shared__ uint32_t dks[];                 // [max_blocks] keys, the probabilities, [G][P] merge weights
    __shared__ float s_lse, s_inv[16];
    __shared__ uint32_t cand[8 * 64], s_best[8 * 64], sel[64];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.x / p.Hk, h = blockIdx.x % p.Hk;
    follow();
    const int len = p.seq_len[b], t = len - 1;
    const int ncmp = len >= p.ks ? (len - p.ks) / p.stride + 1 : 0;
    const int bq = t / p.BK, nb = t >= 0 ? min(bq + 1, p.max_blocks) : 0;
    const int bstride = p.BK / p.stride, pad = p.ks / p.stride - 1;
    const int cmax = min(min(ncmp, nb * bstride + p.nw), (int)p.ld);
    const float* row = p.scores + ((int64_t)b * p.Hk + h) * p.ld;
    float* pv = reinterpret_cast<float*>(dks + p.max_blocks);
    float* s_w = pv + p.max_blocks * bstride + p.nw;
    // the first scores are on their way while the partials are merged
    float v0[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v0[j] = j * 256 + tid < cmax ? row[j * 256 + tid] : 0.f;
    // ---- merge: statistics and weights of a head by a warp, then the rows by all threads
    const int64_t row0 = (int64_t)b * p.Hk * p.G + h * p.G;
    for (int g = warp; g < p.G; g += 8) {
        const float2* mlr = p.ml + (row0 + g) * p.P;
        float M = -INFINITY;
        for (int i = lane; i < p.P; i += 32) {
            const float2 v = mlr[i];
            if (v.y > 0.f) M = fmaxf(M, v.x);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        float L = 0.f;
        for (int i = lane; i < p.P; i += 32) {
            const float2 v = mlr[i];
            const float wt = v.y > 0.f ? exp2f(v.x - M) : 0.f;
            L += wt * v.y;
            s_w[g * p.P + i] = wt;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
        if (lane == 0) {
            s_inv[g] = L > 0.f ? 1.f / L : 0.f;
            if (g == 0) s_lse = L > 0.f ? M + log2f(L) : -INFINITY;
        }
    }
    __syncthreads();
    const float lse = s_lse;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (j * 256 + tid < cmax) pv[j * 256 + tid] = exp2f(v0[j] - lse);
    for (int c = 2048 + tid; c < cmax; c += 256) pv[c] = exp2f(row[c] - lse);
    for (int i = tid; i < p.G * (p.D / 4); i += 256) {
        const int g = i / (p.D / 4), d = (i - g * (p.D / 4)) * 4;
        const float* src = p.o_part + (row0 + g) * p.P * p.D + d;
        const float* wg = s_w + g * p.P;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i0 = 0; i0 < p.P; i0 += 8) {
            float4 x[8];
            float wt[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                wt[j] = i0 + j < p.P ? wg[i0 + j] : 0.f;
                x[j] = wt[j] > 0.f ? *reinterpret_cast<const float4*>(src + (int64_t)(i0 + j) * p.D) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                acc.x = fmaf(wt[j], x[j].x, acc.x); acc.y = fmaf(wt[j], x[j].y, acc.y);
                acc.z = fmaf(wt[j], x[j].z, acc.z); acc.w = fmaf(wt[j], x[j].w, acc.w);
            }
        }
        const float inv = s_inv[g];
        *reinterpret_cast<uint2*>((ET*)p.o_cmp + (row0 + g) * p.D + d) =
            make_uint2(ElemTraits<ET>::pack2(acc.x * inv, acc.y * inv), ElemTraits<ET>::pack2(acc.z * inv, acc.w * inv));
    }
    __syncthreads();
    // ---- block scores
    for (int blk = tid; blk < nb; blk += 256) {
        float s = 0.f;
        for (int o = 0; o < p.nw; ++o) {
            const int c = blk * bstride - pad + o;
            const float v = (c >= 0 && c < cmax) ? pv[c] : 0.f;
            s += v * p.w[o];
        }
        if (blk < p.init_blocks || (bq >= blk && bq < blk + p.local_blocks)) s = INFINITY;
        // scores are >= 0: their bf16 words order like the scores
        dks[blk] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16(s)) << 16 | (uint32_t)(65535 - blk);
    }
    __syncthreads();
    // ---- top-k: the best T of every warp's share of the blocks, then the best T of those
    const int nsel = min(p.T, nb);
    const int share = (nb + 7) / 8, s0 = min(nb, warp * share), s1 = min(nb, s0 + share);
    warp_largest(dks + s0, s1 - s0, nsel, cand + warp * 64, lane);
    __syncthreads();
    // the eight lists without the zeros behind them
    if (tid < nsel)
        for (int w = 0; w < 8; ++w) s_best[w * nsel + tid] = cand[w * 64 + tid];
    __syncthreads();
    if (warp == 0) warp_largest(s_best, 8 * nsel, nsel, sel, lane);
    __syncthreads();
    int32_t* out = p.topk + ((int64_t)b * p.Hk + h) * p.T;
    int* s_id = reinterpret_cast<int*>(cand);          // ascending ids, -1 behind them
    if (tid < p.T) {
        int id = -1, at = tid;
        if (tid < nsel) {
            id = 65535 - (int)(sel[tid] & 0xffffu);
            at = 0;
            for (int j = 0; j < nsel; ++j) at += 65535 - (int)(sel[j] & 0xffffu) < id;
        }
        s_id[at] = id;
        out[at] = id;
    }
    __syncthreads();
    // ---- cache rows of the selected blocks and of the window [max(0, t - window), t] in pieces of BK rows
    const int R = p.T + p.npieces;
    const int64_t r0 = ((int64_t)b * p.Hk + h) * R;
    for (int r = tid; r < R; r += 256) {
        int a = 0, e = 0;
        if (len > 0) {
            if (r < p.T) {
                const int id = s_id[r];
                if (id >= 0 && id <= t / p.BK) { a = id * p.BK; e = min(a + p.BK, len); }
            } else {
                a = max(0, t - p.window) + (r - p.T) * p.BK;
                e = min(a + p.BK, len);
            }
        }
        p.rng_lo[r0 + r] = a < e ? p.seq_row0[b] + a : -1;
        p.rng_hi[r0 + r] = a < e ? p.seq_row0[b] + e : -1;
    }
}

}  // namespace fsa

using namespace fsa;

static bool misaligned(std::initializer_list<const void*> ps) {
    for (const void* p : ps)
        if ((uintptr_t)p & 15) return true;
    return false;
}

// Shared memory of decode_select_kernel: keys, probabilities that the blocks can touch, merge weights.
static int64_t select_smem(int max_blocks, int taps, int blocks_per, int group, int num_partials) {
    return 4 * ((int64_t)max_blocks + (int64_t)max_blocks * blocks_per + taps + (int64_t)group * num_partials);
}

static bool select_sizes(int num_q_heads, int num_kv_heads, int kernel_size, int kernel_stride, int block_size, int topk, int max_blocks, int num_partials) {
    if (kernel_size % kernel_stride || block_size % kernel_stride || topk > 64 || max_blocks > 65535 || num_q_heads / num_kv_heads > 16) return false;
    const int bb = block_size / kernel_stride, nw = kernel_size / kernel_stride + bb - 1;
    return nw <= 16 && select_smem(max_blocks, nw, bb, num_q_heads / num_kv_heads, num_partials) <= 200 * 1024;
}

static bool compress_sizes(int num_kv_heads, int head_dim, int kernel_size) {
    return (head_dim == 64 || head_dim == 128) && kernel_size % 8 == 0 && kernel_size <= 128 && num_kv_heads <= 65535;
}

extern "C" int fsa_decode_step_sizes(int num_q_heads, int num_kv_heads, int head_dim, int kernel_size, int kernel_stride, int block_size, int topk,
                                     int max_blocks, int num_partials, int gate_dim) {
    if (num_q_heads <= 0 || num_kv_heads <= 0 || num_q_heads % num_kv_heads || head_dim <= 0 || kernel_size <= 0 || kernel_stride <= 0 || block_size <= 0 ||
        topk <= 0 || max_blocks <= 0 || num_partials <= 0 || gate_dim < -1)
        return FSA_ERR_BAD_ARG;
    return (head_dim == 64 || head_dim == 128) && (gate_dim < 0 || (compress_sizes(num_kv_heads, head_dim, kernel_size) && gate_dim % 8 == 0)) &&
                   select_sizes(num_q_heads, num_kv_heads, kernel_size, kernel_stride, block_size, topk, max_blocks, num_partials)
               ? FSA_OK
               : FSA_ERR_UNSUPPORTED;
}

extern "C" int fsa_decode_proj(const void* x, int64_t x_stride, int batch, int k_dim, int num, const void* const* w, const int* rows,
                               void* const* y, const int64_t* y_stride, int dtype, void* stream) {
    if (!x || !w || !rows || !y || !y_stride || batch <= 0 || num <= 0 || k_dim <= 0) return FSA_ERR_BAD_ARG;
    if (dtype != FSA_DTYPE_BF16 && dtype != FSA_DTYPE_FP16) return FSA_ERR_BAD_ARG;
    if (num > 4 || batch > 16 || k_dim % 256) return FSA_ERR_UNSUPPORTED;
    if ((x_stride % 8) || misaligned({x})) return FSA_ERR_BAD_ARG;
    DecodeProjParams p;
    p.n = num; p.x = x; p.x_stride = x_stride; p.B = batch; p.K = k_dim;
    int tiles = 0;
    for (int i = 0; i < num; ++i) {
        if (!w[i] || !y[i] || rows[i] <= 0 || misaligned({w[i]})) return FSA_ERR_BAD_ARG;
        p.w[i] = w[i]; p.y[i] = y[i]; p.y_stride[i] = y_stride[i]; p.rows[i] = rows[i]; p.tile0[i] = tiles;
        tiles += (rows[i] + 15) / 16;
    }
    p.tile0[num] = tiles;
    (void)cudaGetLastError();
    cudaStream_t st = (cudaStream_t)stream;
    auto kern = dtype == FSA_DTYPE_BF16 ? (batch <= 8 ? decode_proj_kernel<1, __nv_bfloat16> : decode_proj_kernel<2, __nv_bfloat16>)
                                        : (batch <= 8 ? decode_proj_kernel<1, __half> : decode_proj_kernel<2, __half>);
    return launch_dependent(kern, dim3((unsigned)tiles), 256, 0, st, 1, p) == cudaSuccess ? FSA_OK : FSA_ERR_CUDA;
}

extern "C" int fsa_copy(int num, const void* const* src, void* const* dst, const int64_t* bytes, void* stream) {
    if (num < 0 || num > 8 || (num > 0 && (!src || !dst || !bytes))) return FSA_ERR_BAD_ARG;
    CopyParams p = {};
    p.n = num;
    for (int i = 0; i < num; ++i) {
        if (bytes[i] < 0 || (bytes[i] > 0 && (!src[i] || !dst[i]))) return FSA_ERR_BAD_ARG;
        p.src[i] = (const char*)src[i]; p.dst[i] = (char*)dst[i]; p.bytes[i] = bytes[i];
        p.first[i + 1] = p.first[i] + (bytes[i] + 15) / 16;
    }
    const int64_t units = p.first[num];
    if (units == 0) return FSA_OK;
    (void)cudaGetLastError();
    const int64_t ctas = (units + 255) / 256;
    copy_kernel<<<(unsigned)(ctas < 4096 ? ctas : 4096), 256, 0, (cudaStream_t)stream>>>(p);
    return cudaGetLastError() == cudaSuccess ? FSA_OK : FSA_ERR_CUDA;
}

extern "C" int fsa_decode_append(const void* q_in, const void* k_in, const void* v_in, void* q_out, void* k_cache, void* v_cache, void* k_tail,
                                 void* v_tail, const float* inv_freq, int32_t* seq_len, const int32_t* seq_row0, int batch, int cap,
                                 int num_q_heads, int num_kv_heads, int head_dim, int kernel_size, const void* gate_logits, const void* gate_x,
                                 const void* gate_w, int gate_dim, void* gate, int dtype, void* stream) {
    if (!k_in || !v_in || !k_cache || !v_cache || !k_tail || !v_tail || !seq_len || !seq_row0 || !gate || batch <= 0 || cap <= 0) return FSA_ERR_BAD_ARG;
    if (num_q_heads <= 0 || num_kv_heads <= 0 || kernel_size <= 0 || (inv_freq && (!q_in || !q_out))) return FSA_ERR_BAD_ARG;
    if (!gate_logits && (!gate_x || !gate_w || gate_dim <= 0 || gate_dim % 8 || misaligned({gate_x, gate_w}))) return FSA_ERR_BAD_ARG;
    if (misaligned({q_in, k_in, v_in, q_out, k_cache, v_cache, k_tail, v_tail})) return FSA_ERR_BAD_ARG;
    if (head_dim % 16 || head_dim > 256) return FSA_ERR_UNSUPPORTED;
    if (dtype != FSA_DTYPE_BF16 && dtype != FSA_DTYPE_FP16) return FSA_ERR_BAD_ARG;
    DecodeAppendParams p;
    p.q_in = q_in; p.k_in = k_in; p.v_in = v_in; p.q_out = q_out; p.k_cache = k_cache; p.v_cache = v_cache; p.k_tail = k_tail; p.v_tail = v_tail;
    p.inv_freq = inv_freq; p.seq_len = seq_len; p.seq_row0 = seq_row0; p.spare_row = (int64_t)batch * cap; p.cap = cap; p.ks = kernel_size;
    p.z = gate_logits; p.gx = gate_x; p.gw = gate_w; p.glen = gate_dim; p.gate = gate; p.Hq = num_q_heads; p.Hk = num_kv_heads; p.D = head_dim;
    (void)cudaGetLastError();
    auto kern = dtype == FSA_DTYPE_BF16 ? decode_append_kernel<__nv_bfloat16> : decode_append_kernel<__half>;
    return launch_dependent(kern, dim3((unsigned)batch), 256, 0, (cudaStream_t)stream, 1, p) == cudaSuccess ? FSA_OK : FSA_ERR_CUDA;
}

template <int D, typename ET>
static cudaError_t launch_compress(const DecodeCompressParams& p, cudaStream_t stream) {
    constexpr int smem = dc_smem<D>();
    static_assert(kDcRows * D * 4 <= kDcRows * (kDcChunk + kDcPad) * 2 && smem <= 225 * 1024, "shared memory");
    auto kern = decode_compress_kernel<D, ET>;
    cudaError_t e = allow_smem((const void*)kern, smem);
    if (e != cudaSuccess) return e;
    return launch_dependent(kern, dim3(kDcSplit, (unsigned)p.Hk, 2), 256, smem, stream, kDcSplit, p);
}

extern "C" int fsa_decode_compress(const void* k_tail, const void* v_tail, const void* w_key, const void* w_value, const void* pe,
                                   const float* inv_freq, const int32_t* seq_len, const int32_t* cmp_row0, void* cmp_k, void* cmp_v, int batch,
                                   int num_kv_heads, int head_dim, int kernel_size, int kernel_stride, int cmp_cap, int dtype, void* stream) {
    if (!k_tail || !v_tail || !w_key || !w_value || !seq_len || !cmp_row0 || !cmp_k || !cmp_v || batch <= 0 || num_kv_heads <= 0) return FSA_ERR_BAD_ARG;
    if (kernel_size <= 0 || kernel_stride <= 0 || misaligned({w_key, w_value})) return FSA_ERR_BAD_ARG;
    if (!compress_sizes(num_kv_heads, head_dim, kernel_size)) return FSA_ERR_UNSUPPORTED;
    if (dtype != FSA_DTYPE_BF16 && dtype != FSA_DTYPE_FP16) return FSA_ERR_BAD_ARG;
    DecodeCompressParams p;
    p.k_tail = k_tail; p.v_tail = v_tail; p.wk = w_key; p.wv = w_value; p.pe = pe; p.inv_freq = inv_freq; p.seq_len = seq_len; p.cmp_row0 = cmp_row0;
    p.cmp_k = cmp_k; p.cmp_v = cmp_v; p.B = batch; p.Hk = num_kv_heads; p.ks = kernel_size; p.stride = kernel_stride; p.cmp_cap = cmp_cap;
    (void)cudaGetLastError();
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e;
    if (dtype == FSA_DTYPE_BF16) e = head_dim == 128 ? launch_compress<128, __nv_bfloat16>(p, st) : launch_compress<64, __nv_bfloat16>(p, st);
    else e = head_dim == 128 ? launch_compress<128, __half>(p, st) : launch_compress<64, __half>(p, st);
    return e == cudaSuccess ? FSA_OK : FSA_ERR_CUDA;
}

extern "C" int fsa_decode_merge_select(const float* o_part, const float* ml, int num_partials, const float* scores, int64_t scores_ld,
                                       const int32_t* seq_len, const int32_t* seq_row0, int batch, int num_q_heads, int num_kv_heads, int head_dim,
                                       int kernel_size, int kernel_stride, int block_size, int init_blocks, int local_blocks, int topk,
                                       int max_blocks, int window, int num_window_pieces, int dtype, void* o_cmp, int32_t* topk_idx,
                                       int32_t* rng_lo, int32_t* rng_hi, void* stream) {
    if (!o_part || !ml || !scores || !seq_len || !seq_row0 || !o_cmp || !topk_idx || !rng_lo || !rng_hi || batch <= 0 || num_partials <= 0) return FSA_ERR_BAD_ARG;
    if (num_kv_heads <= 0 || num_q_heads % num_kv_heads || topk <= 0 || max_blocks <= 0 || num_window_pieces < 0 || kernel_stride <= 0 || block_size <= 0)
        return FSA_ERR_BAD_ARG;
    if (num_window_pieces > 0 && (int64_t)block_size * num_window_pieces < (int64_t)window + 1) return FSA_ERR_BAD_ARG;
    if (head_dim % 4 || misaligned({o_part}) || ((uintptr_t)o_cmp & 7)) return FSA_ERR_BAD_ARG;
    if (!select_sizes(num_q_heads, num_kv_heads, kernel_size, kernel_stride, block_size, topk, max_blocks, num_partials)) return FSA_ERR_UNSUPPORTED;
    if (dtype != FSA_DTYPE_BF16 && dtype != FSA_DTYPE_FP16) return FSA_ERR_BAD_ARG;
    DecodeSelectParams p;
    p.o_part = o_part; p.ml = (const float2*)ml; p.scores = scores; p.ld = scores_ld; p.seq_len = seq_len; p.seq_row0 = seq_row0;
    p.B = batch; p.Hk = num_kv_heads; p.G = num_q_heads / num_kv_heads; p.D = head_dim; p.P = num_partials;
    p.ks = kernel_size; p.stride = kernel_stride; p.BK = block_size; p.init_blocks = init_blocks; p.local_blocks = local_blocks; p.T = topk;
    p.max_blocks = max_blocks; p.window = window; p.npieces = num_window_pieces;
    const int a = kernel_size / kernel_stride, bb = block_size / kernel_stride;
    p.nw = a + bb - 1;
    for (int i = 0; i < 16; ++i) p.w[i] = 0.f;
    for (int i = 0; i < a; ++i)
        for (int j = 0; j < bb; ++j) p.w[i + j] += 1.f;
    p.o_cmp = o_cmp; p.topk = topk_idx; p.rng_lo = rng_lo; p.rng_hi = rng_hi;
    const int64_t smem = select_smem(max_blocks, p.nw, bb, p.G, num_partials);
    (void)cudaGetLastError();
    const void* kern = dtype == FSA_DTYPE_BF16 ? (const void*)decode_select_kernel<__nv_bfloat16> : (const void*)decode_select_kernel<__half>;
    if (smem > 48 * 1024 && allow_smem(kern, (int)smem) != cudaSuccess) return FSA_ERR_CUDA;
    const unsigned grid = (unsigned)(batch * num_kv_heads);
    auto run = dtype == FSA_DTYPE_BF16 ? decode_select_kernel<__nv_bfloat16> : decode_select_kernel<__half>;
    return launch_dependent(run, dim3(grid), 256, smem, (cudaStream_t)stream, 1, p) == cudaSuccess ? FSA_OK : FSA_ERR_CUDA;
}
