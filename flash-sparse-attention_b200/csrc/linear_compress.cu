// K/V compression by a strided linear projection (forward), as a tcgen05 GEMM that reads the overlapping token windows
// in place.
//
// Replaces linear_compress_fwd_kernel of the reference (nsa_ref/ops/linear_compress.py:28-131, launched at :334-398):
//     y[c, h, :] = sum_{k < ks} x[s_b + c * stride + k, h, :] @ W[h, k * d : (k + 1) * d, :]      c < n_b
//     n_b = floor((L_b - ks) / stride) + 1, or 0 when L_b < ks                                     (:334-337)
// and the bias of the intra-block position embedding, bias[h, :] = sum_{k, d'} pe[h, k, d'] W[h, k * d + d', :], which the
// reference adds to the rounded product in the activation dtype (:497-501).
//
// Per head this is the GEMM [n_b, ks * d] x [ks * d, d] whose left operand is never materialised: a 3-D tensor map over
// the sequence's rows of x -- dims (column, window c, offset k), strides (1, stride * row, row): overlapping -- lets TMA
// fetch the 64-column slab (k, half of d) of 128 consecutive windows straight into a swizzled K-major tile; windows
// past n_b are out of the map's bounds and read as zero.  One CTA = 128 windows of one sequence x one head of one tensor (K and
// V in the same launch) x a share of the reduction; a producer warp streams (A slab, W slab) stages through a six-stage
// mbarrier ring, one elected thread issues the MMAs (M = 128, N = d, fp32 in TMEM), four warps round the sum to the
// activation dtype, add the bias and store the rows.
//
// The reduction over ks * d is one serial chain of MMAs behind a ring of loads: 26 us at ks * d = 4096 however few windows
// there are.  When short sequences leave SMs idle the chain is cut in up to eight, one CTA of a cluster each, whose fp32 sums meet
// through distributed shared memory (517 tokens, 8 heads, K and V, inside a layer: 11 us for both; two launches of 26 us before; 19 us with
// six stages, an SM for every CTA, and the sums read one after the other).  One launch takes up to
// kLcSeqs sequences, whose tensor maps travel as kernel parameters.
#include "../../include/fsa_sm100.h"
#include <cooperative_groups.h>

#include "sm100_prims.cuh"

namespace fsa {

int make_tile_map(CUtensorMap* map, const void* base, int dtype, int64_t rows, int64_t cols, int64_t row_stride, int box_rows);
int make_tile_map_3d(CUtensorMap* map, const void* base, int dtype, int64_t d0, int64_t d1, int64_t d2, int64_t stride1,
                     int64_t stride2, int box1);

constexpr int kLcStages = 6, kLcStagesSplit = 3, kLcSeqs = 12, kLcTensors = 2, kLcSplits = 8, kLcShort = 64;

struct LcMaps {
    CUtensorMap a[kLcTensors][kLcSeqs];      // overlapping windows of every sequence
    CUtensorMap w[kLcTensors];
};
struct LcParams {
    int n_seq, H, ks;
    int tile0[kLcSeqs + 1];     // first 128-window tile of every sequence
    int n_cmp[kLcSeqs];         // windows of every sequence
    int y_row0[kLcSeqs];        // first output row
    const void* bias[kLcTensors];    // null, or [H, D] in the activation dtype, or with bias_parts > 0 fp32 [bias_parts, H, D] to be summed
    int bias_parts[kLcTensors];
    void* y[kLcTensors];        // [sum n_b, H, D]
    int* status;
};
static_assert(sizeof(LcMaps) + sizeof(LcParams) <= 4096, "kernel parameters");

template <int D, typename ET, int ST>
__global__ void __launch_bounds__(192) linear_compress_fwd_kernel(const __grid_constant__ LcMaps maps, const LcParams p) {
    namespace cg = cooperative_groups;
    constexpr int kA = 128 * 128, kB = 64 * D * 2;        // one stage: 128 windows x 64 columns, 64 weight rows x D columns
    constexpr int kSlabsPerK = D / 64;
    constexpr int kPitch = D + 4;                         // floats per row of a partial tile (16-byte aligned, fewer bank conflicts)
    static_assert(128 * kPitch * 4 <= ST * (kA + kB), "the partial tile reuses the ring");
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sA = smem;
    uint8_t* sB = sA + ST * kA;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sB + ST * kB);
    uint64_t* full = bars;                  // [stages]
    uint64_t* empty = bars + ST;     // [stages]
    uint64_t* acc_full = bars + 2 * ST;
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 2 * ST + 1);
    float* s_bias = reinterpret_cast<float*>(bars + 2 * ST + 2);      // [D] rounded to the activation dtype
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = (int)gridDim.x, rank = (int)blockIdx.x;            // CTAs that share the reduction (= cluster size), this one
    const int tn = (int)blockIdx.z / p.H, h = (int)blockIdx.z % p.H;
    int seq = 0;
    while (seq + 1 < p.n_seq && (int)blockIdx.y >= p.tile0[seq + 1]) ++seq;
    const int c0 = ((int)blockIdx.y - p.tile0[seq]) * 128;
    const int nvalid = min(128, p.n_cmp[seq] - c0);
    const int nslab = p.ks * kSlabsPerK / S, slab0 = rank * nslab;
    const CUtensorMap* amap = &maps.a[tn][seq];
    const CUtensorMap* wmap = &maps.w[tn];
    int* status = p.status;
    const uint32_t limit = wait_limit(status);
    if (tid == 0) {
        for (int i = 0; i < ST; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        mbar_init(acc_full, 1);
        mbar_init_fence();
        tma_prefetch_desc(amap);
        tma_prefetch_desc(wmap);
    }
    if (warp == 0) tmem_alloc(&tmem_slot, D);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tmem_slot;
    const int quarter = warp & 3, r = quarter * 32 + lane;           // (epilogue warps) this thread's window
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    bool ok = true;
    if (warp == 0) {
        // ---- producer
        for (int i = 0; i < nslab && ok; ++i) {
            const int st = i % ST;
            if (lane == 0) {
                ok = ok && mbar_wait(&empty[st], ((i / ST) & 1) ^ 1, status, limit);
                if (ok) {
                    mbar_expect_tx(&full[st], (uint32_t)(kA + kB));
                    const int k = (slab0 + i) / kSlabsPerK, dh = (slab0 + i) % kSlabsPerK;
                    tma_load_3d(smem_u32(sA + st * kA), amap, h * D + dh * 64, c0, k, &full[st]);
#pragma unroll
                    for (int nh = 0; nh < D / 64; ++nh)
                        tma_load_2d(smem_u32(sB + st * kB + nh * (64 * 128)), wmap, nh * 64, (h * p.ks * D) + (slab0 + i) * 64, &full[st]);
                }
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        }
    } else if (warp == 1) {
        // ---- MMA issuer
        const bool leader = elect_one();
        constexpr uint32_t idesc = umma_idesc(ElemTraits<ET>::kIsBF16, 128, D, false, true);
        for (int i = 0; i < nslab && ok; ++i) {
            const int st = i % ST;
            ok = ok && mbar_wait(&full[st], (i / ST) & 1, status, limit);
            ok = warp_ok(ok);
            if (!ok) break;
            tc_fence_after();
            if (leader) {
#pragma unroll
                for (int k16 = 0; k16 < 4; ++k16) {
                    const uint64_t ad = umma_desc_sw128(smem_u32(sA + st * kA) + k16 * 32, 16, 1024);
                    const uint64_t bd = umma_desc_sw128(smem_u32(sB + st * kB) + k16 * 2048, 64 * 128, 1024);
                    umma_ss(tbase, ad, bd, idesc, (i > 0 || k16 > 0) ? 1u : 0u);
                }
                umma_commit(&empty[st]);
                if (i == nslab - 1) umma_commit(acc_full);
            }
            __syncwarp();
        }
    } else {
        // ---- bias of this head (while the products run), then the accumulator
        const int t = tid - 64;
        if (t < D) {
            float v = 0.f;
            if (p.bias_parts[tn] > 0) {
                const float* bp = reinterpret_cast<const float*>(p.bias[tn]) + h * D + t;
                for (int i = 0; i < p.bias_parts[tn]; ++i) v += __ldg(bp + (int64_t)i * p.H * D);
                v = ElemTraits<ET>::unpack2(ElemTraits<ET>::pack2(v, 0.f)).x;
            } else if (p.bias[tn]) {
                v = (float)reinterpret_cast<const ET*>(p.bias[tn])[h * D + t];
            }
            s_bias[t] = v;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        ok = ok && mbar_wait(acc_full, 0, status, limit);
        tc_fence_after();
    }
    ET* y = reinterpret_cast<ET*>(p.y[tn]) + ((int64_t)(p.y_row0[seq] + c0) * p.H + h) * D;      // row r at r * H * D
    // the sum rounded to the activation dtype, then the bias added in that dtype
    auto finish = [&](const float* v, int col) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            w[j] = ElemTraits<ET>::pack2(v[2 * j], v[2 * j + 1]);
            if (p.bias[tn]) {
                const float2 f = ElemTraits<ET>::unpack2(w[j]);
                w[j] = ElemTraits<ET>::pack2(f.x + s_bias[col + 2 * j], f.y + s_bias[col + 2 * j + 1]);
            }
        }
        return make_uint4(w[0], w[1], w[2], w[3]);
    };
    if (S == 1) {
        if (warp >= 2) {
#pragma unroll
            for (int cc = 0; cc < D; cc += 32) {
                uint32_t v[32];
                tmem_ld32(tbase + lane_off + cc, v);
                tmem_ld_wait();
                if (ok && r < nvalid) {
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4)
                        *reinterpret_cast<uint4*>(y + (int64_t)r * p.H * D + cc + q4 * 8) =
                            finish(reinterpret_cast<const float*>(&v[q4 * 8]), cc + q4 * 8);
                }
            }
        }
    } else {
        float* part = reinterpret_cast<float*>(smem);      // [128][kPitch] (every product has read its operands: the ring is free)
        if (warp >= 2) {
#pragma unroll
            for (int cc = 0; cc < D; cc += 32) {
                uint32_t v[32];
                tmem_ld32(tbase + lane_off + cc, v);
                tmem_ld_wait();
                if (r < nvalid) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) *reinterpret_cast<uint4*>(part + r * kPitch + cc + q * 4) = *reinterpret_cast<uint4*>(&v[q * 4]);
                }
            }
        }
        ok = __syncthreads_and(ok);
        cluster.sync();
        // this CTA's rows of the tile: eight columns per thread, summed over the cluster in rank order
        const int per = (nvalid + S - 1) / S, r_lo = rank * per, r_hi = min(nvalid, r_lo + per);
        for (int i = tid; i < (r_hi - r_lo) * (D / 8) && ok; i += 192) {
            const int row = r_lo + i / (D / 8), col = (i % (D / 8)) * 8;
            float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            float4 a[kLcSplits], b[kLcSplits];                   // all reads in flight at once: one after the other they took 3 us
#pragma unroll
            for (int q = 0; q < kLcSplits; ++q)
                if (q < S) {
                    const float* src = cluster.map_shared_rank(part, q) + row * kPitch + col;
                    a[q] = *reinterpret_cast<const float4*>(src);
                    b[q] = *reinterpret_cast<const float4*>(src + 4);
                }
#pragma unroll
            for (int q = 0; q < kLcSplits; ++q)
                if (q < S) {
                    sum[0] += a[q].x; sum[1] += a[q].y; sum[2] += a[q].z; sum[3] += a[q].w;
                    sum[4] += b[q].x; sum[5] += b[q].y; sum[6] += b[q].z; sum[7] += b[q].w;
                }
            *reinterpret_cast<uint4*>(y + (int64_t)row * p.H * D + col) = finish(sum, col);
        }
        cluster.sync();                                    // nobody leaves while its partial tile is being read
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, D);
}

// Partial sums of the bias of the position embedding, part[i, h, :] = sum over the i-th share of the ks * D rows of
// pe[h, row] W[h, row, :] (fp32, added in a fixed order by the kernel above).  Bound by reading W (8 MB at 8 heads, 32-token
// windows); as a broadcast product and a column sum in torch it took five passes and 60 us.
constexpr int kPeParts = 16;

template <int D, typename ET>
__global__ void __launch_bounds__(256) compress_bias_kernel(const ET* __restrict__ pe, const ET* __restrict__ w, int rows, float* __restrict__ part,
                                                           int* __restrict__ status) {
    constexpr int CG = D / 8, KL = 256 / CG;
    __shared__ float red[8][D];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y, cgi = tid % CG, kl = tid / CG;
    if (tid == 0 && blockIdx.x == 0 && h == 0) *status = kStatusOk;
    const int share = rows / kPeParts, r0 = blockIdx.x * share;
    const ET* wr = w + ((int64_t)h * rows + r0) * D + cgi * 8;
    const ET* pr = pe + (int64_t)h * rows + r0;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int i = kl; i < share; i += KL) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(wr + (int64_t)i * D));
        const float x = (float)pr[i];
        const uint32_t* pv = &v.x;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = ElemTraits<ET>::unpack2(pv[j]);
            acc[2 * j] = fmaf(x, f.x, acc[2 * j]);
            acc[2 * j + 1] = fmaf(x, f.y, acc[2 * j + 1]);
        }
    }
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
        for (int v = 0; v < 8; ++v) s += red[v][tid];
        part[((int64_t)blockIdx.x * gridDim.y + h) * D + tid] = s;
    }
}

template <int D, typename ET>
static cudaError_t launch_lc(const LcMaps& maps, const LcParams& p, int tiles, int nt, cudaStream_t stream) {
    // CTAs per tile: as many as still find an SM of their own (the ring takes one SM's shared memory).  Short sequences only: another
    // order of the sum moves the last bit of a compressed row, and with it near ties of a block selection.  Up to kLcShort windows
    // (about 1000 tokens at stride 16, 16 blocks of 64) a selection of 16 blocks of 64 takes them all; a smaller one, or one of 32-key
    // blocks, does choose there.  The split goes by all sequences of the launch, so a sequence's last bits may depend on its batch.
    int S = 1, longest = 0;
    for (int b = 0; b < p.n_seq; ++b) longest = p.n_cmp[b] > longest ? p.n_cmp[b] : longest;
    while (longest <= kLcShort && S < kLcSplits && (p.ks * (D / 64)) % (2 * S) == 0 && 2 * S * tiles * p.H * nt <= sm_count()) S *= 2;
    // Three stages where the reduction is split, so that two CTAs share an SM: clusters of eight that need an SM for each CTA do not all
    // find one at once (a GPU processing cluster has 16 to 20 SMs), and sixteen of them took two rounds.
    const int stages = S > 1 ? kLcStagesSplit : kLcStages;
    const int smem = stages * (128 * 128 + 64 * D * 2) + 128 + D * 4;
    auto kern = S > 1 ? linear_compress_fwd_kernel<D, ET, kLcStagesSplit> : linear_compress_fwd_kernel<D, ET, kLcStages>;
    cudaError_t e = allow_smem((const void*)kern, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)S, (unsigned)tiles, (unsigned)(p.H * nt));
    cfg.blockDim = dim3(192);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)S; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, maps, p);
}

// One tensor of the launch (K or V).
struct LcTensor {
    const void* x;
    int64_t x_sn;
    const void* w;
    const void* bias;
    int bias_parts;
    void* y;
};

static int run_compress(const LcTensor* t, int nt, const int32_t* seqlens, int batch, int H, int D, int ks, int stride, int dtype, int32_t* status,
                        cudaStream_t stream) {
    int rc = ensure_context();
    if (rc) return rc;
    LcMaps maps;
    LcParams p;
    p.H = H; p.ks = ks; p.status = status;
    for (int i = 0; i < nt; ++i) {
        rc = make_tile_map(&maps.w[i], t[i].w, dtype, (int64_t)H * ks * D, D, D, 64);
        if (rc) return rc;
        p.bias[i] = t[i].bias; p.bias_parts[i] = t[i].bias_parts; p.y[i] = t[i].y;
    }
    int64_t tok0 = 0;
    int y_row0 = 0;
    p.n_seq = 0; p.tile0[0] = 0;
    for (int b = 0; b < batch; ++b) {
        const int L = seqlens[b];
        if (L < 0) return FSA_ERR_BAD_ARG;
        const int n = L >= ks ? (L - ks) / stride + 1 : 0;
        if (n > 0) {
            const int q = p.n_seq;
            for (int i = 0; i < nt; ++i) {
                if (!t[i].y || ((uintptr_t)t[i].y & 15)) return FSA_ERR_BAD_ARG;
                rc = make_tile_map_3d(&maps.a[i][q], (const char*)t[i].x + tok0 * t[i].x_sn * 2, dtype, (int64_t)H * D, n, ks,
                                      (int64_t)stride * t[i].x_sn, t[i].x_sn, 128);
                if (rc) return rc;
            }
            p.n_cmp[q] = n; p.y_row0[q] = y_row0;
            p.tile0[q + 1] = p.tile0[q] + (n + 127) / 128;
            ++p.n_seq;
        }
        tok0 += L;
        y_row0 += n;
        if (p.n_seq == kLcSeqs || (b == batch - 1 && p.n_seq > 0)) {
            const int tiles = p.tile0[p.n_seq];
            if (tiles > 65535 || H * nt > 65535) return FSA_ERR_UNSUPPORTED;
            cudaError_t e;
            if (dtype == FSA_DTYPE_BF16)
                e = D == 128 ? launch_lc<128, __nv_bfloat16>(maps, p, tiles, nt, stream) : launch_lc<64, __nv_bfloat16>(maps, p, tiles, nt, stream);
            else
                e = D == 128 ? launch_lc<128, __half>(maps, p, tiles, nt, stream) : launch_lc<64, __half>(maps, p, tiles, nt, stream);
            if (e != cudaSuccess) return FSA_ERR_CUDA;
            p.n_seq = 0;
        }
    }
    return FSA_OK;
}

static int check_compress(const void* x, int64_t x_sn, const void* w, const int32_t* seqlens, int batch, int H, int D, int ks, int stride, int dtype) {
    if (!x || !w || !seqlens || batch < 0 || H <= 0 || ks <= 0 || stride <= 0) return FSA_ERR_BAD_ARG;
    if (dtype != FSA_DTYPE_BF16 && dtype != FSA_DTYPE_FP16) return FSA_ERR_BAD_ARG;
    if (D != 64 && D != 128) return FSA_ERR_UNSUPPORTED;
    if (((uintptr_t)x & 15) || ((uintptr_t)w & 15) || (x_sn % 8)) return FSA_ERR_BAD_ARG;
    if (x_sn < (int64_t)H * D) return FSA_ERR_BAD_ARG;
    return FSA_OK;
}

}  // namespace fsa

using namespace fsa;

extern "C" int fsa_linear_compress_fwd(const void* x, int64_t x_stride_n, const void* w, const void* bias, const int32_t* seqlens_host,
                                       int batch, int num_heads, int head_dim, int kernel_size, int kernel_stride, int dtype, void* y,
                                       int32_t* status, void* stream) {
    int rc = check_compress(x, x_stride_n, w, seqlens_host, batch, num_heads, head_dim, kernel_size, kernel_stride, dtype);
    if (rc) return rc;
    if (bias && ((uintptr_t)bias & 15)) return FSA_ERR_BAD_ARG;
    (void)cudaGetLastError();
    const LcTensor t{x, x_stride_n, w, bias, 0, y};
    return run_compress(&t, 1, seqlens_host, batch, num_heads, head_dim, kernel_size, kernel_stride, dtype, status, (cudaStream_t)stream);
}

extern "C" int64_t fsa_compress_bias_scratch_bytes(int num_heads, int head_dim) { return (int64_t)kPeParts * num_heads * head_dim * 4 + 16; }

extern "C" int fsa_compress_kv_fwd(const void* k, int64_t k_stride_n, const void* v, int64_t v_stride_n, const void* w_key, const void* w_value,
                                   const void* pe, const int32_t* seqlens_host, int batch, int num_heads, int head_dim, int kernel_size,
                                   int kernel_stride, int dtype, void* yk, void* yv, float* scratch, void* stream_) {
    int rc = check_compress(k, k_stride_n, w_key, seqlens_host, batch, num_heads, head_dim, kernel_size, kernel_stride, dtype);
    if (rc) return rc;
    if (v && (rc = check_compress(v, v_stride_n, w_value, seqlens_host, batch, num_heads, head_dim, kernel_size, kernel_stride, dtype))) return rc;
    if (pe && (!scratch || (kernel_size * head_dim) % kPeParts)) return FSA_ERR_BAD_ARG;
    (void)cudaGetLastError();
    cudaStream_t stream = (cudaStream_t)stream_;
    int* status = pe ? (int*)(scratch + (int64_t)kPeParts * num_heads * head_dim) : nullptr;
    if (pe) {
        const dim3 grid(kPeParts, (unsigned)num_heads);
        const int rows = kernel_size * head_dim;
        if (dtype == FSA_DTYPE_BF16) {
            if (head_dim == 128) compress_bias_kernel<128, __nv_bfloat16><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)pe, (const __nv_bfloat16*)w_key, rows, scratch, status);
            else compress_bias_kernel<64, __nv_bfloat16><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)pe, (const __nv_bfloat16*)w_key, rows, scratch, status);
        } else {
            if (head_dim == 128) compress_bias_kernel<128, __half><<<grid, 256, 0, stream>>>((const __half*)pe, (const __half*)w_key, rows, scratch, status);
            else compress_bias_kernel<64, __half><<<grid, 256, 0, stream>>>((const __half*)pe, (const __half*)w_key, rows, scratch, status);
        }
        if (cudaGetLastError() != cudaSuccess) return FSA_ERR_CUDA;
    }
    const LcTensor t[2] = {{k, k_stride_n, w_key, pe ? scratch : nullptr, pe ? kPeParts : 0, yk}, {v, v_stride_n, w_value, nullptr, 0, yv}};
    return run_compress(t, v ? 2 : 1, seqlens_host, batch, num_heads, head_dim, kernel_size, kernel_stride, dtype, status, stream);
}
