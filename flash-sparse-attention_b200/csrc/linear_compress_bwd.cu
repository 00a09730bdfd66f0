// K/V compression by a strided linear projection (backward), two tcgen05 GEMM kernels without atomics.
//
// Replaces linear_compress_bwd_kernel of the reference (nsa_ref/ops/linear_compress.py:135-292, launched at :401-470),
// which scatters both gradients with fp32 tl.atomic_add (:275, :292).  With
//     y[c, h, :] = sum_{k < ks} x[s_b + c * stride + k, h, :] @ W[h, k * d : (k + 1) * d, :]
// the gradients are
//     dx[s_b + t, h, :]          = sum_{j < ks / stride} dy[m - j, h, :] @ W[h, (p + j * stride) * d : ..., :]^T      t = m * stride + p
//     dW[h, k * d + a, :]        = sum_b sum_c x[s_b + c * stride + k, h, a] * dy[y_b + c, h, :]
//
// dx: a token belongs to ks / stride windows, and tokens with the same phase p = t mod stride meet the same slices of W.
// One CTA = 128 consecutive m of one sequence x one head x a group of phases; per phase it runs the GEMM
// [128, (ks / stride) * d] x [(ks / stride) * d, d] whose left operand is dy shifted by j rows (TMA; rows outside the
// sequence's windows are out of the map's bounds and read as zero) and writes the rows m * stride + p once, in the
// activation dtype, from an fp32 accumulator in TMEM (two accumulators: the stores of a phase overlap the next phase).
//
// dW: one CTA = one head x one window offset k (two offsets when d = 64): M = input feature, N = output feature, the
// reduction runs over every window of every sequence in 128-window tiles.  Both operands are "MN-major" (the window index
// is the row of both tiles), gathered with 16-byte async copies (rows of x are stride tokens apart; windows past the end
// of a sequence are zero-filled), so no tensor map per sequence is needed and the whole gradient is one launch.
#include "../../include/fsa_sm100.h"
#include "sm100_prims.cuh"

namespace fsa {

int make_tile_map(CUtensorMap* map, const void* base, int dtype, int64_t rows, int64_t cols, int64_t row_stride, int box_rows);

// ------------------------------------------------------------------------------------------------ dx
// One launch takes up to kLbSeqs sequences (their tensor maps travel as kernel parameters) of up to two tensors (K and V).
constexpr int kLbSeqs = 12, kLbTensors = 2;
struct LcDxMaps {
    CUtensorMap y[kLbTensors][kLbSeqs];     // dy of every sequence
    CUtensorMap w[kLbTensors];
};
struct LcDxParams {
    int n_seq, H, ks, stride;
    int phases;                 // phases per CTA
    int tile0[kLbSeqs + 1];     // first tile (128 m) of every sequence
    int n_cmp[kLbSeqs];         // windows of every sequence (0: no product, the gradient is zero)
    int L[kLbSeqs];             // tokens
    int64_t tok0[kLbSeqs];      // first token
    void* dx[kLbTensors];       // [N, H, D] contiguous
    int* status;
};
static_assert(sizeof(LcDxMaps) + sizeof(LcDxParams) <= 4096, "kernel parameters");

constexpr int kLcDxStages = 4;

template <int D, typename ET>
__global__ void __launch_bounds__(192) linear_compress_dx_kernel(const __grid_constant__ LcDxMaps maps, const LcDxParams p) {
    constexpr int kA = 128 * 128, kB = D * 128;           // one stage: 128 rows of dy x 64 columns, D rows of W x 64 columns
    constexpr int KH = D / 64;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sA = smem;
    uint8_t* sB = sA + kLcDxStages * kA;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sB + kLcDxStages * kB);
    uint64_t* full = bars;                      // [stages]
    uint64_t* empty = bars + kLcDxStages;       // [stages]
    uint64_t* acc_full = bars + 2 * kLcDxStages;        // [2]
    uint64_t* acc_empty = bars + 2 * kLcDxStages + 2;   // [2]
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 2 * kLcDxStages + 4);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int seq = 0;
    while (seq + 1 < p.n_seq && (int)blockIdx.x >= p.tile0[seq + 1]) ++seq;
    const int tn = (int)blockIdx.y / p.H, h = (int)blockIdx.y % p.H;
    const int m0 = ((int)blockIdx.x - p.tile0[seq]) * 128, p0 = blockIdx.z * p.phases;
    const bool product = p.n_cmp[seq] > 0;
    const CUtensorMap* ymap = &maps.y[tn][seq];
    const CUtensorMap* wmap = &maps.w[tn];
    const int J = p.ks / p.stride;
    const int per_phase = J * KH;
    int* status = p.status;
    const uint32_t limit = wait_limit(status);
    if (tid == 0) {
        for (int i = 0; i < kLcDxStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 128); }
        mbar_init_fence();
        tma_prefetch_desc(ymap);
        tma_prefetch_desc(wmap);
    }
    if (warp == 0) tmem_alloc(&tmem_slot, 2 * D);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tmem_slot;
    if (warp == 0) {
        // ---- producer: (dy shifted by j, W slice of offset p + j * stride), 64 reduction columns per stage
        bool ok = true;
        int i = 0;
        for (int pi = 0; pi < p.phases && ok && product; ++pi) {
            for (int q = 0; q < per_phase && ok; ++q, ++i) {
                const int st = i % kLcDxStages;
                if (lane == 0) {
                    ok = ok && mbar_wait(&empty[st], ((i / kLcDxStages) & 1) ^ 1, status, limit);
                    if (ok) {
                        mbar_expect_tx(&full[st], (uint32_t)(kA + kB));
                        const int j = q / KH, kh = q % KH;
                        const int k = p0 + pi + j * p.stride;
                        tma_load_2d(smem_u32(sA + st * kA), ymap, h * D + kh * 64, m0 - j, &full[st]);
#pragma unroll
                        for (int nh = 0; nh < KH; ++nh)
                            tma_load_2d(smem_u32(sB + st * kB + nh * (64 * 128)), wmap, kh * 64, (h * p.ks + k) * D + nh * 64, &full[st]);
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer
        const bool leader = elect_one();
        constexpr uint32_t idesc = umma_idesc(ElemTraits<ET>::kIsBF16, 128, D, false, false);
        bool ok = true;
        int i = 0;
        for (int pi = 0; pi < p.phases && ok && product; ++pi) {
            const int buf = pi & 1;
            ok = ok && mbar_wait(&acc_empty[buf], ((pi >> 1) & 1) ^ 1, status, limit);
            tc_fence_after();
            for (int q = 0; q < per_phase; ++q, ++i) {       // (left by all lanes at the vote below)
                const int st = i % kLcDxStages;
                ok = ok && mbar_wait(&full[st], (i / kLcDxStages) & 1, status, limit);
                ok = warp_ok(ok);
                if (!ok) break;
                tc_fence_after();
                if (leader) {
#pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16) {
                        const uint64_t ad = umma_desc_sw128(smem_u32(sA + st * kA) + k16 * 32, 16, 1024);
                        const uint64_t bd = umma_desc_sw128(smem_u32(sB + st * kB) + k16 * 32, 16, 1024);
                        umma_ss(tbase + buf * D, ad, bd, idesc, (q > 0 || k16 > 0) ? 1u : 0u);
                    }
                    umma_commit(&empty[st]);
                    if (q == per_phase - 1) umma_commit(&acc_full[buf]);
                }
                __syncwarp();
            }
        }
    } else {
        // ---- epilogue: thread = one m (TMEM lane quarter = warp % 4), one row of dx per phase
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        bool ok = true;
        for (int pi = 0; pi < p.phases && warp_stays(ok); ++pi) {
            const int buf = pi & 1;
            if (product) ok = ok && mbar_wait(&acc_full[buf], (pi >> 1) & 1, status, limit);
            tc_fence_after();
            const int64_t t = (int64_t)(m0 + r) * p.stride + p0 + pi;
            const bool valid = ok && t < p.L[seq];
            ET* dst = reinterpret_cast<ET*>(p.dx[tn]) + ((p.tok0[seq] + t) * p.H + h) * D;
#pragma unroll
            for (int cc = 0; cc < D; cc += 32) {
                uint32_t v[32];
                if (product) {
                    tmem_ld32(tbase + lane_off + buf * D + cc, v);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = 0u;
                }
                if (valid) {
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) {
                        uint4 u;
                        u.x = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 0]), __uint_as_float(v[q4 * 8 + 1]));
                        u.y = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 2]), __uint_as_float(v[q4 * 8 + 3]));
                        u.z = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 4]), __uint_as_float(v[q4 * 8 + 5]));
                        u.w = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 6]), __uint_as_float(v[q4 * 8 + 7]));
                        *reinterpret_cast<uint4*>(dst + cc + q4 * 8) = u;
                    }
                }
            }
            tc_fence_before();
            mbar_arrive(&acc_empty[buf]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, 2 * D);
}

template <int D, typename ET>
static cudaError_t launch_dx(const LcDxMaps& maps, const LcDxParams& p, int nt, cudaStream_t stream) {
    constexpr int smem = kLcDxStages * (128 * 128 + D * 128) + 256;
    auto kern = linear_compress_dx_kernel<D, ET>;
    cudaError_t e = allow_smem((const void*)kern, smem);
    if (e != cudaSuccess) return e;
    kern<<<dim3((unsigned)p.tile0[p.n_seq], (unsigned)(p.H * nt), (unsigned)(p.stride / p.phases)), 192, smem, stream>>>(maps, p);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------ dW
template <typename ET>
struct LcDwParams {
    const ET* x[kLbTensors];  int64_t x_sn[kLbTensors];     // [N, H, D], token stride in elements
    const ET* dy[kLbTensors];       // [sum n_b, H, D] contiguous
    const int32_t* cu;              // [batch + 1] token offsets
    int batch, H, ks, stride;
    ET* dw[kLbTensors];             // [H, ks * D, D]
    // bias of the position embedding (tensor 0 only; pe null: none): dW[h, r, :] += pe[h, r] dbias[h, :], dpe[h, r] = W[h, r, :] dbias[h, :],
    // with dbias[h, :] the sum of its parts, rounded to the activation dtype
    const ET *pe, *w;
    ET* dpe;
    const float* dbias;             // [parts][H][D]
    int parts;
    int* status;
};

constexpr int kLcDwStages = 3;

template <int D, typename ET>
__global__ void __launch_bounds__(256) linear_compress_dw_kernel(const LcDwParams<ET> p) {
    constexpr int KPC = 128 / D;                  // window offsets per CTA (M = 128 input features in all)
    constexpr int KH = D / 64;                    // 64-column slabs of a dy row
    constexpr int kSlab = 128 * 128;              // 128 windows x 64 elements
    constexpr int kX = 2 * kSlab, kY = KH * kSlab, kStage = kX + kY;
    constexpr int CY = D / 8;                     // 16-byte chunks of a dy row
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kLcDwStages * kStage);
    uint64_t* full = bars;                        // [stages] 128 arrivals (one per producer thread, when its copies landed)
    uint64_t* empty = bars + kLcDwStages;         // [stages]
    uint64_t* acc_full = bars + 2 * kLcDwStages;
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 2 * kLcDwStages + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int k0 = blockIdx.x * KPC, h = blockIdx.y, tn = blockIdx.z;
    const ET* x = p.x[tn];
    const ET* dy = p.dy[tn];
    const int64_t x_sn = p.x_sn[tn];
    const bool with_pe = tn == 0 && p.pe != nullptr;
    float* s_db = reinterpret_cast<float*>(bars + 2 * kLcDwStages + 2);      // [D] gradient of the bias
    int* status = p.status;
    const uint32_t limit = wait_limit(status);
    if (tid == 0) {
        for (int i = 0; i < kLcDwStages; ++i) { mbar_init(&full[i], 128); mbar_init(&empty[i], 1); }
        mbar_init(acc_full, 1);
        mbar_init_fence();
    }
    if (warp == 4) tmem_alloc(&tmem_slot, D < 32 ? 32 : D);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tmem_slot;
    // tiles of 128 windows over all sequences
    int nitems = 0;
    for (int b = 0; b < p.batch; ++b) {
        const int L = __ldg(p.cu + b + 1) - __ldg(p.cu + b);
        const int n = L >= p.ks ? (L - p.ks) / p.stride + 1 : 0;
        nitems += (n + 127) / 128;
    }
    if (warp < 4) {
        // ---- producers: thread t copies 16-byte chunk t % 16 of the rows t / 16 + 8 i of the x tile (a half-warp covers the
        // 256 bytes of one window: both 64-feature halves of offset k0 when d = 128, offsets k0 and k0 + 1 when d = 64),
        // and chunk t % CY of the rows t / CY + (128 / CY) i of the dy tile
        const int xc = tid & 15, xr0 = tid >> 4;
        const int yc = tid % CY, yr0 = tid / CY;
        constexpr int YSTEP = 128 / CY, YIT = 128 / YSTEP;
        // column of x this thread reads, and the window offset it belongs to
        const int x_k = KPC == 1 ? k0 : k0 + (xc >> 3);
        const int x_col = h * D + (KPC == 1 ? xc * 8 : (xc & 7) * 8);
        const uint32_t x_slab = (uint32_t)(xc >> 3) * kSlab;
        const uint32_t y_slab = (uint32_t)(yc >> 3) * kSlab;
        bool ok = true;
        int i = 0;
        int64_t y0 = 0;
        for (int b = 0; b < p.batch && ok; ++b) {
            const int s_b = __ldg(p.cu + b);
            const int L = __ldg(p.cu + b + 1) - s_b;
            const int n = L >= p.ks ? (L - p.ks) / p.stride + 1 : 0;
            for (int c0 = 0; c0 < n && ok; c0 += 128, ++i) {
                const int st = i % kLcDwStages;
                ok = ok && mbar_wait(&empty[st], ((i / kLcDwStages) & 1) ^ 1, status, limit);
                const uint32_t sx = smem_u32(smem + st * kStage) + x_slab;
                const uint32_t sy = smem_u32(smem + st * kStage + kX) + y_slab;
#pragma unroll
                for (int it = 0; it < 16; ++it) {
                    const int r = xr0 + it * 8;
                    const bool valid = c0 + r < n;
                    const int64_t row = valid ? (int64_t)s_b + (int64_t)(c0 + r) * p.stride + x_k : 0;
                    cp_async16(sx + sw128_chunk_off(r, xc & 7), x + row * x_sn + x_col, valid);
                }
#pragma unroll
                for (int it = 0; it < YIT; ++it) {
                    const int r = yr0 + it * YSTEP;
                    const bool valid = c0 + r < n;
                    const int64_t row = valid ? y0 + c0 + r : 0;
                    cp_async16(sy + sw128_chunk_off(r, yc & 7), dy + (row * p.H + h) * D + yc * 8, valid);
                }
                cp_async_mbar_arrive_noinc(&full[st]);
            }
            y0 += n;
        }
    } else {
        if (warp == 4) {
            // ---- MMA issuer: dW^T tile (+)= x_tile^T dy_tile, 16 windows per instruction
            const bool leader = elect_one();
            constexpr uint32_t idesc = umma_idesc(ElemTraits<ET>::kIsBF16, 128, D, true, true);
            constexpr uint32_t hi_1024 = umma_desc_hi(1024);
            bool ok = true;
            for (int i = 0; i < nitems && ok; ++i) {
                const int st = i % kLcDwStages;
                ok = ok && mbar_wait(&full[st], (i / kLcDwStages) & 1, status, limit);
                fence_async_smem();
                ok = warp_ok(ok);
                if (!ok) break;
                tc_fence_after();
                if (leader) {
                    const uint32_t a_lo = umma_desc_lo(smem_u32(smem + st * kStage), kSlab);
                    const uint32_t b_lo = umma_desc_lo(smem_u32(smem + st * kStage + kX), kSlab);
#pragma unroll
                    for (int ks16 = 0; ks16 < 8; ++ks16)
                        umma_ss(tbase, umma_desc_pack(a_lo + ks16 * (2048 >> 4), hi_1024), umma_desc_pack(b_lo + ks16 * (2048 >> 4), hi_1024),
                                idesc, (i > 0 || ks16 > 0) ? 1u : 0u);
                    umma_commit(&empty[st]);
                    if (i == nitems - 1) umma_commit(acc_full);
                }
                __syncwarp();
            }
        }
        // ---- epilogue (warps 4..7): thread = one row of dW (TMEM lane = input feature, or offset and feature when d = 64)
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        bool ok = true;
        const int64_t wrow = (int64_t)(h * p.ks + k0) * D + r;
        float pe_r = 0.f, dpe = 0.f;
        if (with_pe) {
            if (r < D) {
                float v = 0.f;
                for (int i = 0; i < p.parts; ++i) v += __ldg(p.dbias + ((int64_t)i * p.H + h) * D + r);
                s_db[r] = ElemTraits<ET>::unpack2(ElemTraits<ET>::pack2(v, 0.f)).x;
            }
            pe_r = (float)p.pe[wrow];
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        if (nitems > 0) {
            ok = ok && mbar_wait(acc_full, 0, status, limit);
            tc_fence_after();
        }
        ET* dst = p.dw[tn] ? p.dw[tn] + wrow * D : nullptr;
#pragma unroll
        for (int cc = 0; cc < D; cc += 32) {
            uint32_t v[32];
            if (nitems > 0) {
                tmem_ld32(tbase + lane_off + cc, v);
                tmem_ld_wait();
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = 0u;
            }
            if (with_pe) {
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4) {
                    const uint4 wv = __ldg(reinterpret_cast<const uint4*>(p.w + wrow * D + cc + q4 * 8));
                    const uint32_t* pw = &wv.x;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 f = ElemTraits<ET>::unpack2(pw[j]);
                        const float d0 = s_db[cc + q4 * 8 + 2 * j], d1 = s_db[cc + q4 * 8 + 2 * j + 1];
                        dpe = fmaf(f.x, d0, fmaf(f.y, d1, dpe));
                        v[q4 * 8 + 2 * j] = __float_as_uint(fmaf(pe_r, d0, __uint_as_float(v[q4 * 8 + 2 * j])));
                        v[q4 * 8 + 2 * j + 1] = __float_as_uint(fmaf(pe_r, d1, __uint_as_float(v[q4 * 8 + 2 * j + 1])));
                    }
                }
            }
            if (ok && dst) {
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4) {
                    uint4 u;
                    u.x = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 0]), __uint_as_float(v[q4 * 8 + 1]));
                    u.y = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 2]), __uint_as_float(v[q4 * 8 + 3]));
                    u.z = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 4]), __uint_as_float(v[q4 * 8 + 5]));
                    u.w = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 6]), __uint_as_float(v[q4 * 8 + 7]));
                    *reinterpret_cast<uint4*>(dst + cc + q4 * 8) = u;
                }
            }
        }
        if (with_pe && p.dpe) p.dpe[wrow] = (ET)dpe;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 4) tmem_dealloc(tbase, D < 32 ? 32 : D);
}

template <int D, typename ET>
static cudaError_t launch_dw(const LcDwParams<ET>& p, int nt, cudaStream_t stream) {
    constexpr int smem = kLcDwStages * (2 + D / 64) * 128 * 128 + 128 + D * 4;
    auto kern = linear_compress_dw_kernel<D, ET>;
    cudaError_t e = allow_smem((const void*)kern, smem);
    if (e != cudaSuccess) return e;
    kern<<<dim3((unsigned)(p.ks / (128 / D)), (unsigned)p.H, (unsigned)nt), 256, smem, stream>>>(p);
    return cudaGetLastError();
}

// One tensor of a backward (K or V); dx and dw may be null.
struct LcGrad {
    const void* x;
    int64_t x_sn;
    const void *w, *dy;
    void* dx;
    void* dw;
};
struct LcPeGrad {
    const void* pe;
    void* dpe;
    const float* dbias;
    int parts;
};

template <typename ET>
static int run_bwd(const LcGrad* t, int nt, const LcPeGrad& pe, const int32_t* cu_dev, const int32_t* seqlens, int batch, int H, int D, int ks, int stride,
                   int dtype, int32_t* status, cudaStream_t stream) {
    if (t[0].dx) {
        LcDxMaps maps;
        LcDxParams p;
        p.H = H; p.ks = ks; p.stride = stride; p.phases = stride < 4 ? stride : 4; p.status = status;
        p.n_seq = 0; p.tile0[0] = 0;
        for (int i = 0; i < nt; ++i) {
            int rc = make_tile_map(&maps.w[i], t[i].w, dtype, (int64_t)H * ks * D, D, D, 64);
            if (rc) return rc;
            p.dx[i] = t[i].dx;
        }
        int64_t tok0 = 0, y0 = 0;
        const int64_t row_bytes = (int64_t)H * D * 2;
        for (int b = 0; b < batch; ++b) {
            const int L = seqlens[b];
            if (L < 0) return FSA_ERR_BAD_ARG;
            const int n = L >= ks ? (L - ks) / stride + 1 : 0;
            if (L > 0) {
                const int q = p.n_seq;
                for (int i = 0; i < nt; ++i) {
                    // (a sequence without a window loads nothing: any valid map does)
                    int rc = make_tile_map(&maps.y[i][q], n > 0 ? (const char*)t[i].dy + y0 * row_bytes : (const char*)t[i].w, dtype, n > 0 ? n : 1,
                                           n > 0 ? (int64_t)H * D : D, n > 0 ? (int64_t)H * D : D, 128);
                    if (rc) return rc;
                }
                p.n_cmp[q] = n; p.L[q] = L; p.tok0[q] = tok0;
                p.tile0[q + 1] = p.tile0[q] + ((L + stride - 1) / stride + 127) / 128;
                ++p.n_seq;
            }
            tok0 += L;
            y0 += n;
            if (p.n_seq == kLbSeqs || (b == batch - 1 && p.n_seq > 0)) {
                const cudaError_t e = D == 128 ? launch_dx<128, ET>(maps, p, nt, stream) : launch_dx<64, ET>(maps, p, nt, stream);
                if (e != cudaSuccess) return FSA_ERR_CUDA;
                p.n_seq = 0;
            }
        }
    }
    if (t[0].dw || pe.dpe || (nt > 1 && t[1].dw)) {
        LcDwParams<ET> p = {};
        for (int i = 0; i < nt; ++i) {
            p.x[i] = (const ET*)t[i].x; p.x_sn[i] = t[i].x_sn; p.dy[i] = (const ET*)t[i].dy; p.dw[i] = (ET*)t[i].dw;
        }
        p.cu = cu_dev; p.batch = batch; p.H = H; p.ks = ks; p.stride = stride; p.status = status;
        p.pe = (const ET*)pe.pe; p.w = (const ET*)t[0].w; p.dpe = (ET*)pe.dpe; p.dbias = pe.dbias; p.parts = pe.parts;
        const cudaError_t e = D == 128 ? launch_dw<128, ET>(p, nt, stream) : launch_dw<64, ET>(p, nt, stream);
        if (e != cudaSuccess) return FSA_ERR_CUDA;
    }
    return FSA_OK;
}

cudaError_t launch_column_sum(int dtype, int D, const void* dy, int64_t rows, int H, int parts, float* out, int* status, cudaStream_t stream);

constexpr int kBiasParts = 32;      // shares of the windows in the sum that is the bias's gradient

static int check_bwd(const LcGrad& g, const int32_t* cu, const int32_t* seqlens, int batch, int H, int D, int ks, int stride, int dtype, int64_t* total) {
    if (!g.x || !g.w || !cu || !seqlens || batch < 0 || H <= 0 || ks <= 0 || stride <= 0) return FSA_ERR_BAD_ARG;
    if (dtype != FSA_DTYPE_BF16 && dtype != FSA_DTYPE_FP16) return FSA_ERR_BAD_ARG;
    if (D != 64 && D != 128) return FSA_ERR_UNSUPPORTED;
    if (ks % stride != 0 || (stride & (stride - 1)) != 0 || (ks & 1)) return FSA_ERR_UNSUPPORTED;
    if (((uintptr_t)g.x & 15) || ((uintptr_t)g.w & 15) || ((uintptr_t)g.dy & 15) || ((uintptr_t)g.dx & 15) || ((uintptr_t)g.dw & 15) || (g.x_sn % 8))
        return FSA_ERR_BAD_ARG;
    if (g.x_sn < (int64_t)H * D) return FSA_ERR_BAD_ARG;
    *total = 0;
    for (int b = 0; b < batch; ++b)
        if (seqlens[b] >= ks) *total += (seqlens[b] - ks) / stride + 1;
    return *total > 0 && !g.dy ? FSA_ERR_BAD_ARG : FSA_OK;
}

}  // namespace fsa

using namespace fsa;

extern "C" int fsa_linear_compress_bwd(const void* x, int64_t x_stride_n, const void* w, const void* dy, const int32_t* cu_seqlens,
                                       const int32_t* seqlens_host, int batch, int num_heads, int head_dim, int kernel_size,
                                       int kernel_stride, int dtype, void* dx, void* dw, int32_t* status, void* stream_) {
    const LcGrad g{x, x_stride_n, w, dy, dx, dw};
    int64_t total = 0;
    int rc = check_bwd(g, cu_seqlens, seqlens_host, batch, num_heads, head_dim, kernel_size, kernel_stride, dtype, &total);
    if (rc) return rc;
    (void)cudaGetLastError();
    if ((rc = ensure_context())) return rc;
    const LcPeGrad none{nullptr, nullptr, nullptr, 0};
    cudaStream_t stream = (cudaStream_t)stream_;
    return dtype == FSA_DTYPE_BF16
               ? run_bwd<__nv_bfloat16>(&g, 1, none, cu_seqlens, seqlens_host, batch, num_heads, head_dim, kernel_size, kernel_stride, dtype, status, stream)
               : run_bwd<__half>(&g, 1, none, cu_seqlens, seqlens_host, batch, num_heads, head_dim, kernel_size, kernel_stride, dtype, status, stream);
}

extern "C" int64_t fsa_compress_kv_bwd_scratch_bytes(int num_heads, int head_dim) { return (int64_t)kBiasParts * num_heads * head_dim * 4 + 16; }

extern "C" int fsa_compress_kv_bwd(const void* k, int64_t k_stride_n, const void* v, int64_t v_stride_n, const void* w_key, const void* w_value,
                                   const void* pe, const void* dyk, const void* dyv, const int32_t* cu_seqlens, const int32_t* seqlens_host, int batch, int num_heads, int head_dim, int kernel_size,
                                   int kernel_stride, int dtype, void* dk, void* dv, void* dw_key, void* dw_value, void* dpe, float* scratch,
                                   void* stream_) {
    const LcGrad g[2] = {{k, k_stride_n, w_key, dyk, dk, dw_key}, {v, v_stride_n, w_value, dyv, dv, dw_value}};
    int64_t total = 0;
    for (int i = 0; i < 2; ++i) {
        const int rc = check_bwd(g[i], cu_seqlens, seqlens_host, batch, num_heads, head_dim, kernel_size, kernel_stride, dtype, &total);
        if (rc) return rc;
    }
    if (!dk || !dv || !pe || !scratch) return FSA_ERR_BAD_ARG;
    (void)cudaGetLastError();
    int rc = ensure_context();
    if (rc) return rc;
    cudaStream_t stream = (cudaStream_t)stream_;
    const int parts = total < 32 * kBiasParts ? (total < 32 ? 1 : (int)(total / 32)) : kBiasParts;
    int* status = (int*)(scratch + (int64_t)kBiasParts * num_heads * head_dim);
    if (launch_column_sum(dtype, head_dim, dyk, total, num_heads, parts, scratch, status, stream) != cudaSuccess) return FSA_ERR_CUDA;
    const LcPeGrad pg{pe, dpe, scratch, parts};
    return dtype == FSA_DTYPE_BF16
               ? run_bwd<__nv_bfloat16>(g, 2, pg, cu_seqlens, seqlens_host, batch, num_heads, head_dim, kernel_size, kernel_stride, dtype, status, stream)
               : run_bwd<__half>(g, 2, pg, cu_seqlens, seqlens_host, batch, num_heads, head_dim, kernel_size, kernel_stride, dtype, status, stream);
}
