// Merges of the selected-attention kernels for sm_100a, for tokens of up to 16 partial rows: o from the forward's unnormalised
// partial outputs and their (m, l), dQ as the plain sum of the backward's partial rows.  (In the reference: the reduction of
// fsa/ops/FSA_topk_sparse_attention.py:741-818 and the dQ accumulation of :1416-1545.)
//
// 4 KB (head size 64: 2 KB) have to come in per output row, as 16 pieces of 256 bytes from all over 2 GB.  As one warp per row that
// loads positions, then rows, then sums up and ends, the merge was bound by that chain of round trips, not by memory (partial
// rows laid out in one contiguous piece took it no less time).  Here a CTA stays on its SM and each of 24 warps keeps 8 KB of
// rows in flight: one bulk copy per partial row into the warp's own ring of stages, whose positions were loaded two rows before;
// nothing passes through registers.  (With 12 warps and 16 KB each the arithmetic of a warp holds its stages up: dQ 503 us.)
// 64K tokens x 8 heads x 16 rows of 256 bytes: forward 502 -> 420 us, dQ 476 -> 361 us = 5.1 and 5.9 TB/s of partial rows.  At head size 256 a
// warp per row already moves 5.9 TB/s and keeps the other kernels; at 64 a row's arithmetic is too much for 24 warps (151 -> 193 us
// forward at 16384 tokens x 16 heads), so that half a warp takes a row there (forward 144 us, dQ 157 -> 137 us).
#include "sel_launch.cuh"

namespace fsa {

constexpr int kMgWarps = 24, kMgSlots = 16;
constexpr int64_t kMgRows = 24000;      // output rows from which a warp has enough of them in turn (fewer: a warp each, sel_fwd.cu and sel_bwd.cu)

template <int D>
struct MergeCfg {
    static constexpr int kRow = D * 2;                      // bytes of a partial row
    static constexpr int H = 128 / D;                       // output rows that a warp takes at a time: one, or at head size 64 one per half warp
    static constexpr int kStage = H * kMgSlots * kRow;
    static constexpr int S = 8192 / kStage;                 // stages of a warp
    static constexpr int kBytes = kMgWarps * (S * (kStage + 8 + 4) + H * kMgSlots * 4);
};

// An output row (token, kv head, head of the group) and the step from one of a warp's rows to the next.
struct MergeRow {
    int n, h, g;
    __device__ __forceinline__ void next(const MergeRow& d, int Hk, int G) {
        g += d.g; h += d.h; n += d.n;
        if (g >= G) { g -= G; ++h; }
        if (h >= Hk) { h -= Hk; ++n; }
    }
};
__device__ __forceinline__ MergeRow merge_row(int row, const SelShape& s) {
    MergeRow r;
    r.n = (int)((unsigned)row / (unsigned)s.Hq);
    const int hq = row - r.n * s.Hq;
    r.h = hq / s.G;
    r.g = hq - r.h * s.G;
    return r;
}

template <int D, typename ET, bool FWD>
__global__ void __launch_bounds__(kMgWarps * 32, 1) sel_merge(const ET* __restrict__ part, const float2* __restrict__ ml, const int* __restrict__ pos,
                                                             SelShape s, int nsub, ET* __restrict__ out, int64_t o_sn, int64_t o_sh,
                                                             float* __restrict__ lse, int* status) {
    using C = MergeCfg<D>;
    constexpr int S = C::S, H = C::H, LPR = 32 / H, V = D / LPR;          // LPR: lanes of an output row
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, l = lane % LPR, half = lane / LPR;
    uint8_t* ring = smem + warp * (S * C::kStage);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kMgWarps * S * C::kStage) + warp * S;
    float* wts = reinterpret_cast<float*>(smem + kMgWarps * S * (C::kStage + 8)) + (warp * H + half) * kMgSlots;
    unsigned* masks = reinterpret_cast<unsigned*>(smem + kMgWarps * (S * (C::kStage + 8) + H * kMgSlots * 4)) + warp * S;
    if (lane < S) mbar_init(&bars[lane], 1);
    mbar_init_fence();
    __syncwarp();
    const int rows = (int)(s.N * s.Hq), items = (rows + H - 1) / H, W = (int)gridDim.x * kMgWarps, first = (int)blockIdx.x * kMgWarps + warp;
    const int cnt = first < items ? (items - first + W - 1) / W : 0;
    const MergeRow step = merge_row(W * H, s);
    const int R = s.T * nsub, sl = l % s.T, sub = l / s.T;              // partial rows; lane: row sub * T + sl
    MergeRow at_pos = merge_row(first * H + half, s), at_ml = at_pos, at = at_pos;      // (n = N: the odd row out at the end)
    auto load_pos = [&](int& ps, int& g) {
        ps = l < R && at_pos.n < s.N ? __ldg(pos + ((int64_t)at_pos.h * s.N + at_pos.n) * s.T + sl) : -1;
        g = at_pos.g;
        at_pos.next(step, s.Hk, s.G);
    };
    auto load_ml = [&]() {
        const float2 v = l < s.T && at_ml.n < s.N ? __ldg(ml + ((int64_t)(at_ml.h * s.G + at_ml.g) * s.N + at_ml.n) * s.T + l) : make_float2(0.f, 0.f);
        at_ml.next(step, s.Hk, s.G);
        return v;
    };
    auto issue = [&](int k, int ps, int g) {
        const int st = k % S;
        const unsigned mask = __ballot_sync(0xffffffffu, ps >= 0);
        if (lane == 0) {
            masks[st] = mask;
            mbar_expect_tx(&bars[st], (uint32_t)(__popc(mask) * C::kRow));
        }
        __syncwarp();
        if (ps >= 0) {
            const int tile = ps / s.TPT;
            const int64_t row = ((int64_t)tile * nsub + sub) * kTileRows + g * s.TPT + (ps - tile * s.TPT);
            bulk_load(smem_u32(ring + st * C::kStage + (half * kMgSlots + l) * C::kRow), part + row * D, C::kRow, &bars[st]);
        }
    };
    int ps[S], gs[S];
#pragma unroll
    for (int k = 0; k < S; ++k)
        if (k < cnt) load_pos(ps[k], gs[k]);
    int pA = -1, pB = -1, gA = 0, gB = 0;                     // positions of the next two rows to be copied
    float2 mA = make_float2(0.f, 0.f), mB = mA;               // (m, l) of this row and the next
    if (S < cnt) load_pos(pA, gA);
    if (S + 1 < cnt) load_pos(pB, gB);
    if (FWD && cnt > 0) mA = load_ml();
    if (FWD && cnt > 1) mB = load_ml();
#pragma unroll
    for (int k = 0; k < S; ++k)
        if (k < cnt) issue(k, ps[k], gs[k]);

    int k = 0;
    for (; k < cnt; ++k) {
        const int st = k % S;
        const float2 v = mA;
        if (FWD) {
            mA = mB;
            if (k + 2 < cnt) mB = load_ml();
        }
        if (!__all_sync(0xffffffffu, mbar_wait(&bars[st], (k / S) & 1, status))) break;      // (the warp stays together)
        const unsigned mask = masks[st];
        const ET* src = reinterpret_cast<const ET*>(ring + st * C::kStage) + half * kMgSlots * D + l * V;
        float acc[V];
#pragma unroll
        for (int i = 0; i < V; ++i) acc[i] = 0.f;
        float M = 0.f, L = 1.f;
        if (FWD) {
            // (16 lanes hold the slots of a row: four steps, and at head size 128 the sum handed to the others)
            const float m0 = (mask >> lane & 1u) ? v.x : -INFINITY;
            M = m0;
#pragma unroll
            for (int o = 8; o; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
            const float w = m0 == -INFINITY ? 0.f : exp2f(m0 - M);
            if (l < kMgSlots) wts[l] = w;
            L = m0 == -INFINITY ? 0.f : w * v.y;
#pragma unroll
            for (int o = 8; o; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
            L = __shfl_sync(0xffffffffu, L, lane & ~(LPR - 1));
            __syncwarp();
        }
        const bool all = mask == ((1u << R) - 1u) * (H == 2 ? 0x10001u : 1u) && (R & 3) == 0;
        auto four = [&](int j0) {
            const float4 w = FWD ? *reinterpret_cast<const float4*>(wts + j0) : make_float4(1.f, 1.f, 1.f, 1.f);
            fma_row_vec<V, ET>(acc, ld_row_vec<V, ET>(src + j0 * D), w.x);
            fma_row_vec<V, ET>(acc, ld_row_vec<V, ET>(src + (j0 + 1) * D), w.y);
            fma_row_vec<V, ET>(acc, ld_row_vec<V, ET>(src + (j0 + 2) * D), w.z);
            fma_row_vec<V, ET>(acc, ld_row_vec<V, ET>(src + (j0 + 3) * D), w.w);
        };
        if (all && R == kMgSlots) {
#pragma unroll
            for (int j0 = 0; j0 < kMgSlots; j0 += 4) four(j0);
        } else if (all) {
            for (int j0 = 0; j0 < R; j0 += 4) four(j0);
        } else {
            for (int j = 0; j < R; ++j)
                if (mask >> (half * 16 + j) & 1u) fma_row_vec<V, ET>(acc, ld_row_vec<V, ET>(src + j * D), FWD ? wts[j] : 1.f);
        }
        __syncwarp();                            // the stage has been read
        if (k + S < cnt) {
            issue(k + S, pA, gA);
            pA = pB; gA = gB;
            if (k + S + 2 < cnt) load_pos(pB, gB);
        }
        const int hq = at.h * s.G + at.g;
        const float inv = FWD ? (L > 0.f ? 1.f / L : 0.f) : 1.f;
        ET* dst = out + (int64_t)at.n * o_sn + (int64_t)hq * o_sh + l * V;
        uint32_t x[V / 2];
#pragma unroll
        for (int i = 0; i < V / 2; ++i) x[i] = ElemTraits<ET>::pack2(acc[2 * i] * inv, acc[2 * i + 1] * inv);
        if (at.n < s.N) {
            *reinterpret_cast<uint2*>(dst) = make_uint2(x[0], x[1]);
            if (FWD && l == 0) lse[(int64_t)hq * s.N + at.n] = L > 0.f ? M + log2f(L) : -INFINITY;
        }
        at.next(step, s.Hk, s.G);
    }
    // (on a wait that ran out: the copies in flight, those of this row and the S - 1 behind it, land before the CTA ends)
    for (int j = k; j < cnt && j < k + S; ++j)
        if (lane == 0) mbar_wait(&bars[j % S], (j / S) & 1, nullptr);
}

bool sel_merge_fits(const SelShape& s, int nsub) {
    return s.D <= 128 && s.T * nsub <= kMgSlots && s.N * s.Hq >= kMgRows && s.N * s.Hq < (1ll << 30);
}

template <int D, typename ET, bool FWD>
static cudaError_t launch_merge(const void* part, const float2* ml, const int* pos, const SelShape& s, int nsub, void* out, int64_t o_sn,
                                int64_t o_sh, float* lse, int* status, int sms, cudaStream_t stream) {
    auto kern = sel_merge<D, ET, FWD>;
    cudaError_t e = allow_smem((const void*)kern, MergeCfg<D>::kBytes);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)sms, kMgWarps * 32, MergeCfg<D>::kBytes, stream>>>((const ET*)part, ml, pos, s, nsub, (ET*)out, o_sn, o_sh, lse, status);
    return cudaGetLastError();
}

template <bool FWD>
static cudaError_t merge(int dtype, const void* part, const float2* ml, const int* pos, const SelShape& s, int nsub, void* out, int64_t o_sn,
                         int64_t o_sh, float* lse, int* status, int sms, cudaStream_t stream) {
#define FSA_CASE(DD)                                                                                                                            \
    if (s.D == DD)                                                                                                                              \
        return dtype == kBF16 ? launch_merge<DD, __nv_bfloat16, FWD>(part, ml, pos, s, nsub, out, o_sn, o_sh, lse, status, sms, stream)         \
                              : launch_merge<DD, __half, FWD>(part, ml, pos, s, nsub, out, o_sn, o_sh, lse, status, sms, stream);
    FSA_CASE(64) FSA_CASE(128)
#undef FSA_CASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_sel_merge_fwd(int dtype, const void* part, const float2* ml, const int* pos, const SelShape& s, void* o, int64_t o_sn,
                                 int64_t o_sh, float* lse, int* status, int sms, cudaStream_t stream) {
    return merge<true>(dtype, part, ml, pos, s, 1, o, o_sn, o_sh, lse, status, sms, stream);
}

cudaError_t launch_sel_merge_dq(int dtype, const void* part, const int* pos, const SelShape& s, int nsub, void* dq, int* status, int sms,
                                cudaStream_t stream) {
    return merge<false>(dtype, part, nullptr, pos, s, nsub, dq, (int64_t)s.Hq * s.D, s.D, nullptr, status, sms, stream);
}

}  // namespace fsa
