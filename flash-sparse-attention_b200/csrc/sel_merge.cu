// Merges of the selected-attention kernels for sm_100a, for tokens of up to 16 partial rows: o from the forward's unnormalised
// partial outputs and their (m, l), dQ as the plain sum of the backward's partial rows.  (In the reference: the reduction of
// fsa/ops/FSA_topk_sparse_attention.py:741-818 and the dQ accumulation of :1416-1545.)
//
// 4 KB (head size 64: 2 KB) have to come in per output row, as 16 pieces of 256 bytes from all over 2 GB.  As one warp per row that
// loads positions, then rows, then sums up and ends, the merge was bound by that chain of round trips, not by memory (partial
// rows laid out in one contiguous piece took it no less time).  Here a CTA stays on its SM and each of 24 warps keeps two output rows
// (8 KB) in flight in its own ring; positions and statistics are loaded two rows before.  (With 12 warps and 16 KB each the arithmetic of a
// warp holds its stages up.)  What bounded it then was the issue of instructions: 665 (forward) and 504 (dQ) a row, of which the
// bulk copy per partial row alone took some 200 (the copies of a warp's lanes are issued one after the other).  16-byte asynchronous
// copies, a lane each, take 8 instructions for the 4 KB, fill missing rows with zeros (no case apart for them) and are waited
// for by count; pairs of elements are multiplied and added together (f32x2: the same roundings).
// 64K tokens x 8 heads x 16 rows of 256 bytes: forward 502 (a warp per row) -> 420 (bulk copies) -> 374 us in 418 instructions a row, dQ 476 -> 361 -> 360 us
// in 290 = 6.4 and 6.5 TB/s in all, the rate of a copy; 21K tokens x 4 heads x 8 rows, which L2 holds: forward 60 -> 42 us.  At head size 256 a
// warp per row already moves 5.9 TB/s and keeps the other kernels; at 64 half a warp takes a row.
#include "sel_launch.cuh"

namespace fsa {

constexpr int kMgWarps = 24, kMgSlots = 16;
constexpr int64_t kMgRows = 24000;      // output rows from which a warp has enough of them in turn (fewer: a warp each, sel_fwd.cu and sel_bwd.cu)

template <int D>
struct MergeCfg {
    static constexpr int kRow = D * 2;                      // bytes of a partial row
    static constexpr int H = 128 / D;                       // output rows that a warp takes at a time: one, or at head size 64 one per half warp
    static constexpr int kStage = H * kMgSlots * kRow;      // 4 KB
    static constexpr int kBytes = kMgWarps * (2 * kStage + H * kMgSlots * 8);
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

// two fp32 values side by side in a 64-bit register
__device__ __forceinline__ uint64_t f32x2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 f32x2_get(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// ALL: 13 to 16 partial rows, every copy and addition without a test
template <int D, typename ET, bool FWD, bool ALL>
__global__ void __launch_bounds__(kMgWarps * 32, 1) sel_merge(const ET* __restrict__ part, const float2* __restrict__ ml, const int* __restrict__ pos,
                                                             SelShape s, int nsub, ET* __restrict__ out, int64_t o_sn, int64_t o_sh,
                                                             float* __restrict__ lse) {
    using C = MergeCfg<D>;
    constexpr int H = C::H, LPR = 32 / H;                    // LPR: lanes of an output row
    constexpr int CPR = D / 8, RPI = 32 / CPR;               // 16-byte pieces of a partial row; partial rows that a copy instruction covers
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, l = lane % LPR, half = lane / LPR;
    uint8_t* ring = smem + warp * (2 * C::kStage);
    float2* wts = reinterpret_cast<float2*>(smem + kMgWarps * 2 * C::kStage) + warp * H * kMgSlots;      // every weight twice, a pair's factor
    const int N = (int)s.N, rows = N * s.Hq, W = (int)gridDim.x * kMgWarps * H, first = ((int)blockIdx.x * kMgWarps + warp) * H;
    const int R = s.T * nsub, R4 = (R + 3) & ~3;             // partial rows of an output row
    const int sub = l / s.T, sl = l - sub * s.T;             // lane: partial row l = sub * T + sl (l < R)
    const int shift = 31 - __clz(s.TPT);
    const bool pow2 = s.TPT == 1 << shift;
    const MergeRow step = merge_row(W, s);
    MergeRow next = merge_row(first + half, s);              // (n = N or more: past the last row)
    int row0 = first;                                        // the warp's first row of `next`

    struct Row { int n, hq, g, part; float2 st; };           // output row (n < 0: none); lane: its partial row (-1: none) and its statistics
    auto fetch = [&]() {
        Row r{-1, 0, 0, -1, make_float2(-INFINITY, 0.f)};
        if (row0 < rows && next.n < N) {
            r.n = next.n;
            r.hq = next.h * s.G + next.g;
            r.g = next.g;
            if (l < R) {
                // (rows and entries of a kv head fit 30 bits, their products with T need not)
                r.part = __ldg(pos + (int64_t)(next.h * N + next.n) * s.T + sl);
                if (FWD) r.st = __ldg(ml + (int64_t)(r.hq * N + next.n) * s.T + l);
            }
        }
        row0 += W;
        next.next(step, s.Hk, s.G);
        return r;
    };
    // copies the partial rows of r into a stage (zeros for those that it does not have)
    auto issue = [&](const Row& r, int st) {
        int src = -1;
        if (r.part >= 0) {
            const int tile = pow2 ? r.part >> shift : r.part / s.TPT;
            src = (tile * nsub + sub) * kTileRows + r.g * s.TPT + (r.part - tile * s.TPT);
        }
        const uint32_t dst = smem_u32(ring + st * C::kStage) + lane * 16;
        const ET* base = part + (lane % CPR) * 8;
        if (ALL && __all_sync(0xffffffffu, src >= 0 || l >= kMgSlots)) {
#pragma unroll
            for (int it = 0; it < H * kMgSlots / RPI; ++it)
                cp_async16(dst + it * 512, base + (int64_t)__shfl_sync(0xffffffffu, src, it * RPI + lane / CPR) * D, true);
        } else {
#pragma unroll 1
            for (int it = 0; it < H * kMgSlots / RPI; ++it) {
                if (!ALL && (it * RPI) % kMgSlots >= R4) continue;
                const int row = __shfl_sync(0xffffffffu, src, it * RPI + lane / CPR);
                cp_async16(dst + it * 512, base + (int64_t)max(row, 0) * D, row >= 0);
            }
        }
        cp_async_commit();
    };
    Row q0 = fetch(), q1 = fetch(), q2 = fetch();
    issue(q0, 0);
    issue(q1, 1);
    int st = 0;
    for (int r = first; r < rows; r += W) {
        Row q3 = fetch();
        cp_async_wait<1>();
        __syncwarp();
        float M = 0.f, L = 1.f;
        if (FWD) {
            // (16 lanes hold the slots of a row: four steps, and at head size 128 the sum handed to the others)
            const float m0 = q0.part >= 0 ? q0.st.x : -INFINITY;
            M = m0;
#pragma unroll
            for (int o = 8; o; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
            const float w = m0 == -INFINITY ? 0.f : exp2f(m0 - M);
            if (l < kMgSlots) wts[half * kMgSlots + l] = make_float2(w, w);
            L = m0 == -INFINITY ? 0.f : w * q0.st.y;
#pragma unroll
            for (int o = 8; o; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
            if (H == 1) L = __shfl_sync(0xffffffffu, L, lane & 15);
            __syncwarp();
        }
        const uint8_t* src = ring + st * C::kStage + half * (kMgSlots * C::kRow) + l * 8;
        const float2* wt = wts + half * kMgSlots;
        uint64_t a0 = 0, a1 = 0;                              // the lane's four elements
        auto add = [&](int j, uint64_t w) {
            const uint2 u = *reinterpret_cast<const uint2*>(src + j * C::kRow);
            const float2 x = ElemTraits<ET>::unpack2(u.x), y = ElemTraits<ET>::unpack2(u.y);
            a0 = FWD ? fma_f32x2(f32x2(x.x, x.y), w, a0) : add_f32x2(f32x2(x.x, x.y), a0);
            a1 = FWD ? fma_f32x2(f32x2(y.x, y.y), w, a1) : add_f32x2(f32x2(y.x, y.y), a1);
        };
        auto four = [&](int j) {
            ulonglong2 w01 = make_ulonglong2(0, 0), w23 = w01;
            if (FWD) {
                w01 = *reinterpret_cast<const ulonglong2*>(wt + j);
                w23 = *reinterpret_cast<const ulonglong2*>(wt + j + 2);
            }
            add(j, w01.x); add(j + 1, w01.y); add(j + 2, w23.x); add(j + 3, w23.y);
        };
        if (ALL) {
#pragma unroll
            for (int j = 0; j < kMgSlots; j += 4) four(j);
        } else {
#pragma unroll 1
            for (int j = 0; j < R4; j += 4) four(j);
        }
        __syncwarp();                                         // the stage has been read
        issue(q2, st);
        st ^= 1;
        if (q0.n >= 0) {
            const float inv = FWD ? (L > 0.f ? 1.f / L : 0.f) : 1.f;
            const float2 x = f32x2_get(a0), y = f32x2_get(a1);
            *reinterpret_cast<uint2*>(out + (int64_t)q0.n * o_sn + (int64_t)q0.hq * o_sh + l * 4) =
                make_uint2(ElemTraits<ET>::pack2(x.x * inv, x.y * inv), ElemTraits<ET>::pack2(y.x * inv, y.y * inv));
            if (FWD && l == 0) lse[q0.hq * N + q0.n] = L > 0.f ? M + log2f(L) : -INFINITY;
        }
        q0 = q1; q1 = q2; q2 = q3;
    }
    cp_async_wait<0>();
}

bool sel_merge_fits(const SelShape& s, int nsub) {
    return s.D <= 128 && s.T * nsub <= kMgSlots && s.N * s.Hq >= kMgRows && s.N * s.Hq < (1ll << 30);
}

template <int D, typename ET, bool FWD>
static cudaError_t launch_merge(const void* part, const float2* ml, const int* pos, const SelShape& s, int nsub, void* out, int64_t o_sn,
                                int64_t o_sh, float* lse, int sms, cudaStream_t stream) {
    auto kern = s.T * nsub > 12 ? sel_merge<D, ET, FWD, true> : sel_merge<D, ET, FWD, false>;
    cudaError_t e = allow_smem((const void*)kern, MergeCfg<D>::kBytes);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)sms, kMgWarps * 32, MergeCfg<D>::kBytes, stream>>>((const ET*)part, ml, pos, s, nsub, (ET*)out, o_sn, o_sh, lse);
    return cudaGetLastError();
}

template <bool FWD>
static cudaError_t merge(int dtype, const void* part, const float2* ml, const int* pos, const SelShape& s, int nsub, void* out, int64_t o_sn,
                         int64_t o_sh, float* lse, int sms, cudaStream_t stream) {
#define FSA_CASE(DD)                                                                                                                            \
    if (s.D == DD)                                                                                                                              \
        return dtype == kBF16 ? launch_merge<DD, __nv_bfloat16, FWD>(part, ml, pos, s, nsub, out, o_sn, o_sh, lse, sms, stream)         \
                              : launch_merge<DD, __half, FWD>(part, ml, pos, s, nsub, out, o_sn, o_sh, lse, sms, stream);
    FSA_CASE(64) FSA_CASE(128)
#undef FSA_CASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_sel_merge_fwd(int dtype, const void* part, const float2* ml, const int* pos, const SelShape& s, void* o, int64_t o_sn,
                                 int64_t o_sh, float* lse, int sms, cudaStream_t stream) {
    return merge<true>(dtype, part, ml, pos, s, 1, o, o_sn, o_sh, lse, sms, stream);
}

cudaError_t launch_sel_merge_dq(int dtype, const void* part, const int* pos, const SelShape& s, int nsub, void* dq, int sms, cudaStream_t stream) {
    return merge<false>(dtype, part, nullptr, pos, s, nsub, dq, (int64_t)s.Hq * s.D, s.D, nullptr, sms, stream);
}

}  // namespace fsa
