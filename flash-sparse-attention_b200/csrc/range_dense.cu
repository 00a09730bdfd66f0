// Range attention forward, query-tile-major ("dense") kernel for sm_100a: every token attends one contiguous range of
// K/V rows, as in the compressed branch (replaces the forward of CompressedAttention,
// nsa_ref/ops/compressed_attention.py:762-829, kernel :33-190) and in the sliding-window branch (replaces the
// flash_attn_varlen_func call of fsa/module/fsa.py:149-159).
//
// One item = one tile of <= 128 rows = (query head of a GQA group, TPT consecutive tokens of one sequence) x one KV head.
// The rows of the tile see neighbouring ranges, so the CTA walks the 64-row K/V tiles from the lowest row any of its rows
// sees to the highest, keeps the output accumulator in TMEM across them (online softmax) and writes o and lse once: no
// partial rows, no merge kernel, no index.  Two CTAs share an SM (112 KB of shared memory and 256 TMEM columns each), so
// the softmax of one overlaps the MMAs of the other.  The grid has a CTA per item, but a CTA that runs takes over items whose
// CTA has not started (cluster launch control), one ahead: finding a tile, its ranges and the first loads take 7200 cycles and
// the end of an item 4500, as long as seven of its K/V tiles, and run under the item before.  Measured at sequences
// of 20011 and 12345 tokens, 32 / 8 heads, window of 512 and compressed branch: 788 -> 594 us (a CTA per item before).
//   warp 0      finds the items; TMA producer: the Q tile (3-D box: column, token, head -> head-major rows), K and V tiles through
//               two rings of two stages (K is released by the S product, V by the P V product, so K runs a tile ahead);
//   warp 1      one elected thread issues S(j+1) = Q K^T before the softmax of tile j is done, then O (+)= P(j) V(j);
//   warps 2..5  one row per thread: scaled logits from TMEM, per-row range mask, running max / sum, P -> TMEM (input dtype,
//               over S).  The reference max of a row is only raised when a tile exceeds it by more than 2^8 (the final
//               o = O / l does not depend on the reference); then the warp waits for the previous P V product and
//               rescales its 32 accumulator rows in TMEM.  Epilogue: o = O / l through swizzled staging, 64 columns at a
//               time, and 3-D TMA stores, or plain stores for the last, partial tile of a sequence; lse = m + log2 l.
#include "../../include/fsa_sm100.h"
#include <climits>

#include "sel_launch.cuh"

namespace fsa {

int make_tile_map(CUtensorMap* map, const void* base, int dtype, int64_t rows, int64_t cols, int64_t row_stride, int box_rows);
int make_tile_map_3d_box(CUtensorMap* map, const void* base, int dtype, int64_t d0, int64_t d1, int64_t d2, int64_t stride1,
                         int64_t stride2, int box1, int box2);
int device_sm_count(int* out);

struct RangeDenseParams {
    const int32_t* cu_q;    // [B + 1]
    const int32_t* cu_k;    // [B + 1] first K/V row of every sequence
    const int32_t* kv_lo;   // [N] lowest visible K/V row of every token, or null (the sequence's first row)
    const int32_t* kv_hi;   // [N] highest visible K/V row, lower than kv_lo when the token sees nothing
    int64_t N, Nk;
    int B, Hq, Hk, G, TPT;
    float scale_log2;
    void* o;  int64_t o_sn, o_sh;     // [N, Hq, D]
    float* lse;                       // [Hq, N] log2 units
    int* status;
};

// Up to three problems in one launch (blockIdx.z): branches of a layer that do not wait for one another.  A short prompt has fewer tiles
// than the SMs hold CTAs, and each launch of its own left most of them empty (517 tokens, 32 / 8 heads: 3 x 11 us, together 19: prefill 158 -> 138 us).
constexpr int kRdProblems = 3;
struct RangeDenseLaunch {
    CUtensorMap q[kRdProblems], k[kRdProblems], v[kRdProblems], o[kRdProblems];
    RangeDenseParams p[kRdProblems];
};

constexpr int kRdThreads = 192;
constexpr int kRdBK = 64;
constexpr float kRdLazy = 8.0f;       // raise a row's reference max only when exceeded by more than this (log2 units)

__device__ __forceinline__ float rd_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// One item: a tile of tokens x one KV head of problem z.
struct RdItem {
    int z, h, seq, tok0, ne, row_lo, nblk;
};

// The K/V rows that a row of the item sees: [x, y].
__device__ __forceinline__ int2 rd_row(const RangeDenseLaunch& launch, const RdItem& m, bool valid, int e) {
    if (m.z < 0 || !valid) return make_int2(0, -1);
    const RangeDenseParams& p = launch.p[m.z];
    return make_int2(p.kv_lo ? __ldg(p.kv_lo + m.tok0 + e) : __ldg(p.cu_k + m.seq), __ldg(p.kv_hi + m.tok0 + e));
}

// Takes over a CTA of this launch that has not started yet (cluster launch control): 16 bytes of answer at dst, with bar as the
// transaction barrier.  Not to be called again once the answer was no.
__device__ __forceinline__ void claim_next_cta(uint32_t dst, uint64_t* bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(dst),
                 "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool claimed_cta(uint32_t src, int& x, int& y, int& z) {
    uint32_t yes, cx, cy, cz;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b128 a;\n\t"
        "mov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
        "ld.shared.b128 a, [%4];\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, a;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, _}, a;\n\t}"
        : "=r"(yes), "=r"(cx), "=r"(cy), "=r"(cz) : "r"(src) : "memory");
    x = (int)cx; y = (int)cy; z = (int)cz;
    return yes != 0;
}

template <int D, typename ET>
__global__ void __launch_bounds__(kRdThreads, 2) range_fwd_dense(const __grid_constant__ RangeDenseLaunch launch) {
    constexpr int BK = kRdBK;
    constexpr int kQ = kTileRows * D * 2;
    constexpr int kKt = BK * D * 2;                  // one K (or V) tile
    constexpr int KH = D / 64;
    constexpr uint32_t kCols = (2 * BK + D) <= 128 ? 128 : 256;
    constexpr int cS = 0, cO = 2 * BK;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + kQ;
    uint8_t* sV = sK + 2 * kKt;
    uint8_t* sOut = sV + 2 * kKt;                    // 64 output columns on their way out
    uint64_t* bars = reinterpret_cast<uint64_t*>(sOut + kTileRows * 128);
    uint64_t* q_full = bars;            // [1]
    uint64_t* k_full = bars + 1;        // [2]
    uint64_t* k_empty = bars + 3;       // [2]
    uint64_t* v_full = bars + 5;        // [2]
    uint64_t* v_empty = bars + 7;       // [2]
    uint64_t* s_full = bars + 9;        // [2]
    uint64_t* p_full = bars + 11;       // [2]
    // [2] P V of the even / odd tiles done.  Two, because a row warp may be two products ahead: it can finish the last softmax
    // before the product of the tile before has been issued, and one barrier's parity cannot tell that product from its own
    uint64_t* pv_done = bars + 13;
    uint64_t* q_empty = bars + 15;      // the item's last S product is done
    uint64_t* o_free = bars + 16;       // the 128 row threads have read an item's accumulator
    uint64_t* it_full = bars + 17;      // the next item is known
    uint64_t* it_empty = bars + 18;     // ... has been taken by the five other warps
    uint64_t* claim = bars + 19;        // the answer to a claim has arrived
    int* s_claim = reinterpret_cast<int*>(bars + 20);    // 16 bytes
    int4* s_item = reinterpret_cast<int4*>(bars + 22);   // [2 items][2]
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 30);
    int* status = reinterpret_cast<int*>(bars + 30) + 1;     // of this CTA

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t limit = wait_limit(launch.p[blockIdx.z].status);
    const int G = launch.p[0].G, TPT = launch.p[0].TPT;      // (the same for all problems)
    if (tid == 0) {
        *status = kStatusOk;
        mbar_init(q_full, 1); mbar_init(q_empty, 1); mbar_init(o_free, 128);
        mbar_init(it_full, 1); mbar_init(it_empty, 5); mbar_init(claim, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
            mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
            mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 128);
            mbar_init(&pv_done[i], 1);
        }
        mbar_init_fence();
    }
    if (warp == 0) tmem_alloc(&tmem_slot, kCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tmem_slot;
    // Item n of this CTA.  Each of the five other warps takes every item once, in order; z < 0 ends the list.
    auto read_item = [&](int n) {
        const int4 x = s_item[(n & 1) * 2], y = s_item[(n & 1) * 2 + 1];
        RdItem m;
        m.z = x.x; m.h = x.y; m.seq = x.z; m.tok0 = x.w;
        m.ne = y.x; m.row_lo = y.y; m.nblk = y.z;
        return m;
    };
    auto take_item = [&](int n, bool& ok) {
        ok = ok && mbar_wait(it_full, n & 1, status, limit);
        RdItem m = read_item(n);
        ok = warp_ok(ok);
        if (!ok) m.z = -1;
        if (lane == 0) mbar_arrive(it_empty);
        return m;
    };

    if (warp == 0) {
        // ------------------------------------------------------------------ items and TMA producer
        bool ok = true;
        int n = 0, claims = 0, qi = 0, c = 0;           // items, claims, non-empty items, K/V tiles so far
        int bx = blockIdx.x, h = blockIdx.y, z = blockIdx.z;
        while (ok) {
            const RangeDenseParams& p = launch.p[z];
            bool asked = false;
            auto ask = [&]() {
                mbar_expect_tx(claim, 16);
                claim_next_cta(smem_u32(s_claim), claim);
                asked = true;
            };
            // which tile is this: the heaviest (last) tiles of the list start first
            const int total = count_seq_tiles(p.cu_q, p.B, TPT, lane);
            int seq, tok0, ne;
            find_seq_tile(p.cu_q, p.B, TPT, total - 1 - bx, lane, seq, tok0, ne);
            if (seq >= 0) {
                // lowest and highest K/V row any token of the tile sees
                int lo = INT_MAX, hi = -1;
                const int k0 = __ldg(p.cu_k + seq);
                for (int e = lane; e < ne; e += 32) {
                    const int l = p.kv_lo ? __ldg(p.kv_lo + tok0 + e) : k0;
                    const int u = __ldg(p.kv_hi + tok0 + e);
                    if (u >= l) { lo = min(lo, l); hi = max(hi, u); }
                }
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) {
                    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, d));
                    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, d));
                }
                lo = max(lo, 0);
                hi = min(hi, (int)p.Nk - 1);
                const int nblk = hi >= lo ? (hi - lo) / BK + 1 : 0;
                if (n > 0) ok = ok && mbar_wait(it_empty, (n - 1) & 1, status, limit);
                ok = warp_ok(ok);
                if (ok && lane == 0) {
                    s_item[(n & 1) * 2] = make_int4(z, h, seq, tok0);
                    s_item[(n & 1) * 2 + 1] = make_int4(ne, lo, nblk, 0);
                    mbar_arrive(it_full);
                }
                ++n;
                if (lane == 0 && nblk > 0) {
                    const CUtensorMap *kmap = &launch.k[z], *vmap = &launch.v[z];
                    ok = ok && mbar_wait(q_empty, (qi & 1) ^ 1, status, limit);
                    ask();                  // not earlier: a CTA is to be one item ahead, not to take the share of others
                    if (ok) {
                        mbar_expect_tx(q_full, (uint32_t)(KH * 128 * TPT * G));
#pragma unroll
                        for (int b = 0; b < KH; ++b) tma_load_3d(smem_u32(sQ + b * (kTileRows * 128)), &launch.q[z], b * 64, tok0, h * G, q_full);
                    }
                    // K tile j and V tile j are loaded in the order the MMA warp needs them: K(0), K(1), V(0), K(2), V(1), ...
                    for (int step = 0; step < nblk + 1 && ok; ++step) {
                        const int jk = c + step, jv = jk - 1;
                        if (step < nblk) {
                            const int st = jk & 1;
                            ok = ok && mbar_wait(&k_empty[st], ((jk >> 1) & 1) ^ 1, status, limit);
                            if (!ok) break;
                            mbar_expect_tx(&k_full[st], (uint32_t)kKt);
#pragma unroll
                            for (int b = 0; b < KH; ++b)
                                tma_load_2d(smem_u32(sK + st * kKt + b * (BK * 128)), kmap, h * D + b * 64, lo + step * BK, &k_full[st]);
                        }
                        if (step > 0) {
                            const int st = jv & 1;
                            ok = ok && mbar_wait(&v_empty[st], ((jv >> 1) & 1) ^ 1, status, limit);
                            if (!ok) break;
                            mbar_expect_tx(&v_full[st], (uint32_t)kKt);
#pragma unroll
                            for (int b = 0; b < KH; ++b)
                                tma_load_2d(smem_u32(sV + st * kKt + b * (BK * 128)), vmap, h * D + b * 64, lo + (step - 1) * BK, &v_full[st]);
                        }
                    }
                }
                c += nblk;
                qi += nblk > 0;
            }
            if (lane == 0 && !asked) ask();
            // (the answer is in shared memory before this CTA may end, whatever happened above)
            const bool answered = mbar_wait(claim, claims & 1, status, limit);
            ok = ok && answered;
            ++claims;
            const bool more = claimed_cta(smem_u32(s_claim), bx, h, z);
            ok = warp_ok(ok);
            fence_async_smem();
            if (!more) break;
        }
        if (n > 0) ok = ok && mbar_wait(it_empty, (n - 1) & 1, status, limit);
        ok = warp_ok(ok);
        if (ok && lane == 0) {          // (else the other warps give up by themselves: one may still read this place)
            s_item[(n & 1) * 2] = make_int4(-1, 0, -1, 0);
            s_item[(n & 1) * 2 + 1] = make_int4(0, 0, 0, 0);
            mbar_arrive(it_full);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const bool leader = elect_one();
        constexpr uint32_t idesc_s = umma_idesc(ElemTraits<ET>::kIsBF16, 128, BK, false, false);
        constexpr uint32_t idesc_o = umma_idesc(ElemTraits<ET>::kIsBF16, 128, D, false, true);
        constexpr uint32_t hi_1024 = umma_desc_hi(1024);
        const uint32_t q_lo = umma_desc_lo(smem_u32(sQ), 16);
        const uint32_t k_lo = umma_desc_lo(smem_u32(sK), 16);
        const uint32_t v_lo = umma_desc_lo(smem_u32(sV), BK * 128);     // MN-major: LBO = slab stride
        bool ok = true;
        int n = 0, qi = 0, c = 0;
        // S(t) takes the place of P(t - 2): products of two shapes may run in another order than they were issued, so it waits for the one
        // that reads P(t - 2) (it was issued before the softmax of tile t - 1 began, and is done by the time that this is reached)
        auto issue_s = [&](int t, bool last) {
            const int st = t & 1;
            ok = ok && mbar_wait(&k_full[st], (t >> 1) & 1, status, limit);
            if (t >= 2) ok = ok && mbar_wait(&pv_done[st], ((t - 2) >> 1) & 1, status, limit);
            ok = warp_ok(ok);
            if (!ok) return;
            tc_fence_after();
            if (leader) {
                constexpr int kSlabA = (kTileRows * 128) >> 4, kSlabB = (BK * 128) >> 4;
                const uint32_t b_lo = k_lo + (uint32_t)(st * (kKt >> 4));
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_ss(tbase + cS + st * BK, umma_desc_pack(q_lo + (ks >> 2) * kSlabA + (ks & 3) * 2, hi_1024),
                            umma_desc_pack(b_lo + (ks >> 2) * kSlabB + (ks & 3) * 2, hi_1024), idesc_s, ks > 0);
                umma_commit(&k_empty[st]);
                umma_commit(&s_full[st]);
                if (last) umma_commit(q_empty);
            }
            __syncwarp();
        };
        for (RdItem m = take_item(n, ok); m.z >= 0; m = take_item(++n, ok)) {
            if (m.nblk == 0) continue;
            ok = ok && mbar_wait(q_full, qi & 1, status, limit);
            issue_s(c, m.nblk == 1);
            for (int j = 0; j < m.nblk && ok; ++j, ++c) {
                const int st = c & 1;
                if (j + 1 < m.nblk) issue_s(c + 1, j + 2 == m.nblk);
                if (j == 0 && qi > 0) ok = ok && mbar_wait(o_free, (qi - 1) & 1, status, limit);
                ok = ok && mbar_wait(&p_full[st], (c >> 1) & 1, status, limit);
                ok = ok && mbar_wait(&v_full[st], (c >> 1) & 1, status, limit);
                ok = warp_ok(ok);
                if (!ok) break;
                tc_fence_after();
                if (leader) {
                    const uint32_t b_lo = v_lo + (uint32_t)(st * (kKt >> 4));
#pragma unroll
                    for (int ks = 0; ks < BK / 16; ++ks)
                        umma_ts(tbase + cO, tbase + cS + st * BK + ks * 8, umma_desc_pack(b_lo + ks * (2048 >> 4), hi_1024), idesc_o,
                                (j > 0 || ks > 0) ? 1u : 0u);
                    umma_commit(&v_empty[st]);
                    umma_commit(&pv_done[st]);
                }
                __syncwarp();
            }
            ++qi;
        }
    } else {
        // ------------------------------------------------------------------ softmax and epilogue: one row per thread
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        const int g = r / TPT, e = r - g * TPT;
        bool ok = true;
        int n = 0, c = 0;
        RdItem m = take_item(n, ok);
        int2 sees = rd_row(launch, m, g < G && e < m.ne, e);
        // (the four warps leave the loop together: they meet at barriers in it)
        for (ok = bar_all(1, 128, ok); ok && m.z >= 0;) {
            const float scale_log2 = launch.p[0].scale_log2;                 // (the same for all problems)
            const int lo_r = sees.x - m.row_lo, hi_r = min(sees.y, (int)launch.p[m.z].Nk - 1) - m.row_lo;      // rows past the end of K/V do not exist
            const int nblk = m.nblk;
            float m_ref = -INFINITY, l_run = 0.f;
            for (int j = 0; j < nblk; ++j, ++c) {          // (left by all lanes at the vote below)
                const int st = c & 1;
                const int c_lo = max(0, lo_r - j * BK), c_hi = min(BK, hi_r - j * BK + 1);      // visible columns [c_lo, c_hi)
                ok = ok && mbar_wait(&s_full[st], (c >> 1) & 1, status, limit);
                tc_fence_after();
                uint32_t v[BK];
                tmem_ld32(tbase + lane_off + cS + st * BK, *reinterpret_cast<uint32_t (*)[32]>(&v[0]));
                tmem_ld32(tbase + lane_off + cS + st * BK + 32, *reinterpret_cast<uint32_t (*)[32]>(&v[32]));
                tmem_ld_wait();
                if (c_lo > 0 || c_hi < BK) {
                    // bit i: column i is seen
                    const int v_hi = max(c_hi, 0), v_lo = min(c_lo, BK);
                    const uint64_t vis = v_hi > v_lo ? (~0ull >> (BK - v_hi + v_lo)) << v_lo : 0ull;
                    const uint32_t vis2[2] = {(uint32_t)vis, (uint32_t)(vis >> 32)};
#pragma unroll
                    for (int i = 0; i < BK; ++i)
                        if (!(vis2[i >> 5] >> (i & 31) & 1u)) v[i] = 0xff800000u;      // -inf: exp2 gives exactly 0
                }
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int i = 0; i < BK; i += 4) {
                    mx[0] = fmaxf(mx[0], __uint_as_float(v[i]));
                    mx[1] = fmaxf(mx[1], __uint_as_float(v[i + 1]));
                    mx[2] = fmaxf(mx[2], __uint_as_float(v[i + 2]));
                    mx[3] = fmaxf(mx[3], __uint_as_float(v[i + 3]));
                }
                const float m_blk = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2;
                // raise the reference only when this tile exceeds it by a lot; the first finite maximum sets it
                float alpha = 1.f;
                const bool raise = m_blk > m_ref + kRdLazy;     // false when m_blk is -inf; true when m_ref is -inf and m_blk finite
                if (raise) {
                    alpha = m_ref == -INFINITY ? 0.f : rd_ex2(m_ref - m_blk);
                    m_ref = m_blk;
                }
                // accumulator rows already hold products (j > 0): rescale them when any row of the warp changes reference
                const bool scale_acc = __any_sync(0xffffffffu, (raise && j > 0) || !ok);
                if (scale_acc) {
                    ok = ok && mbar_wait(&pv_done[(c - 1) & 1], ((c - 1) >> 1) & 1, status, limit);
                    if (!warp_stays(ok)) break;
                    tc_fence_after();
#pragma unroll
                    for (int c0 = 0; c0 < D; c0 += 32) {
                        uint32_t a[32];
                        tmem_ld32(tbase + lane_off + cO + c0, a);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) * alpha);
                        tmem_st32(tbase + lane_off + cO + c0, a);
                    }
                }
                l_run *= alpha;
                const float m_use = m_ref == -INFINITY ? 0.f : m_ref;     // all columns masked so far: every p is exp2(-inf) = 0
                float ls[4] = {0.f, 0.f, 0.f, 0.f};
                uint32_t pk[BK / 2];
#pragma unroll
                for (int i = 0; i < BK; i += 4) {
                    const float p0 = rd_ex2(fmaf(__uint_as_float(v[i]), scale_log2, -m_use));
                    const float p1 = rd_ex2(fmaf(__uint_as_float(v[i + 1]), scale_log2, -m_use));
                    const float p2 = rd_ex2(fmaf(__uint_as_float(v[i + 2]), scale_log2, -m_use));
                    const float p3 = rd_ex2(fmaf(__uint_as_float(v[i + 3]), scale_log2, -m_use));
                    ls[0] += p0; ls[1] += p1; ls[2] += p2; ls[3] += p3;
                    pk[i >> 1] = ElemTraits<ET>::pack2(p0, p1);
                    pk[(i >> 1) + 1] = ElemTraits<ET>::pack2(p2, p3);
                }
                l_run += (ls[0] + ls[1]) + (ls[2] + ls[3]);
                tmem_st32(tbase + lane_off + cS + st * BK, *reinterpret_cast<uint32_t (*)[32]>(&pk[0]));
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&p_full[st]);
            }
            m = read_item(n);
            const RangeDenseParams& p = launch.p[m.z];
            const bool row_valid = g < G && e < m.ne;
            const int tok = m.tok0 + e;
            // the next item's numbers arrive under this item's epilogue
            const RdItem next = take_item(++n, ok);
            sees = rd_row(launch, next, g < G && e < next.ne, e);
            // ---- epilogue
            if (m.nblk > 0) {
                ok = ok && mbar_wait(&pv_done[(c - 1) & 1], ((c - 1) >> 1) & 1, status, limit);
                tc_fence_after();
            }
            ok = bar_all(1, 128, ok);
            const float inv_l = l_run > 0.f ? 1.f / l_run : 0.f;
            if (row_valid && ok) p.lse[(int64_t)(m.h * G + g) * p.N + tok] = l_run > 0.f ? m_ref + log2f(l_run) : -INFINITY;
            const bool full_tile = m.ne == TPT && G * TPT == kTileRows;      // whole box inside the sequence, every row staged
            ET* orow = reinterpret_cast<ET*>(p.o) + (int64_t)tok * p.o_sn + (int64_t)(m.h * G + g) * p.o_sh;
#pragma unroll
            for (int c0 = 0; c0 < D; c0 += 32) {
                uint32_t a[32];
                if (m.nblk > 0) {
                    tmem_ld32(tbase + lane_off + cO + c0, a);
                    tmem_ld_wait();
                    if (c0 + 32 == D) {
                        tc_fence_before();
                        mbar_arrive(o_free);            // the accumulator may take the next item
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) a[i] = 0u;
                }
                if (full_tile && c0 % 64 == 0) {        // the columns before have left the staging memory
                    if (quarter == 0 && lane == 0) bulk_wait_read0();
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                }
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4) {
                    uint4 x;
                    x.x = ElemTraits<ET>::pack2(__uint_as_float(a[q4 * 8 + 0]) * inv_l, __uint_as_float(a[q4 * 8 + 1]) * inv_l);
                    x.y = ElemTraits<ET>::pack2(__uint_as_float(a[q4 * 8 + 2]) * inv_l, __uint_as_float(a[q4 * 8 + 3]) * inv_l);
                    x.z = ElemTraits<ET>::pack2(__uint_as_float(a[q4 * 8 + 4]) * inv_l, __uint_as_float(a[q4 * 8 + 5]) * inv_l);
                    x.w = ElemTraits<ET>::pack2(__uint_as_float(a[q4 * 8 + 6]) * inv_l, __uint_as_float(a[q4 * 8 + 7]) * inv_l);
                    if (full_tile) *reinterpret_cast<uint4*>(sOut + sw128_chunk_off(r, (c0 % 64) / 8 + q4)) = x;
                    else if (row_valid && ok) *reinterpret_cast<uint4*>(orow + c0 + q4 * 8) = x;
                }
                if (full_tile && c0 % 64 == 32) {
                    // all four warps have staged their rows: one 3-D store of 64 columns
                    fence_async_smem();
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (quarter == 0 && lane == 0) {
                        if (ok) tma_store_3d(&launch.o[m.z], c0 - 32, m.tok0, m.h * G, smem_u32(sOut));
                        bulk_commit();
                    }
                }
            }
            m = next;
        }
        if (quarter == 0 && lane == 0) bulk_wait_read0();      // the last columns have left shared memory
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, kCols);
    // (a CTA has taken over items of every problem of the launch, and gave up those that it would have taken)
    if (tid < kRdProblems && *status != kStatusOk && launch.p[tid].status) atomicMax(launch.p[tid].status, *status);
}

template <int D, typename ET>
static cudaError_t launch_rd(const RangeDenseLaunch& l, int num, int max_tiles, cudaStream_t stream) {
    constexpr int smem = kTileRows * D * 2 + 4 * kRdBK * D * 2 + kTileRows * 128 + 256;
    auto kern = range_fwd_dense<D, ET>;
    cudaError_t e = allow_smem((const void*)kern, smem);
    if (e != cudaSuccess) return e;
    prof_begin(FSA_KERNEL_RANGE_DENSE, stream);
    kern<<<dim3((unsigned)max_tiles, (unsigned)l.p[0].Hk, (unsigned)num), kRdThreads, smem, stream>>>(l);
    prof_end(FSA_KERNEL_RANGE_DENSE, stream);
    return cudaGetLastError();
}


// ------------------------------------------------------------------------------------------------ dQ, query-tile-major
// dQ of range attention with the same tiling as the forward above: per K/V tile S = Q K^T and dP = dO V^T, then
// P = exp2(S c - lse), dS = scale P (dP - delta), dQ (+)= dS K accumulated in TMEM over the tiles and written once.  (In the reference: the dQ part of _backward_kernel, nsa_ref/ops/compressed_attention.py:
// 193-760, and of flash-attn's backward for the sliding window.)  With it the block-major backward kernel computes
// only dK and dV and no partial dQ row is written or merged.  One CTA per SM, 384 threads:
//   warp 0      TMA producer: Q and dO tiles of every item, (K, V) tiles through a four-stage ring (a stage comes free only
//               when the tile's dQ product is done, and the next load needs a microsecond to land);
//   warp 1      one elected thread issues S and dP (two TMEM buffers: they run a tile ahead of the row threads);
//   warp 10     one elected thread issues dQ (a second issuer: see the MMA section);
//   warp 11     finds the items, up to four ahead (the search and its loads take ~3700 cycles, three tiles' worth);
//   warps 2..9  two groups of 128 row threads: Q (group 0) and dO (group 1) of the next item to TMEM when the item's S / dP are
//               done; 32 of the 64 key columns each, dS over dP; epilogue: each group rounds 64 of the dQ columns, stages them
//               and stores its slab by 3-D TMA (plain stores for the last, partial tile of a sequence).
// The left operand of every product (Q, dO, dS) comes from TMEM, so a tile of 64 keys takes three reads of 16 KB from shared
// memory.  With all of them in shared memory it was 128 KB and the writes of dS, twice the cycles that the products take.
// Measured at 2 x 32768 tokens, 32 / 8 heads (window of 512 and compressed branch together): operands in shared memory, items
// found by every warp for itself 3.49 ms; operands in TMEM 2.92; items by a warp of their own and row numbers an item ahead 2.77
// (6.4 thousand cycles between two items before, ten tiles of 1190).  A tile is now bound by its row threads (700 cycles) in
// turn with the S / dP products, which two TMEM buffers let run one tile ahead; the products alone take 770.
struct RangeDqParams {
    const int32_t* cu_q;
    const int32_t* cu_k;
    const int32_t* kv_lo;
    const int32_t* kv_hi;
    int64_t N, Nk;
    int B, Hq, Hk, G, TPT;
    float scale, scale_log2;
    const float* lse;       // [Hq, N] log2 units
    const float* delta;     // [Hq, N] sum_d o dO
    void* dq;               // [N, Hq, D] contiguous
    int* status;
};

constexpr int kDqThreads = 384;     // producer, S/dP issuer, 8 row warps, dQ issuer, item warp
constexpr int kDqStages = 4;
constexpr int kDqItems = 4;         // items known ahead
// The item warp is ahead, so that its wait for a free entry lasts as long as an item: a tile of 64 K/V rows takes some 1200 cycles, and
// 0.2 s would end it at 21 million rows.  This many cycles more for each tile of the longest item so far.
constexpr uint32_t kDqTileClocks = 4096;
static_assert(kMaxTokens / kRdBK * kDqTileClocks + FSA_WAIT_CLOCKS < (int64_t)1 << 32, "the counter comes round");

// One work item of the dQ kernel: a tile of tokens x one KV head.
struct DqItem {
    int seq, tok0, ne, row_lo, nblk, h;
};

// Work item w of the list (heaviest tiles first).  Warp-collective: all 32 lanes call it and get the same answer.
__device__ __forceinline__ DqItem dq_item(const RangeDqParams& p, int ntiles, int w, int lane) {
    DqItem m;
    m.h = w % p.Hk;
    const int want = ntiles - 1 - w / p.Hk;
    m.row_lo = 0; m.nblk = 0;
    find_seq_tile(p.cu_q, p.B, p.TPT, want, lane, m.seq, m.tok0, m.ne);
    if (m.seq < 0) return m;
    int lo = INT_MAX, hi = -1;
    const int k0 = __ldg(p.cu_k + m.seq);
    for (int e = lane; e < m.ne; e += 32) {
        const int l = p.kv_lo ? __ldg(p.kv_lo + m.tok0 + e) : k0;
        const int u = __ldg(p.kv_hi + m.tok0 + e);
        if (u >= l) { lo = min(lo, l); hi = max(hi, u); }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, d));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, d));
    }
    lo = max(lo, 0);
    hi = min(hi, (int)p.Nk - 1);
    m.row_lo = lo;
    m.nblk = hi >= lo ? (hi - lo) / kRdBK + 1 : 0;
    return m;
}

template <typename ET>
__global__ void __launch_bounds__(kDqThreads, 1) range_bwd_dq_dense(const RangeDqParams p, const __grid_constant__ CUtensorMap qmap,
                                                                   const __grid_constant__ CUtensorMap domap,
                                                                   const __grid_constant__ CUtensorMap kmap,
                                                                   const __grid_constant__ CUtensorMap vmap,
                                                                   const __grid_constant__ CUtensorMap dqmap) {
    constexpr int D = 128, BK = kRdBK, KH = D / 64;
    constexpr int kQ = kTileRows * D * 2;            // Q tile, same for dO
    constexpr int kKt = BK * D * 2;
    constexpr int kOut = kTileRows * 128;            // 64 columns of the dQ tile on their way out
    constexpr uint32_t kCols = 512;
    constexpr int cDQ = 256, cQ = 384, cDO = 448;    // S(b) at 128 b, dP(b) / dS(b) at 128 b + 64; Q and dO two values a column
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;
    uint8_t* sDO = sQ + kQ;
    uint8_t* sKV = sDO + kQ;                         // stage: K then V
    uint8_t* sOut = sKV + kDqStages * 2 * kKt;       // two slabs
    uint64_t* bars = reinterpret_cast<uint64_t*>(sOut + 2 * kOut);
    uint64_t* qd_full = bars;           // Q and dO tiles of an item have landed
    uint64_t* qd_empty = bars + 1;      // ... have been read by the 256 row threads
    uint64_t* kv_full = bars + 2;                        // [stages]
    uint64_t* kv_empty = kv_full + kDqStages;            // [stages] the dQ product of the tile is done
    uint64_t* sdp_full = kv_empty + kDqStages;           // [2]
    uint64_t* sdp_free = sdp_full + 2;                   // [2] the 256 row threads have read S and dP
    uint64_t* ds_full = sdp_free + 2;                    // [2] ... have written dS over dP
    uint64_t* ds_empty = ds_full + 2;                    // [2] the dQ product has read dS
    uint64_t* dq_free = ds_empty + 2;                    // the 256 row threads have read an item's dQ accumulator
    uint64_t* qt_full = dq_free + 1;                     // ... have written an item's Q and dO to TMEM
    uint64_t* it_full = qt_full + 1;                     // [items]
    uint64_t* it_empty = it_full + kDqItems;             // [items] the eleven other warps have read the entry
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(it_empty + kDqItems);
    int4* s_item = reinterpret_cast<int4*>(bars + 32);   // [items][2]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int* status = p.status;
    if (tid == 0) {
        mbar_init(qd_full, 1); mbar_init(qd_empty, 256);
        for (int i = 0; i < kDqStages; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sdp_full[i], 1); mbar_init(&sdp_free[i], 256);
            mbar_init(&ds_full[i], 256); mbar_init(&ds_empty[i], 1);
        }
        for (int i = 0; i < kDqItems; ++i) { mbar_init(&it_full[i], 1); mbar_init(&it_empty[i], kDqThreads / 32 - 1); }
        mbar_init(dq_free, 256); mbar_init(qt_full, 256);
        mbar_init_fence();
        tma_prefetch_desc(&qmap);
        tma_prefetch_desc(&domap);
        tma_prefetch_desc(&kmap);
        tma_prefetch_desc(&vmap);
        tma_prefetch_desc(&dqmap);
    }
    if (warp == 0) tmem_alloc(&tmem_slot, kCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tmem_slot;
    const int ntiles = count_seq_tiles(p.cu_q, p.B, p.TPT, lane);
    const int nitems = ntiles * p.Hk;
    // Entry n of this CTA's items: every warp but the one that fills the ring takes each of them once, in order.
    auto take_item = [&](int n, bool& ok) {
        ok = ok && mbar_wait(&it_full[n % kDqItems], (n / kDqItems) & 1, status);
        const int4 x = s_item[(n % kDqItems) * 2], y = s_item[(n % kDqItems) * 2 + 1];
        ok = warp_ok(ok);
        if (lane == 0) mbar_arrive(&it_empty[n % kDqItems]);
        DqItem m;
        m.seq = x.x; m.tok0 = x.y; m.ne = x.z; m.row_lo = x.w; m.nblk = y.x; m.h = y.y;
        if (!ok) m.ne = m.nblk = 0;
        return m;
    };

    if (warp == kDqThreads / 32 - 1) {
        // ------------------------------------------------------------------ items
        bool ok = true;
        int n = 0, longest = 0;
        for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x, ++n) {
            const DqItem m = dq_item(p, ntiles, w, lane);
            ok = ok && mbar_wait(&it_empty[n % kDqItems], ((n / kDqItems) & 1) ^ 1, status, FSA_WAIT_CLOCKS + longest * kDqTileClocks);
            ok = warp_ok(ok);
            longest = max(longest, m.nblk);
            if (ok && lane == 0) {
                s_item[(n % kDqItems) * 2] = make_int4(m.seq, m.tok0, m.ne, m.row_lo);
                s_item[(n % kDqItems) * 2 + 1] = make_int4(m.nblk, m.h, 0, 0);
                mbar_arrive(&it_full[n % kDqItems]);
            }
        }
    } else if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        bool ok = true;
        int kvc = 0, qi = 0, n = 0;    // K/V tiles and non-empty items so far
        for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x, ++n) {
            const DqItem m = take_item(n, ok);
            if (m.nblk == 0) continue;
            if (lane == 0) {
                ok = ok && mbar_wait(qd_empty, (qi & 1) ^ 1, status);
                if (ok) {
                    mbar_expect_tx(qd_full, (uint32_t)(2 * KH * 128 * p.TPT * p.G));
#pragma unroll
                    for (int b = 0; b < KH; ++b) {
                        tma_load_3d(smem_u32(sQ + b * (kTileRows * 128)), &qmap, b * 64, m.tok0, m.h * p.G, qd_full);
                        tma_load_3d(smem_u32(sDO + b * (kTileRows * 128)), &domap, b * 64, m.tok0, m.h * p.G, qd_full);
                    }
                }
            }
            ++qi;
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            for (int j = 0; j < m.nblk && ok; ++j, ++kvc) {
                if (lane == 0) {
                    const int st = kvc % kDqStages;
                    ok = ok && mbar_wait(&kv_empty[st], ((kvc / kDqStages) & 1) ^ 1, status);
                    if (ok) {
                        mbar_expect_tx(&kv_full[st], (uint32_t)(2 * kKt));
                        uint8_t* dK = sKV + st * 2 * kKt;
                        uint8_t* dV = dK + kKt;
#pragma unroll
                        for (int b = 0; b < KH; ++b) {
                            tma_load_2d(smem_u32(dK + b * (BK * 128)), &kmap, m.h * D + b * 64, m.row_lo + j * BK, &kv_full[st]);
                            tma_load_2d(smem_u32(dV + b * (BK * 128)), &vmap, m.h * D + b * 64, m.row_lo + j * BK, &kv_full[st]);
                        }
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            }
        }
    } else if (warp == 1 || warp == kDqThreads / 32 - 2) {
        // ------------------------------------------------------------------ MMA issuers
        // Two warps: a single issuing thread waits on barriers between products; with dQ on a warp of its own its chain overlaps
        // the S / dP chains of the next tile (measured: 20 % faster).  Warp 1 issues S and dP, warp 10 dQ.  The K/V tiles of all
        // items form one sequence c = 0, 1, ...; S / dP run ahead of dQ as far as their two TMEM buffers and the K/V ring allow,
        // also across the boundary between two items (the next item's Q / dO replace this item's when its last S / dP are done).
        const bool leader = elect_one();
        constexpr uint32_t idesc_s = umma_idesc(ElemTraits<ET>::kIsBF16, 128, BK, false, false);
        constexpr uint32_t idesc_dq = umma_idesc(ElemTraits<ET>::kIsBF16, 128, D, false, true);     // dS (K-major) x K (MN-major)
        constexpr uint32_t hi_1024 = umma_desc_hi(1024);
        constexpr int kSlabB = (BK * 128) >> 4;
        const uint32_t kv_lo_ = umma_desc_lo(smem_u32(sKV), 16);
        const uint32_t k_mn_lo = umma_desc_lo(smem_u32(sKV), BK * 128);
        bool ok = true;
        int c = 0, qi = 0, n = 0;
        for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x, ++n) {
            const DqItem m = take_item(n, ok);
            if (m.nblk == 0) continue;
            if (warp == 1) {
                ok = ok && mbar_wait(qt_full, qi & 1, status);
                ok = warp_ok(ok);
                for (int j = 0; j < m.nblk && ok; ++j, ++c) {
                    const int b = c & 1, st = c % kDqStages;
                    const uint32_t k_lo = kv_lo_ + (uint32_t)(st * ((2 * kKt) >> 4));
                    const uint32_t v_lo = k_lo + (uint32_t)(kKt >> 4);
                    ok = ok && mbar_wait(&kv_full[st], (c / kDqStages) & 1, status);
                    ok = ok && mbar_wait(&sdp_free[b], ((c >> 1) & 1) ^ 1, status);     // S / dP of tile c - 2 have been read
                    ok = warp_ok(ok);
                    if (!ok) break;
                    tc_fence_after();
                    if (leader) {
#pragma unroll
                        for (int ks = 0; ks < D / 16; ++ks)
                            umma_ts(tbase + b * 128, tbase + cQ + ks * 8, umma_desc_pack(k_lo + (ks >> 2) * kSlabB + (ks & 3) * 2, hi_1024),
                                    idesc_s, ks > 0);
                    }
                    __syncwarp();
                    ok = ok && mbar_wait(&ds_empty[b], ((c >> 1) & 1) ^ 1, status);     // the dQ product of tile c - 2 has read dS
                    ok = warp_ok(ok);
                    if (!ok) break;
                    tc_fence_after();
                    if (leader) {
#pragma unroll
                        for (int ks = 0; ks < D / 16; ++ks)
                            umma_ts(tbase + b * 128 + BK, tbase + cDO + ks * 8, umma_desc_pack(v_lo + (ks >> 2) * kSlabB + (ks & 3) * 2, hi_1024),
                                    idesc_s, ks > 0);
                        umma_commit(&sdp_full[b]);
                    }
                    __syncwarp();
                }
            } else {
                for (int j = 0; j < m.nblk && ok; ++j, ++c) {
                    const int b = c & 1, st = c % kDqStages;
                    ok = ok && mbar_wait(&ds_full[b], (c >> 1) & 1, status);      // (implies S / dP of the tile are done with K and V)
                    if (j == 0 && qi > 0) ok = ok && mbar_wait(dq_free, (qi - 1) & 1, status);     // the previous item's dQ has been read
                    ok = warp_ok(ok);
                    if (!ok) break;
                    tc_fence_after();
                    if (leader) {
                        const uint32_t b_lo = k_mn_lo + (uint32_t)(st * ((2 * kKt) >> 4));
#pragma unroll
                        for (int ks = 0; ks < BK / 16; ++ks)      // the two row groups keep their halves 32 columns apart
                            umma_ts(tbase + cDQ, tbase + b * 128 + BK + (ks >> 1) * 32 + (ks & 1) * 8,
                                    umma_desc_pack(b_lo + ks * (2048 >> 4), hi_1024), idesc_dq, (j > 0 || ks > 0) ? 1u : 0u);
                        umma_commit(&kv_empty[st]);
                        umma_commit(&ds_empty[b]);
                    }
                    __syncwarp();
                }
            }
            ++qi;
        }
    } else {
        // ------------------------------------------------------------------ dS and the epilogue: one row, half the columns
        const int sb = (warp - 2) >> 2;               // column half of this group
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        const int g = r / p.TPT, e = r - g * p.TPT;
        constexpr int HC = BK / 2;
        const int cb = sb * HC;
        bool ok = true;
        int c = 0, qi = 0;
        // One row of an item's Q (group 0) or dO (group 1) to TMEM.  Not before the last S / dP products of the item before are done.
        auto take_row = [&]() {
            ok = ok && mbar_wait(qd_full, qi & 1, status);
            ++qi;
            const uint8_t* src = sb ? sDO : sQ;
            uint32_t x[2][32];
#pragma unroll
            for (int i = 0; i < D / 8; ++i)
                *reinterpret_cast<uint4*>(&x[i >> 3][(i & 7) * 4]) = *reinterpret_cast<const uint4*>(src + (i >> 3) * (kTileRows * 128) + sw128_chunk_off(r, i & 7));
            tmem_st32(tbase + lane_off + (sb ? cDO : cQ), x[0]);
            tmem_st32(tbase + lane_off + (sb ? cDO : cQ) + 32, x[1]);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(qd_empty);
            mbar_arrive(qt_full);
        };
        // This row's numbers, loaded an item ahead: item numbers and loads of their own between two items were a third of the kernel.
        struct Row { int lo, hi; float lse, delta; };
        auto load_numbers = [&](const DqItem& m) {
            Row x = {0, -1, 0.f, 0.f};
            if (g < p.G && e < m.ne) {
                x.lo = p.kv_lo ? __ldg(p.kv_lo + m.tok0 + e) : __ldg(p.cu_k + m.seq);
                x.hi = __ldg(p.kv_hi + m.tok0 + e);
                const int64_t idx = (int64_t)(m.h * p.G + g) * p.N + m.tok0 + e;
                x.lse = __ldg(p.lse + idx);
                x.delta = __ldg(p.delta + idx);
            }
            return x;
        };
        DqItem m;
        m.nblk = m.ne = 0;
        int n = 0;
        if ((int)blockIdx.x < nitems) {
            m = take_item(n, ok);
            if (m.nblk > 0) take_row();
        }
        Row row = load_numbers(m);
        ok = bar_all(3, 256, ok);       // (the eight warps enter the loop together: they meet at barriers in it)
        for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
            const bool row_valid = g < p.G && e < m.ne;
            const int tok = m.tok0 + e;
            const int lo_r = row.lo;
            const float lse_r = row.lse, delta_s = row.delta * p.scale;
            int hi_r = min(row.hi, (int)p.Nk - 1);              // rows past the end of K/V do not exist
            if (!(lse_r > -INFINITY)) hi_r = lo_r - 1;          // a row that saw nothing in the forward sees nothing here
            DqItem next;
            next.nblk = next.ne = 0;
            if (w + (int)gridDim.x < nitems) next = take_item(++n, ok);
            row = load_numbers(next);
            for (int j = 0; j < m.nblk; ++j, ++c) {        // (left by all lanes at the vote below)
                const int b = c & 1;
                const int R0 = m.row_lo + j * BK;
                const int c_lo = max(0, lo_r - R0), c_hi = min(BK, hi_r - R0 + 1);
                ok = ok && mbar_wait(&sdp_full[b], (c >> 1) & 1, status);
                tc_fence_after();
                uint32_t dd[HC / 2];
                const bool all_visible = __all_sync(0xffffffffu, ok && c_lo == 0 && c_hi == BK);
                if (!all_visible && !warp_stays(ok)) break;
                {
                    uint32_t sv[32], dv[32];
                    tmem_ld32(tbase + lane_off + b * 128 + cb, sv);
                    tmem_ld32(tbase + lane_off + b * 128 + BK + cb, dv);
                    tmem_ld_wait();
                    tc_fence_before();
                    mbar_arrive(&sdp_free[b]);       // both rows are in registers: the buffer may take tile c + 2
                    if (j + 1 == m.nblk && next.nblk > 0) take_row();      // the next item's S / dP run under this item's end
                    if (all_visible) {
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const float p0 = rd_ex2(fmaf(__uint_as_float(sv[i]), p.scale_log2, -lse_r));
                            const float p1 = rd_ex2(fmaf(__uint_as_float(sv[i + 1]), p.scale_log2, -lse_r));
                            dd[i >> 1] = ElemTraits<ET>::pack2(p0 * fmaf(__uint_as_float(dv[i]), p.scale, -delta_s),
                                                               p1 * fmaf(__uint_as_float(dv[i + 1]), p.scale, -delta_s));
                        }
                    } else {
                        // bit i: column cb + i is seen
                        const int v_lo = min(max(c_lo - cb, 0), HC), v_hi = min(max(c_hi - cb, 0), HC);
                        const uint32_t vis = v_hi > v_lo ? (0xffffffffu >> (HC - v_hi + v_lo)) << v_lo : 0u;
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const float p0 = rd_ex2(fmaf(__uint_as_float(sv[i]), p.scale_log2, -lse_r));
                            const float p1 = rd_ex2(fmaf(__uint_as_float(sv[i + 1]), p.scale_log2, -lse_r));
                            const float d0 = (vis >> i & 1u) && p0 > 0.f ? p0 * fmaf(__uint_as_float(dv[i]), p.scale, -delta_s) : 0.f;
                            const float d1 = (vis >> (i + 1) & 1u) && p1 > 0.f ? p1 * fmaf(__uint_as_float(dv[i + 1]), p.scale, -delta_s) : 0.f;
                            dd[i >> 1] = ElemTraits<ET>::pack2(d0, d1);
                        }
                    }
                }
                tmem_st16(tbase + lane_off + b * 128 + BK + cb, dd);
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&ds_full[b]);
            }
            if (m.nblk == 0 && next.nblk > 0) take_row();
            // ---- epilogue of the item: this group's 64 of the 128 dQ columns
            const bool full_tile = m.ne == p.TPT && p.G * p.TPT == kTileRows && m.nblk > 0;
            if (m.nblk > 0) {
                ok = ok && mbar_wait(&ds_empty[(c - 1) & 1], ((c - 1) >> 1) & 1, status);      // the item's last dQ product is done
                tc_fence_after();
            }
            ET* drow = reinterpret_cast<ET*>(p.dq) + ((int64_t)tok * p.Hq + (m.h * p.G + g)) * D + sb * 64;
            uint8_t* stage = sOut + sb * kOut;
            // the slab of the item before has left its place; and the four warps go on, or give up, together
            if (quarter == 0 && lane == 0) bulk_wait_read0();
            ok = bar_all(1 + sb, 128, ok);
#pragma unroll
            for (int c0 = 0; c0 < 64; c0 += 32) {
                uint32_t a[32];
                if (m.nblk > 0) {
                    tmem_ld32(tbase + lane_off + cDQ + sb * 64 + c0, a);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) a[i] = 0u;
                }
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4) {
                    uint4 x;
                    x.x = ElemTraits<ET>::pack2(__uint_as_float(a[q4 * 8 + 0]), __uint_as_float(a[q4 * 8 + 1]));
                    x.y = ElemTraits<ET>::pack2(__uint_as_float(a[q4 * 8 + 2]), __uint_as_float(a[q4 * 8 + 3]));
                    x.z = ElemTraits<ET>::pack2(__uint_as_float(a[q4 * 8 + 4]), __uint_as_float(a[q4 * 8 + 5]));
                    x.w = ElemTraits<ET>::pack2(__uint_as_float(a[q4 * 8 + 6]), __uint_as_float(a[q4 * 8 + 7]));
                    const int chunk = (c0 >> 3) + q4;       // 16-byte chunk inside this group's 128-byte half row
                    if (full_tile) {
                        *reinterpret_cast<uint4*>(stage + sw128_chunk_off(r, chunk)) = x;
                    } else if (row_valid && ok) {
                        *reinterpret_cast<uint4*>(drow + chunk * 8) = x;
                    }
                }
            }
            if (m.nblk > 0) {
                tc_fence_before();
                mbar_arrive(dq_free);            // the accumulator may take the next item
            }
            if (full_tile) {
                fence_async_smem();
                if (sb == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
                else asm volatile("bar.sync 2, 128;" ::: "memory");
                if (quarter == 0 && lane == 0) {
                    if (ok) tma_store_3d(&dqmap, sb * 64, m.tok0, m.h * p.G, smem_u32(stage));
                    bulk_commit();
                }
            }
            m = next;
        }
        if (quarter == 0 && lane == 0) bulk_wait_read0();      // the last slab has left shared memory
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, kCols);
}

// dQ of a range-attention backward (head_dim 128).  q / dO strided, dq contiguous [N, Hq, 128].
cudaError_t launch_range_bwd_dq(int dtype, const SelBwdArgs& a, const SelShape& s, const CUtensorMap& kmap, const CUtensorMap& vmap,
                                int* status, cudaStream_t stream) {
    CUtensorMap qmap, domap, dqmap;
    if (make_tile_map_3d_box(&qmap, a.q, dtype, 128, s.N, s.Hq, a.q_sn, a.q_sh, s.TPT, s.G)) return cudaErrorInvalidValue;
    if (make_tile_map_3d_box(&domap, a.d_o, dtype, 128, s.N, s.Hq, a.do_sn, a.do_sh, s.TPT, s.G)) return cudaErrorInvalidValue;
    if (make_tile_map_3d_box(&dqmap, a.dq, dtype, 128, s.N, s.Hq, (int64_t)s.Hq * 128, 128, s.TPT, s.G)) return cudaErrorInvalidValue;
    RangeDqParams p;
    p.cu_q = a.cu; p.cu_k = a.bd.cu_k ? a.bd.cu_k : a.cu; p.kv_lo = a.bd.kv_lo; p.kv_hi = a.bd.kv_hi;
    p.N = s.N; p.Nk = s.Nk; p.B = s.B; p.Hq = s.Hq; p.Hk = s.Hk; p.G = s.G; p.TPT = s.TPT;
    p.scale = a.sm_scale; p.scale_log2 = a.sm_scale * 1.4426950408889634f;
    p.lse = a.lse; p.delta = a.delta; p.dq = a.dq; p.status = status;
    constexpr int smem = 2 * kTileRows * 128 * 2 + kDqStages * 2 * kRdBK * 128 * 2 + 2 * kTileRows * kRdBK * 2 + 256 + kDqItems * 32;
    const int64_t max_items = ((s.N + s.TPT - 1) / s.TPT + s.B) * (int64_t)s.Hk;
    int sms = 0;
    if (device_sm_count(&sms) != 0 || sms <= 0) return cudaErrorInvalidValue;
    const unsigned grid = (unsigned)(max_items < sms ? max_items : sms);
    cudaError_t e;
    if (dtype == kBF16) {
        auto kern = range_bwd_dq_dense<__nv_bfloat16>;
        e = allow_smem((const void*)kern, smem);
        if (e != cudaSuccess) return e;
        prof_begin(FSA_KERNEL_SEL_BWD_DQ_REDUCE, stream);
        kern<<<grid, kDqThreads, smem, stream>>>(p, qmap, domap, kmap, vmap, dqmap);
        prof_end(FSA_KERNEL_SEL_BWD_DQ_REDUCE, stream);
    } else {
        auto kern = range_bwd_dq_dense<__half>;
        e = allow_smem((const void*)kern, smem);
        if (e != cudaSuccess) return e;
        prof_begin(FSA_KERNEL_SEL_BWD_DQ_REDUCE, stream);
        kern<<<grid, kDqThreads, smem, stream>>>(p, qmap, domap, kmap, vmap, dqmap);
        prof_end(FSA_KERNEL_SEL_BWD_DQ_REDUCE, stream);
    }
    return cudaGetLastError();
}

}  // namespace fsa

using namespace fsa;

extern "C" int fsa_range_attn_fwd_dense_several(int num, const fsa_range_problem* problems, int B, int Hq, int Hk, int D, int dtype, float sm_scale,
                                                void* stream_) {
    if (num <= 0 || !problems || B < 0 || Hq <= 0 || Hk <= 0 || Hq % Hk != 0) return FSA_ERR_BAD_ARG;
    if (dtype != FSA_DTYPE_BF16 && dtype != FSA_DTYPE_FP16) return FSA_ERR_BAD_ARG;
    const int G = Hq / Hk;
    for (int i = 0; i < num; ++i)
        if (problems[i].N < 0 || problems[i].Nk < 0) return FSA_ERR_BAD_ARG;
    if ((D != 64 && D != 128) || G > 32 || num > kRdProblems) return FSA_ERR_UNSUPPORTED;
    if (!(sm_scale > 0.f)) return FSA_ERR_BAD_ARG;
    const int TPT = (kTileRows / G) & ~3;
    RangeDenseLaunch l = {};
    int used = 0, max_tiles = 0, rc;
    for (int i = 0; i < num; ++i) {
        const fsa_range_problem& a = problems[i];
        if (a.N == 0 || B == 0) continue;
        if (!a.q || !a.k || !a.v || !a.cu_seqlens_q || !a.cu_seqlens_k || !a.kv_hi || !a.o || !a.lse || a.Nk == 0) return FSA_ERR_BAD_ARG;
        if (((uintptr_t)a.q & 15) || ((uintptr_t)a.k & 15) || ((uintptr_t)a.v & 15) || ((uintptr_t)a.o & 15)) return FSA_ERR_BAD_ARG;
        if ((a.q_stride_n % 8) || (a.q_stride_h % 8) || (a.k_stride_n % 8) || (a.v_stride_n % 8) || (a.o_stride_n % 8) || (a.o_stride_h % 8))
            return FSA_ERR_BAD_ARG;
        if (a.k_stride_n < (int64_t)Hk * D || a.v_stride_n < (int64_t)Hk * D) return FSA_ERR_BAD_ARG;
        if (used == 0) {
            (void)cudaGetLastError();
            if ((rc = ensure_context())) return rc;
        }
        if ((rc = make_tile_map_3d_box(&l.q[used], a.q, dtype, D, a.N, Hq, a.q_stride_n, a.q_stride_h, TPT, G))) return rc;
        if ((rc = make_tile_map_3d_box(&l.o[used], a.o, dtype, D, a.N, Hq, a.o_stride_n, a.o_stride_h, TPT, G))) return rc;
        if ((rc = make_tile_map(&l.k[used], a.k, dtype, a.Nk, (int64_t)Hk * D, a.k_stride_n, 64))) return rc;
        if ((rc = make_tile_map(&l.v[used], a.v, dtype, a.Nk, (int64_t)Hk * D, a.v_stride_n, 64))) return rc;
        RangeDenseParams& p = l.p[used++];
        p.cu_q = a.cu_seqlens_q; p.cu_k = a.cu_seqlens_k; p.kv_lo = a.kv_lo; p.kv_hi = a.kv_hi;
        p.N = a.N; p.Nk = a.Nk; p.B = B; p.Hq = Hq; p.Hk = Hk; p.G = G; p.TPT = TPT;
        p.scale_log2 = sm_scale * 1.4426950408889634f;
        p.o = a.o; p.o_sn = a.o_stride_n; p.o_sh = a.o_stride_h; p.lse = a.lse; p.status = a.status;
        const int tiles = (int)((a.N + TPT - 1) / TPT) + B;
        if (tiles > max_tiles) max_tiles = tiles;
    }
    if (used == 0) return FSA_OK;
    cudaStream_t stream = (cudaStream_t)stream_;
    const cudaError_t e = dtype == FSA_DTYPE_BF16 ? (D == 128 ? launch_rd<128, __nv_bfloat16>(l, used, max_tiles, stream) : launch_rd<64, __nv_bfloat16>(l, used, max_tiles, stream))
                                                  : (D == 128 ? launch_rd<128, __half>(l, used, max_tiles, stream) : launch_rd<64, __half>(l, used, max_tiles, stream));
    return e == cudaSuccess ? FSA_OK : FSA_ERR_CUDA;
}

extern "C" int fsa_range_attn_fwd_dense(const void* q, const void* k, const void* v, const int32_t* cu_seqlens_q,
                                        const int32_t* cu_seqlens_k, const int32_t* kv_lo, const int32_t* kv_hi, int64_t N, int64_t Nk,
                                        int B, int Hq, int Hk, int D, int dtype, int64_t q_sn, int64_t q_sh, int64_t k_sn, int64_t v_sn,
                                        float sm_scale, void* o, int64_t o_sn, int64_t o_sh, float* lse, int32_t* status, void* stream) {
    const fsa_range_problem a = {q, k, v, cu_seqlens_q, cu_seqlens_k, kv_lo, kv_hi, N, Nk, q_sn, q_sh, k_sn, v_sn, o, o_sn, o_sh, lse, status};
    return fsa_range_attn_fwd_dense_several(1, &a, B, Hq, Hk, D, dtype, sm_scale, stream);
}
