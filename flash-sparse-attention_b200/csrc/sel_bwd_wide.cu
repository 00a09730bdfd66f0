// Selected-attention backward at head size 256, pipelined: the roles and the math of sel_bwd_pipe.cu (same partial rows, same
// slabs), laid out for rows of 512 bytes.
//
// What bounds it: 128 rows of Q and dO are 128 KB, so one stage of each and one K/V block fill shared memory, and dK^T, dV^T
// (256 TMEM columns) leave 256 columns for S, dP and dQ together.  A tile is therefore a chain -- gather, S / dP, P / dS,
// dK / dV / dQ -- that overlaps with its neighbours only where a resource is given back early:
//   * dK first: it frees the Q stage, whose next rows are on their way while dV and dQ run; dV frees dO;
//   * dQ takes the columns of S and dP (they have been read when dS is there).  The P / dS warps, which have nothing to do until
//     the next S, read it into registers as one, so that S may follow at once, and stage it from there in the P / dS buffers (their
//     readers are done).  Four drain warps that staged it half a row at a time held the columns for 4000 of a tile's 9300 cycles.
// The unpipelined kernel walked the same chain with 128 threads and no overlap at all: 17.5 us a tile.
// 16384 tokens, 4 KV heads, G = 2: 1967 -> 736 -> 704 us, with an even share of the tiles (sched_run) 598.
// Blocks of more than 64 keys are walked in 64-key parts as in sel_bwd_pipe.cu.
#include "sel_launch.cuh"

namespace fsa {

template <typename ET>
struct SelBwdWideParams {
    const ET* q;   int64_t q_sn, q_sh;
    const ET* d_o; int64_t do_sn, do_sh;
    const float* lse;
    const float* delta;
    SelShape s;
    SelIndex ix;
    float scale, scale_log2;
    int run, nsub;
    SelBounds bd;
    float* slabs;      // [segments][nsub][2 (dK, dV)][64 keys][256] fp32
};

namespace bwdwide {
constexpr int D = 256, KT = 64;
constexpr int kThreads = 768, kLoaders = 256;
constexpr int kWLoad = kLoaders / 32, kWMma1 = kWLoad, kWMma2 = kWLoad + 1, kWPrep = kWLoad + 2, kWDrain = kWLoad + 4,
              kWGroups = kWLoad + 8;
constexpr int kRegLoad = 40, kRegMma = 48, kRegDrain = 96, kRegGroup = 128;
static_assert(8 * kRegLoad + 4 * kRegMma + 4 * kRegDrain + 8 * kRegGroup <= 24 * 80, "register budget");
constexpr int kSlab = kTileRows * 128;           // 64 columns of 128 rows
constexpr int kQ = 4 * kSlab;                    // Q (or dO): 64 KB
constexpr int kK = KT * D * 2;                   // K (or V): 32 KB
constexpr int kP = kTileRows * KT * 2;           // P (or dS): 16 KB; the two stage 128 columns of dQ, 8 KB per warp
constexpr int kRing = 2;                         // prepared tiles: row offsets of Q and dO
constexpr int kTail = 3072;
constexpr int kBytes = 2 * kQ + 2 * kK + 2 * kP + kTail;
static_assert(kBytes <= 227 * 1024, "smem budget");
constexpr int cS = 0, cDP = 64, cDQ = 0;         // dQ: 256 columns over S, dP and the 128 behind them
constexpr int cDK = 256, cDV = 384;              // two halves of the head dimension, 64 columns each
constexpr uint32_t kCols = 512;
}  // namespace bwdwide

__device__ __forceinline__ float ex2_approx_w(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <typename ET>
__global__ void __launch_bounds__(bwdwide::kThreads, 1) sel_bwd_wide(const SelBwdWideParams<ET> p, const __grid_constant__ CUtensorMap kmap,
                                                                     const __grid_constant__ CUtensorMap vmap,
                                                                     const __grid_constant__ CUtensorMap dqmap) {
    using namespace bwdwide;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;
    uint8_t* sDO = sQ + kQ;
    uint8_t* sK = sDO + kQ;
    uint8_t* sV = sK + kK;
    uint8_t* sP = sV + kK;
    uint8_t* sDS = sP + kP;
    uint8_t* tail = sDS + kP;
    int (*s_off)[2][kTileRows] = reinterpret_cast<int (*)[2][kTileRows]>(tail);    // [ring][Q, dO][row] element offset / 8, -1: padding
    uint64_t* bars = reinterpret_cast<uint64_t*>(tail + kRing * 2 * kTileRows * 4);
    uint64_t* q_full = bars;             // Q rows have landed
    uint64_t* q_empty = bars + 1;        // ... have been read by S and dK
    uint64_t* do_full = bars + 2;
    uint64_t* do_empty = bars + 3;
    uint64_t* kv_full = bars + 4;
    uint64_t* kv_empty = bars + 5;       // every product of the segment is done
    uint64_t* sdp_full = bars + 6;
    uint64_t* pds_full = bars + 7;       // the 256 row threads have written P and dS
    uint64_t* pds_free = bars + 8;       // the stores of dQ have read their staging (the P / dS buffers)
    uint64_t* dq_full = bars + 9;        // every product of the tile is done
    uint64_t* dq_empty = bars + 10;      // dQ has been read: its columns may take the next S and dP
    uint64_t* acc_full = bars + 11;
    uint64_t* acc_empty = bars + 12;
    uint64_t* off_full = bars + 13;      // [ring]
    uint64_t* off_empty = bars + 15;     // [ring]
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 17);
    int4* s_rec = reinterpret_cast<int4*>(bars + 18);  // [8] prepared tiles: {bit 0: first tile of a segment (it loads its K/V block), bit 1: last
                                                       // one, tile of partial dQ rows, tile, run}
    static_assert(kRing * 2 * kTileRows * 4 + 18 * 8 + 8 * 16 <= kTail, "tail budget");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const SelShape& s = p.s;
    int* status = p.ix.header;
    if (smem_u32(smem) & 1023u) {
        if (tid == 0) atomicMax(status, (int)kStatusBadIndex);
        return;
    }
    if (tid == 0) {
        mbar_init(q_full, kLoaders); mbar_init(q_empty, 1);
        mbar_init(do_full, kLoaders); mbar_init(do_empty, 1);
        mbar_init(kv_full, 1); mbar_init(kv_empty, 1);
        mbar_init(sdp_full, 1); mbar_init(pds_full, 256); mbar_init(pds_free, 8);
        mbar_init(dq_full, 1); mbar_init(dq_empty, 256 + 4);
        mbar_init(acc_full, 1); mbar_init(acc_empty, 128);
        for (int i = 0; i < kRing; ++i) { mbar_init(&off_full[i], 1); mbar_init(&off_empty[i], kWLoad + 1); }
        mbar_init_fence();
        tma_prefetch_desc(&kmap);
        tma_prefetch_desc(&vmap);
        tma_prefetch_desc(&dqmap);
    }
    if (warp == 0) tmem_alloc(&tmem_slot, kCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tmem_slot;
    const TileScheduleT<true> sched(p.ix.header[1], p.run, p.nsub);
    const int nloc = sched.nloc;
    const int key_lim = min(KT, s.BK);
    bool ok = true;                          // no wait of this thread has run out

    if (warp < kWLoad) {
        // ------------------------------------------------------------------ gather warps: a warp copies whole 512-byte rows
        reg_dec<kRegLoad>();
        constexpr int NIT = kTileRows / kWLoad;                  // rows per warp
        const uint32_t slab_off = (uint32_t)(lane >> 3) * kSlab;
        auto copy = [&](const ET* base, uint8_t* dst, const int* off) {
            const ET* src = base + lane * 8;
            const uint32_t d = smem_u32(dst) + slab_off;
#pragma unroll 1
            for (int i0 = 0; i0 < NIT; i0 += 8) {                // (the offsets of eight rows are read ahead of their copies)
                int o[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = off[warp + (i0 + i) * kWLoad];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    cp_async16(d + sw128_chunk_off(warp + (i0 + i) * kWLoad, lane & 7), src + ((int64_t)max(o[i], 0) << 3), o[i] >= 0);
            }
        };
        for (int k = 0; k < nloc; ++k) {                         // (left by all lanes at the vote below)
            const int slot = k % kRing;
            ok = ok && mbar_poll(&off_full[slot], (k / kRing) & 1);
            ok = ok && mbar_poll(q_empty, (k & 1) ^ 1);
            ok = warp_ok(ok);
            if (!ok) break;
            copy(p.q, sQ, s_off[slot][0]);
            cp_async_mbar_arrive_noinc(q_full);
            ok = ok && mbar_poll(do_empty, (k & 1) ^ 1);
            copy(p.d_o, sDO, s_off[slot][1]);
            cp_async_mbar_arrive_noinc(do_full);
            __syncwarp();
            if (lane == 0) mbar_arrive(&off_empty[slot]);
        }
    } else if (warp >= kWDrain && warp < kWDrain + 4) {
        // ------------------------------------------------------------------ drain: dK / dV per segment
        reg_inc<kRegDrain>();
        const int quarter = warp & 3;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        int nflush = 0;
#pragma unroll 1
        for (int k = 0; k < nloc; ++k) {                         // (left by all lanes at the vote below)
            ok = ok && mbar_poll(dq_full, k & 1);
            const int4 rec = s_rec[k & 7];
            ok = warp_ok(ok);
            if (!ok) break;
            if (lane == 0) mbar_arrive(dq_empty);                // (no tile gets two ahead of this warp)
            if (!(rec.x & 2)) continue;
            const int seg = load_tile(p.ix, rec.z).seg0 + rec.w - __ldg(p.ix.tile_aux + rec.z).x / sched.run;
            float* slab = p.slabs + ((int64_t)seg * p.nsub + (rec.y - rec.z * p.nsub)) * (2 * KT * D) + quarter * 32 + lane;
            ok = ok && mbar_poll(acc_full, nflush & 1);
            tc_fence_after();
#pragma unroll 1
            for (int part = 0; part < 4; ++part) {               // dK low, dK high, dV low, dV high half of the head dimension
                uint32_t v[KT];
#pragma unroll
                for (int c0 = 0; c0 < KT; c0 += 32)
                    tmem_ld32(tbase + lane_off + cDK + part * KT + c0, *reinterpret_cast<uint32_t (*)[32]>(&v[c0]));
                tmem_ld_wait();
                if (part == 3) {
                    tc_fence_before();
                    mbar_arrive(acc_empty);
                    ++nflush;
                }
                float* dst = slab + (part >> 1) * (KT * D) + (part & 1) * 128;
#pragma unroll
                for (int key = 0; key < KT; ++key) dst[key * D] = __uint_as_float(v[key]);
            }
        }
    } else if (warp < kWDrain) {
        reg_dec<kRegMma>();
        if (warp == kWMma1) {
            // -------------------------------------------------------------- MMA issuer 1: S, dP
            const bool leader = elect_one();
            constexpr uint32_t idesc = umma_idesc(ElemTraits<ET>::kIsBF16, 128, KT, false, false);
            constexpr uint32_t hi_1024 = umma_desc_hi(1024);
            constexpr int kSlabA = kSlab >> 4, kSlabB = (KT * 128) >> 4;
            const uint32_t q_lo = umma_desc_lo(smem_u32(sQ), 16), do_lo = umma_desc_lo(smem_u32(sDO), 16);
            const uint32_t k_lo = umma_desc_lo(smem_u32(sK), 16), v_lo = umma_desc_lo(smem_u32(sV), 16);
            int kvn = -1;
            for (int k = 0; k < nloc && ok; ++k) {
                const int slot = k % kRing;
                ok = ok && mbar_poll(&off_full[slot], (k / kRing) & 1);
                const int seg = s_rec[k & 7].x;
                __syncwarp();
                if (lane == 0) mbar_arrive(&off_empty[slot]);
                if (seg & 1) {
                    ++kvn;
                    ok = ok && mbar_poll(kv_full, kvn & 1);
                }
                ok = ok && mbar_poll(dq_empty, (k & 1) ^ 1);
                ok = ok && mbar_poll(q_full, k & 1);
                fence_async_smem();
                ok = warp_ok(ok);
                if (!ok) break;
                tc_fence_after();
                if (leader) {
#pragma unroll 4
                    for (int ks = 0; ks < D / 16; ++ks)
                        umma_ss(tbase + cS, umma_desc_pack(q_lo + (ks >> 2) * kSlabA + (ks & 3) * 2, hi_1024),
                                umma_desc_pack(k_lo + (ks >> 2) * kSlabB + (ks & 3) * 2, hi_1024), idesc, ks > 0);
                }
                __syncwarp();
                ok = ok && mbar_poll(do_full, k & 1);
                fence_async_smem();
                ok = warp_ok(ok);
                if (!ok) break;
                tc_fence_after();
                if (leader) {
#pragma unroll 4
                    for (int ks = 0; ks < D / 16; ++ks)
                        umma_ss(tbase + cDP, umma_desc_pack(do_lo + (ks >> 2) * kSlabA + (ks & 3) * 2, hi_1024),
                                umma_desc_pack(v_lo + (ks >> 2) * kSlabB + (ks & 3) * 2, hi_1024), idesc, ks > 0);
                    umma_commit(sdp_full);
                }
                __syncwarp();
            }
        } else if (warp == kWMma2) {
            // -------------------------------------------------------------- MMA issuer 2: dK^T, dV^T, dQ
            const bool leader = elect_one();
            constexpr uint32_t idesc_dq = umma_idesc(ElemTraits<ET>::kIsBF16, 128, D, false, true);     // dS (K-major) x K (MN-major)
            constexpr uint32_t idesc_dk = umma_idesc(ElemTraits<ET>::kIsBF16, 128, KT, true, true);     // Q^T / dO^T x dS / P
            constexpr uint32_t hi_1024 = umma_desc_hi(1024);
            const uint32_t ds_k_lo = umma_desc_lo(smem_u32(sDS), 16);
            const uint32_t ds_mn_lo = umma_desc_lo(smem_u32(sDS), 8192), p_mn_lo = umma_desc_lo(smem_u32(sP), 8192);
            const uint32_t k_mn_lo = umma_desc_lo(smem_u32(sK), KT * 128);
            const uint32_t q_mn_lo = umma_desc_lo(smem_u32(sQ), kSlab), do_mn_lo = umma_desc_lo(smem_u32(sDO), kSlab);
            int blk = -1;
#pragma unroll 1
            for (int k = 0; k < nloc && ok; ++k) {
                // (the record is complete: its tile has been through the S / dP issuer when P is there)
                ok = ok && mbar_poll(pds_full, k & 1);
                const int seg = s_rec[k & 7].x;
                const bool first = seg & 1, last = seg & 2;
                if (first) ++blk;
                // (complete already: acquire only)
                ok = ok && mbar_poll(kv_full, blk & 1);
                ok = ok && mbar_poll(q_full, k & 1);
                ok = ok && mbar_poll(do_full, k & 1);
                if (first && blk > 0) ok = ok && mbar_poll(acc_empty, (blk - 1) & 1);
                fence_async_smem();
                ok = warp_ok(ok);
                if (!ok) break;
                tc_fence_after();
                if (leader) {
#pragma unroll 2
                    for (int ks = 0; ks < kTileRows / 16; ++ks)
#pragma unroll
                        for (int half = 0; half < 2; ++half)
                            umma_ss(tbase + cDK + half * KT, umma_desc_pack(q_mn_lo + half * ((2 * kSlab) >> 4) + ks * (2048 >> 4), hi_1024),
                                    umma_desc_pack(ds_mn_lo + ks * (2048 >> 4), hi_1024), idesc_dk, (!first || ks > 0) ? 1u : 0u);
                    umma_commit(q_empty);
#pragma unroll 2
                    for (int ks = 0; ks < kTileRows / 16; ++ks)
#pragma unroll
                        for (int half = 0; half < 2; ++half)
                            umma_ss(tbase + cDV + half * KT, umma_desc_pack(do_mn_lo + half * ((2 * kSlab) >> 4) + ks * (2048 >> 4), hi_1024),
                                    umma_desc_pack(p_mn_lo + ks * (2048 >> 4), hi_1024), idesc_dk, (!first || ks > 0) ? 1u : 0u);
                    umma_commit(do_empty);
                    if (last) umma_commit(acc_full);
#pragma unroll
                    for (int ks = 0; ks < KT / 16; ++ks)
                        umma_ss(tbase + cDQ, umma_desc_pack(ds_k_lo + ks * 2, hi_1024), umma_desc_pack(k_mn_lo + ks * (2048 >> 4), hi_1024), idesc_dq,
                                ks > 0);
                    umma_commit(dq_full);
                    if (last) umma_commit(kv_empty);
                }
                __syncwarp();
            }
        } else if (warp == kWPrep) {
            // -------------------------------------------------------------- tile preparation: row offsets, two tiles ahead of the copies
            int gg[4], ee[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = lane + 32 * i;
                gg[i] = r / s.TPT;
                ee[i] = r - gg[i] * s.TPT;
            }
            const int qsn8 = (int)(p.q_sn >> 3), dsn8 = (int)(p.do_sn >> 3), qsh8 = (int)(p.q_sh >> 3), dsh8 = (int)(p.do_sh >> 3);
            int prev_hg = -1;
            // (two tiles in turn: handing the registers on would wait for the loads)
            struct Pre { int h, hg; uint32_t e[4]; };
            TileCursorT<true> ahead(sched), cur(sched);
            auto fetch = [&](Pre& m) {
                const TileInfo ti = load_tile(p.ix, ahead.j);
                m.h = ti.h; m.hg = ti.hg;
#pragma unroll
                for (int i = 0; i < 4; ++i) m.e[i] = gg[i] < s.G ? __ldg(p.ix.entries + (int64_t)ahead.j * s.TPT + ee[i]) : 0xFFFFFFFFu;
                ahead.next(sched);
            };
            auto publish = [&](int k, Pre& m, const Pre& next) {
                const int slot = k % kRing;
                ok = ok && mbar_poll(&off_empty[slot], ((k / kRing) & 1) ^ 1);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int tok = (int)(m.e[i] >> kSlotBits), hq = m.h * s.G + gg[i];
                    s_off[slot][0][lane + 32 * i] = m.e[i] != 0xFFFFFFFFu ? tok * qsn8 + hq * qsh8 : -1;
                    s_off[slot][1][lane + 32 * i] = m.e[i] != 0xFFFFFFFFu ? tok * dsn8 + hq * dsh8 : -1;
                }
                if (lane == 0)
                    s_rec[k & 7] = make_int4((m.hg != prev_hg || cur.r == 0 ? 1 : 0) | (k + 1 >= nloc || next.hg != m.hg || cur.r + 1 == sched.run ? 2 : 0),
                                             cur.j * p.nsub + cur.sub(sched), cur.j, cur.run(sched));
                cur.next(sched);
                prev_hg = m.hg;
                ok = warp_ok(ok);
                if (lane == 0) mbar_arrive(&off_full[slot]);
                if (k + 2 < nloc) fetch(m);
            };
            Pre m1{0, -1, {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}}, m2 = m1;
            if (nloc > 0) fetch(m1);
            if (nloc > 1) fetch(m2);
#pragma unroll 1
            for (int k = 0; k < nloc && ok; k += 2) {
                publish(k, m1, m2);
                if (k + 1 < nloc) publish(k + 1, m2, m1);
            }
        } else {
            // -------------------------------------------------------------- K/V blocks by TMA
            int kvn = -1, prev_hg = -1;
            TileCursorT<true> cur(sched);
#pragma unroll 1
            for (int k = 0; k < nloc && ok; ++k) {
                const TileInfo ti = load_tile(p.ix, cur.j);
                const int row = ti.row0 + cur.sub(sched) * KT;
                const bool first = ti.hg != prev_hg || cur.r == 0;
                cur.next(sched);
                if (!first) continue;
                prev_hg = ti.hg;
                ++kvn;
                if (lane == 0) {
                    ok = ok && mbar_poll(kv_empty, (kvn & 1) ^ 1);
                    if (ok) {
                        mbar_expect_tx(kv_full, (uint32_t)(2 * kK));
#pragma unroll
                        for (int b = 0; b < D / 64; ++b) {
                            tma_load_2d(smem_u32(sK + b * KT * 128), &kmap, ti.h * D + b * 64, row, kv_full);
                            tma_load_2d(smem_u32(sV + b * KT * 128), &vmap, ti.h * D + b * 64, row, kv_full);
                        }
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            }
        }
    } else {
        // ------------------------------------------------------------------ P / dS: one row per thread, half of the columns per group
        reg_inc<kRegGroup>();
        const int sb = (warp - kWGroups) >> 2;
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        const int g = r / s.TPT, e = r - g * s.TPT;
        const bool row_exists = g < s.G;
        constexpr int HC = KT / 2;
        const int cb = sb * HC;
        uint32_t ent = 0xFFFFFFFFu;
        int row0 = 0, h = 0;
        TileCursorT<true> ahead(sched);
        auto fetch_ent = [&]() {
            const TileInfo ti = load_tile(p.ix, ahead.j);
            row0 = ti.row0 + ahead.sub(sched) * KT;
            h = ti.h;
            ent = row_exists ? __ldg(p.ix.entries + (int64_t)ahead.j * s.TPT + e) : 0xFFFFFFFFu;
            ahead.next(sched);
        };
        if (nloc > 0) fetch_ent();
        // lse, delta and visible columns of the next tile's row (padding rows: zero Q and dO rows, any finite P will do)
        float lse_n = 0.f, delta_n = 0.f;
        int lo_n = 0, hi_n = key_lim;
        auto fetch_stats = [&]() {
            lse_n = 0.f; delta_n = 0.f; lo_n = 0; hi_n = key_lim;
            if (ent != 0xFFFFFFFFu) {
                const int tok = (int)(ent >> kSlotBits);
                const int64_t idx = (int64_t)(h * s.G + g) * s.N + tok;
                lse_n = __ldg(p.lse + idx);
                delta_n = __ldg(p.delta + idx);
                visible_cols(p.bd, tok, row0, key_lim, lo_n, hi_n);
            }
        };
        if (nloc > 0) fetch_stats();
        uint8_t* my_stage = sP + (sb * 4 + quarter) * (32 * 128);        // 32 rows x 64 columns
#pragma unroll 1
        for (int k = 0; k < nloc && warp_stays(ok); ++k) {
            const float lse_r = lse_n, delta_s = delta_n * p.scale;
            const int c_lo = lo_n, c_hi = hi_n;
            if (k + 1 < nloc) fetch_ent();
            ok = ok && mbar_poll(sdp_full, k & 1);
            tc_fence_after();
            uint32_t pp[HC / 2], dd[HC / 2];
            {
                uint32_t sv[32], dv[32];
                tmem_ld32(tbase + lane_off + cS + cb, sv);
                tmem_ld32(tbase + lane_off + cDP + cb, dv);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) sv[i] = __float_as_uint(ex2_approx_w(fmaf(__uint_as_float(sv[i]), p.scale_log2, -lse_r)));
                if (!__all_sync(0xffffffffu, c_lo <= cb && c_hi >= cb + HC)) {
                    // (bit i: column cb + i is visible)
                    const int lo = min(max(c_lo - cb, 0), 32), hi = min(max(c_hi - cb, 0), 32);
                    const uint32_t vis = (uint32_t)((1ull << hi) - 1) & ~(uint32_t)((1ull << lo) - 1);
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (!(vis >> i & 1u)) sv[i] = 0u;
                }
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float p0 = __uint_as_float(sv[i]), p1 = __uint_as_float(sv[i + 1]);
                    pp[i >> 1] = ElemTraits<ET>::pack2(p0, p1);
                    dd[i >> 1] = ElemTraits<ET>::pack2(p0 * fmaf(__uint_as_float(dv[i]), p.scale, -delta_s), p1 * fmaf(__uint_as_float(dv[i + 1]), p.scale, -delta_s));
                }
            }
            tc_fence_before();
            if (k > 0) ok = ok && mbar_poll(pds_free, (k - 1) & 1);
#pragma unroll
            for (int c4 = 0; c4 < HC / 8; ++c4) {
                const uint32_t off = sw128_chunk_off(r, sb * (HC / 8) + c4);
                *reinterpret_cast<uint4*>(sP + off) = make_uint4(pp[c4 * 4], pp[c4 * 4 + 1], pp[c4 * 4 + 2], pp[c4 * 4 + 3]);
                *reinterpret_cast<uint4*>(sDS + off) = make_uint4(dd[c4 * 4], dd[c4 * 4 + 1], dd[c4 * 4 + 2], dd[c4 * 4 + 3]);
            }
            fence_async_smem();
            mbar_arrive(pds_full);
            if (k + 1 < nloc) fetch_stats();
            // ---- dQ of the tile: this group's 128 columns to registers, which frees its TMEM columns for the next S and dP, and from
            // there 64 at a time through the P / dS buffers, which the products have read
            ok = ok && mbar_poll(dq_full, k & 1);
            tc_fence_after();
            const int row = s_rec[k & 7].y * kTileRows + quarter * 32;
            uint32_t x[64];
#pragma unroll
            for (int c0 = 0; c0 < 128; c0 += 32) {
                uint32_t v[32];
                tmem_ld32(tbase + lane_off + cDQ + sb * 128 + c0, v);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; ++i) x[c0 / 2 + i] = ElemTraits<ET>::pack2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
            }
            tc_fence_before();
            mbar_arrive(dq_empty);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<uint4*>(my_stage + sw128_chunk_off(lane, c)) =
                        make_uint4(x[half * 32 + c * 4], x[half * 32 + c * 4 + 1], x[half * 32 + c * 4 + 2], x[half * 32 + c * 4 + 3]);
                fence_async_smem();
                __syncwarp();
                if (lane == 0) {
                    if (ok) tma_store_2d(&dqmap, sb * 128 + half * 64, row, smem_u32(my_stage));
                    bulk_commit();
                    bulk_wait_read0();
                    if (half == 1) mbar_arrive(pds_free);
                }
                __syncwarp();
            }
        }
        if (lane == 0) bulk_wait0();
    }
    if (!ok) atomicMax(status, (int)kStatusWaitTimeout);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, bwdwide::kCols);
}

template <typename ET>
static cudaError_t launch_wide(const SelBwdArgs& a, const SelShape& s, const SelIndex& ix, const CUtensorMap& kmap, const CUtensorMap& vmap,
                               const CUtensorMap& dqmap, int num_sms, cudaStream_t stream) {
    SelBwdWideParams<ET> p;
    p.q = (const ET*)a.q; p.q_sn = a.q_sn; p.q_sh = a.q_sh;
    p.d_o = (const ET*)a.d_o; p.do_sn = a.do_sn; p.do_sh = a.do_sh;
    p.lse = a.lse; p.delta = a.delta;
    p.s = s; p.ix = ix;
    p.scale = a.sm_scale; p.scale_log2 = a.sm_scale * 1.4426950408889634f;
    p.run = s.RB; p.nsub = s.BK > bwdwide::KT ? s.BK / bwdwide::KT : 1;
    p.bd = a.bd; p.slabs = a.slabs;
    auto kern = sel_bwd_wide<ET>;
    cudaError_t e = allow_smem((const void*)kern, bwdwide::kBytes);
    if (e != cudaSuccess) return e;
    prof_begin(2, stream);
    kern<<<num_sms, bwdwide::kThreads, bwdwide::kBytes, stream>>>(p, kmap, vmap, dqmap);
    prof_end(2, stream);
    return cudaGetLastError();
}

cudaError_t launch_sel_bwd_wide(int dtype, const SelBwdArgs& a, const SelShape& s, const SelIndex& ix, const CUtensorMap& kmap,
                                const CUtensorMap& vmap, const CUtensorMap& dqmap, int num_sms, cudaStream_t stream) {
    return dtype == kBF16 ? launch_wide<__nv_bfloat16>(a, s, ix, kmap, vmap, dqmap, num_sms, stream)
                          : launch_wide<__half>(a, s, ix, kmap, vmap, dqmap, num_sms, stream);
}

}  // namespace fsa
