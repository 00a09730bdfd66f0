// Selected-attention backward, pipelined kernel for head_dim 64 and 128 (256: sel_bwd_wide.cu).  Blocks of 128 and 256 keys are
// walked as independent 64-key parts, every part a pass over the tiles of its own (the gathers are repeated, which costs less
// than the registers and TMEM of a wider tile: 21008 tokens, 128-key blocks, 734 us in the unpipelined kernel before).
// Per tile of <= 128 (head, token) rows of one part of a KV block
//     S = Q K^T, dP = dO V^T | P = exp2(S c - lse), dS = scale P (dP - delta) | dQ = dS K,
//     dK^T += Q^T dS, dV^T += dO^T P
// Warp roles (768 threads in six warpgroups whose register budgets are rebalanced with setmaxnreg; one CTA per SM,
// persistent over a round-robin run schedule):
//   warps 0..7   gather the dO rows, then the Q rows with 16-byte async copies (two stages);
//   warp 8       issues dP, then S (tcgen05, fp32 in TMEM, two buffers);
//   warp 9       issues dV^T, dK^T, dQ;
//   warp 10      prepares, two tiles ahead, the offset of every tile row (the gather warps then run without
//                any global load of their own: a plain load issued behind a burst of async copies waits for it);
//   warp 11      loads the K/V block of every segment by TMA;
//   warps 12..15 the accumulator drain, one row / one head-dim index per thread: for every tile the dQ partial from TMEM
//                through a swizzled staging area to global memory by TMA store (input dtype, tile order: the load/store
//                unit is left to the row gathers); at the end of a segment (the tiles of one block inside one
//                scheduling run) the finished dK^T / dV^T accumulators from TMEM to registers (freeing them for the next
//                segment at once) and on to the segment's own fp32 slab while the next segment computes; a second kernel
//                sums the slabs of a block in segment order, so dK and dV do not depend on the order in which CTAs
//                finish (no atomics);
//   warps 16..23 two groups, one row per thread, each on half of the 64 key columns of every tile: P / dS to swizzled smem
//                and nothing else -- they are the critical path of a tile (the exp2 and the dS arithmetic between two
//                MMA phases), so both groups shorten the same tile instead of alternating tiles.
// What bounds it: the dependent chain of a tile (gather of 64 KB, S / dP, P / dS, dV / dK) with two stages of Q / dO.  Hence
//   - dO and Q are separate stages: dV is issued before dK and gives dO back first, the gather brings dO back first, and dP,
//     the factor scale (dP - delta) and the product of the tile before run under the gather of Q (in one stage, and with dK
//     and dV interleaved: 1115 and 1060 us instead of 1000);
//   - K has two stages and V is given back after the last dP of a segment, so that a segment starts while the one before it
//     ends; the 16 KB come from staging dQ 64 columns at a time;
//   - the loops of all roles together stay in the SM's instruction cache: no division per tile (cursors), rolled loops where
//     nothing waits for the issue, short waits, segment records from the preparation warp instead of in every role.  With
//     65 KB of code the issue slots found no instruction 1.7 times per instruction issued, with 43 KB 0.2 times; the new
//     stages in 74 KB of code: 7.6 times, 1600 us.
// 64K tokens x 8 heads x 16 blocks (CUDA events): 1190 us; with the short waits alone 1099; now 1000.  21K ragged tokens,
// 128-key blocks: 235 -> 205 us.
#include "sel_launch.cuh"

namespace fsa {

template <typename ET>
struct SelBwdPipeParams {
    const ET* q;   int64_t q_sn, q_sh;
    const ET* d_o; int64_t do_sn, do_sh;
    const float* lse;
    const float* delta;
    SelShape s;
    SelIndex ix;
    float scale, scale_log2;
    int run;
    SelBounds bd;      // visible K/V rows per token
    ET* dq_part;       // [max_tiles][nsub][128, D] (written through dqmap)
    int nsub;          // 64-key parts of a block
    float* slabs;      // [segments][nsub][2 (dK, dV)][64 keys][D] fp32: the partial sums of every segment of tiles
};

namespace bwdpipe {
constexpr int KT = 64;
constexpr int kKStages = 2;                      // K; V has one: its last reader, dP, is early in a tile
constexpr int kThreads = 768, kLoaders = 256;
constexpr int kWLoad = kLoaders / 32, kWMma1 = kWLoad, kWMma2 = kWLoad + 1, kWFlush = kWLoad + 4, kWGroups = kWLoad + 8;
// registers per thread of each role (multiples of 8); 32 * sum over warps <= 768 * 80 = the CTA's allocation
constexpr int kRegLoad = 32, kRegMma = 64, kRegFlush = 96, kRegGroup = 128;
static_assert(8 * kRegLoad + 4 * kRegMma + 4 * kRegFlush + 8 * kRegGroup <= 24 * 80, "register budget");
constexpr int kPS = 2 * kTileRows * KT * 2;      // P then dS: 32 KB
constexpr int kTail = 2624;
constexpr int cS = 0, cDP = 64;                  // + 128 * buffer
constexpr int cDQ = 256, cDK = 384, cDV = 448;
constexpr uint32_t kCols = 512;
template <int D> struct Cfg {
    static constexpr int kK = KT * D * 2;                   // one of K, V
    static constexpr int kQD = 2 * kTileRows * D * 2;       // Q then dO
    static constexpr int kDQ = kTileRows * 64 * 2;          // dQ staging, 64 columns at a time, a quarter per TMEM lane quarter
    static constexpr int kBytes = (kKStages + 1) * kK + 2 * kQD + kPS + kDQ + kTail;
    static_assert(kBytes <= 227 * 1024, "smem budget");
};
}  // namespace bwdpipe

// Optional cycle accounting per role (debug builds only, -DFSA_TIMING): a table [gridDim.x][64] of accumulated
// clock64() deltas, read back with fsa_debug_read_bwd_timing.
#ifdef FSA_TIMING
__device__ unsigned long long g_bwd_timing[512 * 64];
#define BT_DECL unsigned long long _t0 = clock64(), _acc[8] = {0, 0, 0, 0, 0, 0, 0, 0}
#define BT_TOC(i) do { unsigned long long _t1 = clock64(); _acc[i] += _t1 - _t0; _t0 = _t1; } while (0)
#define BT_DUMP(base, n) do { for (int _i = 0; _i < (n); ++_i) g_bwd_timing[blockIdx.x * 64 + (base) + _i] = _acc[_i]; } while (0)
// Event trace of eight consecutive tiles of CTA 0 (absolute clock64() values), [tile][16 events].
__device__ unsigned long long g_bwd_trace[8 * 16];
constexpr int kTraceTile0 = 200;
#define BT_EV(k, ev, who) do { if (blockIdx.x == 0 && (k) >= kTraceTile0 && (k) < kTraceTile0 + 8 && (who)) \
        g_bwd_trace[((k) - kTraceTile0) * 16 + (ev)] = clock64(); } while (0)
#else
#define BT_DECL
#define BT_TOC(i)
#define BT_DUMP(base, n)
#define BT_EV(k, ev, who)
#endif

__device__ __forceinline__ float ex2_approx_b(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <int D, bool PARTS, typename ET>
__global__ void __launch_bounds__(bwdpipe::kThreads, 1) sel_bwd_pipe(const SelBwdPipeParams<ET> p,
                                                                     const __grid_constant__ CUtensorMap kmap,
                                                                     const __grid_constant__ CUtensorMap vmap,
                                                                     const __grid_constant__ CUtensorMap dqmap) {
    using namespace bwdpipe;
    constexpr int kK = Cfg<D>::kK, kQD = Cfg<D>::kQD, kDQ = Cfg<D>::kDQ;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sK = smem;                                     // K stages, then V
    uint8_t* sV = sK + kKStages * kK;
    uint8_t* sQD = sV + kK;
    uint8_t* sP = sQD + 2 * kQD;
    uint8_t* sDS = sP + kTileRows * KT * 2;
    uint8_t* sDQ = sP + kPS;
    uint8_t* tail = sDQ + kDQ;
    int2 (*s_off)[kTileRows] = reinterpret_cast<int2 (*)[kTileRows]>(tail);              // [2][128] offset of every tile row in q and dO (units of
                                                                                        // 8 elements), -1: padding
    uint64_t* bars = reinterpret_cast<uint64_t*>(tail + 2048);
    uint64_t* do_full = bars;            // [2] the dO rows of a stage have landed
    uint64_t* do_empty = bars + 2;       // [2] ... have been read (dV)
    uint64_t* q_full = bars + 4;         // [2]
    uint64_t* q_empty = bars + 6;        // [2] (dK)
    uint64_t* k_full = bars + 8;         // [2]
    uint64_t* k_empty = bars + 10;       // [2]
    uint64_t* v_full = bars + 12;
    uint64_t* v_empty = bars + 13;
    uint64_t* dp_full = bars + 14;       // [2]
    uint64_t* s_full = bars + 16;        // [2]
    uint64_t* sdp_empty = bars + 18;     // [2]
    uint64_t* p_full = bars + 20;
    uint64_t* p_empty = bars + 21;
    uint64_t* ds_full = bars + 22;
    uint64_t* ds_empty = bars + 23;
    uint64_t* dq_full = bars + 24;
    uint64_t* dq_empty = bars + 25;
    uint64_t* acc_full = bars + 26;
    uint64_t* acc_empty = bars + 27;
    uint64_t* off_full = bars + 28;      // [2] ring of prepared tiles: row offsets and record are valid
    uint64_t* off_empty = bars + 32;     // [2] ... have been read by the eight gather warps and the S/dP issuer
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 36);
    int4* s_rec = reinterpret_cast<int4*>(bars + 38);    // [16] prepared tiles: {bit 0: first tile of a segment (K and V are loaded for it),
                                                         // bit 1: last one, tile of partial dQ rows, tile, run}.  16: the drain may be eight behind
    static_assert(2 * kTileRows * 8 + 38 * 8 + 16 * 16 <= kTail, "tail budget");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const SelShape& s = p.s;
    int* status = p.ix.header;
    if (smem_u32(smem) & 1023u) {
        if (tid == 0) atomicMax(status, (int)kStatusBadIndex);
        return;
    }
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&do_full[i], kLoaders); mbar_init(&do_empty[i], 1);
            mbar_init(&q_full[i], kLoaders); mbar_init(&q_empty[i], 1);
            mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
            mbar_init(&dp_full[i], 1); mbar_init(&s_full[i], 1); mbar_init(&sdp_empty[i], 256);
        }
        mbar_init(v_full, 1); mbar_init(v_empty, 1);
        mbar_init(p_full, 256); mbar_init(p_empty, 1);
        mbar_init(ds_full, 256); mbar_init(ds_empty, 1);
        mbar_init(dq_full, 1); mbar_init(dq_empty, 128);
        mbar_init(acc_full, 1); mbar_init(acc_empty, 128);
        for (int i = 0; i < 2; ++i) { mbar_init(&off_full[i], 1); mbar_init(&off_empty[i], kWLoad + 1); }
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
    const TileScheduleT<PARTS> sched(p.ix.header[1], p.run, p.nsub);
    const int nsub = PARTS ? p.nsub : 1;
    const int nloc = sched.nloc;
    const int key_lim = min(KT, s.BK);
    bool ok = true;                         // no wait of this thread has run out

    if (warp < kWLoad) {
        // ------------------------------------------------------------------ gather warps
        // (D = 128) thread t copies 16-byte chunk t % 16 of the rows t / 16 + 16 i (a half-warp covers one 256-byte row) of Q and
        // dO.  The rows' offsets come from the prepared ring.
        reg_dec<kRegLoad>();
        const int t = tid;
        constexpr int CPR = D / 8, RSTEP = kLoaders / CPR, NIT = kTileRows / RSTEP;   // D = 128: 16 chunks per row, 8 rows per thread
        const int cchunk = t % CPR, rbase = t / CPR;
        const uint32_t slab_off = (uint32_t)(cchunk >> 3) * (kTileRows * 128);
        const ET* qc = p.q + cchunk * 8;
        const ET* dc = p.d_o + cchunk * 8;
        BT_DECL;
#pragma unroll 1
        for (int k = 0; k < nloc; ++k) {                // (left by all lanes at the vote below)
            const int st = k & 1;
            BT_TOC(0);
            ok = ok && mbar_poll(&off_full[st], (k >> 1) & 1);
            BT_TOC(2);
            int2 off[NIT];                              // (all of them ahead of the copies)
#pragma unroll
            for (int it = 0; it < NIT; ++it) off[it] = s_off[st][rbase + it * RSTEP];
            ok = warp_ok(ok);
            if (!ok) break;
            if (lane == 0) mbar_arrive(&off_empty[st]);
            // dO first: dV, its last reader, is issued before dK, the last reader of Q
            // (RSTEP is a multiple of 8: the rows of a thread have one swizzle)
            const uint32_t dq_ = smem_u32(sQD + st * kQD) + slab_off + sw128_chunk_off(rbase, cchunk & 7);
            const uint32_t dd_ = dq_ + kTileRows * D * 2;
            ok = ok && mbar_poll(&do_empty[st], ((k >> 1) & 1) ^ 1);
            BT_EV(k, 0, t == 0);
            BT_TOC(1);
#pragma unroll
            for (int it = 0; it < NIT; ++it) {
                const int o = off[it].y;
                cp_async16(dd_ + it * (RSTEP * 128), dc + ((int64_t)max(o, 0) << 3), o >= 0);
            }
            cp_async_mbar_arrive_noinc(&do_full[st]);
            BT_TOC(4);
            ok = ok && mbar_poll(&q_empty[st], ((k >> 1) & 1) ^ 1);
            BT_TOC(1);
#pragma unroll
            for (int it = 0; it < NIT; ++it) {
                const int o = off[it].x;
                cp_async16(dq_ + it * (RSTEP * 128), qc + ((int64_t)max(o, 0) << 3), o >= 0);
            }
            cp_async_mbar_arrive_noinc(&q_full[st]);
            BT_EV(k, 1, t == 0);
            BT_TOC(4);
        }
        if (t == 0) BT_DUMP(0, 5);
    } else if (warp >= kWFlush && warp < kWFlush + 4) {
        // ------------------------------------------------------------------ accumulator drain: dQ per tile, dK / dV per segment
        // Walks the CTA's tiles in order.  Per tile: wait for its dQ product, move it TMEM -> registers -> swizzled staging
        // (this warp's 32 rows) -> TMA store.  At the last tile of a segment: wait for the segment's last products, pull
        // dK^T / dV^T (lane = head-dim index, columns = keys) into registers, release the TMEM accumulators, store them to
        // the segment's slab.
        reg_inc<kRegFlush>();
        const int quarter = warp & 3;
        const int d_idx = quarter * 32 + lane;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        uint8_t* my_stage = sDQ + quarter * (32 * 128);
        int nflush = 0;
        BT_DECL;
#pragma unroll 1
        for (int k = 0; k < nloc && ok; ++k) {
            // ---- dQ partial of this tile
            BT_TOC(0);
            ok = ok && mbar_poll(dq_full, k & 1);
            BT_EV(k, 13, warp == kWFlush && lane == 0);
            BT_TOC(1);
            ok = warp_ok(ok);
            tc_fence_after();
            const int4 rec = s_rec[k & 15];
            // (rolled loops here and below: see the note on code size)
#pragma unroll 1
            for (int b = 0; b < D / 64; ++b) {
                if (lane == 0) bulk_wait_read0();          // the store before this one has read this warp's staging rows
                __syncwarp();
#pragma unroll 1
                for (int c0 = 0; c0 < 64; c0 += 32) {
                    uint32_t v[32];
                    tmem_ld32(tbase + lane_off + cDQ + b * 64 + c0, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) {
                        uint4 u;
                        u.x = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 0]), __uint_as_float(v[q4 * 8 + 1]));
                        u.y = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 2]), __uint_as_float(v[q4 * 8 + 3]));
                        u.z = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 4]), __uint_as_float(v[q4 * 8 + 5]));
                        u.w = ElemTraits<ET>::pack2(__uint_as_float(v[q4 * 8 + 6]), __uint_as_float(v[q4 * 8 + 7]));
                        *reinterpret_cast<uint4*>(my_stage + sw128_chunk_off(lane, (c0 >> 3) + q4)) = u;
                    }
                }
                if (b == D / 64 - 1) {
                    tc_fence_before();
                    mbar_arrive(dq_empty);
                    BT_EV(k, 14, warp == kWFlush && lane == 0);
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) {
                    if (ok) tma_store_2d(&dqmap, b * 64, rec.y * kTileRows + quarter * 32, smem_u32(my_stage));
                    bulk_commit();
                }
            }
            BT_TOC(2);
            if (!ok || !(rec.x & 2)) continue;
            // ---- dK^T / dV^T of the finished segment (the segments of a key are numbered by the scheduling run they fall into)
            const int seg = load_tile(p.ix, rec.z).seg0 + rec.w - __ldg(p.ix.tile_aux + rec.z).x / sched.run;
            float* slab = p.slabs + ((int64_t)seg * nsub + (rec.y - rec.z * nsub)) * (2 * KT * D) + d_idx;
            ok = ok && mbar_poll(acc_full, nflush & 1);
            ok = warp_ok(ok);
            BT_TOC(3);
            tc_fence_after();
#pragma unroll 1
            for (int which = 0; which < 2; ++which) {
                uint32_t v[KT];
                tmem_ld32(tbase + lane_off + (which == 0 ? cDK : cDV), *reinterpret_cast<uint32_t (*)[32]>(&v[0]));
                tmem_ld32(tbase + lane_off + (which == 0 ? cDK : cDV) + 32, *reinterpret_cast<uint32_t (*)[32]>(&v[32]));
                tmem_ld_wait();
                if (which == 1) {
                    // both accumulators have been read: the next segment may overwrite them
                    tc_fence_before();
                    mbar_arrive(acc_empty);
                    ++nflush;
                }
                // (D = 64: the upper accumulator rows are products of whatever follows the tile in shared memory)
                if (quarter * 32 < D) {
#pragma unroll
                    for (int key = 0; key < KT; ++key) slab[key * D] = __uint_as_float(v[key]);
                }
                slab += KT * D;
            }
            BT_TOC(4);
        }
        if (lane == 0) bulk_wait0();
        if (warp == kWFlush && lane == 0) BT_DUMP(8, 5);
    } else if (warp < kWFlush) {
      reg_dec<kRegMma>();
      if (warp == kWMma1) {
        // ------------------------------------------------------------------ MMA issuer 1: S and dP
        const bool leader = elect_one();
        constexpr uint32_t idesc_s = umma_idesc(ElemTraits<ET>::kIsBF16, 128, KT, false, false);
        constexpr uint32_t hi_1024 = umma_desc_hi(1024);
        const uint32_t qd_lo = umma_desc_lo(smem_u32(sQD), 16);
        const uint32_t k_lo = umma_desc_lo(smem_u32(sK), 16), v_lo = umma_desc_lo(smem_u32(sV), 16);
        int kvn = -1;
        BT_DECL;
#pragma unroll 1
        for (int k = 0; k < nloc && ok; ++k) {
            const int st = k & 1;
            BT_TOC(0);
            ok = ok && mbar_poll(&off_full[st], (k >> 1) & 1);
            BT_TOC(1);
            const int seg = s_rec[k & 15].x;
            __syncwarp();
            if (lane == 0) mbar_arrive(&off_empty[st]);
            if (seg & 1) {
                ++kvn;
                ok = ok && mbar_poll(v_full, kvn & 1);
            }
            BT_TOC(2);
            ok = ok && mbar_poll(&sdp_empty[st], ((k >> 1) & 1) ^ 1);
            BT_EV(k, 3, lane == 0);
            BT_TOC(4);
            ok = ok && mbar_poll(&do_full[st], (k >> 1) & 1);
            BT_EV(k, 2, lane == 0);
            BT_TOC(3);
            fence_async_smem();
            ok = warp_ok(ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t aq = qd_lo + (uint32_t)(st * (kQD >> 4));
            const uint32_t ad = aq + (uint32_t)((kTileRows * D * 2) >> 4);
            const uint32_t bk = k_lo + (uint32_t)((kvn % kKStages) * (kK >> 4));
            const uint32_t dS_ = tbase + cS + st * 128, dP_ = tbase + cDP + st * 128;
            constexpr int kSlabA = (kTileRows * 128) >> 4, kSlabB = (KT * 128) >> 4;
            if (leader) {
#pragma unroll 4
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_ss(dP_, umma_desc_pack(ad + (ks >> 2) * kSlabA + (ks & 3) * 2, hi_1024),
                            umma_desc_pack(v_lo + (ks >> 2) * kSlabB + (ks & 3) * 2, hi_1024), idesc_s, ks > 0);
                umma_commit(&dp_full[st]);
                if (seg & 2) umma_commit(v_empty);
            }
            __syncwarp();
            BT_TOC(5);
            if (seg & 1) ok = ok && mbar_poll(&k_full[kvn % kKStages], (kvn / kKStages) & 1);
            BT_TOC(2);
            ok = ok && mbar_poll(&q_full[st], (k >> 1) & 1);
            BT_TOC(3);
            fence_async_smem();
            ok = warp_ok(ok);
            if (!ok) break;
            tc_fence_after();
            if (leader) {
#pragma unroll 4
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_ss(dS_, umma_desc_pack(aq + (ks >> 2) * kSlabA + (ks & 3) * 2, hi_1024),
                            umma_desc_pack(bk + (ks >> 2) * kSlabB + (ks & 3) * 2, hi_1024), idesc_s, ks > 0);
                umma_commit(&s_full[st]);
            }
            __syncwarp();
            BT_EV(k, 4, lane == 0);
            BT_TOC(5);
        }
        if (lane == 0) BT_DUMP(16, 6);
      } else if (warp == kWMma2) {
        // ------------------------------------------------------------------ MMA issuer 2: dQ, dK^T, dV^T
        const bool leader = elect_one();
        constexpr uint32_t idesc_dq = umma_idesc(ElemTraits<ET>::kIsBF16, 128, D, false, true);     // dS (K-major) x K (MN-major)
        constexpr uint32_t idesc_dk = umma_idesc(ElemTraits<ET>::kIsBF16, 128, KT, true, true);     // Q^T / dO^T x dS / P
        constexpr uint32_t hi_1024 = umma_desc_hi(1024);
        const uint32_t ds_k_lo = umma_desc_lo(smem_u32(sDS), 16);                       // dS as K-major A
        const uint32_t ds_mn_lo = umma_desc_lo(smem_u32(sDS), 8192);                    // dS as MN-major B (one slab)
        const uint32_t p_mn_lo = umma_desc_lo(smem_u32(sP), 8192);
        const uint32_t k_mn_lo = umma_desc_lo(smem_u32(sK), KT * 128);                  // K as MN-major B: slabs KT*128 apart
        const uint32_t qd_mn_lo = umma_desc_lo(smem_u32(sQD), kTileRows * 128);         // Q / dO as MN-major A
        int kvn = -1, blk = -1;            // K/V loads, segments
        BT_DECL;
#pragma unroll 1
        for (int k = 0; k < nloc && ok; ++k) {
            const int st = k & 1;
            BT_TOC(0);
            // (the record is complete: its tile has been through the S / dP issuer when P is there)
            ok = ok && mbar_poll(p_full, k & 1);
            BT_EV(k, 9, lane == 0);
            BT_TOC(1);
            const int seg = s_rec[k & 15].x;
            const bool first_of_block = seg & 1, last_of_block = seg & 2;
            if (first_of_block) { ++kvn; ++blk; }
            if (first_of_block && blk > 0) ok = ok && mbar_poll(acc_empty, (blk - 1) & 1);
            BT_TOC(4);
            ok = ok && mbar_poll(&do_full[st], (k >> 1) & 1);     // already complete: acquire only
            ok = ok && mbar_poll(&q_full[st], (k >> 1) & 1);
            ok = ok && mbar_poll(&k_full[kvn % kKStages], (kvn / kKStages) & 1);
            BT_TOC(3);
            fence_async_smem();
            ok = warp_ok(ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t bk = k_mn_lo + (uint32_t)((kvn % kKStages) * (kK >> 4));
            const uint32_t aq = qd_mn_lo + (uint32_t)(st * (kQD >> 4));
            const uint32_t ad = aq + (uint32_t)((kTileRows * D * 2) >> 4);
            // dV, then dK: they are the last readers of the dO and Q rows, which go back to the gather warps as soon as each is
            // done; dQ (which reads dS and K only) follows
            if (leader) {
#pragma unroll 4
                for (int ks = 0; ks < kTileRows / 16; ++ks)
                    umma_ss(tbase + cDV, umma_desc_pack(ad + ks * (2048 >> 4), hi_1024), umma_desc_pack(p_mn_lo + ks * (2048 >> 4), hi_1024),
                            idesc_dk, (!first_of_block || ks > 0) ? 1u : 0u);
                umma_commit(&do_empty[st]);
                umma_commit(p_empty);
            }
            __syncwarp();
            BT_TOC(5);
            ok = ok && mbar_poll(ds_full, k & 1);
            BT_TOC(2);
            fence_async_smem();
            ok = warp_ok(ok);
            if (!ok) break;
            tc_fence_after();
            if (leader) {
#pragma unroll 4
                for (int ks = 0; ks < kTileRows / 16; ++ks)
                    umma_ss(tbase + cDK, umma_desc_pack(aq + ks * (2048 >> 4), hi_1024), umma_desc_pack(ds_mn_lo + ks * (2048 >> 4), hi_1024),
                            idesc_dk, (!first_of_block || ks > 0) ? 1u : 0u);
                umma_commit(&q_empty[st]);
                if (last_of_block) umma_commit(acc_full);
            }
            __syncwarp();
            BT_EV(k, 10, lane == 0);
            ok = ok && mbar_poll(dq_empty, (k & 1) ^ 1);
            BT_EV(k, 11, lane == 0);
            ok = warp_ok(ok);
            if (!ok) break;
            tc_fence_after();
            if (leader) {
#pragma unroll
                for (int ks = 0; ks < KT / 16; ++ks)
                    umma_ss(tbase + cDQ, umma_desc_pack(ds_k_lo + ks * 2, hi_1024), umma_desc_pack(bk + ks * (2048 >> 4), hi_1024),
                            idesc_dq, ks > 0);
                umma_commit(ds_empty);
                umma_commit(dq_full);
                if (last_of_block) umma_commit(&k_empty[kvn % kKStages]);
            }
            __syncwarp();
            BT_EV(k, 12, lane == 0);
            BT_TOC(5);
        }
        if (lane == 0) BT_DUMP(24, 6);
      } else if (warp == kWMma2 + 1) {
        // ------------------------------------------------------------------ tile preparation (tokens of the rows)
        // lane l owns rows l, l + 32, l + 64, l + 96; records and entries are fetched three tiles ahead
        uint32_t gg = 0;                    // head (of the group) of the lane's rows, a byte each
#pragma unroll
        for (int i = 0; i < 4; ++i) gg |= (uint32_t)((lane + 32 * i) / s.TPT) << (8 * i);
        const int qsn8 = (int)(p.q_sn >> 3), dsn8 = (int)(p.do_sn >> 3), qsh8 = (int)(p.q_sh >> 3), dsh8 = (int)(p.do_sh >> 3);
        struct Pre { int h, hg; uint32_t e[4]; };
        TileCursorT<PARTS> ahead(sched), cur_t(sched);
        auto fetch = [&](Pre& m) {
            const TileInfo ti = load_tile(p.ix, ahead.j);
            m.h = ti.h; m.hg = ti.hg;
            const uint32_t* ent = p.ix.entries + (int64_t)ahead.j * s.TPT + lane;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int g = gg >> (8 * i) & 255;
                m.e[i] = g < s.G ? __ldg(ent + 32 * i - g * s.TPT) : 0xFFFFFFFFu;
            }
            ahead.next(sched);
        };
        Pre m1{0, -1, {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}}, m2 = m1, m3 = m1;
        if (nloc > 0) fetch(m1);
        if (nloc > 1) fetch(m2);
        if (nloc > 2) fetch(m3);
        int prev_hg = -1;
#pragma unroll 1
        for (int k = 0; k < nloc && ok; ++k) {
            const int slot = k & 1;
            const Pre cur = m1;
            m1 = m2; m2 = m3;
            if (k + 3 < nloc) fetch(m3);
            ok = ok && mbar_poll(&off_empty[slot], ((k >> 1) & 1) ^ 1);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int hq = cur.h * s.G + (int)(gg >> (8 * i) & 255), tok = (int)(cur.e[i] >> kSlotBits);
                s_off[slot][lane + 32 * i] = cur.e[i] != 0xFFFFFFFFu ? make_int2(tok * qsn8 + hq * qsh8, tok * dsn8 + hq * dsh8) : make_int2(-1, -1);
            }
            if (lane == 0)
                s_rec[k & 15] = make_int4((cur.hg != prev_hg || cur_t.r == 0 ? 1 : 0) | (k + 1 >= nloc || m1.hg != cur.hg || cur_t.r + 1 == sched.run ? 2 : 0),
                                          cur_t.j * nsub + cur_t.sub(sched), cur_t.j, cur_t.run(sched));
            cur_t.next(sched);
            prev_hg = cur.hg;
            ok = warp_ok(ok);
            if (lane == 0) mbar_arrive(&off_full[slot]);
        }
      } else {
        // ------------------------------------------------------------------ K/V blocks by TMA
        int kvn = -1, prev_hg = -1;
        TileInfo t1{0, 0, 0, -1, 0}, t2 = t1;
        TileCursorT<PARTS> ahead(sched), cur_t(sched);
        auto fetch = [&](TileInfo& t) { t = load_tile(p.ix, ahead.j); ahead.next(sched); };
        if (nloc > 0) fetch(t1);
        if (nloc > 1) fetch(t2);
#pragma unroll 1
        for (int k = 0; k < nloc && ok; ++k) {
            const TileInfo cur = t1;
            t1 = t2;
            if (k + 2 < nloc) fetch(t2);
            const int row = cur.row0 + cur_t.sub(sched) * KT;
            const bool first = cur.hg != prev_hg || cur_t.r == 0;     // (every segment loads its K/V block)
            cur_t.next(sched);
            if (!first) continue;
            prev_hg = cur.hg;
            ++kvn;
            if (lane == 0) {
                const int ks = kvn % kKStages;
                ok = ok && mbar_poll(&k_empty[ks], ((kvn / kKStages) & 1) ^ 1);
                if (ok) {
                    mbar_expect_tx(&k_full[ks], (uint32_t)kK);
#pragma unroll
                    for (int b = 0; b < D / 64; ++b) tma_load_2d(smem_u32(sK + ks * kK + b * KT * 128), &kmap, cur.h * D + b * 64, row, &k_full[ks]);
                }
                ok = ok && mbar_poll(v_empty, (kvn & 1) ^ 1);
                if (ok) {
                    mbar_expect_tx(v_full, (uint32_t)kK);
#pragma unroll
                    for (int b = 0; b < D / 64; ++b) tma_load_2d(smem_u32(sV + b * KT * 128), &vmap, cur.h * D + b * 64, row, v_full);
                }
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        }
      }
    } else {
        // ------------------------------------------------------------------ P / dS
        // Both groups work on every tile, each on its 32 of the 64 key columns: the P / dS step sits on the tile's
        // critical path (between the two MMA phases), so its latency counts, not only its throughput.
        reg_inc<kRegGroup>();
        const int sb = (warp - kWGroups) >> 2;
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        const int g = r / s.TPT;
        const int e = r - g * s.TPT;
        const bool row_exists = g < s.G;
        constexpr int HC = KT / 2;              // columns of this group
        const int cb = sb * HC;
        // software pipeline over the tiles: entries two tiles ahead, lse / delta one ahead
        uint32_t entB = 0xFFFFFFFFu;            // entry of tile k + 2
        uint32_t entA = 0xFFFFFFFFu;            // entry of tile k + 1 (after rotation)
        int row0A = 0, row0B = 0, hA = 0, hB = 0;
        float lseA = 0.f, deltaA = 0.f;
        int cloA = 0, chiA = 0;
        auto fetch_ent = [&](int j, uint32_t& ent, int& row0, int& h) {
            TileInfo ti = load_tile(p.ix, j);
            row0 = ti.row0; h = ti.h;
            ent = 0xFFFFFFFFu;
            if (row_exists) ent = __ldg(p.ix.entries + (int64_t)j * s.TPT + e);
        };
        TileCursorT<PARTS> ahead(sched);
        auto fetch = [&](uint32_t& ent, int& row0, int& h) {      // ... and the first key of the tile's part
            fetch_ent(ahead.j, ent, row0, h);
            row0 += ahead.sub(sched) * KT;
            ahead.next(sched);
        };
        auto fetch_stats = [&](uint32_t ent, int h, int row0, float& lse_, float& delta_, int& c_lo, int& c_hi) {
            // padding rows: their Q and dO rows are zero, so they add nothing to dK / dV whatever P is, and their dQ
            // rows are never read: they count as fully visible with lse = delta = 0 (finite values everywhere)
            lse_ = 0.f; delta_ = 0.f; c_lo = 0; c_hi = key_lim;
            if (ent != 0xFFFFFFFFu) {
                const int tok_ = (int)(ent >> kSlotBits);
                const int64_t idx = (int64_t)(h * s.G + g) * s.N + tok_;
                lse_ = __ldg(p.lse + idx);
                delta_ = __ldg(p.delta + idx) * p.scale;
                visible_cols(p.bd, tok_, row0, key_lim, c_lo, c_hi);
            }
        };
        if (nloc > 0) {
            fetch(entA, row0A, hA);
            fetch_stats(entA, hA, row0A, lseA, deltaA, cloA, chiA);
        }
        if (nloc > 1) fetch(entB, row0B, hB);
        BT_DECL;
#pragma unroll 1
        for (int k = 0; k < nloc; ++k) {               // (left by all lanes at the vote below)
            const int st = k & 1;
            const float lse_r = lseA, delta_s = deltaA;
            const int c_lo = cloA, c_hi = chiA;
            // rotate the prefetch registers
            entA = entB; row0A = row0B; hA = hB;
            if (k + 1 < nloc) fetch_stats(entA, hA, row0A, lseA, deltaA, cloA, chiA);
            if (k + 2 < nloc) fetch(entB, row0B, hB);
            BT_TOC(0);
            // most tiles are fully visible to all their rows (only a token's own block is cut by causality)
            const bool all_visible = __all_sync(0xffffffffu, ok && c_lo == 0 && c_hi == KT);
            if (!all_visible && !warp_stays(ok)) break;
            // dP comes first (its rows are gathered first): scale (dP - delta) is ready when S arrives
            ok = ok && mbar_poll(&dp_full[st], (k >> 1) & 1);
            tc_fence_after();
            uint32_t sv[32], dv[32], pp[HC / 2];
            tmem_ld32(tbase + lane_off + cDP + st * 128 + cb, dv);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) dv[i] = __float_as_uint(fmaf(__uint_as_float(dv[i]), p.scale, -delta_s));
            BT_TOC(5);
            ok = ok && mbar_poll(&s_full[st], (k >> 1) & 1);
            BT_EV(k, 5, sb == 0 && quarter == 0 && lane == 0);
            BT_TOC(1);
            tc_fence_after();
            tmem_ld32(tbase + lane_off + cS + st * 128 + cb, sv);
            tmem_ld_wait();
            tc_fence_before();
            mbar_arrive(&sdp_empty[st]);
#pragma unroll
            for (int i = 0; i < 32; ++i) sv[i] = __float_as_uint(ex2_approx_b(fmaf(__uint_as_float(sv[i]), p.scale_log2, -lse_r)));
            if (!all_visible) {
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
                sv[i >> 1] = ElemTraits<ET>::pack2(p0 * __uint_as_float(dv[i]), p1 * __uint_as_float(dv[i + 1]));      // (dS over what has been read)
            }
            BT_EV(k, 6, sb == 0 && quarter == 0 && lane == 0);
            BT_TOC(2);
            // P first: dV starts while dS is being written
            ok = ok && mbar_poll(p_empty, (k & 1) ^ 1);
            BT_EV(k, 7, sb == 0 && quarter == 0 && lane == 0);
            BT_TOC(3);
#pragma unroll
            for (int c4 = 0; c4 < HC / 8; ++c4)
                *reinterpret_cast<uint4*>(sP + sw128_chunk_off(r, sb * (HC / 8) + c4)) = make_uint4(pp[c4 * 4], pp[c4 * 4 + 1], pp[c4 * 4 + 2], pp[c4 * 4 + 3]);
            fence_async_smem();
            mbar_arrive(p_full);
            BT_TOC(4);
            ok = ok && mbar_poll(ds_empty, (k & 1) ^ 1);
            BT_TOC(3);
#pragma unroll
            for (int c4 = 0; c4 < HC / 8; ++c4)
                *reinterpret_cast<uint4*>(sDS + sw128_chunk_off(r, sb * (HC / 8) + c4)) = make_uint4(sv[c4 * 4], sv[c4 * 4 + 1], sv[c4 * 4 + 2], sv[c4 * 4 + 3]);
            fence_async_smem();
            mbar_arrive(ds_full);
            BT_EV(k, 8, sb == 0 && quarter == 0 && lane == 0);
            BT_TOC(4);
            BT_TOC(6);
        }
        if (quarter == 0 && lane == 0) BT_DUMP(32 + sb * 8, 7);
    }
    if (!ok) atomicMax(status, (int)kStatusWaitTimeout);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, bwdpipe::kCols);
}

template <int D, typename ET>
static cudaError_t launch_pipe(const SelBwdArgs& a, const SelShape& s, const SelIndex& ix, const CUtensorMap& kmap,
                               const CUtensorMap& vmap, const CUtensorMap& dqmap, int num_sms, cudaStream_t stream) {
    SelBwdPipeParams<ET> p;
    p.q = (const ET*)a.q; p.q_sn = a.q_sn; p.q_sh = a.q_sh;
    p.d_o = (const ET*)a.d_o; p.do_sn = a.do_sn; p.do_sh = a.do_sh;
    p.lse = a.lse; p.delta = a.delta;
    p.s = s; p.ix = ix;
    p.scale = a.sm_scale; p.scale_log2 = a.sm_scale * 1.4426950408889634f;
    p.run = s.RB;                      // (long runs: few segments per block)
    p.bd = a.bd;
    p.dq_part = (ET*)a.dq_part; p.slabs = a.slabs;
    p.nsub = s.BK > bwdpipe::KT ? s.BK / bwdpipe::KT : 1;
    auto kern = p.nsub > 1 ? sel_bwd_pipe<D, true, ET> : sel_bwd_pipe<D, false, ET>;
    constexpr int smem = bwdpipe::Cfg<D>::kBytes;
    cudaError_t e = allow_smem((const void*)kern, smem);
    if (e != cudaSuccess) return e;
    prof_begin(2, stream);
    kern<<<num_sms, bwdpipe::kThreads, smem, stream>>>(p, kmap, vmap, dqmap);
    prof_end(2, stream);
    return cudaGetLastError();
}

#ifdef FSA_TIMING
}  // namespace fsa
extern "C" int fsa_debug_read_bwd_timing(unsigned long long* host, int n) {
    return (int)cudaMemcpyFromSymbol(host, fsa::g_bwd_timing, (size_t)n * sizeof(unsigned long long));
}
extern "C" int fsa_debug_read_bwd_trace(unsigned long long* host) {
    return (int)cudaMemcpyFromSymbol(host, fsa::g_bwd_trace, sizeof(fsa::g_bwd_trace));
}
namespace fsa {
#endif

cudaError_t launch_sel_bwd_pipe(int dtype, const SelBwdArgs& a, const SelShape& s, const SelIndex& ix,
                                const CUtensorMap& kmap, const CUtensorMap& vmap, const CUtensorMap& dqmap, int num_sms,
                                cudaStream_t stream) {
    if (s.D == 64)
        return dtype == kBF16 ? launch_pipe<64, __nv_bfloat16>(a, s, ix, kmap, vmap, dqmap, num_sms, stream)
                              : launch_pipe<64, __half>(a, s, ix, kmap, vmap, dqmap, num_sms, stream);
    return dtype == kBF16 ? launch_pipe<128, __nv_bfloat16>(a, s, ix, kmap, vmap, dqmap, num_sms, stream)
                          : launch_pipe<128, __half>(a, s, ix, kmap, vmap, dqmap, num_sms, stream);
}

}  // namespace fsa
