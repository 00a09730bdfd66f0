// dK and dV of range attention (every token attends one contiguous range of K/V rows: the compressed and the sliding-window
// branch), key-tile-major, for sm_100a and head_dim 128.  In the reference: the dK / dV part of _backward_kernel,
// nsa_ref/ops/compressed_attention.py:193-760, and of flash-attn's backward for the window branch.
//
// The tokens that see one of 128 neighbouring K/V rows are (nearly) neighbours too, so a work item is a tile of 128 K/V rows
// of one sequence x one KV head x a stretch of tokens, and walks the stretch in tiles of <= 128 rows (query head of the GQA
// group, token) that TMA reads in place: no index, no gather.  Everything is computed transposed -- a TMEM lane is a K/V row
// -- so that P^T and dS^T are written over S^T and dP^T in TMEM and feed the products from there, never through shared memory:
//   S^T = K Q^T, dP^T = V dO^T, P = exp2(S c - lse), dS = scale P (dP - delta), dV += P^T dO, dK += dS^T Q.
// S^T / P^T, dP^T / dS^T, dV and dK take 128 columns each: all of TMEM, one buffer of each.  The chains dV(i) -> S(i+1) and
// dK(i) -> dP(i+1) go by halves of a row tile: a row group hands its 64 rows on and gets the next ones without waiting for the
// other group, so that one group's exp2 / dS arithmetic runs under the products of the other.  Each chain has an issuing warp.
//   warp 0       TMA producer: K and V of an item, and Q, dO, Q, dO, ... through a ring of five tiles (32 KB each; a tile
//                comes free when both products that read it are done)
//   warp 1       issues S(i) and dV(i)            warp 2    issues dP(i) and dK(i)
//   warp 3       lse, delta and visible rows of every row of a tile, two stages
//   warps 4..11  one K/V row per thread, half of the tile's rows: P and dS; epilogue: warps 4..7 dV, 8..11 dK
// Items of few tiles would leave SMs idle at the end, items of one K/V tile are of very different length (the first
// compressed rows are seen by the whole sequence): a plan on the device cuts the stretches so that an SM gets about eight.  The
// parts of a K/V tile that was cut go to fp32 slabs that the last kernel adds in order (bit-reproducible); others are written in place.
// A tile takes 3100 cycles where every row sees all K/V rows: its products read 256 KB of shared memory and the loads write 64 KB,
// 2560 cycles (the products alone: 2050).  Tiles that need the mask are bound by the row threads.  Measured at 2 x 32768
// tokens, 32 / 8 heads (window of 512 and compressed branch together): whole tiles in turns 4.19 ms, halves 3.93; at four sequences
// of 777 to 3001 tokens, 16 / 4 heads, 119 -> 106 us (104 -> 110 with the waits of a half's S and dP for the product that reads the P
// or dS in their place; nothing at the larger size, 3.85 ms).
#include "../../include/fsa_sm100.h"
#include <climits>

#include "range_bwd.cuh"

namespace fsa {

int make_tile_map_3d_box(CUtensorMap* map, const void* base, int dtype, int64_t d0, int64_t d1, int64_t d2, int64_t stride1,
                         int64_t stride2, int box1, int box2);
int device_sm_count(int* out);

constexpr int kRkThreads = 384;
constexpr int kRkUnits = 5;             // Q / dO tiles in the ring
constexpr int kRkTile = kTileRows * 128 * 2;

// ------------------------------------------------------------------------------------------------ plan
// Tokens that see a row of a K/V tile: [first, last] over the tokens of its sequence (a CTA per tile; the ranges need not be
// monotone, so every token is looked at: 8 loads in flight per thread, 2 x 128 KB of L2 reads at 32768 tokens).  The last CTA
// zeroes the rows of dk and dv past the last sequence and the status word.
__global__ void __launch_bounds__(512) range_key_tiles(const RangeKvPlan p, uint4* __restrict__ dk, uint4* __restrict__ dv, int* __restrict__ status) {
    __shared__ int s_lo[16], s_hi[16];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (blockIdx.x == gridDim.x - 1) {
        if (tid == 0) *status = kStatusOk;
        const int64_t row16 = (int64_t)p.Hk * 128 / 8;
        for (int64_t i = (int64_t)__ldg(p.cu_k + p.B) * row16 + tid; i < p.Nk * row16; i += blockDim.x) {
            dk[i] = make_uint4(0u, 0u, 0u, 0u);
            dv[i] = make_uint4(0u, 0u, 0u, 0u);
        }
        return;
    }
    int seq, key0, nkeys;
    find_seq_tile(p.cu_k, p.B, kTileRows, (int)blockIdx.x, lane, seq, key0, nkeys);
    if (seq < 0) {
        if (tid == 0) p.tiles[blockIdx.x] = make_int4(0, 0, 0, -1);
        return;
    }
    const int t0 = __ldg(p.cu_q + seq), t1 = __ldg(p.cu_q + seq + 1), k0 = __ldg(p.cu_k + seq), key1 = key0 + nkeys - 1;
    int first = INT_MAX, last = -1;
    for (int base = t0 + tid; base < t1; base += 512 * 8) {
        int l[8], u[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int t = base + j * 512;
            l[j] = t < t1 ? (p.kv_lo ? __ldg(p.kv_lo + t) : k0) : 0;
            u[j] = t < t1 ? __ldg(p.kv_hi + t) : -1;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (u[j] >= l[j] && l[j] <= key1 && u[j] >= key0) { first = min(first, base + j * 512); last = max(last, base + j * 512); }
    }
    first = __reduce_min_sync(0xffffffffu, first);
    last = __reduce_max_sync(0xffffffffu, last);
    if (lane == 0) { s_lo[warp] = first; s_hi[warp] = last; }
    __syncthreads();
    if (warp == 0) {
        first = __reduce_min_sync(0xffffffffu, s_lo[lane & 15]);
        last = __reduce_max_sync(0xffffffffu, s_hi[lane & 15]);
        if (lane == 0) p.tiles[blockIdx.x] = make_int4(key0, nkeys, last >= 0 ? first : 0, last);
    }
}

// Work items from the stretches (one CTA): a tile of n row tiles becomes ceil(n / C) items of about equal length, C the
// smallest length that leaves about p.aim items (times heads), and at least kRkMinTiles: below that an item's epilogue weighs
// more than an idle SM.
__global__ void __launch_bounds__(1024) range_plan_items(const RangeKvPlan p) {
    __shared__ int wa[32], wb[32], wc[32];
    __shared__ long long total;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto row_tiles = [&](const int4& t) { return t.w >= 0 ? (t.w - t.z + p.TPT) / p.TPT : 0; };
    if (tid == 0) total = 0;
    __syncthreads();
    int mine = 0;
    for (int i = tid; i < p.max_tiles; i += 1024) mine += row_tiles(p.tiles[i]);
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) atomicAdd(reinterpret_cast<unsigned long long*>(&total), (unsigned long long)mine);
    __syncthreads();
    const int C = max(kRkMinTiles, (int)((total * p.Hk + p.aim - 1) / p.aim));
    int items = 0, slabs = 0, multi = 0;              // so far
    for (int base = 0; base < p.max_tiles; base += 1024) {
        const int i = base + tid;
        const int4 t = i < p.max_tiles ? p.tiles[i] : make_int4(0, 0, 0, -1);
        const int n = row_tiles(t);
        const int nch = t.y > 0 ? max(1, (n + C - 1) / C) : 0;
        const int a = nch, b = nch > 1 ? nch : 0, c = nch > 1;
        int sa = a, sb = b, sc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int ta = __shfl_up_sync(0xffffffffu, sa, o), tb = __shfl_up_sync(0xffffffffu, sb, o), tc = __shfl_up_sync(0xffffffffu, sc, o);
            if (lane >= o) { sa += ta; sb += tb; sc += tc; }
        }
        if (lane == 31) { wa[warp] = sa; wb[warp] = sb; wc[warp] = sc; }
        __syncthreads();
        const int va = wa[lane], vb = wb[lane], vc = wc[lane];
        const int first = items + __reduce_add_sync(0xffffffffu, lane < warp ? va : 0) + sa - a;
        const int slab = slabs + __reduce_add_sync(0xffffffffu, lane < warp ? vb : 0) + sb - b;
        const int list = multi + __reduce_add_sync(0xffffffffu, lane < warp ? vc : 0) + sc - c;
        for (int j = 0; j < nch; ++j) {
            const int r0 = (int)((int64_t)n * j / nch), r1 = (int)((int64_t)n * (j + 1) / nch);
            p.items[first + j] = make_int4(i, r0, r1 - r0, nch > 1 ? slab + j : -1);
        }
        if (nch > 1) p.multi[list] = make_int4(t.x, t.y, slab, nch);
        items += __reduce_add_sync(0xffffffffu, va);
        slabs += __reduce_add_sync(0xffffffffu, vb);
        multi += __reduce_add_sync(0xffffffffu, vc);
        __syncthreads();
    }
    if (tid == 0) { p.counts[0] = items; p.counts[1] = multi; }
}

// dk / dv rows of the K/V tiles that were cut: the sum of the slabs in order.  Slab: [dV, dK][column / 4][row] float4.
template <typename ET>
__global__ void __launch_bounds__(256) range_dkdv_reduce(const RangeKvPlan p, const float4* __restrict__ slabs, ET* __restrict__ dk, ET* __restrict__ dv) {
    const int64_t units = (int64_t)__ldg(p.counts + 1) * p.Hk * 16;       // 2 x 16 x 128 chunks of 8 columns per tile and head, 256 a CTA
    for (int64_t w = blockIdx.x; w < units; w += gridDim.x) {
        const int part = (int)(w & 15), h = (int)((w >> 4) % p.Hk);
        const int4 m = __ldg(p.multi + (w >> 4) / p.Hk);
        const int u = part * 256 + threadIdx.x, key = u & 127, chunk = (u >> 7) & 15, which = u >> 11;
        if (key >= m.y) continue;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const float4* src = slabs + ((int64_t)m.z * p.Hk + h) * (2 * 32 * 128) + (which * 32 + chunk * 2) * 128 + key;
        const int64_t stride = (int64_t)p.Hk * (2 * 32 * 128);
#pragma unroll 4
        for (int j = 0; j < m.w; ++j) {
            const float4 x = __ldcs(src + j * stride), y = __ldcs(src + j * stride + 128);
            acc[0] += x.x; acc[1] += x.y; acc[2] += x.z; acc[3] += x.w;
            acc[4] += y.x; acc[5] += y.y; acc[6] += y.z; acc[7] += y.w;
        }
        ET* dst = (which ? dk : dv) + ((int64_t)(m.x + key) * p.Hk + h) * 128 + chunk * 8;
        *reinterpret_cast<uint4*>(dst) = make_uint4(ElemTraits<ET>::pack2(acc[0], acc[1]), ElemTraits<ET>::pack2(acc[2], acc[3]),
                                                    ElemTraits<ET>::pack2(acc[4], acc[5]), ElemTraits<ET>::pack2(acc[6], acc[7]));
    }
}

// ------------------------------------------------------------------------------------------------ dK and dV
struct RangeKvParams {
    RangeKvPlan plan;
    int Hq, G;
    float scale, scale_log2;
    const float* lse;       // [Hq, N] log2 units
    const float* delta;     // [Hq, N]
    float4* slabs;
    void *dk, *dv;          // [Nk, Hk, 128] contiguous
    int* status;
};

// One work item: K/V rows [key0, key0 + nkeys) of head h, n row tiles of TPT tokens from tok0 on, tokens up to tok_last.
struct RkItem {
    int h, key0, nkeys, tok0, tok_last, n, slab;
};
__device__ __forceinline__ RkItem rk_item(const RangeKvPlan& p, int w) {
    RkItem m;
    const int4 it = __ldg(p.items + w / p.Hk);
    const int4 t = __ldg(p.tiles + it.x);
    m.h = w % p.Hk;
    m.key0 = t.x; m.nkeys = t.y;
    m.tok0 = t.z + it.y * p.TPT;
    m.tok_last = min(t.w, m.tok0 + it.z * p.TPT - 1);
    m.n = it.z;
    m.slab = it.w;
    return m;
}

__device__ __forceinline__ float rk_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <typename ET>
__global__ void __launch_bounds__(kRkThreads, 1) range_bwd_dkdv(const RangeKvParams p, const __grid_constant__ CUtensorMap qmap,
                                                               const __grid_constant__ CUtensorMap domap,
                                                               const __grid_constant__ CUtensorMap kmap,
                                                               const __grid_constant__ CUtensorMap vmap) {
    constexpr int D = 128;
    constexpr int kSlab = kTileRows * 128;           // 64 columns of a tile
    constexpr int cS = 0, cP = 128, cDV = 256, cDK = 384;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sK = smem;
    uint8_t* sV = sK + kRkTile;
    uint8_t* sU = sV + kRkTile;                      // [kRkUnits] Q, dO, Q, dO, ...
    float* sLse = reinterpret_cast<float*>(sU + kRkUnits * kRkTile);      // [2][128]
    float* sDel = sLse + 2 * 128;                                         // [2][128] scale * delta
    uint8_t* sVis = reinterpret_cast<uint8_t*>(sDel + 2 * 128);           // [2][2][128] first visible row; last one | 128
    uint64_t* bars = reinterpret_cast<uint64_t*>(sVis + 4 * 128);
    uint64_t* k_full = bars;            // K of an item has landed
    uint64_t* k_empty = bars + 1;       // ... has been read by the item's last S product
    uint64_t* v_full = bars + 2;
    uint64_t* v_empty = bars + 3;
    uint64_t* u_full = bars + 4;                     // [units]
    uint64_t* u_empty = u_full + kRkUnits;           // [units] the two products that read a Q or dO tile are done
    uint64_t* st_full = u_empty + kRkUnits;          // [2]
    uint64_t* st_empty = st_full + 2;                // [2]
    uint64_t* s_full = st_empty + 2;    // [2 halves] S(i) is done
    uint64_t* p_full = s_full + 2;      // [2] P(i) is in its place
    uint64_t* dp_full = s_full + 4;     // [2]
    uint64_t* ds_full = s_full + 6;     // [2]
    uint64_t* dv_done = s_full + 8;     // the item's last dV product is done
    uint64_t* dk_done = s_full + 9;
    uint64_t* dv_free = s_full + 10;    // the accumulator has been read
    uint64_t* dk_free = s_full + 11;
    uint64_t* p_read = s_full + 12;     // [2 halves] dV(i) has read P
    uint64_t* ds_read = s_full + 14;    // [2] dK(i) has read dS
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(s_full + 16);
    int* s_masked = reinterpret_cast<int*>(s_full + 16) + 2;              // [2] some row of the tile does not see all K/V rows

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int* status = p.status;
    if (tid == 0) {
        mbar_init(k_full, 1); mbar_init(k_empty, 1); mbar_init(v_full, 1); mbar_init(v_empty, 1);
        for (int i = 0; i < kRkUnits; ++i) { mbar_init(&u_full[i], 1); mbar_init(&u_empty[i], 2); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&st_full[i], 32); mbar_init(&st_empty[i], 256);
            mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 128); mbar_init(&dp_full[i], 1); mbar_init(&ds_full[i], 128);
            mbar_init(&p_read[i], 1); mbar_init(&ds_read[i], 1);
        }
        mbar_init(dv_done, 1); mbar_init(dk_done, 1); mbar_init(dv_free, 128); mbar_init(dk_free, 128);
        mbar_init_fence();
        tma_prefetch_desc(&qmap);
        tma_prefetch_desc(&domap);
        tma_prefetch_desc(&kmap);
        tma_prefetch_desc(&vmap);
    }
    // rows past G * TPT of a Q or dO tile are never loaded, but they are multiplied (by P = dS = 0)
    for (int i = p.G * p.plan.TPT * 8 + tid; i < kTileRows * 8; i += kRkThreads)
        for (int u = 0; u < 2 * kRkUnits; ++u) reinterpret_cast<uint4*>(sU + u * kSlab)[i] = make_uint4(0u, 0u, 0u, 0u);
    fence_async_smem();
    if (warp == 0) tmem_alloc(&tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tmem_slot;
    const int nitems = __ldg(p.plan.counts) * p.plan.Hk;
    const int TPT = p.plan.TPT;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            bool ok = true;
            int u = 0, qi = 0;             // Q / dO tiles and non-empty items so far
            const uint32_t unit_bytes = (uint32_t)(2 * 128 * TPT * p.G);
            for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
                const RkItem m = rk_item(p.plan, w);
                if (m.n == 0) continue;
                auto load_unit = [&](const CUtensorMap* map, int tok) {
                    const int st = u % kRkUnits;
                    ok = ok && mbar_wait(&u_empty[st], ((u / kRkUnits) & 1) ^ 1, status);
                    if (!ok) return;
                    mbar_expect_tx(&u_full[st], unit_bytes);
#pragma unroll
                    for (int b = 0; b < 2; ++b) tma_load_3d(smem_u32(sU + st * kRkTile + b * kSlab), map, b * 64, tok, m.h * p.G, &u_full[st]);
                    ++u;
                };
                auto load_kv = [&](const CUtensorMap* map, uint8_t* dst, uint64_t* full, uint64_t* empty) {
                    ok = ok && mbar_wait(empty, (qi & 1) ^ 1, status);
                    if (!ok) return;
                    mbar_expect_tx(full, (uint32_t)kRkTile);
#pragma unroll
                    for (int b = 0; b < 2; ++b)
#pragma unroll
                        for (int r = 0; r < 2; ++r)
                            tma_load_2d(smem_u32(dst + b * kSlab + r * (kSlab / 2)), map, m.h * D + b * 64, m.key0 + r * 64, full);
                };
                load_kv(&kmap, sK, k_full, k_empty);
                load_unit(&qmap, m.tok0);
                load_kv(&vmap, sV, v_full, v_empty);
                load_unit(&domap, m.tok0);
                for (int i = 1; i < m.n && ok; ++i) {
                    load_unit(&qmap, m.tok0 + i * TPT);
                    load_unit(&domap, m.tok0 + i * TPT);
                }
                ++qi;
            }
        }
    } else if (warp == 1 || warp == 2) {
        // ------------------------------------------------------------------ MMA issuers: warp 1 S and dV, warp 2 dP and dK
        const bool first = warp == 1;
        const bool leader = elect_one();
        constexpr uint32_t idesc_s = umma_idesc(ElemTraits<ET>::kIsBF16, 128, 64, false, false);
        constexpr uint32_t idesc_acc = umma_idesc(ElemTraits<ET>::kIsBF16, 128, D, false, true);     // P^T / dS^T (TMEM) x dO / Q (MN-major)
        constexpr uint32_t hi_1024 = umma_desc_hi(1024);
        const uint32_t a_lo = umma_desc_lo(smem_u32(first ? sK : sV), 16);
        const uint32_t b_lo = umma_desc_lo(smem_u32(sU), 16);
        const uint32_t b_mn_lo = umma_desc_lo(smem_u32(sU), kSlab);
        const uint32_t c_s = tbase + (first ? cS : cP), c_acc = tbase + (first ? cDV : cDK);
        uint64_t *kv_full = first ? k_full : v_full, *kv_empty = first ? k_empty : v_empty;
        uint64_t *out_full = first ? s_full : dp_full, *in_full = first ? p_full : ds_full, *in_read = first ? p_read : ds_read;
        uint64_t *acc_done = first ? dv_done : dk_done, *acc_free = first ? dv_free : dk_free;
        bool ok = true;
        int c = 0, qi = 0;
        // S^T (dP^T) of half a row tile t into its place, when the product that reads P^T (dS^T) of the tile before from there is done
        // (products of two shapes may run in another order than they were issued)
        auto issue_s = [&](int t, int half, bool last) {
            const int u = 2 * t + (first ? 0 : 1), st = u % kRkUnits;
            if (half == 0) ok = ok && mbar_wait(&u_full[st], (u / kRkUnits) & 1, status);
            if (t > 0) ok = ok && mbar_wait(&in_read[half], (t - 1) & 1, status);
            ok = warp_ok(ok);
            if (!ok) return;
            tc_fence_after();
            if (leader) {
                const uint32_t bu = b_lo + (uint32_t)(st * (kRkTile >> 4) + half * (8192 >> 4));
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    const uint32_t off = (ks >> 2) * (kSlab >> 4) + (ks & 3) * 2;
                    umma_ss(c_s + half * 64, umma_desc_pack(a_lo + off, hi_1024), umma_desc_pack(bu + off, hi_1024), idesc_s, ks > 0);
                }
                umma_commit(&out_full[half]);
                if (half) umma_commit(&u_empty[st]);
                if (half && last) umma_commit(kv_empty);
            }
            __syncwarp();
        };
        for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
            const RkItem m = rk_item(p.plan, w);
            if (m.n == 0) continue;
            ok = ok && mbar_wait(kv_full, qi & 1, status);
            issue_s(c, 0, m.n == 1);
            issue_s(c, 1, m.n == 1);
            for (int i = 0; i < m.n && ok; ++i, ++c) {
                const int u = 2 * c + (first ? 1 : 0), st = u % kRkUnits;       // dV takes dO, dK takes Q
                ok = ok && mbar_wait(&u_full[st], (u / kRkUnits) & 1, status);
                if (i == 0 && qi > 0) ok = ok && mbar_wait(acc_free, (qi - 1) & 1, status);
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    ok = ok && mbar_wait(&in_full[half], c & 1, status);
                    ok = warp_ok(ok);
                    if (!ok) break;
                    tc_fence_after();
                    if (leader) {
                        const uint32_t bu = b_mn_lo + (uint32_t)(st * (kRkTile >> 4) + half * (8192 >> 4));
#pragma unroll
                        for (int ks = 0; ks < kTileRows / 32; ++ks)
                            umma_ts(c_acc, c_s + half * 64 + ks * 8, umma_desc_pack(bu + ks * (2048 >> 4), hi_1024), idesc_acc,
                                    (i > 0 || half > 0 || ks > 0) ? 1u : 0u);
                        umma_commit(&in_read[half]);
                        if (half) umma_commit(&u_empty[st]);
                        if (half && i + 1 == m.n) umma_commit(acc_done);
                    }
                    __syncwarp();
                    if (i + 1 < m.n) issue_s(c + 1, half, i + 2 == m.n);
                }
            }
            ++qi;
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------------ per-row numbers of the tiles
        bool ok = true;
        int c = 0;
        int g[4], e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) { g[j] = (lane + 32 * j) / TPT; e[j] = lane + 32 * j - g[j] * TPT; }
        for (int w = blockIdx.x; w < nitems && warp_stays(ok); w += gridDim.x) {
            const RkItem m = rk_item(p.plan, w);
            for (int i = 0; i < m.n && warp_stays(ok); ++i, ++c) {
                float lse[4], del[4];
                int lo[4], hi[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int tok = m.tok0 + i * TPT + e[j];
                    lse[j] = INFINITY; del[j] = 0.f; lo[j] = 0; hi[j] = -1;
                    if (g[j] < p.G && tok <= m.tok_last) {
                        const int64_t idx = (int64_t)(m.h * p.G + g[j]) * p.plan.N + tok;
                        lse[j] = __ldg(p.lse + idx);
                        del[j] = __ldg(p.delta + idx) * p.scale;
                        lo[j] = p.plan.kv_lo ? __ldg(p.plan.kv_lo + tok) : m.key0;      // (without kv_lo: the sequence's first row)
                        hi[j] = __ldg(p.plan.kv_hi + tok);
                    }
                }
                bool masked = false;
                int vis[4][2];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int l = max(lo[j] - m.key0, 0), u = min(hi[j] - m.key0, kTileRows - 1);
                    const bool sees = u >= l && lse[j] > -INFINITY && lse[j] < INFINITY;     // a row that saw nothing in the forward sees nothing here
                    masked |= sees && (l > 0 || u < m.nkeys - 1);
                    if (!sees) { lse[j] = INFINITY; del[j] = 0.f; }                          // exp2(s - inf) = 0
                    vis[j][0] = sees ? l : kTileRows - 1;
                    vis[j][1] = sees ? u | 128 : 128;
                }
                masked = __any_sync(0xffffffffu, masked);
                const int b = c & 1;
                ok = ok && mbar_wait(&st_empty[b], ((c >> 1) & 1) ^ 1, status);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    sLse[b * 128 + lane + 32 * j] = lse[j];
                    sDel[b * 128 + lane + 32 * j] = del[j];
                    sVis[b * 256 + lane + 32 * j] = (uint8_t)vis[j][0];
                    sVis[b * 256 + 128 + lane + 32 * j] = (uint8_t)vis[j][1];
                }
                if (lane == 0) s_masked[b] = masked;
                mbar_arrive(&st_full[b]);
            }
        }
    } else {
        // ------------------------------------------------------------------ P, dS and the epilogue: one K/V row, half the tile's rows
        const int grp = (warp - 4) >> 2;
        const int quarter = warp & 3;
        const int key = quarter * 32 + lane;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        const uint32_t tS = tbase + lane_off + cS + grp * 64, tP = tbase + lane_off + cP + grp * 64;
        bool ok = true;
        int c = 0, qi = 0;
        for (int w = blockIdx.x; w < nitems && warp_stays(ok); w += gridDim.x) {
            const RkItem m = rk_item(p.plan, w);
            for (int i = 0; i < m.n && warp_stays(ok); ++i, ++c) {
                const int b = c & 1;
                ok = ok && mbar_wait(&st_full[b], (c >> 1) & 1, status);
                ok = ok && mbar_wait(&s_full[grp], c & 1, status);
                tc_fence_after();
                const bool masked = s_masked[b] != 0;
                const float4* lse4 = reinterpret_cast<const float4*>(sLse + b * 128 + grp * 64);
                const float4* del4 = reinterpret_cast<const float4*>(sDel + b * 128 + grp * 64);
                uint32_t v[64];
                tmem_ld32(tS, *reinterpret_cast<uint32_t (*)[32]>(&v[0]));
                tmem_ld32(tS + 32, *reinterpret_cast<uint32_t (*)[32]>(&v[32]));
                tmem_ld_wait();
                uint32_t pk[32];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float4 l = lse4[j];
                    float x0 = rk_ex2(fmaf(__uint_as_float(v[4 * j]), p.scale_log2, -l.x));
                    float x1 = rk_ex2(fmaf(__uint_as_float(v[4 * j + 1]), p.scale_log2, -l.y));
                    float x2 = rk_ex2(fmaf(__uint_as_float(v[4 * j + 2]), p.scale_log2, -l.z));
                    float x3 = rk_ex2(fmaf(__uint_as_float(v[4 * j + 3]), p.scale_log2, -l.w));
                    v[4 * j] = __float_as_uint(x0); v[4 * j + 1] = __float_as_uint(x1);
                    v[4 * j + 2] = __float_as_uint(x2); v[4 * j + 3] = __float_as_uint(x3);
                }
                if (masked) {
                    // four rows at a time: bit 7 of a byte of (128 | key) - first says key >= first, of (128 | last) - key that key <= last
                    const uint32_t key4 = (uint32_t)key * 0x01010101u;
                    const uint4* first4 = reinterpret_cast<const uint4*>(sVis + b * 256 + grp * 64);
                    const uint4* last4 = first4 + 8;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint4 f = first4[j], l = last4[j];
                        const uint32_t seen[4] = {((key4 | 0x80808080u) - f.x) & (l.x - key4), ((key4 | 0x80808080u) - f.y) & (l.y - key4),
                                                  ((key4 | 0x80808080u) - f.z) & (l.z - key4), ((key4 | 0x80808080u) - f.w) & (l.w - key4)};
#pragma unroll
                        for (int q = 0; q < 16; ++q)
                            if (!(seen[q >> 2] & (0x80u << ((q & 3) * 8)))) v[16 * j + q] = 0u;
                    }
                }
#pragma unroll
                for (int j = 0; j < 32; ++j) pk[j] = ElemTraits<ET>::pack2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                tmem_st32(tS, pk);
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&p_full[grp]);
                ok = ok && mbar_wait(&dp_full[grp], c & 1, status);
                tc_fence_after();
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    uint32_t d[32], dd[16];
                    tmem_ld32(tP + hf * 32, d);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float4 dl = del4[hf * 8 + j];
                        const int k4 = hf * 32 + 4 * j;
                        dd[2 * j] = ElemTraits<ET>::pack2(__uint_as_float(v[k4]) * fmaf(__uint_as_float(d[4 * j]), p.scale, -dl.x),
                                                          __uint_as_float(v[k4 + 1]) * fmaf(__uint_as_float(d[4 * j + 1]), p.scale, -dl.y));
                        dd[2 * j + 1] = ElemTraits<ET>::pack2(__uint_as_float(v[k4 + 2]) * fmaf(__uint_as_float(d[4 * j + 2]), p.scale, -dl.z),
                                                              __uint_as_float(v[k4 + 3]) * fmaf(__uint_as_float(d[4 * j + 3]), p.scale, -dl.w));
                    }
                    tmem_st16(tP + hf * 16, dd);
                }
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&ds_full[grp]);
                mbar_arrive(&st_empty[b]);
            }
            // ---- epilogue of the item: group 0 dV, group 1 dK
            if (m.n > 0) {
                ok = ok && mbar_wait(grp ? dk_done : dv_done, qi & 1, status);
                tc_fence_after();
            }
            const bool write = ok && key < m.nkeys;
            ET* dst = reinterpret_cast<ET*>(grp ? p.dk : p.dv) + ((int64_t)(m.key0 + key) * p.plan.Hk + m.h) * D;
            float4* slab = p.slabs + ((int64_t)m.slab * p.plan.Hk + m.h) * (2 * 32 * 128) + grp * (32 * 128) + key;
#pragma unroll
            for (int c0 = 0; c0 < D; c0 += 32) {
                uint32_t a[32];
                if (m.n > 0) {
                    tmem_ld32(tbase + lane_off + (grp ? cDK : cDV) + c0, a);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) a[j] = 0u;
                }
                if (c0 + 32 == D && m.n > 0) {
                    tc_fence_before();
                    mbar_arrive(grp ? dk_free : dv_free);            // the accumulator may take the next item
                }
                if (write && m.slab >= 0) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        slab[(c0 / 4 + j) * 128] = make_float4(__uint_as_float(a[4 * j]), __uint_as_float(a[4 * j + 1]),
                                                               __uint_as_float(a[4 * j + 2]), __uint_as_float(a[4 * j + 3]));
                } else if (write) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        *reinterpret_cast<uint4*>(dst + c0 + 8 * j) =
                            make_uint4(ElemTraits<ET>::pack2(__uint_as_float(a[8 * j]), __uint_as_float(a[8 * j + 1])),
                                       ElemTraits<ET>::pack2(__uint_as_float(a[8 * j + 2]), __uint_as_float(a[8 * j + 3])),
                                       ElemTraits<ET>::pack2(__uint_as_float(a[8 * j + 4]), __uint_as_float(a[8 * j + 5])),
                                       ElemTraits<ET>::pack2(__uint_as_float(a[8 * j + 6]), __uint_as_float(a[8 * j + 7])));
                }
            }
            if (m.n > 0) ++qi;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, 512);
}

cudaError_t launch_range_bwd_plan(const RangeKvPlan& p, const SelBwdArgs& a, int* status, cudaStream_t stream) {
    range_key_tiles<<<(unsigned)p.max_tiles + 1, 512, 0, stream>>>(p, (uint4*)a.dk, (uint4*)a.dv, status);
    range_plan_items<<<1, 1024, 0, stream>>>(p);
    return cudaGetLastError();
}

template <typename ET>
static cudaError_t launch_rk(const RangeKvParams& p, const CUtensorMap& qmap, const CUtensorMap& domap, const CUtensorMap& kmap, const CUtensorMap& vmap,
                             int sms, int64_t max_items, cudaStream_t stream) {
    constexpr int smem = (2 + kRkUnits) * kRkTile + 2 * 128 * (4 + 4 + 2) + 512;
    auto kern = range_bwd_dkdv<ET>;
    cudaError_t e = allow_smem((const void*)kern, smem);
    if (e != cudaSuccess) return e;
    prof_begin(FSA_KERNEL_SEL_BWD_MAIN, stream);
    kern<<<(unsigned)(max_items < sms ? max_items : sms), kRkThreads, smem, stream>>>(p, qmap, domap, kmap, vmap);
    prof_end(FSA_KERNEL_SEL_BWD_MAIN, stream);
    e = prefer_l1((const void*)range_dkdv_reduce<ET>);
    if (e != cudaSuccess) return e;
    range_dkdv_reduce<ET><<<(unsigned)(4 * sms), 256, 0, stream>>>(p.plan, (const float4*)p.slabs, (ET*)p.dk, (ET*)p.dv);
    return cudaGetLastError();
}

cudaError_t launch_range_bwd_dkdv(int dtype, const RangeKvPlan& plan, const SelBwdArgs& a, const SelShape& s, const CUtensorMap& kmap,
                                  const CUtensorMap& vmap, int* status, cudaStream_t stream) {
    CUtensorMap qmap, domap;
    if (make_tile_map_3d_box(&qmap, a.q, dtype, 128, s.N, s.Hq, a.q_sn, a.q_sh, s.TPT, s.G)) return cudaErrorInvalidValue;
    if (make_tile_map_3d_box(&domap, a.d_o, dtype, 128, s.N, s.Hq, a.do_sn, a.do_sh, s.TPT, s.G)) return cudaErrorInvalidValue;
    RangeKvParams p;
    p.plan = plan;
    p.Hq = s.Hq; p.G = s.G;
    p.scale = a.sm_scale; p.scale_log2 = a.sm_scale * 1.4426950408889634f;
    p.lse = a.lse; p.delta = a.delta; p.slabs = (float4*)a.slabs; p.dk = a.dk; p.dv = a.dv; p.status = status;
    int sms = 0;
    if (device_sm_count(&sms) != 0 || sms <= 0) return cudaErrorInvalidValue;
    const int64_t max_items = (range_kv_max_tiles(s) + range_kv_max_cut(s)) * s.Hk;
    return dtype == kBF16 ? launch_rk<__nv_bfloat16>(p, qmap, domap, kmap, vmap, sms, max_items, stream)
                          : launch_rk<__half>(p, qmap, domap, kmap, vmap, sms, max_items, stream);
}

}  // namespace fsa
