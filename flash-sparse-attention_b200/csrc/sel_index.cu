// Index inversion for selected attention: from topk_idx[Hk, N, T] (token -> KV blocks) build the CSR
// "KV block -> (token, slot) entries", cut into the tiles the persistent kernels walk, and the inverse map `pos`.
// Replaces the reference's block_to_token / index_mapping kernels, its bincount + boolean-mask compaction
// (fsa/ops/FSA_topk_sparse_attention.py:60-135, 622-668, 951-1020) and, for the backward, reorder_topk_idx
// (nsa_ref/ops/topk_sparse_attention.py:412-476): one structure serves forward and backward, its size is O(N*Hk*T),
// and no step syncs with the host.
//
// The build is a counting sort without global atomics, so the same input always gives the same list (the backward's
// dK / dV sums depend on the order of the entries):
//   1. count   one CTA per (kv head, chunk of C tokens): its warps take contiguous token ranges of the chunk and count
//              the entries per block into private shared-memory histograms; the chunk's totals go to chunk_cnt;
//   2. keys    one thread per (kv head, block): exclusive prefix of chunk_cnt over the chunks (every chunk's first
//              position inside the key) and the key's total;
//   3. scan    one CTA: first tile and first segment of every key;
//   4. fill    the CTAs of step 1 again: tile records and the padding of a key's last tile (a warp per key); then every warp's
//              first position inside each key is known, and a second pass over the same tokens writes entries and positions.
// Where a thread has few chunks to add up, step 3 does step 2 as well (a launch costs about 4 us of a short build).
// Entries of a key are in ascending order of (chunk, warp range, 32-token group): ascending token groups, and inside a group
// ascending tokens (short lists without repeated ids), else slot by slot.
// Short problems run all steps in one launch (sel_index_small).
#include <cooperative_groups.h>

#include "sel_launch.cuh"

namespace fsa {

constexpr int kIdxMaxWarps = 8;     // (8 warps x 512-token chunks keep four CTAs resident per SM: the kernels are latency-bound)
constexpr int kIdxMaxSlots = 16;   // top-k lists up to this length are held in registers

// Count (FILL = false: hw[gb] += entries) or place (FILL = true: hw[gb] is this warp's next position in the
// tile-ordered entry list) the entries of this warp's share of the chunk [n0, n1).
// Bound by the latency of a warp's chain through shared memory.  Counts are shared-memory adds that nothing waits for.  To place
// a group of 32 tokens, every lane sets its bit in the word mk[gb] of each of its blocks; a token's place among the
// group's entries of a block is the number of bits below its own, so the slots do not wait for one another: three round trips
// a group.  (Slot by slot, with __match_any_sync and a running position, took 16 dependent rounds: 89 us for 3661 tokens x 2
// heads in the one-launch build.)  A list that names a block twice finds the bit set already; its group, long lists,
// ranges and tables of more keys than have room for mk (null) go slot by slot.
template <bool FILL>
__device__ __forceinline__ void chunk_pass(const int* __restrict__ topk_idx, const int* __restrict__ cu, const SelBounds& bd,
                                           const SelShape& s, const SelIndex& ix, int h, int c, int n0, int n1, int* hw, unsigned* mk,
                                           int warp, int nwarps, int lane) {
    const int ngroups = (n1 - n0 + 31) >> 5;
    const int gpw = (ngroups + nwarps - 1) / nwarps;
    const int g_lo = warp * gpw, g_hi = min(ngroups, g_lo + gpw);
    const bool list = bd.kv_hi == nullptr;
    const bool in_regs = list && s.T <= kIdxMaxSlots, by4 = (s.T & 3) == 0 && (reinterpret_cast<uintptr_t>(topk_idx) & 15) == 0;
    const unsigned lt = (1u << lane) - 1;
    auto store_pos = [&](const int (&ids)[kIdxMaxSlots], int n) {
        int* prow = ix.pos + ((int64_t)h * s.N + n) * s.T;
        if (!by4) {
#pragma unroll
            for (int j = 0; j < kIdxMaxSlots; ++j)
                if (j < s.T) prow[j] = ids[j];
        }
#pragma unroll
        for (int i = 0; i < kIdxMaxSlots / 4; ++i)
            if (by4 && i * 4 < s.T) reinterpret_cast<int4*>(prow)[i] = make_int4(ids[i * 4], ids[i * 4 + 1], ids[i * 4 + 2], ids[i * 4 + 3]);
    };
    for (int g = g_lo; g < g_hi; ++g) {
        const int n = n0 + g * 32 + lane;
        const bool active = n < n1;
        TokenCtx tc{0, 0, 0, 0, -1, 0};
        if (active) tc = token_ctx(cu, bd, s.B, s.BK, n);
        const int* row = topk_idx + ((int64_t)h * s.N + n) * s.T;
        int ids[kIdxMaxSlots];
        if (in_regs && active) {
            // the whole list in one round trip (by4: rows are 16-byte aligned)
            if (!by4) {
#pragma unroll
                for (int j = 0; j < kIdxMaxSlots; ++j) ids[j] = j < s.T ? __ldg(row + j) : -1;
            }
#pragma unroll
            for (int i = 0; i < kIdxMaxSlots / 4; ++i) {
                if (by4 && i * 4 < s.T) {
                    const int4 v = __ldg(reinterpret_cast<const int4*>(row) + i);
                    ids[i * 4] = v.x; ids[i * 4 + 1] = v.y; ids[i * 4 + 2] = v.z; ids[i * 4 + 3] = v.w;
                }
            }
        }
        if (FILL && in_regs && mk) {
            int gb[kIdxMaxSlots];
            unsigned twice = 0;
#pragma unroll
            for (int j = 0; j < kIdxMaxSlots; ++j) {
                int r0;
                gb[j] = active && j < s.T ? entry_block_ctx(tc, bd, s.BK, n, j, ids[j], &r0) : -1;
                if (gb[j] >= 0) twice |= atomicOr(&mk[gb[j]], 1u << lane) >> lane & 1u;
            }
            __syncwarp();
            const bool again = __any_sync(0xffffffffu, twice);
            unsigned leads = 0;                    // slots in which this lane is the first of its block's entries
#pragma unroll
            for (int j = 0; j < kIdxMaxSlots; ++j) {
                const int key = gb[j];
                if (key >= 0 && !again) {
                    const unsigned m = mk[key];
                    const int ps = hw[key] + __popc(m & lt);
                    if ((m & lt) == 0) leads |= 1u << j;
                    ix.entries[ps] = ((uint32_t)n << kSlotBits) | (uint32_t)j;
                    ids[j] = ps;
                } else if (!again) {
                    ids[j] = -1;
                }
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < kIdxMaxSlots; ++j) {
                if (again ? gb[j] >= 0 : (leads >> j & 1u) != 0) {
                    if (!again) hw[gb[j]] += __popc(mk[gb[j]]);
                    mk[gb[j]] = 0u;
                }
            }
            __syncwarp();
            if (!again) {
                if (active) store_pos(ids, n);
                continue;
            }
        }
#pragma unroll 1
        for (int sl0 = 0; sl0 < s.T; sl0 += kIdxMaxSlots) {
#pragma unroll
            for (int j = 0; j < kIdxMaxSlots; ++j) {
                const int sl = sl0 + j;
                if (sl >= s.T) break;
                int r0 = 0;
                const int id = !active ? -1 : in_regs ? ids[j] : list ? __ldg(row + sl) : 0;
                int gb = active ? entry_block_ctx(tc, bd, s.BK, n, sl, id, &r0) : -1;
                if (gb >= s.NBmax) {   // only a malformed range can do this: skip the entry, record it (once: the header is
                    if (FILL) atomicMax(ix.header, (int)kStatusBadIndex);      // cleared between the two passes)
                    gb = -1;
                }
                if (!FILL) {
                    if (gb >= 0) atomicAdd(&hw[gb], 1);
                } else {
                    __syncwarp();
                    const unsigned m = __match_any_sync(0xffffffffu, gb);
                    const int leader = __ffs(m) - 1;
                    int base = 0;
                    if (gb >= 0 && lane == leader) {
                        base = hw[gb];
                        hw[gb] = base + __popc(m);
                    }
                    base = __shfl_sync(m, base, leader);
                    if (active) {
                        int ps = -1;
                        if (gb >= 0) {
                            ps = base + __popc(m & lt);
                            ix.entries[ps] = ((uint32_t)n << kSlotBits) | (uint32_t)sl;
                        }
                        if (in_regs) ids[j] = ps;      // the slot's id is used up: keep its position, written as whole rows below
                        else ix.pos[((int64_t)h * s.N + n) * s.T + sl] = ps;
                    }
                    __syncwarp();
                }
            }
        }
        if (FILL && in_regs && active) store_pos(ids, n);
    }
}

// Tile records of one key (a warp), and the unused slots of its last tile.
__device__ __forceinline__ void write_tiles(const SelShape& s, const SelIndex& ix, const int* __restrict__ ck, int h, int gb, int cnt,
                                            int t0, int seg0, int lane) {
    const int hg = h * s.NBmax + gb, nt = (cnt + s.TPT - 1) / s.TPT;
    const int row0 = block_rows(ck, s.B, s.BK, gb).x;
    for (int t = lane; t < nt; t += 32) {
        ix.tile_rec[t0 + t] = make_int4(row0, min(s.TPT, cnt - t * s.TPT) | (h << 8), hg, seg0);
        ix.tile_aux[t0 + t] = make_int2(t0, nt);
    }
    const int used = cnt - (nt - 1) * s.TPT;
    for (int e = used + lane; e < s.TPT; e += 32) ix.entries[(int64_t)(t0 + nt - 1) * s.TPT + e] = 0xFFFFFFFFu;
}

// Is there room for the words of lane bits?
constexpr int kIdxSmem = 200 * 1024;
__host__ __device__ __forceinline__ bool sel_index_masks(const SelShape& s, int nwarps) {
    return (int64_t)nwarps * s.NBmax * 8 <= kIdxSmem && s.T <= kIdxMaxSlots;
}

// Step 1 (FILL = false) and step 4 (FILL = true).
template <bool FILL>
__global__ void __launch_bounds__(kIdxMaxWarps * 32) sel_index_chunk(const int* __restrict__ topk_idx, const int* __restrict__ cu,
                                                                     SelBounds bd, SelShape s, SelIndex ix) {
    extern __shared__ int sm[];   // [nwarps][NBmax] counts or positions, then, if there is room, [nwarps][NBmax] words of lane bits
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nthreads = blockDim.x, nwarps = nthreads >> 5;
    const int c = blockIdx.x, h = blockIdx.y;
    const int n0 = (int)min((int64_t)c * s.C, s.N), n1 = (int)min((int64_t)(c + 1) * s.C, s.N);
    int* cc = ix.chunk_cnt + ((int64_t)h * s.NC + c) * s.NBmax;
    int* wo = ix.warp_off + ((int64_t)h * s.NC + c) * nwarps * s.NBmax;
    if (!FILL) {
        for (int i = tid; i < nwarps * s.NBmax; i += nthreads) sm[i] = 0;
        __syncthreads();
        chunk_pass<false>(topk_idx, cu, bd, s, ix, h, c, n0, n1, sm + warp * s.NBmax, nullptr, warp, nwarps, lane);
        __syncthreads();
        for (int gb = tid; gb < s.NBmax; gb += nthreads) {
            int run = 0;
            for (int i = 0; i < nwarps; ++i) {
                const int v = sm[i * s.NBmax + gb];
                wo[i * s.NBmax + gb] = run;        // this warp's first position inside the key, relative to the chunk
                run += v;
            }
            cc[gb] = run;
        }
    } else {
        // the tile records of this warp's share of the keys
        const int* ck = bd.cu_k ? bd.cu_k : cu;
        for (int gb = c * nwarps + warp; gb < s.NBmax; gb += gridDim.x * nwarps) {
            const int hg = h * s.NBmax + gb, cnt = ix.key_cnt[hg];
            if (cnt > 0) write_tiles(s, ix, ck, h, gb, cnt, ix.key_tile[hg], ix.key_seg[hg], lane);
        }
        // every warp's first position in the tile-ordered entry list: first entry of the key (step 3) + the chunk's first
        // position inside the key (step 2) + the warp's inside the chunk (step 1)
        const int* kt = ix.key_tile + (int64_t)h * s.NBmax;
        for (int gb = tid; gb < s.NBmax; gb += nthreads) {
            const int base = kt[gb] * s.TPT + cc[gb];
            for (int i = 0; i < nwarps; ++i) sm[i * s.NBmax + gb] = base + wo[i * s.NBmax + gb];
        }
        unsigned* mk = sel_index_masks(s, nwarps) ? reinterpret_cast<unsigned*>(sm) + nwarps * s.NBmax : nullptr;
        if (mk)
            for (int i = tid; i < nwarps * s.NBmax; i += nthreads) mk[i] = 0u;
        __syncthreads();
        chunk_pass<true>(topk_idx, cu, bd, s, ix, h, c, n0, n1, sm + warp * s.NBmax, mk ? mk + warp * s.NBmax : nullptr, warp, nwarps, lane);
    }
}

// Exclusive prefix of the chunks' counts of one key, and the total (eight loads in flight).
__device__ __forceinline__ int prefix_chunks(const SelShape& s, const SelIndex& ix, int k) {
    const int h = k / s.NBmax, gb = k - h * s.NBmax;
    int* p = ix.chunk_cnt + (int64_t)h * s.NC * s.NBmax + gb;
    int run = 0;
    for (int c0 = 0; c0 < s.NC; c0 += 8) {
        int v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = c0 + j < s.NC ? p[(int64_t)(c0 + j) * s.NBmax] : 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (c0 + j < s.NC) p[(int64_t)(c0 + j) * s.NBmax] = run;
            run += v[j];
        }
    }
    return run;
}

// Step 2: per key, exclusive prefix of the chunks' counts and the total (thread per key; eight loads in flight).
__global__ void __launch_bounds__(64) sel_index_keys(SelShape s, SelIndex ix) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= s.Hk * s.NBmax) return;
    ix.key_cnt[k] = prefix_chunks(s, ix, k);
}

// Step 3: exclusive scans over the keys (a single CTA): first tile, then -- it depends on the first tile -- first segment.
// A key with tiles [t0, t0 + nt) is cut by the backward's schedule at every multiple of RB.
template <bool KEYS>
__global__ void __launch_bounds__(1024) sel_index_scan(SelShape s, SelIndex ix) {
    __shared__ int wsum_a[32], wsum_b[32], wsum_c[32];
    __shared__ int carry_a, carry_b, carry_c;
    const int HG = s.Hk * s.NBmax;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) { carry_a = 0; carry_b = 0; carry_c = 0; }
    __syncthreads();
    for (int base = 0; base < HG; base += 1024) {
        const int i = base + tid;
        const int a = i >= HG ? 0 : KEYS ? prefix_chunks(s, ix, i) : ix.key_cnt[i];
        if (KEYS && i < HG) ix.key_cnt[i] = a;
        const int b = (a + s.TPT - 1) / s.TPT;
        int sa = a, sb = b;
        for (int o = 1; o < 32; o <<= 1) {
            const int ta = __shfl_up_sync(0xffffffffu, sa, o), tb = __shfl_up_sync(0xffffffffu, sb, o);
            if (lane >= o) { sa += ta; sb += tb; }
        }
        if (lane == 31) { wsum_a[warp] = sa; wsum_b[warp] = sb; }
        __syncthreads();
        if (warp == 0) {
            int va = wsum_a[lane], vb = wsum_b[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int ta = __shfl_up_sync(0xffffffffu, va, o), tb = __shfl_up_sync(0xffffffffu, vb, o);
                if (lane >= o) { va += ta; vb += tb; }
            }
            wsum_a[lane] = va; wsum_b[lane] = vb;
        }
        __syncthreads();
        const int pa = carry_a + (warp ? wsum_a[warp - 1] : 0);
        const int t0 = carry_b + (warp ? wsum_b[warp - 1] : 0) + sb - b;     // first tile of this key
        if (i < HG) ix.key_tile[i] = t0;
        const int cseg = b > 0 ? (t0 + b - 1) / s.RB - t0 / s.RB + 1 : 0;
        int sc = cseg;
        for (int o = 1; o < 32; o <<= 1) {
            const int tc = __shfl_up_sync(0xffffffffu, sc, o);
            if (lane >= o) sc += tc;
        }
        if (lane == 31) wsum_c[warp] = sc;
        __syncthreads();
        if (warp == 0) {
            int vc = wsum_c[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int tc = __shfl_up_sync(0xffffffffu, vc, o);
                if (lane >= o) vc += tc;
            }
            wsum_c[lane] = vc;
        }
        __syncthreads();
        const int pc = carry_c + (warp ? wsum_c[warp - 1] : 0);
        if (i < HG) ix.key_seg[i] = pc + sc - cseg;
        __syncthreads();
        if (tid == 1023) { carry_a = pa + sa; carry_b = t0 + b; carry_c = pc + sc; }
        __syncthreads();
    }
    if (tid == 0) {
        ix.key_tile[HG] = carry_b;
        ix.key_seg[HG] = carry_c;
        ix.header[0] = kStatusOk;
        ix.header[1] = carry_b;
        ix.header[2] = carry_a;
        ix.header[3] = carry_c;
    }
}

// All steps in one launch, for short problems: one CTA per kv head, the CTAs of a cluster exchange the numbers of tiles
// and segments of their heads through distributed shared memory.  What bounds a short build is the latency of its launches
// and dependent steps: 512 tokens x 2 heads took 24 us in five kernels and a memset.  The list is the same one (a warp takes
// a contiguous range of 32-token groups either way).  A head's entries all leave through one SM, scattered, at about one a clock:
// used up to kSmallEntries of them (6 us + 1.1 ns each, against 20-28 us for the launches of the steps), and up to 8 heads (the cluster) and
// kSmallKeys blocks (a thread each).
constexpr int kSmallEntries = 16000, kSmallKeys = 700, kSmallWarps = 32;

// Exclusive prefix of v over the CTA's 1024 threads; *total = the sum.
__device__ __forceinline__ int cta_prefix(int v, int* wsum, int tid, int* total) {
    const int lane = tid & 31, warp = tid >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int base = 0, all = 0;
    const int w = wsum[lane];
    all = __reduce_add_sync(0xffffffffu, w);
    base = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0);
    __syncthreads();
    *total = all;
    return base + incl - v;
}

__global__ void __launch_bounds__(kSmallWarps * 32) sel_index_small(const int* __restrict__ topk_idx, const int* __restrict__ cu, SelBounds bd,
                                                                  SelShape s, SelIndex ix) {
    namespace cg = cooperative_groups;
    extern __shared__ int sm[];   // [warps][NBmax] counts, then positions; [warps][NBmax] lane bits; [NBmax] entries, first tile, first segment of a key
    __shared__ int wsum[32], mine[3];       // tiles, entries, segments of this head
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y, NB = s.NBmax;
    unsigned* mk = reinterpret_cast<unsigned*>(sm) + kSmallWarps * NB;
    int *s_cnt = sm + 2 * kSmallWarps * NB, *s_t0 = s_cnt + NB, *s_seg = s_t0 + NB;
    const int* ck = bd.cu_k ? bd.cu_k : cu;
    for (int i = tid; i < 2 * kSmallWarps * NB; i += blockDim.x) sm[i] = 0;
    __syncthreads();
    chunk_pass<false>(topk_idx, cu, bd, s, ix, h, 0, 0, (int)s.N, sm + warp * NB, nullptr, warp, kSmallWarps, lane);
    __syncthreads();
    // a warp per key: lane w turns warp w's count into its first position inside the key
    for (int gb = warp; gb < NB; gb += kSmallWarps) {
        const int v = sm[lane * NB + gb];
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        sm[lane * NB + gb] = incl - v;
        if (lane == 31) s_cnt[gb] = incl;
    }
    __syncthreads();
    const int cnt = tid < NB ? s_cnt[tid] : 0;
    int entries = 0, tiles = 0, segs = 0;
    cta_prefix(cnt, wsum, tid, &entries);
    const int nt = (cnt + s.TPT - 1) / s.TPT;
    int t0 = cta_prefix(nt, wsum, tid, &tiles);
    // tiles and entries of the heads before this one, and of all
    if (tid == 0) { mine[0] = tiles; mine[1] = entries; }
    cluster.sync();
    const int v0 = lane < s.Hk ? cluster.map_shared_rank(mine, lane)[0] : 0, v1 = lane < s.Hk ? cluster.map_shared_rank(mine, lane)[1] : 0;
    t0 += __reduce_add_sync(0xffffffffu, lane < h ? v0 : 0);
    const int all_tiles = __reduce_add_sync(0xffffffffu, v0), all_entries = __reduce_add_sync(0xffffffffu, v1);
    int seg = cta_prefix(nt > 0 ? (t0 + nt - 1) / s.RB - t0 / s.RB + 1 : 0, wsum, tid, &segs);
    if (tid == 0) mine[2] = segs;
    if (tid == 0 && h == 0) {
        ix.header[0] = kStatusOk; ix.header[1] = all_tiles; ix.header[2] = all_entries;
        ix.key_tile[s.Hk * NB] = all_tiles;
    }
    cluster.sync();
    const int v2 = lane < s.Hk ? cluster.map_shared_rank(mine, lane)[2] : 0;
    seg += __reduce_add_sync(0xffffffffu, lane < h ? v2 : 0);
    const int all_segs = __reduce_add_sync(0xffffffffu, v2);
    cluster.barrier_arrive();                  // (nothing of another CTA is read from here on; none leaves before all have come here)
    if (tid < NB) {
        const int hg = h * NB + tid;
        ix.key_cnt[hg] = cnt; ix.key_tile[hg] = t0; ix.key_seg[hg] = seg;
        s_t0[tid] = t0; s_seg[tid] = seg;
    }
    if (tid == 0 && h == 0) { ix.header[3] = all_segs; ix.key_seg[s.Hk * NB] = all_segs; }
    __syncthreads();
    for (int gb = warp; gb < NB; gb += kSmallWarps)
        if (s_cnt[gb] > 0) write_tiles(s, ix, ck, h, gb, s_cnt[gb], s_t0[gb], s_seg[gb], lane);
    for (int gb = lane; gb < NB; gb += 32) sm[warp * NB + gb] += s_t0[gb] * s.TPT;
    __syncwarp();
    chunk_pass<true>(topk_idx, cu, bd, s, ix, h, 0, 0, (int)s.N, sm + warp * NB, mk + warp * NB, warp, kSmallWarps, lane);
    cluster.barrier_wait();
}

// warps per CTA of the chunk kernels so that the per-warp histograms fit in shared memory; 0: the problem does not fit
int sel_index_warps(const SelShape& s) {
    const int64_t ints = kIdxSmem / 4;
    int64_t nw = ints / (s.NBmax > 0 ? s.NBmax : 1);
    if (nw < 1) return 0;
    if (nw > kIdxMaxWarps) nw = kIdxMaxWarps;
    const int64_t groups = (s.C + 31) / 32;    // no more warps than 32-token groups in a chunk
    if (nw > groups) nw = groups;
    return (int)nw;
}

cudaError_t sel_build_index(const int* topk_idx, const int* cu, const SelBounds& bd, const SelShape& s, const SelIndex& ix,
                            cudaStream_t stream) {
    cudaError_t e;
    if ((int64_t)s.Hk * s.N == 0) return cudaMemsetAsync(ix.header, 0, 64 * 4, stream);
    if (s.N * s.T <= kSmallEntries && s.Hk <= 8 && s.NBmax <= kSmallKeys) {
        const int smem = (2 * kSmallWarps + 3) * s.NBmax * 4;
        e = allow_smem((const void*)sel_index_small, smem);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, (unsigned)s.Hk);
        cfg.blockDim = dim3(kSmallWarps * 32);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = 1; at.val.clusterDim.y = (unsigned)s.Hk; at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, sel_index_small, topk_idx, cu, bd, s, ix);
    }
    const int nw = s.IW;
    if (nw == 0) return cudaErrorInvalidValue;
    const int smem = nw * s.NBmax * 4, smem_fill = sel_index_masks(s, nw) ? 2 * smem : smem;
    e = allow_smem((const void*)sel_index_chunk<false>, smem);
    if (e != cudaSuccess) return e;
    e = allow_smem((const void*)sel_index_chunk<true>, smem_fill);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)s.NC, (unsigned)s.Hk);
    const int HG = s.Hk * s.NBmax;
    sel_index_chunk<false><<<grid, nw * 32, smem, stream>>>(topk_idx, cu, bd, s, ix);
    if ((HG + 1023) / 1024 * s.NC <= 16) {                  // (two rounds of loads a thread)
        sel_index_scan<true><<<1, 1024, 0, stream>>>(s, ix);
    } else {
        sel_index_keys<<<(unsigned)((HG + 63) / 64), 64, 0, stream>>>(s, ix);
        sel_index_scan<false><<<1, 1024, 0, stream>>>(s, ix);
    }
    sel_index_chunk<true><<<grid, nw * 32, smem_fill, stream>>>(topk_idx, cu, bd, s, ix);
    return cudaGetLastError();
}

}  // namespace fsa
