// Blackwell (sm_100a) primitives used by every tensor-core kernel in this library:
// mbarrier (with bounded waits), TMA tiled loads, tcgen05 MMA / TMEM access, and the
// shared-memory layouts the UMMA descriptors describe.
//
// Shared-memory operand tiles use the 128-byte swizzle: a tile is a stack of rows of
// 128 bytes (64 16-bit elements); 8 rows form a 1024-byte atom; inside an atom the
// 16-byte chunk c of row r is stored at chunk position (c ^ (r & 7)).  Tile bases are
// 1024-byte aligned so that "row & 7" equals address bits [7,10), which is what both the
// TMA engine and the tensor core use when they swizzle.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace fsa {

// Host side of every launch (fsa_api.cu).
// cudaFuncSetAttribute(MaxDynamicSharedMemorySize), once per thread, device and kernel (the driver call costs about as much
// as a launch)
cudaError_t allow_smem(const void* kern, int bytes);
// Gives a kernel that streams from global memory and has no shared memory to speak of the whole L1 (once per thread, device and
// kernel).  Without a preference the SMs keep the split of the kernel before, and after one with 227 KB of shared memory the
// 28 KB that are left hold too few loads in flight: the merges of the partial rows took 467 us instead of 390 us (16K tokens,
// 32 heads, 16 rows each).
// smem_percent: the share that stays shared memory, for a kernel that uses some.
cudaError_t prefer_l1(const void* kern, int smem_percent = 0);
// SMs of this process's device, for the rules that sizes and launches share; a B200's where no device answers (size queries need none).
int sm_count();
// Launch of a kernel that begins with follow(): its CTAs are brought up, and its weights fetched, while the kernel before it ends.
// cluster: CTAs (in x) of a cluster.
template <typename... KA, typename... A>
static inline cudaError_t launch_dependent(void (*kern)(KA...), dim3 grid, unsigned block, size_t smem, cudaStream_t stream, unsigned cluster, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[2] = {};
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KA>(args)...);
}
// Binds the current device's primary context to the calling thread: tensor-map encoding is a driver call and needs one.
int ensure_context();

// ----------------------------------------------------------------------------------------
// status word: kernels never trap and never spin forever.  A wait that runs out records
// where it gave up; the host reads the word after the launch.
// ----------------------------------------------------------------------------------------
enum : int {
    kStatusOk = 0,
    kStatusWaitTimeout = 1,    // an mbarrier wait ran out of iterations
    kStatusBadIndex = 2,       // an index outside its table was seen and skipped
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// One lane of a fully converged warp (predicate true in exactly one lane).  Code that must be
// issued by a single thread (tcgen05.mma, TMA) is wrapped in `if (elect_one())` inside
// warp-uniform control flow, so that addresses and descriptors stay in uniform registers.
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(pred));
    return pred != 0;
}

// ---------------------------------------------------------------- dependent launches
// A kernel launched by launch_dependent (below) may start while the one before it in the stream still runs.  Every thread of it calls
// follow() before it reads or writes anything of a kernel before it, and before it may return: from there on all of them have
// ended and their writes are seen.  The kernel after it may start from then on too, so that only one kernel is ever ahead.  What the
// kernel before wrote is not read through the non-coherent path (__ldg, const __restrict__): such a load may be moved before this.
__device__ __forceinline__ void follow() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok;
}
__device__ __forceinline__ uint32_t clock32() {
    uint32_t t;
    asm volatile("mov.u32 %0, %%clock;" : "=r"(t)::"memory");
    return t;
}
// Bounded wait: polls until the phase completes or `limit` cycles of the SM have passed (each try_wait already sleeps for a
// while in hardware) and returns false in the second case.  A role's first wait that runs out is its last (`ok = ok && ...`): from
// there on it issues nothing and uses no address that the wait was for, and leaves its loop, so that TMEM is freed and the
// kernel returns.  mbar_wait records the failure in the status word; mbar_poll leaves that to the caller, once for all its
// waits.  Kept short on purpose: a warp-specialised kernel has some 25 waits, and the loops of its roles together have to
// stay in the SM's instruction cache (sel_bwd_pipe.cu).
#ifndef FSA_WAIT_CLOCKS
#define FSA_WAIT_CLOCKS 400000000u   // 0.2 s at 1.965 GHz; less than the 2^32 at which the counter comes round
#endif
__device__ __forceinline__ bool mbar_poll(uint64_t* bar, uint32_t parity, uint32_t limit = FSA_WAIT_CLOCKS) {
    const uint32_t t0 = clock32();
#pragma unroll 1
    do {
        if (mbar_try_wait(bar, parity)) return true;
    } while (clock32() - t0 < limit);
    return false;
}
// The limit of a CTA's waits in kernels of many waves of CTAs: 3 ms where the status word says that a wait has run out already (of a
// CTA before it, as far as the launch's word was zero).  Read once, by every thread for itself, and not waited for until a wait is slow.
__device__ __forceinline__ uint32_t wait_limit(const int* status) {
    const int failed = status ? *reinterpret_cast<const volatile int*>(status) : 0;
    return failed ? FSA_WAIT_CLOCKS / 64 : FSA_WAIT_CLOCKS;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status, uint32_t limit = FSA_WAIT_CLOCKS) {
    if (mbar_poll(bar, parity, limit)) return true;
    if (status) atomicMax(status, (int)kStatusWaitTimeout);
    return false;
}

// Whether no wait of any lane of a warp has run out, for all its lanes alike.  Stands between waits that the whole warp makes and what an
// elected lane then issues or announces: a phase that this leads to may be the next one of a barrier just waited for, and a lane that
// has yet to look at the one before would see its parity gone by and wait until its limit.  And a lane that gave up must not
// leave a loop in which the others go on to meet it.  (The vote alone does not order the lanes' accesses to shared memory.)
__device__ __forceinline__ bool warp_ok(bool ok) {
    const bool all = __all_sync(0xffffffffu, ok);
    __syncwarp();
    return all;
}

// The condition of a loop in which the lanes of a warp meet (TMEM accesses, votes, shuffles) while each of them waits for itself: they
// leave it together.  A lane that gave up alone would leave the others to wait for it without end.  (A loop that votes in each turn on
// something else counts `!ok` there and asks this only then: a vote more between two tiles cost the row threads up to 1 %.)
__device__ __forceinline__ bool warp_stays(bool& ok) {
    ok = __all_sync(0xffffffffu, ok);
    return ok;
}

// Barrier `id` of `threads` threads that tells whether v held for all of them.
__device__ __forceinline__ bool bar_all(int id, int threads, bool v) {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all) : "r"((uint32_t)v), "r"(id), "r"(threads) : "memory");
    return all != 0;
}

// ---------------------------------------------------------------- proxies / fences
// Generic-proxy writes to shared memory (st.shared, cp.async) must be made visible to the
// async proxy (TMA, tcgen05.mma operand reads) before those engines read them.
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---------------------------------------------------------------- cp.async (16-byte gathers)
__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void* src, bool valid) {
    int sz = valid ? 16 : 0;   // src-size 0 zero-fills the 16 bytes
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst_smem), "l"(src), "r"(sz) : "memory");
}
// The mbarrier receives one arrival (counted in its expected count) when all cp.async issued so
// far by this thread have completed; the thread itself does not wait.
__device__ __forceinline__ void cp_async_mbar_arrive_noinc(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A hint: the line of p into L2.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ---------------------------------------------------------------- TMA
// 2-D tiled load: box of the tensor map starting at (x = innermost element, y = row).
// x * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(uint32_t dst_smem, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
// 3-D tiled load: box starting at (x = innermost element, y, z).  x * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_3d(uint32_t dst_smem, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
// 2-D tiled store smem -> global (bulk async-group completion).  x and y must be non-negative.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, uint32_t src_smem) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(src_smem)
                 : "memory");
}
// 3-D tiled store smem -> global.  Coordinates must be non-negative.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, int x, int y, int z, uint32_t src_smem) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(z), "r"(src_smem)
                 : "memory");
}
// L2 eviction policies for data with a known lifetime: evict_first for rows that are written once and read once much
// later (they should not push anything else out), evict_last for lines that are completed by many small writes.
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void st_float2_hint(float2* ptr, float a, float b, uint64_t policy) {
    asm volatile("st.global.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;" ::"l"(ptr), "f"(a), "f"(b), "l"(policy) : "memory");
}
// 2-D tiled store with an L2 policy
__device__ __forceinline__ void tma_store_2d_hint(const CUtensorMap* map, int x, int y, uint32_t src_smem, uint64_t policy) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group.L2::cache_hint [%0, {%1, %2}], [%3], %4;" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(src_smem), "l"(policy)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// all but the newest 0 groups have finished READING their smem source
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bulk_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// ---------------------------------------------------------------- TMEM
// Allocation is a warp-wide operation; ncols is a power of two in [32, 512].
__device__ __forceinline__ void tmem_alloc(uint32_t* slot_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_smem)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 32 lanes x 32 bit: thread i of warp w reads TMEM lane 32*(w%4)+i, N consecutive columns.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------- UMMA descriptors
// Shared-memory matrix descriptor, 128-byte swizzle.
//   bits [0,14)  start address >> 4
//   bits [16,30) leading-dimension byte offset >> 4
//   bits [32,46) stride-dimension byte offset >> 4
//   bits [46,48) descriptor version (1 on sm_100)
//   bits [61,64) layout type (2 = 128-byte swizzle)
// K-major operand (rows = M or N index, 128 bytes of K per row): SBO = 1024 (next 8 rows);
// the leading offset is not used by the hardware for swizzled K-major tiles.
// MN-major operand (rows = K index, 128 bytes = 64 MN elements per row): SBO = 1024 (next
// 8 K rows), LBO = distance between consecutive 64-element MN slabs.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// The same descriptor split for cheap per-k-step updates: the high word is constant for a tile
// layout, the low word is (address >> 4) | (lbo >> 4) << 16 and advances by (bytes >> 4).
__device__ __forceinline__ constexpr uint32_t umma_desc_hi(uint32_t sbo_bytes) {
    return ((sbo_bytes >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
}
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
    return ((smem_addr & 0x3FFFFu) >> 4) | (((lbo_bytes >> 4) & 0x3FFFu) << 16);
}
__device__ __forceinline__ uint64_t umma_desc_pack(uint32_t lo, uint32_t hi) {
    return ((uint64_t)hi << 32) | lo;
}

// Instruction descriptor for kind::f16 (fp16/bf16 inputs, fp32 accumulate).
//   bits [4,6) D format (1 = f32); [7,10) A format; [10,13) B format (0 = f16, 1 = bf16)
//   bit 15 A major, bit 16 B major (0 = K-major, 1 = MN-major)
//   bits [17,23) N >> 3; bits [24,29) M >> 4
__host__ __device__ constexpr uint32_t umma_idesc(bool bf16, int M, int N, bool a_mn_major, bool b_mn_major) {
    return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((a_mn_major ? 1u : 0u) << 15) |
           ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]; one thread issues for the whole CTA.
__device__ __forceinline__ void umma_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Make the mbarrier track completion of all MMAs issued so far by this thread.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// ---------------------------------------------------------------- swizzled tile addressing
// Byte offset of the 16-byte chunk `chunk` (0..7) of row `row` inside a 128-byte-swizzled tile.
__device__ __forceinline__ uint32_t sw128_chunk_off(int row, int chunk) {
    return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4));
}

// ---------------------------------------------------------------- register budgets of warpgroups
template <int N> __device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

// ---------------------------------------------------------------- element types
template <typename ET> struct ElemTraits;
template <> struct ElemTraits<__nv_bfloat16> {
    static constexpr bool kIsBF16 = true;
    __device__ static __forceinline__ uint32_t pack2(float lo, float hi) {
        __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&v);
    }
    __device__ static __forceinline__ float2 unpack2(uint32_t u) {
        return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
    }
};
template <> struct ElemTraits<__half> {
    static constexpr bool kIsBF16 = false;
    __device__ static __forceinline__ uint32_t pack2(float lo, float hi) {
        __half2 v = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&v);
    }
    __device__ static __forceinline__ float2 unpack2(uint32_t u) {
        return __half22float2(*reinterpret_cast<__half2*>(&u));
    }
};

}  // namespace fsa
