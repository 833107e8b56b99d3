// Blackwell (sm_100a) building blocks as inline PTX: mbarriers with BOUNDED waits, TMA tile loads (each CTA fetches
// its own tiles), tensor-memory allocation, tcgen05 MMA/commit/ld, and shared-memory matrix descriptors.
//
// Every wait on an mbarrier here gives up after a bounded number of polls and reports failure instead of spinning forever: the
// callers raise a status word the host reads (LB_ERR_TIMEOUT) and wind the kernel down. Without a bound of their own are the waits
// that the hardware has as one instruction: tensor-memory allocation (tmem_alloc, tmem_alloc_pair), the cluster barrier (cluster_sync),
// block and named barriers, setmaxnreg.inc, the waits for tensor-memory loads and stores and for bulk copies.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace sm100 {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// The next 1024-byte boundary at or after `p`, which points into shared memory. An offset is added instead of rounding the
// address, so that the compiler still sees where the pointer leads and loads and stores through it are those of shared memory.
// (Through generic pointers every read waits behind stores it might alias. Attention forward and backward, us: 8 x 16 heads x 2048 x
// 64 causal 488 -> 449, 8 x 32 x 4096 x 128 5156 -> 4765; prefill of 2 x 32 heads x 1531 x 128 57.0 -> 54.2.)
__device__ __forceinline__ uint8_t* align_1024(uint8_t* p) { return p + ((0u - smem_u32(p)) & 1023u); }

__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(pred));
    return pred != 0;
}

// ---- mbarrier -----------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// One try: the hardware may suspend the thread until the phase completes or `kSuspendNs` have passed, whichever is
// first. The suspension matters: a warp that spins on a barrier takes issue slots from the warps that work (two CTAs
// share an SM in the attention kernels, and one's waiting warps slowed the other's element-wise work).
constexpr uint32_t kSuspendNs = 20000;
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(kSuspendNs)
        : "memory");
    return ok != 0;
}

// Waits until the phase completes or `budget` cycles of SM clock have passed (by default about a second), checking
// the CTA's abort flag after every (suspended) try so that one role's timeout ends every role's loops. Returns false
// when it gave up (and raises the abort flag).
constexpr long long kWaitCycles = 2000000000LL;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, long long budget = kWaitCycles) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > budget) break;
    }
    *abort_flag = 1;
    return false;
}

// Waits until the last commits aimed at a ring of barriers have arrived, `next` tiles having passed through it: what the producer does
// before it leaves. A commit arrives on its own, and nothing says in which order two of them do, so that a later one's arrival (the
// accumulator's) does not show that an earlier one will not reach shared memory that belongs to another block by then.
template <int STAGES>
__device__ __forceinline__ bool mbar_wait_ring(uint64_t* empty, uint32_t next, volatile int* abort_flag) {
    for (int i = 0; i < STAGES; i++, next++)
        if (!mbar_wait(&empty[next % STAGES], (next / STAGES & 1) ^ 1, abort_flag)) return false;
    return true;
}

// ---- TMA --------------------------------------------------------------------------------------------------
// Tile load into this CTA's shared memory, completion counted in bytes on `bar`. Coordinates innermost first; the
// innermost one times the element size must be a multiple of 16 bytes (callers only pass multiples of the box).
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
// `bytes` contiguous bytes into this CTA's shared memory, counted on `bar`: addresses and size are multiples of 16.
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(smem_dst)), "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---- dynamic work: a running CTA takes over the work of one that has not been launched ----------------------------
// Asks for the next CTA of this grid; the 16-byte answer lands at `slot` and counts on `bar` (expect 16 bytes first).
// Not to be asked again once an answer said that none was left.
__device__ __forceinline__ void next_cta_request(void* slot, uint64_t* bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
                 ::"r"(smem_u32(slot)), "r"(smem_u32(bar))
                 : "memory");
}
// The answer: false when every CTA of the grid has been launched, else the (x) index of the one taken over.
__device__ __forceinline__ bool next_cta_answer(const void* slot, int& x) {
    uint32_t got, cx = 0, cy = 0, cz = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b128 h;\n\t"
        "ld.shared.b128 h, [%4];\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
        "selp.u32 %3, 1, 0, p;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, %1, %2, _}, h;\n\t}"
        : "+r"(cx), "+r"(cy), "+r"(cz), "=r"(got)
        : "r"(smem_u32(slot))
        : "memory");
    x = (int)cx;
    return got != 0;
}

// ---- arithmetic ----
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// ---- registers ----
// Register budget of the calling warpgroup (all four of its warps execute this). An increase draws on what the block was
// launched with and waits until it is there: the warpgroups' budgets may not add up to more.
template <int N>
__device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

// ---- tensor memory ------------------------------------------------------------------------------------------
// Executed by ONE full warp; writes the base address (lane 0, column c) to `smem_out`. `cols` is a power of two >= 32.
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_out, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_out)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem], one CTA, 16-bit inputs: executed by a whole convergent warp, of which the lane with `leader`
// set (elect_one) issues it. The operands then stay in the warp's uniform registers, where the instruction wants them; in a
// branch of one lane every operand of every product is moved there first (head dim 128, forward: 114 cycles per 128 x 128 x 16 product in the issuing thread).
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate, bool leader) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"((uint32_t)leader)
        : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]: the A operand (128 x 16 of 16-bit values per instruction) is read from tensor memory.
__device__ __forceinline__ void mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate, bool leader) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"((uint32_t)leader)
        : "memory");
}
// Arrives on `bar` once every tcgen05.mma issued so far by the leader lane has completed (implies fence::before_thread_sync).
__device__ __forceinline__ void mma_commit(uint64_t* bar, bool leader) {
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "setp.ne.b32 e, %1, 0;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(smem_u32(bar)), "r"((uint32_t)leader)
        : "memory");
}
// mbar_wait of a convergent warp with a warp-uniform answer.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}
// 32 consecutive fp32 columns of this thread's TMEM lane (the warp's 32-lane quarter) into registers.
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 16 consecutive 32-bit columns of this thread's lane from registers into tensor memory.
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
// 8 consecutive 32-bit columns of this thread's lane from registers into tensor memory.
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
// 32 consecutive 32-bit columns of this thread's lane from registers into tensor memory.
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
          "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
          "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- CTA pairs (cta_group::2) -------------------------------------------------------------------------------
// Two CTAs of a cluster, ranks 0 (the leader) and 1, run one MMA over both SMs: each holds its 128 rows of A and
// half of B's columns in shared memory at the same offsets, and receives its 128 accumulator rows in its own tensor
// memory. Only the leader issues MMAs and commits; both CTAs issue their own TMA loads, whose completion bytes are
// counted on the LEADER's barrier.
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Hardware barrier over every thread of the cluster (all threads must call it).
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// `bytes` contiguous bytes of this CTA's shared memory into that of CTA `rank` of the cluster, to where `dst` lies here, counted on the barrier
// at `bar`'s offset there, which alone says when it has arrived. Addresses and size are multiples of 16; fence_proxy_async first by those who
// wrote the source. Neither CTA may leave before it has arrived.
__device__ __forceinline__ void bulk_push(void* dst, const void* src, uint32_t bytes, uint64_t* bar, uint32_t rank) {
    asm volatile(
        "{\n\t.reg .b32 rd, rb;\n\t"
        "mapa.shared::cluster.u32 rd, %0, %4;\n\t"
        "mapa.shared::cluster.u32 rb, %3, %4;\n\t"
        "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [rd], [%1], %2, [rb];\n\t}"
        ::"r"(smem_u32(dst)), "r"(smem_u32(src)), "r"(bytes), "r"(smem_u32(bar)), "r"(rank)
        : "memory");
}
// cluster_sync in two halves, for the end of what other CTAs of the cluster read from this one's shared memory: it orders no memory (a release
// would wait, about a microsecond, for the thread's global stores), but a thread has what it has used of another CTA's when it arrives.
__device__ __forceinline__ void cluster_arrive_done() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_done() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }
// Shared-memory addresses in the cluster window carry the CTA rank from bit 24 up; clearing bit 24 of this CTA's
// barrier address names the barrier at the same offset in the pair's even CTA.
constexpr uint32_t kLeaderMask = 0xFEFFFFFFu;
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar) & kLeaderMask), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
// Arrives on the barrier at `bar`'s offset in CTA `rank` of the cluster. Orders tensor-memory accesses only (with the tcgen05
// fences on both sides): a release at cluster scope would first wait, about a microsecond, for the thread's global stores.
__device__ __forceinline__ void mbar_arrive_cluster(uint64_t* bar, uint32_t rank) {
    asm volatile(
        "{\n\t.reg .b32 ra;\n\t"
        "mapa.shared::cluster.u32 ra, %0, %1;\n\t"
        "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [ra];\n\t}"
        ::"r"(smem_u32(bar)), "r"(rank)
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(kSuspendNs)
        : "memory");
    return ok != 0;
}
// mbar_wait for a barrier that threads of the other CTA arrive on.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (mbar_try_wait_cluster(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > kWaitCycles) break;
    }
    *abort_flag = 1;
    return false;
}
// Tensor-memory allocation of a pair: the same warp of BOTH CTAs executes these, with the same `smem_out` offset.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_out, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_out)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ bool mbar_wait_cluster_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait_cluster(bar, parity, abort_flag));
}
// D[tmem of both CTAs] (+)= A * B over the pair (M = 256: 128 rows per CTA), executed by a whole convergent warp of the leader
// CTA and issued by its lane with `leader` set, as mma_f16.
__device__ __forceinline__ void mma_f16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate, bool leader) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"((uint32_t)leader)
        : "memory");
}
// Arrives on the barrier at `bar`'s offset in every CTA of `cta_mask` once the pair's MMAs issued so far have completed.
__device__ __forceinline__ void mma_commit_pair(uint64_t* bar, uint16_t cta_mask, bool leader) {
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "setp.ne.b32 e, %2, 0;\n\t"
        "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
        ::"r"(smem_u32(bar)), "h"(cta_mask), "r"((uint32_t)leader)
        : "memory");
}

// ---- descriptors --------------------------------------------------------------------------------------------
// Shared-memory matrix descriptor for 128-byte-swizzled tiles (as TMA writes them with CU_TENSOR_MAP_SWIZZLE_128B):
// start address, leading-dimension and stride byte offsets in 16-byte units, descriptor version 1, layout type 2.
//  K-major operand  (rows of 64 k-elements = 128 B): 8-row groups `sbo` bytes apart (1024 for a dense tile); lbo unused.
//  MN-major operand (rows of 64 mn-elements = 128 B, one row per k): 8-k groups `sbo` bytes apart, 64-element mn blocks
//  `lbo` bytes apart.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// The descriptor of the same tile layout `byte_offset` bytes further (a multiple of 16; the address field does not
// overflow inside one CTA's shared memory). One add instead of rebuilding the descriptor: the single MMA-issuing
// thread is otherwise bound by its own integer instructions (measured: 171 cycles per 128x256x16 MMA with
// descriptors rebuilt per instruction, 128 - the tensor pipe's own rate - with descriptors advanced like this).
__device__ __forceinline__ uint64_t desc_advance(uint64_t desc, uint32_t byte_offset) { return desc + (uint64_t)(byte_offset >> 4); }

// Instruction descriptor of tcgen05.mma kind::f16: fp32 accumulate, bf16 (1) or f16 (0) operands, operand majors
// (0 = K-major, 1 = MN-major), N/8 and M/16.
__host__ __device__ constexpr uint32_t make_idesc(int m, int n, bool bf16, bool a_mn_major, bool b_mn_major) {
    return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((a_mn_major ? 1u : 0u) << 15) |
           ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Writes 32 rows x SEGS 16-byte segments - lane l holds row l in w[0..SEGS) - through the warp's staging area in
// shared memory, so that one store instruction covers whole rows of SEGS * 16 contiguous bytes (four 128-byte lines
// for SEGS = 8) instead of one 16-byte piece of 32 different lines. Segments are XOR-swizzled within a row: both the
// row-per-lane writes and the segment-per-lane reads are free of bank conflicts. Called by all lanes of the warp; the first `rows_valid`
// rows are written, the first `segs_valid` segments of each.
// The area is addressed in the shared window: through generic pointers each read waited for the global store before it, which might
// have gone to the same place (64 columns of a 256 x 256 product tile took 3000 cycles, most of them such waits).
constexpr int kStageBytesPerWarp = 4096;
__device__ __forceinline__ void st_shared(uint32_t addr, uint4 x) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x.x), "r"(x.y), "r"(x.z), "r"(x.w) : "memory");
}
__device__ __forceinline__ uint4 ld_shared(uint32_t addr) {
    uint4 x;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(addr) : "memory");
    return x;
}
template <int SEGS>
__device__ __forceinline__ void store_rows_coalesced(uint4* stage, const uint4* w, uint8_t* out0, long long ld_bytes, int rows_valid, int lane,
                                                     int segs_valid = SEGS) {
    constexpr int RP = 32 / SEGS;  // rows per store instruction
    auto swz = [](int row) { return SEGS == 8 ? (row & 7) : ((row >> 1) & 3); };
    const uint32_t area = smem_u32(stage);
    __syncwarp();  // the previous pass has been read out
#pragma unroll
    for (int q = 0; q < SEGS; q++) st_shared(area + (lane * SEGS + (q ^ swz(lane))) * 16, w[q]);
    __syncwarp();
    const int q = lane % SEGS, sub = lane / SEGS;
    uint4 x[SEGS];
#pragma unroll
    for (int t = 0; t < SEGS; t++) x[t] = ld_shared(area + ((t * RP + sub) * SEGS + (q ^ swz(t * RP + sub))) * 16);
    uint8_t* out = out0 + (long long)sub * ld_bytes + q * 16;
#pragma unroll
    for (int t = 0; t < SEGS; t++, out += RP * ld_bytes)
        if (t * RP + sub < rows_valid && q < segs_valid) *(uint4*)out = x[t];
}

}  // namespace sm100
