// dQ = dS K from the dS that the dK/dV kernel has left in memory (attention_bwd.cu, head dim 128).
//
// The kernel that computed dS again executed three products and the exponentials for the one product that is asked for, at the rate of
// the tensor cores and of its element-wise chain; read back, dS costs four bytes of HBM traffic a score, of which the writing half runs
// under the products of the dK/dV kernel, which leaves the memory idle.
//
// What bounds it: HBM (4.4 GB of dS in 725 us at batch 8, 32 heads, sequence 4096, causal: 94 % of a copy's bandwidth). A CTA takes 256
// queries of a head (two accumulators of 128 x 128 in tensor memory) so that a key tile is fetched from the L2 for two query tiles, walks
// its keys 64 at a time - one copy of up to 32 KB of dS, which lies in memory as the product reads it, and two boxes of K - and two CTAs
// share an SM, so that one's prologue and epilogue lie under the other's loads. Fewer CTAs than twice the SMs take 128 queries each: the
// backward of 1 x 8 heads x 2048 63 -> 53 us, of 1 x 8 x 512 21 -> 18.5.
#include "attention_dq.h"

#include "launch.cuh"
#include "sm100.cuh"

namespace lb {
namespace {

using namespace sm100;

constexpr int D = 128, kKeys = 64;
constexpr int kThreads = 192;  // warp 0: copies, warp 1: products + TMEM owner, warps 2..5: epilogue
constexpr int kStageB = kKeys * D * 2;
// TILES: tiles of 128 queries of a CTA
template <int TILES>
struct DqConfig {
    static constexpr int kStages = TILES == 2 ? 2 : 3;
    static constexpr int kStageA = 2 * TILES * kDsHalfBytes;
    static constexpr int kSmemBytes = kStages * (kStageA + kStageB) + 1024 /*alignment*/ + 256 /*barriers*/;
    static_assert(2 * (kSmemBytes + 1024) <= 227 * 1024, "two CTAs an SM");
};

// An operand whose rows lie eight to 16 bytes, without a swizzle: blocks of 8 rows x 8 of the contracted index are 128 contiguous bytes,
// `mn_bytes` apart along the rows and `k_bytes` along the contracted index.
__device__ __forceinline__ uint64_t plain_desc(uint32_t smem_addr, uint32_t mn_bytes, uint32_t k_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((k_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((mn_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

template <int TILES>
__global__ void __launch_bounds__(kThreads, 2) attention_dq_kernel(const __grid_constant__ CUtensorMap map_k, const DqArgs p) {
    constexpr int STAGES = DqConfig<TILES>::kStages, kStageA = DqConfig<TILES>::kStageA;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align_1024(smem_raw);
    uint8_t *sa = smem, *sb = smem + STAGES * kStageA;
    uint64_t* full = (uint64_t*)(smem + STAGES * (kStageA + kStageB));
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;
    uint32_t* tmem_slot = (uint32_t*)(acc_full + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp-uniform for the compiler too
    const int tile = (int)(gridDim.x - 1 - blockIdx.x);  // the longest first
    const int head = p.head0 + (int)blockIdx.y, batch = p.batch0 + (int)blockIdx.z;
    const int qb0 = tile * 2 * TILES, blocks = min(2 * TILES, p.ds.query_blocks - qb0);  // two or four
    // key tiles that the first and the second 128 queries see: equal, or one more
    const int seen0 = p.ds.tiles_seen(qb0), seen1 = blocks == 4 ? p.ds.tiles_seen(qb0 + 2) : 0;
    const int n_iter = 2 * max(seen0, seen1);
    const uint8_t* scores = p.scores + ((long long)blockIdx.z * p.heads + blockIdx.y) * p.ds.head_bytes();

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        fence_barrier_init();
        tma_prefetch_desc(&map_k);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, TILES * D);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    grid_wait();

    if (warp == 0) {
        if (lane == 0 && n_iter > 0) {
            bool ok = true;
            const int kv_head = head / (p.N / p.Nkv);
            for (int it = 0; it < n_iter && ok; it++) {
                const int st = it % STAGES, j = it >> 1, half = it & 1;
                if (!(ok = mbar_wait(&empty[st], ((uint32_t)(it / STAGES) & 1) ^ 1, abort_flag))) break;
                const int skip = j < seen0 ? 0 : 2, count = (j < seen1 ? 4 : 2) - skip;  // blocks of 64 queries that see the tile
                mbar_expect_tx(&full[st], count * kDsHalfBytes + kStageB);
                bulk_load(sa + st * kStageA + skip * kDsHalfBytes, scores + p.ds.at(j, half, qb0 + skip), count * kDsHalfBytes, &full[st]);
                for (int d = 0; d < D / 64; d++) tma_load_4d(sb + st * kStageB + d * (kKeys * 128), &map_k, &full[st], d * 64, kv_head, it * kKeys, batch);
            }
            if (ok) mbar_wait_ring<STAGES>(empty, (uint32_t)n_iter, abort_flag);
        }
    } else if (warp == 1) {
        if (n_iter > 0) {  // the whole warp: the operands stay in uniform registers
            const bool leader = elect_one();
            const uint32_t idesc = make_idesc(128, D, true, true, true);
            const uint64_t da0 = plain_desc(smem_u32(sa), 1024, 128);
            const uint64_t db0 = make_smem_desc(smem_u32(sb), kKeys * 128, 1024);
            bool ok = true;
            for (int it = 0; it < n_iter && ok; it++) {
                const int st = it % STAGES, j = it >> 1;
                if (!(ok = mbar_wait_warp(&full[st], (uint32_t)(it / STAGES) & 1, abort_flag))) break;
                tc_fence_after();
                const uint64_t da = desc_advance(da0, (uint32_t)(st * kStageA)), db = desc_advance(db0, (uint32_t)(st * kStageB));
                if (j < seen0) {
#pragma unroll
                    for (int k = 0; k < kKeys / 16; k++) mma_f16(tmem, desc_advance(da, k * 256), desc_advance(db, k * 2048), idesc, (it | k) != 0, leader);
                }
                if (TILES == 2 && j < seen1) {
#pragma unroll
                    for (int k = 0; k < kKeys / 16; k++)
                        mma_f16(tmem + D, desc_advance(da, 2 * kDsHalfBytes + k * 256), desc_advance(db, k * 2048), idesc, (it | k) != 0, leader);
                }
                mma_commit(&empty[st], leader);
            }
            if (ok) mma_commit(acc_full, leader);
        }
    } else {
        const int quarter = warp & 3;
        bool ok = true;
        if (n_iter > 0) ok = mbar_wait_warp(acc_full, 0, abort_flag);
        if (ok) {
            tc_fence_after();
            // every product has completed, so every load has landed: a warp's rows leave through 4 KB of the first stage
#pragma unroll 1
            for (int c = 0; c < blocks / 2 * (D / 64); c++) {
                const int sub = c / (D / 64), col = c % (D / 64) * 64;
                const bool any = (sub ? seen1 : seen0) > 0;
                uint32_t v[64];
                tmem_ld_32x32(tmem + ((uint32_t)(quarter * 32) << 16) + sub * D + col, v);
                tmem_ld_32x32(tmem + ((uint32_t)(quarter * 32) << 16) + sub * D + col + 32, v + 32);
                tmem_ld_wait();
                uint4 packed[8];
#pragma unroll
                for (int i = 0; i < 64; i += 8) {
                    uint32_t w[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[i + 2 * q]), __uint_as_float(v[i + 2 * q + 1]));
                        w[q] = any ? *(const uint32_t*)&h : 0u;
                    }
                    packed[i / 8] = make_uint4(w[0], w[1], w[2], w[3]);
                }
                const long long row0 = (long long)tile * (TILES * 128) + sub * 128 + quarter * 32;
                uint8_t* out = (uint8_t*)((uint16_t*)p.dq + batch * p.sb + row0 * p.ss + head * p.sn + col);
                store_rows_coalesced<8>((uint4*)(sa + (warp - 2) * kStageBytesPerWarp), packed, out, p.ss * 2, (int)max(0LL, min(32LL, p.Sq - row0)), lane);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) atomicExch(p.status, LB_ERR_TIMEOUT);
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {
        }
        __syncthreads();
    }
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, TILES * D);
    }
}

}  // namespace

template <int TILES>
static void launch_dq(const CUtensorMap& keys, int batches, const DqArgs& p, cudaStream_t s) {
    if (first_use_on_device((const void*)attention_dq_kernel<TILES>))
        LB_CUDA(cudaFuncSetAttribute(attention_dq_kernel<TILES>, cudaFuncAttributeMaxDynamicSharedMemorySize, DqConfig<TILES>::kSmemBytes));
    launch_overlapped(attention_dq_kernel<TILES>, dim3((unsigned)((p.Sq + TILES * 128 - 1) / (TILES * 128)), (unsigned)p.heads, (unsigned)batches), dim3(kThreads),
                      DqConfig<TILES>::kSmemBytes, s, 0, keys, p);
}

void attention_dq_launch(const CUtensorMap& keys, int batches, const DqArgs& p, cudaStream_t s) {
    const long long ctas = (long long)(p.Sq + 255) / 256 * p.heads * batches;
    if (ctas >= 2 * device_info().sms) launch_dq<2>(keys, batches, p, s);
    else launch_dq<1>(keys, batches, p, s);
}

}  // namespace lb
