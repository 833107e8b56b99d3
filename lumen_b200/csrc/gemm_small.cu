// 16-bit matrix products too small for 256 x 256 tiles to fill the GPU: 128 x 64 tiles, the K range of a tile cut over a
// thread-block cluster of up to eight CTAs.
//
// What bounds it: the latency of one pass - first TMA load, the ring, the accumulator's way out - and how many SMs pull
// operands meanwhile. A product of 200 x 4096 with K = 1024 has 16 tiles of 256 x 256 (32 of 148 SMs), one of 200 x 1024
// with K = 4096 four. Narrow tiles and split K ranges give every SM work; the partial sums of a tile meet in distributed
// shared memory, added in rank order (no scratch memory, no second kernel, the same bits every run), each CTA of the
// cluster writing its share of the rows in whole 128-byte lines. Where there is room for them to land (one CTA to an SM), a warp's rows are sent
// to the rank whose they are as soon as they are in shared memory; fetched behind a barrier of the cluster, a line at a time, they took a
// microsecond longer: 512^3 6.1 -> 5.3 us, 200 x 1024 K 4096 8.5 -> 7.8, 400 x 1024 K 4096 10.9 -> 10.5, 300 x 512 K 2048 7.1 -> 6.4.
//
// A block runs its last part once, and its instructions come from the L2, so that part is kept short: one conversion of eight columns for each
// type, the operand of an epilogue fetched in one piece before the ranks' sums, which are fetched four ranks at a time, and a kernel without
// clusters where no K range is cut. us a product, before -> so: 200 x 4096 K 1024 8.1 -> 5.9 (with a mask 9.4 -> 6.8), 64^3 4.3 -> 3.1,
// 128 x 8192 K 1024 8.5 -> 6.3, 1024^3 8.5 -> 6.2; with ranges 704 x 1024 K 4096 16.8 -> 14.6, 200 x 1024 K 4096 9.1 -> 8.5.
#include <cuda_fp16.h>

#include "gemm.h"
#include "launch.cuh"
#include "sm100.cuh"

namespace lb {
namespace {

using namespace sm100;

constexpr int BM = 128, BN = 64, BK = 64;
constexpr int kThreads = 192;  // warp 0: TMA, warp 1: MMA + TMEM owner, warps 2..5: accumulator rows; all: sums and stores
constexpr int kStageA = BM * BK * 2, kStageB = BN * BK * 2;
// A load takes about a microsecond to arrive, a stage's products 0.15: eight stages where an SM has one CTA, four where two
constexpr int kLanding = 7 * (BM / 8) * BN * 4;  // the other ranks' sums of this one's rows: most where there are eight
constexpr int smem_bytes(int stages, bool ranks) { return stages * (kStageA + kStageB) + 1024 /*alignment*/ + 256 /*barriers*/ + (stages == 8 && ranks ? kLanding : 0); }
static_assert(smem_bytes(8, true) <= 227 * 1024 && BM / 2 * BN * 4 <= kLanding && 3 * (BM / 4) * BN * 4 <= kLanding, "shared memory");
static_assert(BM * BN * 4 <= 4 * (kStageA + kStageB), "the partial tile takes the drained ring's place");

__device__ __forceinline__ float4 load_cluster(uint32_t addr, uint32_t rank) {
    float4 v;
    asm volatile(
        "{\n\t.reg .b32 ra;\n\t"
        "mapa.shared::cluster.u32 ra, %4, %5;\n\t"
        "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n\t}"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "r"(addr), "r"(rank)
        : "memory");
    return v;
}
// byte offset of 16-byte chunk `c` of row `r` of the partial tile: eight rows' equal chunks fall in different banks
__device__ __forceinline__ uint32_t chunk_at(int r, int c) { return (uint32_t)(r * BN * 4 + ((c ^ (r & 7)) << 4)); }

// RANKS: a tile's K range is cut over a cluster
template <int STAGES, bool RANKS>
__global__ void __launch_bounds__(kThreads, 8 / STAGES)
gemm_small_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const SmallGemmArgs p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align_1024(smem_raw);
    uint8_t *sa = smem, *sb = smem + STAGES * kStageA;
    uint64_t* full = (uint64_t*)(smem + STAGES * (kStageA + kStageB));
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;
    uint64_t* landed = acc_full + 1;
    uint32_t* tmem_slot = (uint32_t*)(landed + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    constexpr bool PUSH = RANKS && STAGES == 8;  // ranks send one another their sums; else (no room to land) they fetch them
    uint8_t* landing = smem + STAGES * (kStageA + kStageB) + 256;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp-uniform for the compiler too
    const int splits = RANKS ? p.splits : 1, rank = RANKS ? (int)cluster_ctarank() : 0, unit = blockIdx.x / splits;
    const int n_blk = unit % p.tiles_n, m_blk = unit / p.tiles_n % p.tiles_m, b = unit / (p.tiles_n * p.tiles_m);
    const int total_kb = (p.K + BK - 1) / BK;
    const int kb0 = total_kb * rank / splits, num_kb = total_kb * (rank + 1) / splits - kb0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(landed, 1);
        *abort_flag = 0;
        fence_barrier_init();
        if (PUSH) mbar_expect_tx(landed, (splits - 1) * (BM / splits) * (BN * 4));
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, BN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    if (PUSH) cluster_sync();  // every rank's barriers are there before anything is sent
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    grid_wait();

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            for (int i = 0; i < num_kb; i++) {
                const int st = i % STAGES, k = (kb0 + i) * BK;
                if (!(ok = mbar_wait(&empty[st], ((uint32_t)(i / STAGES) & 1) ^ 1, abort_flag))) break;
                mbar_expect_tx(&full[st], kStageA + kStageB);
                if (!p.a_mn_major) {
                    tma_load_3d(sa + st * kStageA, &map_a, &full[st], k, m_blk * BM, b);  // box {64 k, 128 m}
                } else {
                    for (int j = 0; j < BM / 64; j++) tma_load_3d(sa + st * kStageA + j * (64 * BK * 2), &map_a, &full[st], m_blk * BM + j * 64, k, b);
                }
                if (!p.b_mn_major) tma_load_3d(sb + st * kStageB, &map_b, &full[st], k, n_blk * BN, b);  // box {64 k, 64 n}
                else tma_load_3d(sb + st * kStageB, &map_b, &full[st], n_blk * BN, k, b);                 // box {64 n, 64 k}
            }
            if (ok) mbar_wait_ring<STAGES>(empty, (uint32_t)num_kb, abort_flag);
        }
    } else if (warp == 1) {  // the whole warp: the operands stay in uniform registers
        const bool leader = elect_one();
        const uint32_t idesc = make_idesc(BM, BN, p.in_bf16 != 0, p.a_mn_major, p.b_mn_major);
        const uint64_t da0 = make_smem_desc(smem_u32(sa), p.a_mn_major ? 64 * BK * 2 : 16, 1024);
        const uint64_t db0 = make_smem_desc(smem_u32(sb), p.b_mn_major ? 64 * BK * 2 : 16, 1024);
        const uint32_t a_step = p.a_mn_major ? 2048u : 32u, b_step = p.b_mn_major ? 2048u : 32u;
        bool ok = true;
        for (int i = 0; i < num_kb && ok; i++) {
            const int st = i % STAGES;
            if (!(ok = mbar_wait_warp(&full[st], (uint32_t)(i / STAGES) & 1, abort_flag))) break;
            tc_fence_after();
            const uint64_t da = desc_advance(da0, (uint32_t)(st * kStageA)), db = desc_advance(db0, (uint32_t)(st * kStageB));
#pragma unroll
            for (int k = 0; k < BK / 16; k++) mma_f16(tmem, desc_advance(da, k * a_step), desc_advance(db, k * b_step), idesc, (i | k) != 0, leader);
            mma_commit(&empty[st], leader);
        }
        if (ok) mma_commit(acc_full, leader);
    } else {
        // every product has completed, so every load has landed: the ring is free for the partial tile
        const int quarter = warp & 3, row = quarter * 32 + lane;
        if (mbar_wait_warp(acc_full, 0, abort_flag)) {
            tc_fence_after();
            uint32_t v[BN];
            tmem_ld_32x32(tmem + ((uint32_t)(quarter * 32) << 16), v);
            tmem_ld_32x32(tmem + ((uint32_t)(quarter * 32) << 16) + 32, v + 32);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < BN / 4; c++) *(uint4*)(smem + chunk_at(row, c)) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
            if (PUSH) {  // a warp's rows go to the rank or, of eight, the two ranks whose they are
                fence_proxy_async();
                __syncwarp();
                const int share = BM / splits, part = min(32, share), r = quarter * 32 + lane * part, to = r / share;
                if (lane * part < 32 && to != rank)
                    bulk_push(landing + ((rank < to ? rank : rank - 1) * share + r % share) * (BN * 4), smem + r * (BN * 4), part * (BN * 4), landed, to);
            }
            tc_fence_before();
        }
    }
    __syncwarp();
    if (RANKS && !PUSH) cluster_sync();
    else __syncthreads();
    if (PUSH) mbar_wait_cluster_warp(landed, 0, abort_flag);

    // this CTA's share of the rows: eight columns per thread
    const int rows = BM / splits;
    const bool good = !*abort_flag;
    for (int i = threadIdx.x; i < rows * (BN / 8); i += kThreads) {
        const int r = rank * rows + i / (BN / 8), q = i % (BN / 8);
        const long long row = (long long)m_blk * BM + r;
        const int col = n_blk * BN + q * 8;
        const int live = good && row < p.M ? min(8, p.N - col) : 0;
        if (live <= 0) continue;
        const bool whole = p.vec && live == 8;
        uint32_t a[4] = {0u, 0u, 0u, 0u};  // the epilogue's operand is on its way while the ranks' sums are
        if (p.epilogue >= EPI_ADD && live > 0) {
            const uint16_t* aux = (const uint16_t*)p.aux + (long long)b * p.aux_batch_stride + row * p.ld_aux + col;
            if (p.aux_vec && live == 8) {
                const uint4 t = *(const uint4*)aux;
                a[0] = t.x, a[1] = t.y, a[2] = t.z, a[3] = t.w;
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (j < live) a[j / 2] |= (uint32_t)aux[j] << (j % 2 * 16);
            }
        }
        const uint32_t at0 = smem_u32(smem) + chunk_at(r, 2 * q), at1 = smem_u32(smem) + chunk_at(r, 2 * q + 1);
        float x[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (PUSH) {
            const uint32_t at = chunk_at(i / (BN / 8), 2 * q), beside = at ^ 16;
            for (int s = 0; s < splits; s++) {
                const uint32_t from = s == rank ? smem_u32(smem) + rank * rows * (BN * 4) : smem_u32(landing) + (s < rank ? s : s - 1) * rows * (BN * 4);
                const uint4 u = ld_shared(from + at), w = ld_shared(from + beside);
                x[0] += __uint_as_float(u.x), x[1] += __uint_as_float(u.y), x[2] += __uint_as_float(u.z), x[3] += __uint_as_float(u.w);
                x[4] += __uint_as_float(w.x), x[5] += __uint_as_float(w.y), x[6] += __uint_as_float(w.z), x[7] += __uint_as_float(w.w);
            }
        } else if (RANKS) {
            for (int s0 = 0; s0 < splits; s0 += 4) {  // up to four ranks' at once
                float4 u[4], w[4];
#pragma unroll
                for (int s = 0; s < 4; s++)
                    if (s0 + s < splits) u[s] = load_cluster(at0, s0 + s), w[s] = load_cluster(at1, s0 + s);
#pragma unroll
                for (int s = 0; s < 4; s++)
                    if (s0 + s < splits) {
                        x[0] += u[s].x, x[1] += u[s].y, x[2] += u[s].z, x[3] += u[s].w;
                        x[4] += w[s].x, x[5] += w[s].y, x[6] += w[s].z, x[7] += w[s].w;
                    }
            }
        } else {
            const uint4 u = ld_shared(at0), w = ld_shared(at1);
            x[0] = __uint_as_float(u.x), x[1] = __uint_as_float(u.y), x[2] = __uint_as_float(u.z), x[3] = __uint_as_float(u.w);
            x[4] = __uint_as_float(w.x), x[5] = __uint_as_float(w.y), x[6] = __uint_as_float(w.z), x[7] = __uint_as_float(w.w);
        }
        if (p.epilogue == EPI_RELU) {
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] = fmaxf(x[j], 0.0f);
        }
        const long long at = (long long)b * p.d_batch_stride + row * p.ldd + col;
        if (p.d_bf16 || p.d_f16) {
            uint32_t h[4];
            if (p.d_bf16) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const __nv_bfloat162 t = __floats2bfloat162_rn(x[2 * j], x[2 * j + 1]);
                    h[j] = *(const uint32_t*)&t;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const __half2 t = __floats2half2_rn(x[2 * j], x[2 * j + 1]);
                    h[j] = *(const uint32_t*)&t;
                }
            }
            if (p.epilogue >= EPI_ADD) {  // 16-bit outputs only; the product is rounded first, as its own primitive
#pragma unroll
                for (int j = 0; j < 4; j++) h[j] = tail_pair(h[j], a[j], p.epilogue == EPI_ADD, p.d_bf16);
            }
            uint16_t* out = (uint16_t*)p.d + at;
            if (whole) {
                *(uint4*)out = make_uint4(h[0], h[1], h[2], h[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (j < live) out[j] = (uint16_t)(h[j / 2] >> (j % 2 * 16));
            }
        } else {
            float* out = (float*)p.d + at;
            if (whole) {
                *(float4*)out = make_float4(x[0], x[1], x[2], x[3]);
                *(float4*)(out + 4) = make_float4(x[4], x[5], x[6], x[7]);
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (j < live) out[j] = x[j];
            }
        }
    }
    __syncwarp();
    if (RANKS) cluster_arrive_done();
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) atomicExch(p.status, LB_ERR_TIMEOUT);
        // give copies and products still in flight a bounded time to land before shared and tensor memory are released
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {
        }
    }
    __syncwarp();
    if (RANKS) cluster_wait_done();  // no CTA leaves while another reads its partial tile, or before what it sent has landed (each has waited for that)
    else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, BN);
    }
}

}  // namespace

template <int STAGES, bool RANKS>
static void launch_small(const CUtensorMap& map_a, const CUtensorMap& map_b, const SmallGemmArgs& p, int batch, cudaStream_t s) {
    if (first_use_on_device((const void*)gemm_small_kernel<STAGES, RANKS>))
        LB_CUDA(cudaFuncSetAttribute(gemm_small_kernel<STAGES, RANKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(STAGES, RANKS)));
    launch_overlapped(gemm_small_kernel<STAGES, RANKS>, dim3((unsigned)((long long)p.tiles_m * p.tiles_n * batch * p.splits)), dim3(kThreads), smem_bytes(STAGES, RANKS), s,
                      (unsigned)p.splits, map_a, map_b, p);
}

void gemm_small(const CUtensorMap& map_a, const CUtensorMap& map_b, SmallGemmArgs p, int batch, int sms, cudaStream_t s) {
    p.tiles_m = (p.M + BM - 1) / BM, p.tiles_n = (p.N + BN - 1) / BN;
    const int per_line = p.d_bf16 || p.d_f16 ? 8 : 4;
    p.aux_vec = (uintptr_t)p.aux % 16 == 0 && p.ld_aux % 8 == 0 && p.aux_batch_stride % 8 == 0;
    p.vec = (uintptr_t)p.d % 16 == 0 && p.ldd % per_line == 0 && p.d_batch_stride % per_line == 0;
    if ((long long)p.tiles_m * p.tiles_n * batch * p.splits > sms) launch_small<4, true>(map_a, map_b, p, batch, s);
    else if (p.splits > 1) launch_small<8, true>(map_a, map_b, p, batch, s);
    else launch_small<8, false>(map_a, map_b, p, batch, s);
}

}  // namespace lb
