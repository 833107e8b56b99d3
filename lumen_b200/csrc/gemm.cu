// GEMM for lumen's dot_general (one contracting dimension, optional leading batch), the counterpart of the
// reference's Ampere `mma.sync` CuTe kernel behind its GEMM hook (lumen/codegen/dot_general/cuda/ampere.py:35-904,
// lumen/codegen/dot_general/cuda/mod.rs:658-757) rebuilt for Blackwell:
//
//  * gemm_tcgen05: 16-bit operands, explicit fp32 accumulation in tensor memory. Persistent, warp-specialised:
//    warp 0 issues TMA tile loads into a 4-stage ring of 128-byte-swizzled shared-memory tiles, warp 1 (its elected lane)
//    issues tcgen05.mma (128x256x16 per instruction) and commits stage/accumulator barriers, warps 2-9 drain the
//    previous tile's accumulator (tcgen05.ld) through the epilogue while the next tile's MMAs run into the other
//    half of the 512 TMEM columns. All four operand majors (row- or column-major A and B) are handled by the tensor
//    maps and the descriptor major bits, so the transposed *views* of the backward GEMMs (dA = dY.B^T, dB = A^T.dY)
//    need no copies. Every CTA loads its own operand tiles.
//  * gemm_simt: any float dtype and any strides, one thread per output element group, products and partial sums
//    rounded to fp32 one by one in contracting order (__fmul_rn / __fadd_rn): exactly the reference interpreter's
//    accumulation (lumen/reference/mod.rs:958-970). float32 operands always take this path: there is no hidden
//    TF32/bf16 narrowing.
#include <algorithm>
#include <map>
#include <mutex>

#include "gemm.h"
#include "launch.cuh"
#include "sm100.cuh"

namespace lb {
namespace {

using namespace sm100;

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 4;
constexpr int kThreads = 320;  // warp 0: TMA, warp 1: MMA + TMEM owner, warps 2..9: epilogue
constexpr int kEpilogueWarps = 8;
constexpr int kStageBytesA = BM * BK * 2, kStageBytesB = BN * BK * 2;
constexpr int kEpilogueStageBytes = 8 * 4096;  // one 4 KB staging area per epilogue warp (store_rows_coalesced)
constexpr int kSmemBytes = STAGES * (kStageBytesA + kStageBytesB) + 1024 /*alignment slack*/ + 256 /*barriers*/ + kEpilogueStageBytes;

// n / d for 0 <= n < 2^31 as a multiply and a shift (Granlund and Montgomery's round-up method): where a tile lies is worked out by
// every warp between two tiles, and six integer divisions took 1200 cycles there.
struct Divisor {
    uint32_t d = 1, mul = 1, shift = 0;
    void set(uint32_t by) {
        d = by, shift = 0;
        while ((1ull << shift) < d) shift++;
        mul = (uint32_t)(((1ull << 32) * ((1ull << shift) - d)) / d + 1);
    }
    __device__ __forceinline__ uint32_t div(uint32_t n) const { return (__umulhi(n, mul) + n) >> shift; }
};
struct GemmArgs {
    int M, N, K, batch;
    int a_mn_major, b_mn_major;
    void* d;
    int d_bf16;           // output rounded once to bf16 (else fp32)
    int d_f16;
    int in_bf16;          // operands bfloat16 (else float16): the MMA's operand format
    long long ldd, d_batch_stride;
    int epilogue;
    const void* aux;      // EPI_ADD / EPI_MASK operand: same dtype as the output, row-major [batch, M, N] view
    long long ld_aux, aux_batch_stride;
    int* status;          // device word: set to LB_ERR_TIMEOUT when a bounded wait gave up
    int tiles_m, tiles_n, group_m;
    Divisor by_tiles, by_batch, by_group, by_rows, by_last_rows;  // all tiles; tiles of a batch entry; of a group; a group's rows, the last one's
    // split-K: the K loop of every tile is cut into `splits` ranges of `kb_per_split` 64-wide blocks; each (tile, range)
    // unit writes a float32 partial tile to `partial` [splits][batch][M][N] and splitk_reduce adds them in order
    int splits, kb_per_split;
    float* partial;
};

// Unit `unit` of the grid: split * tiles + tile, neighbours share a K range.
__device__ __forceinline__ int tile_coords(const GemmArgs& p, int unit, int& b, int& m_blk, int& n_blk) {
    const int split = p.by_tiles.div(unit), tile = unit - split * (int)p.by_tiles.d;
    b = p.by_batch.div(tile);
    const int t = tile - b * (int)p.by_batch.d;
    // grouped raster: GROUP_M row-blocks share each column-block while they are resident together in L2
    const int g = p.by_group.div(t), first_m = g * p.group_m, in_group = t - g * (int)p.by_group.d;
    const bool last = p.tiles_m - first_m < p.group_m;
    const int rows = last ? p.tiles_m - first_m : p.group_m;
    n_blk = last ? p.by_last_rows.div(in_group) : p.by_rows.div(in_group);
    m_blk = first_m + in_group - n_blk * rows;
    return split;
}

// The cold paths of what follows lie behind the others: a block of one tile runs its way out once, and its instructions come from the L2.
#define LB_RARELY(x) __builtin_expect(!!(x), 0)

// Drains 128 accumulator columns (this warp's half of a 256-wide tile) of the thread's row from tensor memory and
// stores them with the epilogue and one rounding to the output dtype. `release` hands the accumulator back to the MMA warp, once its
// last columns are in registers. Rows leave through the staging area, 128 contiguous bytes of each or, at the end of rows whose length is a
// multiple of 16 bytes, as many 16-byte pieces as there are; other rows by the element.
template <class Release>
__device__ __forceinline__ void drain_tile(const GemmArgs& p, uint32_t tbase, int row, long long row_off, int col_base, int b,
                                           bool vec_ok, uint4* stage, int lane, Release release) {
    const int rows = p.M - (row - lane);
#pragma unroll 1
    for (int c2 = 0; c2 < BN / 2 / 64; c2++) {
        const int col0 = col_base + c2 * 64, span = p.N - col0;  // warp-uniform
        uint32_t v[64];
        tmem_ld_32x32(tbase + c2 * 64, v);  // two loads in flight, one wait
        tmem_ld_32x32(tbase + c2 * 64 + 32, v + 32);
        tmem_ld_wait();
        if (c2 == BN / 2 / 64 - 1) release();
        if (LB_RARELY(span <= 0)) continue;
        if (p.epilogue == EPI_RELU) {
#pragma unroll
            for (int j = 0; j < 64; j++) v[j] = __float_as_uint(fmaxf(__uint_as_float(v[j]), 0.0f));
        }
        if (p.d_bf16 || p.d_f16) {
            uint4 packed[8];
            uint32_t* w = (uint32_t*)packed;
            if (LB_RARELY(p.d_f16)) {
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const __half2 h = __floats2half2_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                    w[j] = *(const uint32_t*)&h;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                    w[j] = *(const uint32_t*)&h;
                }
            }
            if (LB_RARELY(p.epilogue >= EPI_ADD && row < p.M)) {
                // 16-bit outputs only (checked by the host). The product is rounded first, as its own primitive.
                const uint16_t* ax = (const uint16_t*)p.aux + (long long)b * p.aux_batch_stride + (long long)row * p.ld_aux + col0;
                const bool whole = (span >= 64 || p.N % 8 == 0) && p.ld_aux % 8 == 0 && p.aux_batch_stride % 8 == 0 && ((uintptr_t)p.aux & 15) == 0;
#pragma unroll
                for (int j0 = 0; j0 < 64; j0 += 8) {
                    uint32_t aw[4] = {0u, 0u, 0u, 0u};
                    if (whole && j0 < span) {
                        const uint4 t = *(const uint4*)(ax + j0);
                        aw[0] = t.x, aw[1] = t.y, aw[2] = t.z, aw[3] = t.w;
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; j++)
                            if (j0 + j < span) aw[j / 2] |= (uint32_t)ax[j0 + j] << (j % 2 * 16);
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) w[j0 / 2 + j] = tail_pair(w[j0 / 2 + j], aw[j], p.epilogue == EPI_ADD, p.d_bf16);
                }
            }
            uint16_t* out = (uint16_t*)p.d + row_off + col0;
            if (LB_RARELY(!vec_ok || (span < 64 && p.N % 8 != 0))) {
#pragma unroll
                for (int j = 0; j < 64; j++)  // unrolled with a predicate: keeps the fragment in registers
                    if (row < p.M && j < span) out[j] = (uint16_t)(w[j / 2] >> (j % 2 * 16));
            } else {
                store_rows_coalesced<8>(stage, packed, (uint8_t*)(out - (long long)lane * p.ldd), p.ldd * 2, rows, lane, span / 8);
            }
        } else {
            float* out = (float*)p.d + row_off + col0;
            if (LB_RARELY(!vec_ok || (span < 64 && p.N % 4 != 0))) {
#pragma unroll
                for (int j = 0; j < 64; j++)
                    if (row < p.M && j < span) out[j] = __uint_as_float(v[j]);
            } else {
#pragma unroll
                for (int h = 0; h < 2; h++)
                    store_rows_coalesced<8>(stage, (const uint4*)(v + h * 32), (uint8_t*)(out - (long long)lane * p.ldd + h * 32), p.ldd * 4, rows, lane,
                                            (span - h * 32) / 4);
            }
        }
    }
}

// The same where K is split: float32 partial sums, dense [split][batch][M][N]; the epilogue and the rounding happen in splitk_reduce.
// Whole pieces of 32 columns leave as 128-byte lines through the staging area.
template <class Release>
__device__ __forceinline__ void drain_partial(const GemmArgs& p, uint32_t tbase, int row, int col_base, int b, int split, uint4* stage, int lane,
                                              Release release) {
    float* row0 = p.partial + ((long long)(split * p.batch + b) * p.M + (row - lane)) * p.N;  // the warp's first row
#pragma unroll 1
    for (int c = 0; c < BN / 2 / 32; c++) {
        const int col0 = col_base + c * 32;
        uint32_t v[32];
        tmem_ld_32x32(tbase + c * 32, v);
        tmem_ld_wait();
        if (c == BN / 2 / 32 - 1) release();
        if (p.N % 4 == 0) {
            uint4 packed[8];
#pragma unroll
            for (int j = 0; j < 32; j += 4) packed[j / 4] = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            store_rows_coalesced<8>(stage, packed, (uint8_t*)(row0 + col0), (long long)p.N * 4, p.M - (row - lane), lane, (p.N - col0) / 4);
        } else if (row < p.M) {
            float* out = row0 + (long long)lane * p.N + col0;
#pragma unroll
            for (int j = 0; j < 32; j++)
                if (col0 + j < p.N) out[j] = __uint_as_float(v[j]);
        }
    }
}

// The add / mask epilogues on the fast path (unsplit K, a full 128-column span inside N, 16-byte aligned rows of the
// operand and the output): the operand's 32-column chunks are loaded one chunk ahead - the first one before the
// warp waits for the tile's MMAs - so that their global-memory latency never sits between the accumulator load
// and the store.
__device__ __forceinline__ bool aux_fast_path(const GemmArgs& p, int row, int col_base, bool vec_ok) {
    return p.epilogue >= EPI_ADD && p.splits == 1 && vec_ok && row < p.M && col_base + BN / 2 <= p.N && p.ld_aux % 8 == 0 &&
           p.aux_batch_stride % 8 == 0 && ((uintptr_t)p.aux & 15) == 0;
}
// Loads a 32-row x 32-column chunk of the operand with whole 64-byte row pieces per four lanes (eight rows per load
// instruction): lane l gets the 16-byte segment l % 4 of rows l / 4, 8 + l / 4, 16 + l / 4 and 24 + l / 4.
// `ax_warp` points at the warp's first row.
__device__ __forceinline__ void aux_load(const uint16_t* ax_warp, long long ld_aux, int lane, uint4* raw) {
#pragma unroll
    for (int t = 0; t < 4; t++) raw[t] = *(const uint4*)(ax_warp + (long long)(t * 8 + (lane >> 2)) * ld_aux + (lane & 3) * 8);
}
// Turns what aux_load fetched into each lane's own row (16 packed pairs) through 2 KB of the warp's staging area.
__device__ __forceinline__ void aux_to_rows(uint4* stage_aux, const uint4* raw, uint32_t* aw, int lane) {
    const uint32_t area = smem_u32(stage_aux);
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 4; t++) {
        const int r = t * 8 + (lane >> 2), q = lane & 3;
        st_shared(area + (r * 4 + (q ^ ((r >> 1) & 3))) * 16, raw[t]);
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint4 x = ld_shared(area + (lane * 4 + (q ^ ((lane >> 1) & 3))) * 16);
        aw[4 * q] = x.x, aw[4 * q + 1] = x.y, aw[4 * q + 2] = x.z, aw[4 * q + 3] = x.w;
    }
}
template <class Release>
__device__ __forceinline__ void drain_tile_aux(const GemmArgs& p, uint32_t tbase, long long row_off, const uint16_t* ax_warp, uint4* raw,
                                               uint4* stage, int lane, Release release) {
    uint8_t* out0 = (uint8_t*)((uint16_t*)p.d + (row_off - (long long)lane * p.ldd));  // the warp's first row (all 32 are inside M)
#pragma unroll 1
    for (int c = 0; c < BN / 2 / 32; c++) {
        uint32_t v[32], aw[16];
        tmem_ld_32x32(tbase + c * 32, v);
        aux_to_rows(stage + 128, raw, aw, lane);
        if (c + 1 < BN / 2 / 32) aux_load(ax_warp + (c + 1) * 32, p.ld_aux, lane, raw);
        tmem_ld_wait();
        if (c == BN / 2 / 32 - 1) release();
        uint4 packed[4];
        uint32_t* w = (uint32_t*)packed;
        if (LB_RARELY(p.d_f16)) {
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const __half2 h = __floats2half2_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                w[j] = tail_pair(*(const uint32_t*)&h, aw[j], p.epilogue == EPI_ADD, false);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                w[j] = tail_pair(*(const uint32_t*)&h, aw[j], p.epilogue == EPI_ADD, true);
            }
        }
        store_rows_coalesced<4>(stage, packed, out0 + c * 64, p.ldd * 2, 32, lane);
    }
}

__global__ void __launch_bounds__(kThreads, 1)
gemm_tcgen05(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const GemmArgs p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align_1024(smem_raw);
    uint8_t* smem_a = smem;
    uint8_t* smem_b = smem + STAGES * kStageBytesA;
    uint64_t* full = (uint64_t*)(smem + STAGES * (kStageBytesA + kStageBytesB));
    uint64_t* empty = full + STAGES;
    uint64_t* tmem_full = empty + STAGES;
    uint64_t* tmem_empty = tmem_full + 2;
    uint32_t* tmem_base_slot = (uint32_t*)(tmem_empty + 2);
    volatile int* abort_flag = (volatile int*)(tmem_base_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp-uniform for the compiler too
    const int num_tiles = p.tiles_m * p.tiles_n * p.batch;
    const int total_kb = (p.K + BK - 1) / BK;
    const int num_units = num_tiles * p.splits;  // unit = split * num_tiles + tile: neighbours share a K range

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(&tmem_full[s], 1);
            mbar_init(&tmem_empty[s], kEpilogueWarps);  // one arrival per epilogue warp
        }
        *abort_flag = 0;
        fence_barrier_init();
        tma_prefetch_desc(&map_a);
        tma_prefetch_desc(&map_b);
    }
    if (warp == 1) {
        tmem_alloc(tmem_base_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_base_slot, 0);
    grid_wait();

    if (warp == 0) {
        // ---- TMA producer ----
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int unit = blockIdx.x; unit < num_units && ok; unit += gridDim.x) {
                int b, m_blk, n_blk;
                const int kb0 = tile_coords(p, unit, b, m_blk, n_blk) * p.kb_per_split, kb1 = min(total_kb, kb0 + p.kb_per_split);
                for (int kb = kb0; kb < kb1; kb++) {
                    if (!(ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag))) break;
                    mbar_expect_tx(&full[stage], kStageBytesA + kStageBytesB);
                    uint8_t* sa = smem_a + stage * kStageBytesA;
                    uint8_t* sb = smem_b + stage * kStageBytesB;
                    if (!p.a_mn_major) {
                        tma_load_3d(sa, &map_a, &full[stage], kb * BK, m_blk * BM, b);  // box {64 k, 128 m}
                    } else {
                        for (int j = 0; j < BM / 64; j++)  // boxes {64 m, 64 k}
                            tma_load_3d(sa + j * (64 * BK * 2), &map_a, &full[stage], m_blk * BM + j * 64, kb * BK, b);
                    }
                    if (!p.b_mn_major) {
                        tma_load_3d(sb, &map_b, &full[stage], kb * BK, n_blk * BN, b);  // box {64 k, 256 n}
                    } else {
                        for (int j = 0; j < BN / 64; j++)  // boxes {64 n, 64 k}
                            tma_load_3d(sb + j * (64 * BK * 2), &map_b, &full[stage], n_blk * BN + j * 64, kb * BK, b);
                    }
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (ok) mbar_wait_ring<STAGES>(empty, phase * STAGES + stage, abort_flag);
        }
    } else if (warp == 1) {
        // ---- MMA issuer: the whole warp, so that the operands stay in uniform registers ----
        {
            const bool leader = elect_one();
            const uint32_t idesc = make_idesc(BM, BN, p.in_bf16 != 0, p.a_mn_major, p.b_mn_major);
            // descriptors of stage 0; a stage and a 16-wide k step only move the address field.
            // K-major: 16 k-elements = 32 bytes further inside the swizzled 128-byte row.
            // MN-major: 16 k-rows of 128 bytes = 2048 bytes further; 64-element blocks 8 KB apart.
            const uint64_t da0 = p.a_mn_major ? make_smem_desc(smem_u32(smem_a), 64 * BK * 2, 1024) : make_smem_desc(smem_u32(smem_a), 16, 1024);
            const uint64_t db0 = p.b_mn_major ? make_smem_desc(smem_u32(smem_b), 64 * BK * 2, 1024) : make_smem_desc(smem_u32(smem_b), 16, 1024);
            const uint32_t a_step = p.a_mn_major ? 2048u : 32u, b_step = p.b_mn_major ? 2048u : 32u;
            int stage = 0;
            uint32_t phase = 0;
            int local = 0;
            bool ok = true;
            for (int unit = blockIdx.x; unit < num_units && ok; unit += gridDim.x, local++) {
                const int buf = local & 1;
                const uint32_t use = (uint32_t)(local >> 1);
                if (!(ok = mbar_wait_warp(&tmem_empty[buf], (use & 1) ^ 1, abort_flag))) break;
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + (uint32_t)(buf * BN);
                const int kb0 = (int)p.by_tiles.div(unit) * p.kb_per_split;
                const int num_kb = min(total_kb, kb0 + p.kb_per_split) - kb0;
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!(ok = mbar_wait_warp(&full[stage], phase, abort_flag))) break;
                    tc_fence_after();
                    uint64_t da = desc_advance(da0, (uint32_t)(stage * kStageBytesA)), db = desc_advance(db0, (uint32_t)(stage * kStageBytesB));
#pragma unroll
                    for (int k = 0; k < BK / 16; k++) {
                        mma_f16(tmem_d, da, db, idesc, (kb | k) != 0, leader);
                        da = desc_advance(da, a_step), db = desc_advance(db, b_step);
                    }
                    mma_commit(&empty[stage], leader);  // frees the stage once these MMAs have read it
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (ok) mma_commit(&tmem_full[buf], leader);
            }
        }
    } else {
        // ---- epilogue: warps 2..9. A warp may only read TMEM lanes 32*(warp%4) .. +31; the two warps sharing a lane
        // quarter split the tile's 256 columns between them. ----
        const int quarter = warp & 3;
        const int col_half = (warp - 2) >> 2;
        uint4* stage = (uint4*)(smem + STAGES * (kStageBytesA + kStageBytesB) + 256) + (warp - 2) * (kStageBytesPerWarp / 16);
        int local = 0;
        bool ok = true;
        const bool vec_ok = p.d_bf16 || p.d_f16 ? (p.ldd % 8 == 0 && p.d_batch_stride % 8 == 0 && ((uintptr_t)p.d & 15) == 0)
                                                : (p.ldd % 4 == 0 && p.d_batch_stride % 4 == 0 && ((uintptr_t)p.d & 15) == 0);
        for (int unit = blockIdx.x; unit < num_units && ok; unit += gridDim.x, local++) {
            const int buf = local & 1;
            const uint32_t use = (uint32_t)(local >> 1);
            int b, m_blk, n_blk;
            const int split = tile_coords(p, unit, b, m_blk, n_blk);
            const int row = m_blk * BM + quarter * 32 + lane;
            const int col_base = n_blk * BN + col_half * (BN / 2);
            const long long row_off = (long long)b * p.d_batch_stride + (long long)row * p.ldd;
            const bool fast = __all_sync(0xffffffffu, aux_fast_path(p, row, col_base, vec_ok));  // warp-uniform: both drains load tensor memory warp-wide
            const uint16_t* ax_warp = (const uint16_t*)p.aux + (long long)b * p.aux_batch_stride + (long long)(row - lane) * p.ld_aux + col_base;
            uint4 raw[4];
            if (fast) aux_load(ax_warp, p.ld_aux, lane, raw);
            if (!(ok = mbar_wait(&tmem_full[buf], use & 1, abort_flag))) break;
            __syncwarp();
            tc_fence_after();
            const uint32_t tbase = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + col_half * (BN / 2));
            auto release = [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&tmem_empty[buf]);
            };
            if (fast) drain_tile_aux(p, tbase, row_off + col_base, ax_warp, raw, stage, lane, release);
            else if (LB_RARELY(p.splits > 1)) drain_partial(p, tbase, row, col_base, b, split, stage, lane, release);
            else drain_tile(p, tbase, row, row_off, col_base, b, vec_ok, stage, lane, release);
        }
    }

    // ---- teardown: every role leaves its loop (normally, or because the abort flag was raised) ----
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) atomicExch(p.status, LB_ERR_TIMEOUT);
        // give copies and MMAs still in flight a bounded time to land before shared/tensor memory is released
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {
        }
        __syncthreads();
    }
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// ---- the same GEMM on CTA pairs ---------------------------------------------------------------------------------
// A cluster of two CTAs computes a 256 x 256 tile with tcgen05.mma.cta_group::2: CTA `rank` holds rows
// [128 rank, 128 rank + 128) of the A tile and columns [128 rank, 128 rank + 128) of the B tile, so every SM fetches
// only half of B from shared memory per instruction (8 KB instead of 12 KB), which lifts the one-CTA kernel's
// operand-fetch ceiling. The leader (rank 0) issues all MMAs; its commits arrive on the barriers of both CTAs. Both
// CTAs load their own tiles with TMA, counting bytes on the leader's `full` barrier. Each CTA drains its own 128
// accumulator rows; "accumulator drained" arrivals from both CTAs go to the leader's `tmem_empty` barrier.
//
// What bounds it: with K of 2048 and more the products (16384 x 4096 x 4096: 91 % of the tensor pipe's rate between two tiles, then
// the power cap); with shorter K the time a tile needs for its way out, so that the hand-over is kept short: the accumulator goes back
// once its last columns are in registers, by an arrival that waits for no global store; where a tile lies is found without
// divisions; the staging area is addressed as shared memory; and products are issued warp-wide. Together, us a product, bfloat16:
// 16384 x 4096 with K = 64 92 -> 45, K = 512 108 -> 74, K = 1024 142 -> 119; 16384 x 32768 x 1024 1100 -> 920; 6442 x 1120 x 280
// 17.8 -> 12.9; 3000 x 3000 x 600 23.8 -> 18.8; 16384 x 1024 x 4096 121 -> 117; 8192^3 885 -> 858.
// What a block runs once comes from the L2 instruction by instruction, and most products are a tile or two to a block: the way out is
// kept short and its cold paths behind the others, row pieces at the end of rows leave through the staging area like whole ones (one store an
// element of a thread's row stood in line for them), and the add and mask tails are packed. us a product: 1024 x 4096 K 200 8.3 -> 6.4, 704 x 3072
// K 1024 11.8 -> 9.8, 2048^3 17.4 -> 15.2, 4096 x 4096 K 1024 with a mask 32.8 -> 31.2, 1000 x 3000 K 704 12.2 -> 9.7, 6442 x 1120 x 280 12.4 -> 9.4.
constexpr int PSTAGES = 6;
constexpr int kPairStageBytesA = BM * BK * 2, kPairStageBytesB = (BN / 2) * BK * 2;
constexpr int kPairSmemBytes = PSTAGES * (kPairStageBytesA + kPairStageBytesB) + 1024 + 256 + kEpilogueStageBytes;

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_tcgen05_pair(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const GemmArgs p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align_1024(smem_raw);
    uint8_t* smem_a = smem;
    uint8_t* smem_b = smem + PSTAGES * kPairStageBytesA;
    uint64_t* full = (uint64_t*)(smem + PSTAGES * (kPairStageBytesA + kPairStageBytesB));
    uint64_t* empty = full + PSTAGES;
    uint64_t* tmem_full = empty + PSTAGES;
    uint64_t* tmem_empty = tmem_full + 2;
    uint32_t* tmem_base_slot = (uint32_t*)(tmem_empty + 2);
    volatile int* abort_flag = (volatile int*)(tmem_base_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp-uniform for the compiler too
    const uint32_t rank = cluster_ctarank();
    const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
    const int num_tiles = p.tiles_m * p.tiles_n * p.batch;  // tiles_m counts 256-row pair tiles here
    const int total_kb = (p.K + BK - 1) / BK;
    const int num_units = num_tiles * p.splits;

    if (threadIdx.x == 0) {
        for (int s = 0; s < PSTAGES; s++) {
            mbar_init(&full[s], 1);   // the leader's expect_tx arrival; bytes of both CTAs
            mbar_init(&empty[s], 1);  // one commit from the leader's MMA thread
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(&tmem_full[s], 1);
            mbar_init(&tmem_empty[s], 2 * kEpilogueWarps);  // used in the leader only: every epilogue warp of the pair
        }
        *abort_flag = 0;
        fence_barrier_init();
        tma_prefetch_desc(&map_a);
        tma_prefetch_desc(&map_b);
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_base_slot, 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // barriers of both CTAs are initialised and both allocations are done before anyone signals across
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_base_slot, 0);
    grid_wait();

    if (warp == 0) {
        // ---- TMA producer (both CTAs) ----
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int unit = pair; unit < num_units && ok; unit += num_pairs) {
                int b, m_blk, n_blk;
                const int kb0 = tile_coords(p, unit, b, m_blk, n_blk) * p.kb_per_split;
                const int row0 = m_blk * 2 * BM + (int)rank * BM, col0 = n_blk * BN + (int)rank * (BN / 2);
                const int kb1 = min(total_kb, kb0 + p.kb_per_split);
                for (int kb = kb0; kb < kb1; kb++) {
                    if (!(ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag))) break;
                    if (rank == 0) mbar_expect_tx(&full[stage], 2 * (kPairStageBytesA + kPairStageBytesB));
                    uint8_t* sa = smem_a + stage * kPairStageBytesA;
                    uint8_t* sb = smem_b + stage * kPairStageBytesB;
                    if (!p.a_mn_major) {
                        tma_load_3d_pair(sa, &map_a, &full[stage], kb * BK, row0, b);  // box {64 k, 128 m}
                    } else {
                        for (int j = 0; j < BM / 64; j++)  // boxes {64 m, 64 k}
                            tma_load_3d_pair(sa + j * (64 * BK * 2), &map_a, &full[stage], row0 + j * 64, kb * BK, b);
                    }
                    if (!p.b_mn_major) {
                        tma_load_3d_pair(sb, &map_b, &full[stage], kb * BK, col0, b);  // box {64 k, 128 n}
                    } else {
                        for (int j = 0; j < BN / 2 / 64; j++)  // boxes {64 n, 64 k}
                            tma_load_3d_pair(sb + j * (64 * BK * 2), &map_b, &full[stage], col0 + j * 64, kb * BK, b);
                    }
                    if (++stage == PSTAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (ok) mbar_wait_ring<PSTAGES>(empty, phase * PSTAGES + stage, abort_flag);
        }
    } else if (warp == 1) {
        // ---- MMA issuer (leader CTA only): the whole warp, so that the operands stay in uniform registers ----
        if (rank == 0) {
            const bool leader = elect_one();
            const uint32_t idesc = make_idesc(2 * BM, BN, p.in_bf16 != 0, p.a_mn_major, p.b_mn_major);
            const uint64_t da0 = p.a_mn_major ? make_smem_desc(smem_u32(smem_a), 64 * BK * 2, 1024) : make_smem_desc(smem_u32(smem_a), 16, 1024);
            const uint64_t db0 = p.b_mn_major ? make_smem_desc(smem_u32(smem_b), 64 * BK * 2, 1024) : make_smem_desc(smem_u32(smem_b), 16, 1024);
            const uint32_t a_step = p.a_mn_major ? 2048u : 32u, b_step = p.b_mn_major ? 2048u : 32u;
            int stage = 0;
            uint32_t phase = 0;
            int local = 0;
            bool ok = true;
            for (int unit = pair; unit < num_units && ok; unit += num_pairs, local++) {
                const int buf = local & 1;
                const uint32_t use = (uint32_t)(local >> 1);
                if (!(ok = mbar_wait_cluster_warp(&tmem_empty[buf], (use & 1) ^ 1, abort_flag))) break;
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + (uint32_t)(buf * BN);
                const int kb0 = (int)p.by_tiles.div(unit) * p.kb_per_split;
                const int num_kb = min(total_kb, kb0 + p.kb_per_split) - kb0;
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!(ok = mbar_wait_warp(&full[stage], phase, abort_flag))) break;
                    tc_fence_after();
                    uint64_t da = desc_advance(da0, (uint32_t)(stage * kPairStageBytesA)), db = desc_advance(db0, (uint32_t)(stage * kPairStageBytesB));
#pragma unroll
                    for (int k = 0; k < BK / 16; k++) {
                        mma_f16_pair(tmem_d, da, db, idesc, (kb | k) != 0, leader);
                        da = desc_advance(da, a_step), db = desc_advance(db, b_step);
                    }
                    mma_commit_pair(&empty[stage], 3, leader);  // frees the stage in both CTAs
                    if (++stage == PSTAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (ok) mma_commit_pair(&tmem_full[buf], 3, leader);
            }
        }
    } else {
        // ---- epilogue: warps 2..9 of both CTAs, each CTA on its own 128 rows ----
        const int quarter = warp & 3;
        const int col_half = (warp - 2) >> 2;
        uint4* stage = (uint4*)(smem + PSTAGES * (kPairStageBytesA + kPairStageBytesB) + 256) + (warp - 2) * (kStageBytesPerWarp / 16);
        int local = 0;
        bool ok = true;
        const bool vec_ok = p.d_bf16 || p.d_f16 ? (p.ldd % 8 == 0 && p.d_batch_stride % 8 == 0 && ((uintptr_t)p.d & 15) == 0)
                                                : (p.ldd % 4 == 0 && p.d_batch_stride % 4 == 0 && ((uintptr_t)p.d & 15) == 0);
        for (int unit = pair; unit < num_units && ok; unit += num_pairs, local++) {
            const int buf = local & 1;
            const uint32_t use = (uint32_t)(local >> 1);
            int b, m_blk, n_blk;
            const int split = tile_coords(p, unit, b, m_blk, n_blk);
            const int row = m_blk * 2 * BM + (int)rank * BM + quarter * 32 + lane;
            const int col_base = n_blk * BN + col_half * (BN / 2);
            const long long row_off = (long long)b * p.d_batch_stride + (long long)row * p.ldd;
            const bool fast = __all_sync(0xffffffffu, aux_fast_path(p, row, col_base, vec_ok));  // warp-uniform: both drains load tensor memory warp-wide
            const uint16_t* ax_warp = (const uint16_t*)p.aux + (long long)b * p.aux_batch_stride + (long long)(row - lane) * p.ld_aux + col_base;
            uint4 raw[4];
            if (fast) aux_load(ax_warp, p.ld_aux, lane, raw);
            if (!(ok = mbar_wait(&tmem_full[buf], use & 1, abort_flag))) break;
            __syncwarp();
            tc_fence_after();
            const uint32_t tbase = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + col_half * (BN / 2));
            auto release = [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(&tmem_empty[buf], 0);
            };
            if (fast) drain_tile_aux(p, tbase, row_off + col_base, ax_warp, raw, stage, lane, release);
            else if (LB_RARELY(p.splits > 1)) drain_partial(p, tbase, row, col_base, b, split, stage, lane, release);
            else drain_tile(p, tbase, row, row_off, col_base, b, vec_ok, stage, lane, release);
        }
    }

    // ---- teardown: every role of both CTAs leaves its loop (normally, or because an abort flag was raised) ----
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) atomicExch(p.status, LB_ERR_TIMEOUT);
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {
        }
        __syncthreads();
    }
    cluster_sync();  // neither CTA releases shared or tensor memory while the other may still signal or compute into it
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

// Adds the split-K partial tiles in split order (fixed, so results are reproducible), applies the epilogue and rounds once. Bound by
// memory: four elements of a row a thread (VEC: N is a multiple of four, rows of the result and of the epilogue's operand are aligned),
// found by one division where twelve 64-bit ones took most of the time. With the partial tiles stored in whole lines, us a product:
// 1192 x 1736 x 6944 46.9 -> 40.4, 704 x 1504 x 8000 32.7 -> 23.0, 1024 x 1024 x 8192 30.5 -> 24.0.
template <bool VEC>
__global__ void __launch_bounds__(256) splitk_reduce(const float* __restrict__ partial, GemmArgs p) {
    grid_wait(partial);
    constexpr int W = VEC ? 4 : 1;
    const long long per = (long long)p.batch * p.M * p.N;
    for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * W; i < per; i += (long long)gridDim.x * blockDim.x * W) {
        float acc[W] = {};
#pragma unroll 4
        for (int s = 0; s < p.splits; s++) {
            if constexpr (VEC) {
                const float4 v = *(const float4*)(partial + s * per + i);
                acc[0] += v.x, acc[1] += v.y, acc[2] += v.z, acc[3] += v.w;
            } else {
                acc[0] += partial[s * per + i];
            }
        }
        const long long row = i / p.N, b = p.batch > 1 ? row / p.M : 0, r = row - b * p.M, c = i - row * p.N;
        const uint16_t* aux = (const uint16_t*)p.aux + b * p.aux_batch_stride + r * p.ld_aux + c;
        __align__(8) uint16_t a16[W], out16[W];
        if (p.epilogue >= EPI_ADD) {
            if constexpr (VEC) *(uint2*)a16 = *(const uint2*)aux;
            else a16[0] = *aux;
        }
#pragma unroll
        for (int j = 0; j < W; j++) {
            float x = acc[j];
            if (p.epilogue == EPI_RELU) x = fmaxf(x, 0.0f);
            if (p.epilogue >= EPI_ADD) {
                float prod, other;
                if (p.d_bf16) prod = __bfloat162float(__float2bfloat16_rn(x)), other = __uint_as_float((uint32_t)a16[j] << 16);
                else prod = __half2float(__float2half_rn(x)), other = __half2float(__ushort_as_half(a16[j]));
                x = p.epilogue == EPI_ADD ? __fadd_rn(other, prod) : (other > 0.0f ? prod : 0.0f);
            }
            acc[j] = x;
            out16[j] = p.d_bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(x)) : __half_as_ushort(__float2half_rn(x));
        }
        const long long at = b * p.d_batch_stride + r * p.ldd + c;
        if (p.d_bf16 || p.d_f16) {
            if constexpr (VEC) *(uint2*)((uint16_t*)p.d + at) = make_uint2(out16[0] | (uint32_t)out16[1] << 16, out16[2] | (uint32_t)out16[3] << 16);
            else ((uint16_t*)p.d)[at] = out16[0];
        } else {
            if constexpr (VEC) *(float4*)((float*)p.d + at) = make_float4(acc[0], acc[1], acc[2], acc[3]);
            else ((float*)p.d)[at] = acc[0];
        }
    }
}

// [batch, rows, cols] view of a rank-2/3 tensor
struct View3 {
    void* ptr;
    int dtype;
    long long batch, rows, cols, sb, sr, sc;
};
View3 view3(const lb_tensor& t, const char* what) {
    if (t.rank != 2 && t.rank != 3) fail(LB_ERR_INVALID, format("gemm: %s must have rank 2 or 3, got %d", what, t.rank));
    View3 v;
    v.ptr = t.ptr;
    v.dtype = t.dtype;
    int o = t.rank - 2;
    v.batch = o ? t.shape[0] : 1;
    v.sb = o ? t.stride[0] : 0;
    v.rows = t.shape[o];
    v.cols = t.shape[o + 1];
    v.sr = t.stride[o];
    v.sc = t.stride[o + 1];
    return v;
}

CUtensorMap make_map(const View3& v, bool contiguous_is_cols, int box_inner, int box_outer) {
    // dims innermost first: {contiguous, strided, batch}
    long long inner = contiguous_is_cols ? v.cols : v.rows, outer = contiguous_is_cols ? v.rows : v.cols;
    long long outer_stride = contiguous_is_cols ? v.sr : v.sc;
    cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)outer, (cuuint64_t)v.batch};
    if (outer == 1) outer_stride = inner;
    cuuint64_t strides[2] = {(cuuint64_t)outer_stride * 2, (cuuint64_t)(v.batch > 1 ? v.sb : outer_stride * outer) * 2};
    cuuint32_t box[3] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer, 1};
    cuuint32_t elem[3] = {1, 1, 1};
    CUtensorMap map;
    check_cu(driver().cuTensorMapEncodeTiled(&map, v.dtype == LB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                                             3, v.ptr, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE),
             "cuTensorMapEncodeTiled");
    return map;
}

}  // namespace

// Number of K ranges for a GEMM with few output tiles and a long K (weight gradients), with one CTA to a 128 x 256 tile. 1 = no split. A cost
// model picks it: waves of (tile, range) units times the k-blocks of a range, at the measured 4 x 171 cycles per k-block, plus the float32
// partial tiles written by the GEMM and re-read by the reduction kernel at HBM speed and that kernel's launch. A split has to win by a tenth
// to be taken; each range keeps at least 16 k-blocks.
size_t gemm_scratch_bytes(long long M, long long N, long long K, long long batch);
static int gemm_tile_splits(long long M, long long N, long long K, long long batch, int sms) {
    const long long tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN) * batch, total_kb = (K + BK - 1) / BK;
    if (tiles >= 4LL * sms || total_kb < 32) return 1;
    const double us_per_kb = 0.36, bytes_per_us = 5.0e6, launch_us = 6.0;
    auto cost = [&](int s) {
        const long long waves = (tiles * s + sms - 1) / sms, kb = (total_kb + s - 1) / s;
        double us = (double)waves * (double)kb * us_per_kb;
        if (s > 1) us += ((2.0 * s * 4 + 2) * (double)(batch * M * N)) / bytes_per_us + launch_us;
        return us;
    };
    int best = 1;
    double best_us = cost(1) * 0.9;
    for (int s = 2; s <= 32 && total_kb / s >= 16; s++)
        if (cost(s) < best_us) best = s, best_us = cost(s);
    return best;
}

// The same for what runs: CTA pairs take 256 x 256 tiles of more than 128 rows. us: 3 a product, 0.3 a k-block and 2 a unit of each wave, 0.1 a
// k-block shared by all pairs (the L2's part and the power's), 3.5 for the reduction and, a million elements of the result, 0.45 a range and 0.6:
// a fit to 714 shapes of 129 to 9000 rows and columns and K of 500 to 30000 under 1 to 8 ranges (half of them within 6 %). Against the
// model above, on those and 404 other shapes: 55 are cut otherwise and take 0.69 - 1.08 of the time, 0.84 in the mean, three of them more than
// 1.03; 1500 x 1024 K 4096 24.2 -> 18.4, 1530 x 1536 K 6144 0.83, 768 x 3072 K 4096 26.4 -> 23.4, 357 x 4096 K 4096 0.86. (The former number where
// this model puts another less than a tenth below it is no better line: 64 such shapes, every operand major, 0.84 - 1.14 of these counts' time for a product alone,
// 1.007 in the mean, and 0.84 - 1.37, 0.99, one after another under the power cap.) Which products stay on narrow tiles is left to the model above, which
// that line was measured with.
int gemm_splits(long long M, long long N, long long K, long long batch, int sms) {
    if (M <= BM) return gemm_tile_splits(M, N, K, batch, sms);
    const int pairs = sms / 2;
    const long long tiles = ((M + 2 * BM - 1) / (2 * BM)) * ((N + BN - 1) / BN) * batch, total_kb = (K + BK - 1) / BK;
    if (tiles >= 4LL * pairs || total_kb < 32) return 1;
    const double millions = (double)(batch * M * N) * 1e-6;
    auto cost = [&](int s) {
        const double kb = (double)((total_kb + s - 1) / s), waves = (double)((tiles * s + pairs - 1) / pairs);
        return 3.0 + waves * (0.3 * kb + 2.0) + 0.1 * kb * (double)(tiles * s) / pairs + (s > 1 ? 3.5 + millions * (0.45 * s + 0.6) : 0.0);
    };
    int best = 1;
    double best_us = cost(1) * 0.9;
    for (int s = 2; s <= 32 && total_kb / s >= 16; s++)
        if (cost(s) < best_us) best = s, best_us = cost(s);
    return best;
}

// K ranges (CTAs of a cluster) with which a product runs on the 128 x 64 tiles of gemm_small.cu, 0 where 256 x 256 tiles are
// better. The line is one CTA per SM: with no more tiles than SMs, ranges are doubled while they still have an SM each and
// two 64-wide blocks of K, and once more, two CTAs to an SM, where a range would be longer than 64 blocks. Measured (us, large
// tiles -> these), bfloat16: 64^3 8.2 -> 6.2, 512^3 13.5 -> 8.5, 200 x 4096 K 1024 16.4 -> 11.5, 200 x 1024 K 4096 24.6 -> 12.3
// (4 ranges), 1000^3 18.5 -> 12.3, 128 x 8192 K 8192 49 -> 35, 1024 x 1024 K 8192 35 -> 28 (39 with one range); beyond the line
// 4096 x 1024 K 200 12.3 -> 16.4, 700 x 4096 K 1024 16.4 -> 20.5, 2048^3 22.6 -> 32.7.
// Where scratch lets large tiles cut K into `large_split` ranges, ranges that would be 64 blocks and longer with one CTA to an SM may go
// there, since a narrow tile fetches twice the bytes per product: 1024 x 1024 (us, these -> large) K 16384 43.7 -> 32.7, 8192 29.0 -> 23.5,
// 4096 22.1 -> 17.9, 768 x 768 x 8192 20.8 -> 16.8, 768 x 1024 x 16384 41.6 -> 26.7; but 32 blocks: 512 x 512 x 8192 14.6 -> 15.7,
// 1024 x 1024 x 2048 13.0 -> 17.1. They do where the large tiles are CTA pairs' and on the GPU all at once (235 shapes of 136 to 2900
// rows, 128 to 4400 columns and K of 4096 to 30000, every operand major, operands in the L2 or not: 0.40 - 0.87 of the time), and else
// where an SM would walk 130 blocks of narrow tiles, 105 where pairs' tiles cover hardly more than the result, and two and a quarter times
// those of large ones (143 shapes of 16 rows and more: 0.53 - 1.03; 1664 x 256 x 14296 41.5 -> 27.8). What is left to narrow tiles (213
// shapes) takes 0.56 to 1.35 times as long on large ones, a fifth of it longer: 384 x 3072 x 6144 (two row tiles, two waves) 22.2 ->
// 26.3, 384 x 1536 x 8192 18.4 -> 21.6, on the one-CTA kernel 128 x 9216 x 4096 23.2 -> 27.9, 16 x 9216 x 4096 16.4 -> 19.3.
int gemm_small_splits(long long M, long long N, long long K, long long batch, int sms, int large_split) {
    const long long tiles = (M + 127) / 128 * ((N + 63) / 64) * batch, total_kb = (K + BK - 1) / BK;
    if (tiles > sms) return 0;
    int s = 1;
    while (s < 8 && tiles * 2 * s <= sms && total_kb >= 4 * s) s *= 2;
    const bool long_ranges = total_kb >= 64 * s;
    if (s < 8 && total_kb > 64 * s && tiles * s <= sms) s *= 2;
    if (total_kb > 128 * s) return 0;  // longer ranges: not measured, left to the split-K kernels
    if (large_split > 1 && long_ranges) {
        const bool pairs = M > BM;
        const int at_once = pairs ? sms / 2 : sms, rows = pairs ? 2 * BM : BM;
        const long long large_tiles = (M + rows - 1) / rows * ((N + BN - 1) / BN) * batch, units = large_tiles * large_split;
        if (pairs && units <= at_once) return 0;
        const long long narrow_kb = (tiles * s + sms - 1) / sms * ((total_kb + s - 1) / s);
        const long long large_kb = (units + at_once - 1) / at_once * ((total_kb + large_split - 1) / large_split);
        const bool well_filled = pairs && 20 * (large_tiles * rows * BN) <= 23 * (tiles * 128 * 64);  // at most 1.15 times the narrow tiles' area
        if (narrow_kb >= (well_filled ? 105 : 130) && 4 * narrow_kb >= 9 * large_kb) return 0;
    }
    return s;
}

// CTA pairs of gemm_tcgen05_pair that can be resident on `dev` at once (asked of the runtime once per device).
static int resident_pairs(const DeviceInfo& dev) {
    static std::mutex mutex;
    static std::map<int, int> cache;
    std::lock_guard<std::mutex> lock(mutex);
    auto it = cache.find(dev.device);
    if (it != cache.end()) return it->second;
    int pairs = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (dev.sms / 2), 1, 1), cfg.blockDim = dim3(kThreads, 1, 1), cfg.dynamicSmemBytes = kPairSmemBytes;
    if (cudaOccupancyMaxActiveClusters(&pairs, gemm_tcgen05_pair, &cfg) != cudaSuccess || pairs <= 0) {
        cudaGetLastError();
        pairs = 0;
    }
    return cache[dev.device] = pairs;
}

int gemm_model_splits(long long M, long long N, long long K, long long batch) { return gemm_splits(M, N, K, batch, sm_count_hint()); }

size_t gemm_scratch_bytes(long long M, long long N, long long K, long long batch) {
    const int s = gemm_splits(M, N, K, batch, sm_count_hint());
    return s > 1 ? (size_t)s * batch * M * N * 4 : 0;
}

// Scratch a plan's product step takes: none where the narrow tiles run.
static size_t gemm_step_scratch_bytes(long long M, long long N, long long K, long long batch) {
    const int sms = sm_count_hint(), split = gemm_splits(M, N, K, batch, sms);
    return gemm_small_splits(M, N, K, batch, sms, split > 1 ? gemm_tile_splits(M, N, K, batch, sms) : 1) ? 0 : gemm_scratch_bytes(M, N, K, batch);
}

// Where a product of 16-bit operands runs: on narrow tiles with `ranges` CTAs a cluster, or (ranges 0) on large tiles with K cut into
// `splits` ranges of `kb_per_split` 64-wide blocks.
struct GemmRoute {
    int ranges, splits, kb_per_split;
};
static GemmRoute gemm_route(long long M, long long N, long long K, long long batch, int sms, int kernel_choice, size_t scratch_bytes, const GemmTuning* tuning) {
    const int model = scratch_bytes ? gemm_splits(M, N, K, batch, sms) : 1;
    auto holds = [&](int s) { return s > 1 && scratch_bytes >= (size_t)s * batch * M * N * 4; };
    // no kernel asked for and no split or raster tuned: narrow tiles where they fit
    if (kernel_choice == 0 && !(tuning && (tuning->splits > 0 || tuning->group_m > 0))) {
        const int large = scratch_bytes ? gemm_tile_splits(M, N, K, batch, sms) : 1;
        if (const int ranges = gemm_small_splits(M, N, K, batch, sms, holds(model) || holds(large) ? large : 1)) return {ranges, 1, 0};
    }
    // no more ranges than the scratch holds (a saved plan's is what another model asked for), or as many as were tuned if it holds those
    const int split = (int)std::min<size_t>(model, scratch_bytes / ((size_t)batch * M * N * 4));
    const int want = tuning && tuning->splits > 0 ? tuning->splits : split;
    const int total_kb = (int)((K + BK - 1) / BK), kb = holds(want) ? (total_kb + want - 1) / want : total_kb;
    return {0, (total_kb + kb - 1) / kb, kb};
}

// Whether two operands can be read by the tensor-core kernels, and which of their axes is contiguous.
static bool tensor_core_operands(const View3& a, const View3& b, bool& a_cols, bool& b_cols) {
    auto major = [](const View3& v, bool& cols_contig) {
        if (v.sc == 1 || v.cols == 1) { cols_contig = true; return true; }
        if (v.sr == 1 || v.rows == 1) { cols_contig = false; return true; }
        return false;
    };
    // TMA: 16-byte aligned base, strides multiples of 16 bytes
    auto aligned = [](const View3& v, bool cols_contig) {
        long long inner = cols_contig ? v.cols : v.rows, outer = cols_contig ? v.rows : v.cols;
        long long ld = outer == 1 ? inner : (cols_contig ? v.sr : v.sc);
        return ((uintptr_t)v.ptr & 15) == 0 && ld % 8 == 0 && ld >= inner && (v.batch == 1 || v.sb % 8 == 0);
    };
    return (a.dtype == LB_BF16 || a.dtype == LB_F16) && a.cols > 0 && major(a, a_cols) && major(b, b_cols) && aligned(a, a_cols) && aligned(b, b_cols) &&
           a.rows <= INT32_MAX && b.cols <= INT32_MAX && a.cols <= INT32_MAX;
}

// Kernels that gemm launches.
int gemm_launches(const lb_tensor& a_t, const lb_tensor& b_t, size_t scratch_bytes, int kernel_choice, const GemmTuning* tuning) {
    const View3 a = view3(a_t, "a"), b = view3(b_t, "b");
    if (a.rows == 0 || b.cols == 0 || a.batch == 0) return 0;
    bool a_cols, b_cols;
    if (kernel_choice == 2 || !tensor_core_operands(a, b, a_cols, b_cols)) return 1;
    return gemm_route(a.rows, b.cols, a.cols, a.batch, sm_count_hint(), kernel_choice, scratch_bytes, tuning).splits > 1 ? 2 : 1;
}

// The sizes of a product of float32 operands, which decide its tiles; false if there is nothing to do.
bool gemm_held(const lb_tensor& a_t, const lb_tensor& b_t, SimtProblem& q) {
    const View3 a = view3(a_t, "a"), b = view3(b_t, "b");
    q.p.M = (int)a.rows, q.p.N = (int)b.cols, q.p.K = (int)a.cols, q.p.batch = (int)a.batch;
    return a.rows && b.cols && a.batch;
}

// With `held`, a product of the CUDA cores is written there instead of launched, and the answer is true.
bool gemm(const lb_tensor& a_t, const lb_tensor& b_t, const lb_tensor& d_t, int epilogue, int kernel_choice, void* stream,
          void* scratch, size_t scratch_bytes, const lb_tensor* aux_t, const GemmTuning* tuning, SimtProblem* held) {
    View3 a = view3(a_t, "a"), b = view3(b_t, "b"), d = view3(d_t, "output");
    if (epilogue < EPI_NONE || epilogue > EPI_MASK) fail(LB_ERR_INVALID, "gemm: unknown epilogue");
    View3 aux{};
    if (epilogue >= EPI_ADD) {
        if (!aux_t || !aux_t->ptr) fail(LB_ERR_INVALID, "gemm: the add / mask epilogue needs its operand tensor");
        aux = view3(*aux_t, "epilogue operand");
        if (aux.dtype != d.dtype || aux.rows != d.rows || aux.cols != d.cols || aux.batch != d.batch || (aux.sc != 1 && aux.cols > 1))
            fail(LB_ERR_INVALID, "gemm: the epilogue operand must be a row-major tensor of the output's shape and dtype");
        if (d.dtype != LB_BF16 && d.dtype != LB_F16 && !(a.dtype == LB_F32 && held))  // float32 products take one in plans alone
            fail(LB_ERR_UNSUPPORTED, "gemm: the add / mask epilogue is built for 16-bit outputs of the tensor-core kernels");
    }
    if (a.dtype != b.dtype) fail(LB_ERR_INVALID, "gemm: operands must share a dtype (no hidden casts)");
    if (a.cols != b.rows || a.batch != b.batch || d.rows != a.rows || d.cols != b.cols || d.batch != a.batch)
        fail(LB_ERR_INVALID, format("gemm: shapes [%lld,%lld,%lld] x [%lld,%lld,%lld] -> [%lld,%lld,%lld] do not match",
                                    a.batch, a.rows, a.cols, b.batch, b.rows, b.cols, d.batch, d.rows, d.cols));
    if (d.sc != 1 && d.cols > 1) fail(LB_ERR_UNSUPPORTED, "gemm: the output must be row-major");
    if (a.dtype != LB_F32 && a.dtype != LB_BF16 && a.dtype != LB_F16) fail(LB_ERR_UNSUPPORTED, "gemm: float16, bfloat16 or float32 operands");
    if (d.dtype != LB_F32 && d.dtype != a.dtype) fail(LB_ERR_INVALID, "gemm: the output is float32 (the accumulator) or the operands' dtype");
    const long long M = a.rows, N = b.cols, K = a.cols, batch = a.batch;
    if (M == 0 || N == 0 || batch == 0) return false;
    driver();
    cudaStream_t s = (cudaStream_t)stream;

    bool a_cols, b_cols;
    const bool tc_ok = kernel_choice != 2 && tensor_core_operands(a, b, a_cols, b_cols);
    if (kernel_choice == 1 && !tc_ok) fail(LB_ERR_UNSUPPORTED, "gemm: the tcgen05 kernels need bfloat16 or float16 operands with a unit stride and 16-byte aligned rows");

    if (tc_ok) {
        GemmArgs p{};
        p.M = (int)M, p.N = (int)N, p.K = (int)K, p.batch = (int)batch;
        p.a_mn_major = !a_cols;  // A [M, K]: contiguous columns = K-major
        p.b_mn_major = b_cols;   // B [K, N]: contiguous columns = N-major
        p.d = d.ptr;
        p.d_bf16 = d.dtype == LB_BF16;
        p.d_f16 = d.dtype == LB_F16;
        p.in_bf16 = a.dtype == LB_BF16;
        p.ldd = d.sr;
        p.d_batch_stride = d.batch > 1 ? d.sb : 0;
        p.epilogue = epilogue;
        p.aux = aux.ptr, p.ld_aux = aux.sr, p.aux_batch_stride = aux.batch > 1 ? aux.sb : 0;
        p.status = status_word();
        // CTA pairs (256 x 256 tiles over two SMs) whenever there is more than one 128-row block; kernel_choice 3 keeps
        // the one-CTA kernel
        const bool pairs = M > BM && kernel_choice != 3;
        const int tile_rows = pairs ? 2 * BM : BM;
        p.tiles_m = (int)((M + tile_rows - 1) / tile_rows);
        p.tiles_n = (int)((N + BN - 1) / BN);
        p.group_m = tuning && tuning->group_m > 0 ? tuning->group_m : (pairs ? 8 : 16);
        // K-major operands: box {64 k, rows}; MN-major: box {64 mn, 64 k}
        CUtensorMap map_a = p.a_mn_major ? make_map(a, false, 64, BK) : make_map(a, true, BK, BM);
        // B as the N x K operand: "rows" of the operand are B's columns
        View3 bt = b;  // transposed view: rows = N, cols = K
        bt.rows = b.cols, bt.cols = b.rows, bt.sr = b.sc, bt.sc = b.sr;
        CUtensorMap map_b = p.b_mn_major ? make_map(bt, false, 64, BK) : make_map(bt, true, BK, pairs ? BN / 2 : BN);
        const DeviceInfo& dev = device_info();
        const GemmRoute route = gemm_route(M, N, K, batch, dev.sms, kernel_choice, ((uintptr_t)scratch & 15) == 0 && scratch ? scratch_bytes : 0, tuning);
        if (route.ranges) {
            SmallGemmArgs q{};
            q.M = p.M, q.N = p.N, q.K = p.K, q.a_mn_major = p.a_mn_major, q.b_mn_major = p.b_mn_major, q.in_bf16 = p.in_bf16;
            q.d = p.d, q.d_bf16 = p.d_bf16, q.d_f16 = p.d_f16, q.ldd = p.ldd, q.d_batch_stride = p.d_batch_stride;
            q.epilogue = p.epilogue, q.aux = p.aux, q.ld_aux = p.ld_aux, q.aux_batch_stride = p.aux_batch_stride, q.status = p.status;
            q.splits = route.ranges;
            gemm_small(map_a, p.b_mn_major ? map_b : make_map(bt, true, BK, 64), q, (int)batch, dev.sms, s);
            return false;
        }
        if (first_use_on_device((const void*)gemm_tcgen05_pair)) {
            LB_CUDA(cudaFuncSetAttribute(gemm_tcgen05, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
            LB_CUDA(cudaFuncSetAttribute(gemm_tcgen05_pair, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemBytes));
        }
        const int max_pairs = resident_pairs(dev);
        long long tiles = (long long)p.tiles_m * p.tiles_n * batch;
        const int sms = dev.sms;
        p.splits = route.splits, p.kb_per_split = route.kb_per_split;
        p.partial = (float*)scratch;
        if (tiles * p.splits > INT32_MAX) fail(LB_ERR_UNSUPPORTED, "gemm: too many output tiles for one launch");
        p.by_tiles.set((uint32_t)tiles), p.by_batch.set((uint32_t)(p.tiles_m * p.tiles_n));
        p.group_m = std::min(p.group_m, p.tiles_m);
        p.by_group.set((uint32_t)(p.group_m * p.tiles_n)), p.by_rows.set((uint32_t)p.group_m);
        p.by_last_rows.set((uint32_t)(p.tiles_m % p.group_m ? p.tiles_m % p.group_m : p.group_m));
        if (pairs) {
            const int resident = max_pairs > 0 ? max_pairs : sms / 2;
            int grid = 2 * (int)std::min<long long>(tiles * p.splits, resident);
            launch_overlapped(gemm_tcgen05_pair, dim3((unsigned)grid), dim3(kThreads), kPairSmemBytes, s, 0, map_a, map_b, p);
        } else {
            int grid = (int)std::min<long long>(tiles * p.splits, sms);
            launch_overlapped(gemm_tcgen05, dim3((unsigned)grid), dim3(kThreads), kSmemBytes, s, 0, map_a, map_b, p);
        }
        if (p.splits > 1) {
            const size_t quad = d.dtype == LB_F32 ? 16 : 8;  // bytes of four elements
            const bool vec = N % 4 == 0 && p.ldd % 4 == 0 && p.d_batch_stride % 4 == 0 && (uintptr_t)p.d % quad == 0 &&
                             (epilogue < EPI_ADD || (p.ld_aux % 4 == 0 && p.aux_batch_stride % 4 == 0 && (uintptr_t)p.aux % 8 == 0));
            const long long items = (long long)batch * M * N / (vec ? 4 : 1);
            const dim3 blocks((unsigned)std::min<long long>((items + 255) / 256, sms * 8));
            if (vec) launch_overlapped(splitk_reduce<true>, blocks, dim3(256), 0, s, 0, (const float*)p.partial, p);
            else launch_overlapped(splitk_reduce<false>, blocks, dim3(256), 0, s, 0, (const float*)p.partial, p);
        }
        return false;
    }

    SimtArgs p{};
    if (epilogue >= EPI_ADD) p.aux = aux.ptr, p.ld_aux = aux.sr, p.aux_sb = aux.batch > 1 ? aux.sb : 0;
    p.M = (int)M, p.N = (int)N, p.K = (int)K, p.batch = (int)batch;
    p.a_sm = a.sr, p.a_sk = a.sc, p.a_sb = a.batch > 1 ? a.sb : 0;
    p.b_sk = b.sr, p.b_sn = b.sc, p.b_sb = b.batch > 1 ? b.sb : 0;
    p.ldd = d.sr, p.d_sb = d.batch > 1 ? d.sb : 0;
    p.d = d.ptr, p.d_dtype = d.dtype, p.epilogue = epilogue;
    auto vec = [](const View3& v, long long along, long long across) {  // the strides the kernel fetches along and across
        const uintptr_t group = v.dtype == LB_F32 ? 16 : 8;
        return along == 1 && across % 4 == 0 && (v.batch == 1 || v.sb % 4 == 0) && (uintptr_t)v.ptr % group == 0;
    };
    p.a_vec = p.a_sk == 1 ? vec(a, p.a_sk, p.a_sm) : vec(a, p.a_sm, p.a_sk);
    p.b_vec = p.b_sn == 1 ? vec(b, p.b_sn, p.b_sk) : vec(b, p.b_sk, p.b_sn);
    if (held) {
        *held = SimtProblem{a.ptr, b.ptr, p};
        return true;
    }
    gemm_simt(a.ptr, b.ptr, a.dtype, p, device_info().sms, s);
    return false;
}

}  // namespace lb

extern "C" {

int lb_gemm(const lb_tensor* a, const lb_tensor* b, const lb_gemm_out* out, const lb_gemm_cfg* cfg, void* stream) {
    return lb::guarded([&] {
        if (!a || !b || !out) lb::fail(LB_ERR_INVALID, "lb_gemm: null argument");
        lb::GemmTuning tuning{cfg ? cfg->splits : 0, cfg ? cfg->group_m : 0};
        lb::gemm(*a, *b, out->product, out->epilogue, cfg ? cfg->kernel : 0, stream, cfg ? cfg->scratch : nullptr,
                 cfg ? cfg->scratch_bytes : 0, out->epilogue >= 2 ? &out->aux : nullptr, &tuning, nullptr);
    });
}

size_t lb_gemm_scratch_bytes(int64_t m, int64_t n, int64_t k, int64_t batch) { return lb::gemm_scratch_bytes(m, n, k, batch); }

size_t lb_gemm_step_scratch_bytes(int64_t m, int64_t n, int64_t k) { return lb::gemm_step_scratch_bytes(m, n, k, 1); }

size_t lb_gemm_operands_scratch_bytes(const lb_tensor* a, const lb_tensor* b) {
    size_t bytes = 0;
    lb::guarded([&] {
        if (!a || !b) lb::fail(LB_ERR_INVALID, "lb_gemm_operands_scratch_bytes: null argument");
        const lb::View3 x = lb::view3(*a, "a"), y = lb::view3(*b, "b");
        bool a_cols, b_cols;
        if (lb::tensor_core_operands(x, y, a_cols, b_cols)) bytes = lb::gemm_step_scratch_bytes(x.rows, y.cols, x.cols, x.batch);
    });
    return bytes;
}

int lb_device_status(void) {
    int status = 0;
    int rc = lb::guarded([&] { status = lb::read_status(); });
    if (rc != LB_OK) return rc;
    if (status != 0) lb::set_last_error("a device-side wait ran out of its poll budget (kernel wound down early)");
    return status;
}
}
