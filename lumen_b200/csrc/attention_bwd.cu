// Flash-attention backward for sm_100a: FlashAttention-2's recompute-from-log-sum-exp backward as the reference
// traces it (lumen/functional/attention/flash.py:51-85) and as its Triton backend runs it in deterministic mode
// (dkdv_kernel + dq_kernel, lumen/codegen/attention/triton/kernel.py:108-264); the reference's CUDA backend has a
// backward kernel that is never launched (lumen/codegen/attention/README.md:27-28).
//
//   delta = rowsum(dO * O)                                    attention_delta (CUDA cores, HBM bound)
//   P^T   = exp(scale * K Q^T - lse),  dP^T = V dO^T           per (key tile, query tile)
//   dS^T  = P^T * (dP^T - delta) * scale   (rounded to bf16),  P^T rounded to bf16
//   dV   += P^T dO,  dK += dS^T Q,  dQ += dS K
//
// One kernel template runs in two modes. Both keep a 128-row pair of tiles resident in shared memory, stream tile pairs
// through a TMA ring, compute X = R1 T1^T and Y = R2 T2^T with tcgen05.mma into tensor memory, turn them into bf16 P and
// Z = dS (one row per thread, written back to tensor memory as operands) and accumulate in tensor memory:
//   dK/dV mode: CTA = (key tile, kv head, batch); R = (K, V), T = (Q, dO) over every query head of the group and
//               every query tile that sees the keys; acc_a = dK += Z Q, acc_b = dV += P dO.
//   dQ mode:    CTA = (query tile, head, batch); R = (Q, dO), T = (K, V) over the visible key tiles; acc_a = dQ += Z K.
// No atomics: every output element is produced by one CTA in a fixed order (bit-reproducible run to
// run, as the reference's deterministic mode requires, tests/functional/test_attention.py:403-407).
//
// Head dim 128, with scratch for it: dK/dV mode leaves dS in memory and attention_dq.cu takes dQ from it, in place of dQ mode, which
// computes it again (every bit the same). us of the kernels at batch 8, 32 heads, sequence 4096, causal: 1750 + 1365 -> 2020 + 725, the
// whole backward 3140 -> 2900; 4 x 32 heads on 8, 512 tokens 70.6 -> 58.7; 2 x 16, 1024 63.8 -> 54.5; 1 x 8, 256 17.1 -> 14.1; over 44
// shapes of 128 to 8192 tokens 0.80 - 1.02 of the time.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "attention_dq.h"
#include "device.h"
#include "launch.cuh"
#include "sm100.cuh"

namespace lb {
CUtensorMap attention_map_rows(const lb_tensor& t, const char* what, int box_rows);
// attention_bwd_atomic.cu: the single-kernel form (head dim 64) that adds dQ into a zeroed float32 accumulator
bool attention_bwd_atomic_supported(const lb_tensor& q, const lb_tensor& dq);
size_t attention_bwd_atomic_scratch_bytes(const lb_tensor& q);
void attention_bwd_atomic_launch(const lb_attn_desc& desc, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mq,
                                 const CUtensorMap& mdo, const lb_tensor& q, const lb_tensor& k, const float* lse, const float* delta,
                                 float* dq_acc, const lb_tensor& dq, const lb_tensor& dk, const lb_tensor& dv, cudaStream_t s);
namespace {

using namespace sm100;

constexpr int BR = 128;  // resident rows (thread = row)
// warp 0: TMA, warp 1: MMA + TMEM owner, then two compute warpgroups, each on half of the BT streamed columns of every
// iteration. X is free as soon as every thread has loaded it: the next tile's X product is issued while this tile's
// element-wise phase runs, and the exponentials (X alone) do not wait for Y.
//  dK/dV mode: P and Z are written over Y's columns (each thread's over the columns it read), so the next Y follows the
//  accumulation products that read them - the tensor pipe runs in order - and the serial chain per tile is accumulate,
//  Y, signalling and the Z half of the element-wise work.
//  dQ mode: the second accumulator's columns hold Z, Y is handed back like X, and both products of the next tile run
//  under this tile's element-wise phase.
//
//  BT = 128 (head dim 128): one CTA per SM on all 512 columns (X 128, Y 128, accumulators 2 x 128). A product with both
//  operands in shared memory reads its 128 x 16 A operand in about 68 cycles whatever N is, so 64 streamed columns - as
//  the two-buffer form this replaces had, on alternating warpgroups - paid for 128: the tensor unit was busy for 67 %
//  of the kernels' time at 41 % of its rate. Batch 8, 32 heads, sequence 4096, causal: backward 4.66 -> 3.48 ms
//  (790 TFLOP/s), of which 0.26 came from issuing the products warp-wide.
//  BT = 64 at head dim 128: one, three or five blocks of 64 streamed rows, which 128-row tiles would fill to a half at the end
//  (launch_bwd).
//  BT = 64 (head dim 64): 256 columns and half the shared memory, so that TWO CTAs share an SM and one CTA's prologue,
//  epilogue and element-wise latency are covered by the other's products (128 and one CTA: 470 -> 548 us at batch 8,
//  16 heads, sequence 2048).

struct BwdArgs {
    int B, N, Nkv, Sq, Sk;
    int causal;
    long long causal_offset;
    float scale, scale_log2;
    const float* lse;    // [B, N, Sq]
    const float* delta;  // [B, N, Sq]
    void* out_a;         // dK (dkdv mode) or dQ (dq mode): bf16 [B, S, heads, D] view
    long long a_sb, a_ss, a_sn;
    void* out_b;         // dV (dkdv mode)
    long long b_sb, b_ss, b_sn;
    int batch0, head0;   // the launch's first batch entry and first head (kv head in dkdv mode)
    uint8_t* scores;     // with kHands: where dS is left for attention_dq
    DsLayout ds;
    int* status;
};

// TILE: the streamed rows of a tile, BT, and kHands where dK/dV mode leaves dS. Chosen at run time, the 32 registers and the stores of dS cost
// the kernel of plans and of calls without scratch up to 7 % (the whole backward, us, 4 x 32 heads on 8 x 512 69.7 -> 74.8, 1 x 8 x 8192 404 ->
// 431, 8 x 32 x 4096 3234 -> 3285).
constexpr int kHands = 1;
template <int D, bool DKDV, int TILE>
struct BwdConfig {
    static constexpr int BT = TILE & ~kHands;
    static constexpr int kCtas = D == 64 ? 2 : 1;        // per SM
    static constexpr int kFirst = BT == 64 ? 2 : 4;      // first compute warp (register budgets are set per aligned group of four warps)
    static constexpr int kThreads = 32 * kFirst + 256;
    static constexpr int kTmemCols = 512 / kCtas;
    static constexpr int kResident = BR * D * 2, kStream = BT * D * 2;
    // rings of streamed tiles: T1 is read until the tile's accumulation has completed, T2 in dQ mode only by Y
    static constexpr int S1 = BT == 64 ? 4 : (DKDV ? 2 : 3), S2 = BT == 64 ? 4 : 2;
    static constexpr int kCols = BT / 2;                 // streamed columns of one thread
    static constexpr int kStats = DKDV ? 8 * 2 * kCols * 4 : 0;
    static constexpr int kBytes = 2 * kResident + (S1 + S2) * kStream + 1024 + 256 + kStats;  // tiles, alignment, barriers, column statistics
    // BT = 128: what the compiler assigns under __launch_bounds__(384, 1) and the roles' budgets (setmaxnreg)
    static constexpr int kLaunchRegs = 168, kRegsLight = 72, kRegsCompute = 216;
    static_assert(BT == 64 || 128 * kRegsLight + 256 * kRegsCompute <= kLaunchRegs * kThreads, "register budgets exceed the launch allocation");
    static_assert(2 * BT + 2 * D <= kTmemCols && (2 * (S1 + S2) + 9) * 8 + 8 <= 256, "tensor memory / barrier space");
};

template <int D, bool DKDV, int TILE>
__global__ void __launch_bounds__(BwdConfig<D, DKDV, TILE>::kThreads, BwdConfig<D, DKDV, TILE>::kCtas)
attention_bwd_kernel(const __grid_constant__ CUtensorMap map_r1, const __grid_constant__ CUtensorMap map_r2,
                     const __grid_constant__ CUtensorMap map_t1, const __grid_constant__ CUtensorMap map_t2, const BwdArgs p) {
    using C = BwdConfig<D, DKDV, TILE>;
    constexpr bool HANDS = (TILE & kHands) != 0;
    static_assert(!HANDS || (D == 128 && DKDV && C::BT == 128), "what attention_dq reads");
    constexpr int BT = C::BT, kResident = C::kResident, kStream = C::kStream, S1 = C::S1, S2 = C::S2, kTmemCols = C::kTmemCols, COLS = C::kCols;
    constexpr int kRBlock = BR * 128, kTBlock = BT * 128;  // bytes of one 64-wide head-dim block of a tile
    constexpr int DB = D / 64;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align_1024(smem_raw);
    uint8_t* sr1 = smem;
    uint8_t* sr2 = smem + kResident;
    uint8_t* st1 = smem + 2 * kResident;
    uint8_t* st2 = st1 + S1 * kStream;
    uint64_t* bars = (uint64_t*)(st2 + S2 * kStream);
    uint64_t* r_full = bars;             // 1
    uint64_t* t1_full = bars + 1;        // S1
    uint64_t* t1_empty = t1_full + S1;   // S1
    uint64_t* t2_full = t1_empty + S1;   // S2
    uint64_t* t2_empty = t2_full + S2;   // S2
    uint64_t* x_full = t2_empty + S2;    // X is in tensor memory
    uint64_t* y_full = x_full + 1;       // Y is
    uint64_t* x_empty = y_full + 1;      // every compute thread has loaded its X values
    uint64_t* y_empty = x_empty + 1;     // dQ mode: ... its Y values
    uint64_t* pz_ready = y_empty + 1;    // every compute thread has written P and Z
    uint64_t* z_free = pz_ready + 1;     // dQ mode: the accumulation that read Z has completed
    uint64_t* acc_full = z_free + 1;     // everything has
    uint32_t* tmem_slot = (uint32_t*)(acc_full + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    // dkdv mode: minus the log-sum-exp (in log2 units) and minus delta * scale of a compute warp's streamed columns, one
    // private copy per warp ([warp][lse|delta][COLS]) so that staging needs no barrier across warps
    float* col_stats = (float*)((uint8_t*)bars + 256);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp-uniform for the compiler too
    const int tile = DKDV ? (int)blockIdx.x : (int)(gridDim.x - 1 - blockIdx.x);
    const int head = p.head0 + (int)blockIdx.y, batch = p.batch0 + (int)blockIdx.z;  // kv head in dkdv mode, query head in dq mode
    const int group = p.N / p.Nkv;
    const int r0 = tile * BR;

    // streamed rows, per head: tiles of BT from stream0 on; heads_here heads are walked in dkdv mode. Whole blocks of 64 rows that
    // no resident row sees (or that see none) are left out at either tile height: their weights would be 0, but 0 times a NaN is not.
    int stream0, per_head, heads_here;
    if (DKDV) {
        // queries that see at least the first key of this tile: i >= r0 - offset
        const long long first_q = p.causal ? min((long long)p.Sq, max(0LL, (long long)r0 - p.causal_offset)) : 0LL;
        stream0 = (int)(first_q / 64) * 64;
        per_head = (p.Sq - stream0 + BT - 1) / BT;
        if (first_q >= p.Sq) per_head = 0;
        heads_here = group;
    } else {
        const long long last_key = p.causal ? min((long long)p.Sk - 1, (long long)r0 + BR - 1 + p.causal_offset) : (long long)p.Sk - 1;
        const int blocks = last_key < 0 ? 0 : (int)(last_key / 64) + 1;
        stream0 = BT == 128 && blocks % 2 ? -64 : 0;  // an odd block: the first tile starts before the keys (TMA reads zeros there)
        per_head = (blocks * 64 - stream0) / BT;
        heads_here = 1;
    }
    const int n_iter = per_head * heads_here;
    const int r_head = head;                          // resident tiles: kv head (dkdv) / query head (dq)
    const int kv_head_of_q = DKDV ? head : head / group;

    if (threadIdx.x == 0) {
        mbar_init(r_full, 1);
        for (int s = 0; s < S1; s++) {
            mbar_init(&t1_full[s], 1);
            mbar_init(&t1_empty[s], 1);
        }
        for (int s = 0; s < S2; s++) {
            mbar_init(&t2_full[s], 1);
            mbar_init(&t2_empty[s], 1);
        }
        mbar_init(x_full, 1);
        mbar_init(y_full, 1);
        mbar_init(x_empty, 256);
        mbar_init(y_empty, 256);
        mbar_init(pz_ready, 256);
        mbar_init(z_free, 1);
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    grid_wait();
    const uint32_t tmem_x = tmem_base;
    const uint32_t tmem_y = tmem_base + BT;
    const uint32_t tmem_a = tmem_base + 2 * BT;  // acc_a: D columns
    const uint32_t tmem_b = tmem_a + D;          // acc_b: D columns (dkdv mode)
    // bf16 values of 16 streamed rows take 8 columns; a warpgroup's lie within the COLS columns it read: in dkdv mode P in
    // the first and Z in the second half of them
    auto pz_col = [](int k) { return k / (COLS / 16) * COLS + k % (COLS / 16) * 8; };  // k-th group of 16 streamed rows
    const uint32_t tmem_p = tmem_y;
    const uint32_t tmem_z = DKDV ? tmem_y + COLS / 2 : tmem_b;

    // each register budget is set inside the branch it governs: code after a join is compiled for the smallest one
    if (warp < C::kFirst) {
      if constexpr (BT == 128) regs_dec<C::kRegsLight>();
      if (warp == 0) {
        if (lane == 0 && n_iter > 0) {
            tma_prefetch_desc(&map_r1);
            tma_prefetch_desc(&map_r2);
            tma_prefetch_desc(&map_t1);
            tma_prefetch_desc(&map_t2);
            mbar_expect_tx(r_full, 2 * kResident);
            for (int d = 0; d < DB; d++) {
                tma_load_4d(sr1 + d * kRBlock, &map_r1, r_full, d * 64, r_head, r0, batch);
                tma_load_4d(sr2 + d * kRBlock, &map_r2, r_full, d * 64, r_head, r0, batch);
            }
            bool ok = true;
            for (int it = 0; it < n_iter && ok; it++) {
                const int a = it % S1, b = it % S2;
                const int hh = it / per_head;
                const int row0 = stream0 + (it - hh * per_head) * BT;
                const int t_head = DKDV ? head * group + hh : kv_head_of_q;
                if (!(ok = mbar_wait(&t1_empty[a], ((uint32_t)(it / S1) & 1) ^ 1, abort_flag))) break;
                mbar_expect_tx(&t1_full[a], kStream);
                for (int d = 0; d < DB; d++) tma_load_4d(st1 + a * kStream + d * kTBlock, &map_t1, &t1_full[a], d * 64, t_head, row0, batch);
                if (!(ok = mbar_wait(&t2_empty[b], ((uint32_t)(it / S2) & 1) ^ 1, abort_flag))) break;
                mbar_expect_tx(&t2_full[b], kStream);
                for (int d = 0; d < DB; d++) tma_load_4d(st2 + b * kStream + d * kTBlock, &map_t2, &t2_full[b], d * 64, t_head, row0, batch);
            }
            ok = ok && mbar_wait_ring<S1>(t1_empty, (uint32_t)n_iter, abort_flag) && mbar_wait_ring<S2>(t2_empty, (uint32_t)n_iter, abort_flag);
            if (!DKDV && ok) mbar_wait(z_free, (uint32_t)(n_iter - 1) & 1, abort_flag);
        }
      } else if (warp == 1) {
        if (n_iter > 0) {  // the whole warp: the operands stay in uniform registers
            const bool leader = elect_one();
            const uint32_t idesc_xy = make_idesc(BR, BT, true, false, false);
            const uint32_t idesc_acc = make_idesc(BR, D, true, false, true);
            bool ok = mbar_wait_warp(r_full, 0, abort_flag);
            // descriptors are built once and advanced by adds
            const uint64_t dr1 = make_smem_desc(smem_u32(sr1), 16, 1024), dr2 = make_smem_desc(smem_u32(sr2), 16, 1024);
            const uint64_t dt1 = make_smem_desc(smem_u32(st1), 16, 1024), dt2 = make_smem_desc(smem_u32(st2), 16, 1024);
            const uint64_t dt1_mn = make_smem_desc(smem_u32(st1), kTBlock, 1024), dt2_mn = make_smem_desc(smem_u32(st2), kTBlock, 1024);
            auto issue_x = [&](int it) -> bool {
                const int stage = it % S1;
                if (!mbar_wait_warp(&t1_full[stage], (uint32_t)(it / S1) & 1, abort_flag)) return false;
                tc_fence_after();
                const uint64_t t1 = desc_advance(dt1, (uint32_t)(stage * kStream));
#pragma unroll
                for (int k = 0; k < D / 16; k++) {
                    const uint32_t roff = (uint32_t)((k / 4) * kRBlock + (k % 4) * 32), toff = (uint32_t)((k / 4) * kTBlock + (k % 4) * 32);
                    mma_f16(tmem_x, desc_advance(dr1, roff), desc_advance(t1, toff), idesc_xy, k != 0, leader);
                }
                mma_commit(x_full, leader);
                return true;
            };
            auto issue_y = [&](int it) -> bool {
                const int stage = it % S2;
                if (!mbar_wait_warp(&t2_full[stage], (uint32_t)(it / S2) & 1, abort_flag)) return false;
                tc_fence_after();
                const uint64_t t2 = desc_advance(dt2, (uint32_t)(stage * kStream));
#pragma unroll
                for (int k = 0; k < D / 16; k++) {
                    const uint32_t roff = (uint32_t)((k / 4) * kRBlock + (k % 4) * 32), toff = (uint32_t)((k / 4) * kTBlock + (k % 4) * 32);
                    mma_f16(tmem_y, desc_advance(dr2, roff), desc_advance(t2, toff), idesc_xy, k != 0, leader);
                }
                mma_commit(y_full, leader);
                if (!DKDV) mma_commit(&t2_empty[stage], leader);
                return true;
            };
            if (ok) ok = issue_x(0) && issue_y(0);
            for (int it = 0; it < n_iter && ok; it++) {
                const uint32_t par = (uint32_t)it & 1;
                if (it + 1 < n_iter) {
                    if (!(ok = mbar_wait_warp(x_empty, par, abort_flag))) break;
                    tc_fence_after();
                    if (!(ok = issue_x(it + 1))) break;
                    if (!DKDV) {
                        if (!(ok = mbar_wait_warp(y_empty, par, abort_flag))) break;
                        tc_fence_after();
                        if (!(ok = issue_y(it + 1))) break;
                    }
                }
                if (!(ok = mbar_wait_warp(pz_ready, par, abort_flag))) break;
                tc_fence_after();
                const int a = it % S1, b = it % S2;
                const uint64_t t1 = desc_advance(dt1_mn, (uint32_t)(a * kStream)), t2 = desc_advance(dt2_mn, (uint32_t)(b * kStream));
#pragma unroll
                for (int k = 0; k < BT / 16; k++)  // acc_a += Z . T1   (T1 as an MN-major operand: 16 rows = 2048 bytes per step)
                    mma_f16_ts(tmem_a, tmem_z + pz_col(k), desc_advance(t1, k * 2048), idesc_acc, (it | k) != 0, leader);
                mma_commit(&t1_empty[a], leader);
                if (DKDV) {
#pragma unroll
                    for (int k = 0; k < BT / 16; k++)  // acc_b += P . T2
                        mma_f16_ts(tmem_b, tmem_p + pz_col(k), desc_advance(t2, k * 2048), idesc_acc, (it | k) != 0, leader);
                    mma_commit(&t2_empty[b], leader);
                    if (it + 1 < n_iter) ok = issue_y(it + 1);  // behind the products that read P and Z in Y's columns: the tensor pipe runs in order
                } else {
                    mma_commit(z_free, leader);
                }
            }
            if (ok) mma_commit(acc_full, leader);
        }
      }
    } else {
        if constexpr (BT == 128) regs_inc<C::kRegsCompute>();
        // ---- compute warps: thread = resident row, warpgroup = half of the streamed columns ----
        const int wg = (warp - C::kFirst) >> 2;
        const int quarter = warp & 3;
        const int row_in_tile = quarter * 32 + lane;
        const long long row = (long long)r0 + row_in_tile;  // key index (dkdv) or query index (dq)
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        const uint32_t my_x = tmem_x + lane_addr + wg * COLS, my_y = tmem_y + lane_addr + wg * COLS;
        const float LOG2E = 1.4426950408889634f;
        float row_lse = 0.0f, row_delta = 0.0f;  // negated, as the staged columns' are
        if (!DKDV && row < p.Sq) {
            const long long at = ((long long)batch * p.N + head) * p.Sq + row;
            row_lse = -(p.lse[at] * LOG2E);
            row_delta = -(p.delta[at] * p.scale);
        }
        // dkdv: the lane's share of the next tile's column statistics is fetched one iteration ahead
        float next_lse[COLS / 32], next_delta[COLS / 32];
        auto fetch_stats = [&](int it) {
            const int hh = it / per_head;
            const long long at = ((long long)batch * p.N + (head * group + hh)) * p.Sq;
            const long long c = stream0 + (long long)(it - hh * per_head) * BT + wg * COLS + lane;
#pragma unroll
            for (int u = 0; u < COLS / 32; u++) {
                const long long cc = min(c + 32 * u, (long long)p.Sq - 1);
                next_lse[u] = p.lse[at + cc];
                next_delta[u] = p.delta[at + cc];
            }
        };
        if (DKDV && n_iter > 0) fetch_stats(0);
        uint8_t* scores = nullptr;  // dS of this thread's key and its warpgroup's first block of queries
        if constexpr (HANDS)
            scores = p.scores + ((long long)blockIdx.z * gridDim.y + blockIdx.y) * group * p.ds.head_bytes() + p.ds.at(tile, row_in_tile / 64, stream0 / 64) +
                     wg * kDsHalfBytes + row_in_tile % 64 * 16;
        // A tile's dS leaves between the next one's exponentials, a store for every eight of them: in a row, right behind the hand-over of P and
        // Z, the stores hold up those (the backward of 1 x 8 heads x 4096 157 -> 135 us, of 8 x 32 x 4096 2990 -> 2900).
        uint32_t left[HANDS ? COLS / 2 : 1];
        uint8_t* left_to = nullptr;
        auto leave = [&](int c) { *(uint4*)(left_to + c * 1024) = make_uint4(left[4 * c], left[4 * c + 1], left[4 * c + 2], left[4 * c + 3]); };
        float* stat_lse = col_stats + (warp - C::kFirst) * 2 * COLS;
        float* stat_delta = stat_lse + COLS;
        bool ok = true;
        for (int it = 0; it < n_iter && ok; it++) {
            const uint32_t par = (uint32_t)it & 1;
            const int hh = it / per_head;
            const long long c0 = stream0 + (long long)(it - hh * per_head) * BT + wg * COLS;  // this thread's first streamed index: query (dkdv) or key (dq)
            if (DKDV) {
                // each warp stages its columns' log-sum-exps and deltas once; its lanes then read them as shared-memory
                // broadcasts instead of two global loads per score
                __syncwarp();  // every lane is done with the previous tile's values
#pragma unroll
                for (int u = 0; u < COLS / 32; u++) {
                    stat_lse[lane + 32 * u] = -(next_lse[u] * LOG2E);
                    stat_delta[lane + 32 * u] = -(next_delta[u] * p.scale);
                }
                __syncwarp();
                if (it + 1 < n_iter) fetch_stats(it + 1);
            }
            // columns visible to this row: dkdv: query i sees key `row` iff row <= i + off  <=>  i >= row - off, and i < Sq
            //                              dq:   key j visible iff j <= row + off and j < Sk
            long long col_lo, col_hi;  // visible columns are [col_lo, col_hi)
            if (DKDV) {
                col_lo = p.causal ? row - p.causal_offset : 0;
                col_hi = p.Sq;
                if (HANDS && row >= p.Sk) col_hi = 0;  // what is left for these is multiplied by zeros and must be finite
            } else {
                col_lo = 0;
                col_hi = p.causal ? min((long long)p.Sk, row + p.causal_offset + 1) : (long long)p.Sk;
            }
            // visible range [lo, hi) relative to the thread's columns, in 32-bit; no mask is applied unless some row of the
            // warp is cut
            const int lo = (int)max(0LL, min(col_lo - c0, (long long)COLS)), hi = (int)max(0LL, min(col_hi - c0, (long long)COLS));
            const bool masked_tile = __any_sync(0xffffffffu, lo > 0 || hi < COLS);
            if (!(ok = mbar_wait(x_full, par, abort_flag))) break;
            __syncwarp();
            tc_fence_after();
            float pr[COLS];
            {
                uint32_t x[COLS];
#pragma unroll
                for (int c = 0; c < COLS; c += 32) tmem_ld_32x32(my_x + c, x + c);
                tmem_ld_wait();
                tc_fence_before();
                mbar_arrive(x_empty);  // X is handed back for the next tile's product
                // two columns per instruction (packed float32 FMA / MUL of sm_100); each lane's roundings are those of the scalar form
#pragma unroll
                for (int i = 0; i < COLS; i += 4) {
                    float4 l4 = make_float4(row_lse, row_lse, row_lse, row_lse);
                    if (DKDV) l4 = *(const float4*)(stat_lse + i);
                    const float2 s2 = make_float2(p.scale_log2, p.scale_log2);
                    const float2 u = __ffma2_rn(make_float2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])), s2, make_float2(l4.x, l4.y));
                    const float2 v = __ffma2_rn(make_float2(__uint_as_float(x[i + 2]), __uint_as_float(x[i + 3])), s2, make_float2(l4.z, l4.w));
                    pr[i] = fast_exp2(u.x), pr[i + 1] = fast_exp2(u.y), pr[i + 2] = fast_exp2(v.x), pr[i + 3] = fast_exp2(v.y);
                    if (HANDS && it > 0 && i % 8 == 4) leave(i / 8);
                }
                if (masked_tile) {
#pragma unroll
                    for (int i = 0; i < COLS; i++)
                        if (i < lo || i >= hi) pr[i] = 0.0f;
                }
            }
            if (!(ok = mbar_wait(y_full, par, abort_flag))) break;
            __syncwarp();
            tc_fence_after();
            uint32_t y[COLS];
#pragma unroll
            for (int c = 0; c < COLS; c += 32) tmem_ld_32x32(my_y + c, y + c);
            tmem_ld_wait();
            if (!DKDV) {
                tc_fence_before();
                mbar_arrive(y_empty);
            }
            uint32_t pz[DKDV ? COLS : COLS / 2];  // P (dkdv mode), then Z, as bf16 pairs
            constexpr int kZ = DKDV ? COLS / 2 : 0;
#pragma unroll
            for (int i = 0; i < COLS; i += 4) {
                float4 d4 = make_float4(row_delta, row_delta, row_delta, row_delta);
                if (DKDV) d4 = *(const float4*)(stat_delta + i);
                const float2 s2 = make_float2(p.scale, p.scale);
                const float2 u = __ffma2_rn(make_float2(__uint_as_float(y[i]), __uint_as_float(y[i + 1])), s2, make_float2(d4.x, d4.y));
                const float2 v = __ffma2_rn(make_float2(__uint_as_float(y[i + 2]), __uint_as_float(y[i + 3])), s2, make_float2(d4.z, d4.w));
                const float2 zu = __fmul2_rn(make_float2(pr[i], pr[i + 1]), u), zv = __fmul2_rn(make_float2(pr[i + 2], pr[i + 3]), v);  // P * (dP - delta) * scale
                const __nv_bfloat162 hu = __floats2bfloat162_rn(zu.x, zu.y), hv = __floats2bfloat162_rn(zv.x, zv.y);
                pz[kZ + i / 2] = *(const uint32_t*)&hu, pz[kZ + i / 2 + 1] = *(const uint32_t*)&hv;
                if (DKDV) {
                    const __nv_bfloat162 pu = __floats2bfloat162_rn(pr[i], pr[i + 1]), pv = __floats2bfloat162_rn(pr[i + 2], pr[i + 3]);
                    pz[i / 2] = *(const uint32_t*)&pu, pz[i / 2 + 1] = *(const uint32_t*)&pv;
                }
            }
            if constexpr (DKDV) {
#pragma unroll
                for (int c = 0; c < COLS; c += 32) tmem_st_32x32(my_y + c, pz + c);
            } else {
                // Z(it) goes where Z(it - 1) was: the accumulation that read it has completed, unless this warp overtook the tensor pipe
                if (it > 0) {
                    if (!(ok = mbar_wait(z_free, par ^ 1, abort_flag))) break;
                    __syncwarp();
                    tc_fence_after();
                }
                if constexpr (COLS == 64) tmem_st_32x32(tmem_z + lane_addr + wg * COLS, pz);
                else tmem_st_32x16(tmem_z + lane_addr + wg * COLS, pz);
            }
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(pz_ready);
            if constexpr (HANDS) {
                left_to = scores + hh * p.ds.head_bytes() + (long long)(it - hh * per_head) * (2 * kDsHalfBytes);
#pragma unroll
                for (int c = 0; c < COLS / 2; c++) left[c] = pz[kZ + c];
            }
        }
        if (HANDS && n_iter > 0 && ok) {
#pragma unroll
            for (int c = 0; c < 8; c++) leave(c);
        }
        // ---- epilogue: accumulators -> bf16 rows ----
        if (n_iter > 0) ok = ok && mbar_wait(acc_full, 0, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            tc_fence_after();
            const long long limit = DKDV ? p.Sk : p.Sq;
            {
                const int which = DKDV ? wg : 0;  // dkdv: warpgroup 0 writes dK, warpgroup 1 dV
                uint16_t* base = (uint16_t*)(which == 0 ? p.out_a : p.out_b);
                const long long sb = which == 0 ? p.a_sb : p.b_sb, ss = which == 0 ? p.a_ss : p.b_ss, sn = which == 0 ? p.a_sn : p.b_sn;
                uint16_t* out = base + (long long)batch * sb + row * ss + (long long)head * sn;
                const bool vec = (sb % 8 == 0) && (ss % 8 == 0) && (sn % 8 == 0) && (((uintptr_t)base & 15) == 0);
#pragma unroll 1
                for (int c = DKDV ? 0 : wg; c < D / 32; c += DKDV ? 1 : 2) {  // dq: the warpgroups take 32-column chunks in turn
                    uint32_t v[32];
                    if (n_iter > 0) {
                        tmem_ld_32x32((which == 0 ? tmem_a : tmem_b) + lane_addr + c * 32, v);
                        tmem_ld_wait();
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; i++) v[i] = 0u;
                    }
                    if (vec && n_iter > 0) {
                        // The warp's 32 rows leave through 2 KB of the first resident tile's shared memory (every product
                        // that read it has completed): whole 64-byte row pieces, eight rows per store instruction.
                        uint4 packed[4];
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            uint32_t w[4];
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[i + 2 * q]), __uint_as_float(v[i + 2 * q + 1]));
                                w[q] = *(uint32_t*)&h;
                            }
                            packed[i / 8] = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                        store_rows_coalesced<4>((uint4*)(sr1 + (warp - C::kFirst) * 2048), packed, (uint8_t*)(out - (long long)lane * ss + c * 32), ss * 2,
                                                (int)max(0LL, min(32LL, limit - (row - lane))), lane);
                    } else if (row < limit) {
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            uint32_t w[4];
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[i + 2 * q]), __uint_as_float(v[i + 2 * q + 1]));
                                w[q] = *(uint32_t*)&h;
                            }
                            if (vec) {
                                *(uint4*)(out + c * 32 + i) = make_uint4(w[0], w[1], w[2], w[3]);
                            } else {
#pragma unroll
                                for (int q = 0; q < 4; q++) {
                                    out[c * 32 + i + 2 * q] = (uint16_t)(w[q] & 0xffff);
                                    out[c * 32 + i + 2 * q + 1] = (uint16_t)(w[q] >> 16);
                                }
                            }
                        }
                    }
                }
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
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// delta[b, n, s] = sum_d dO[b, s, n, d] * O[b, s, n, d] in fp32. D / 8 lanes per (s, n) row, 16 bytes per lane and
// tensor, several rows per warp; heads of one token are adjacent so a warp reads contiguous memory. One grid row
// (blockIdx.y) per batch entry and 32-bit index arithmetic: the kernel is a pure stream of 2 x 16 bytes per thread,
// and 64-bit divisions per thread used to cost more than the loads. `zeros` (optional): the dense float32 accumulator of dQ,
// cleared on the way by the threads of the same rows: a separate clearing stood between this kernel and the next one's early launch.
// us a backward: 8 x 2048 tokens, 16 heads 312.8 -> 305.4; 4 x 512, 16 heads 33.5 -> 30.3; 300 tokens, 8 heads 30.3 -> 27.7.
__global__ void __launch_bounds__(256) attention_delta(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                                                        float* __restrict__ delta, float* zeros, int S, int N, int D, int n_shift, long long o_sb,
                                                        long long o_ss, long long o_sn, long long g_sb, long long g_ss, long long g_sn) {
    grid_wait(o, d_o);
    const int lanes = D >> 3;  // 8 (D = 64) or 16 (D = 128)
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned row = t / (unsigned)lanes;  // (s, n) of this batch entry; lanes is a power of two
    const int part = (int)(t & (unsigned)(lanes - 1));
    const int b = blockIdx.y;
    const bool live = row < (unsigned)S * (unsigned)N;
    float acc = 0.0f;
    unsigned sq = 0, n = 0;
    if (live) {
        if (n_shift >= 0) sq = row >> n_shift, n = row & ((1u << n_shift) - 1u);
        else sq = row / (unsigned)N, n = row - sq * (unsigned)N;
        const uint4 x = __ldg((const uint4*)(o + b * o_sb + (long long)sq * o_ss + (long long)n * o_sn + part * 8));
        const uint4 y = __ldg((const uint4*)(d_o + b * g_sb + (long long)sq * g_ss + (long long)n * g_sn + part * 8));
        if (zeros) {
            float4* z = (float4*)(zeros + ((long long)b * S * N + row) * D + part * 8);
            z[0] = z[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        const __nv_bfloat162* xp = (const __nv_bfloat162*)&x;
        const __nv_bfloat162* yp = (const __nv_bfloat162*)&y;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            acc = fmaf(__low2float(xp[k]), __low2float(yp[k]), acc);
            acc = fmaf(__high2float(xp[k]), __high2float(yp[k]), acc);
        }
    }
    for (int m = lanes / 2; m >= 1; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if (live && part == 0) delta[((long long)b * N + n) * S + sq] = acc;
}

// Launches attention_delta over [B, S, N, D] views of o and dO.
void launch_delta(const lb_tensor& o, const lb_tensor& d_o, float* delta, float* zeros, cudaStream_t s) {
    const long long B = o.shape[0], S = o.shape[1], N = o.shape[2], D = o.shape[3];
    if (S * N * (D / 8) >= (1LL << 31) || B > 65535) fail(LB_ERR_UNSUPPORTED, "attention backward: sequence x heads or batch too large for the delta kernel's grid");
    int n_shift = -1;
    for (int k = 0; k < 31; k++)
        if ((1LL << k) == N) n_shift = k;
    const unsigned blocks = (unsigned)((S * N * (D / 8) + 255) / 256);
    launch_overlapped(attention_delta, dim3(blocks, (unsigned)B), dim3(256), 0, s, 0, (const __nv_bfloat16*)o.ptr, (const __nv_bfloat16*)d_o.ptr, delta, zeros,
                      (int)S, (int)N, (int)D, n_shift, o.stride[0], o.stride[1], o.stride[2], d_o.stride[0], d_o.stride[1], d_o.stride[2]);
}

template <int D, bool DKDV, int TILE>
void launch_bwd_kernel(const CUtensorMap& r1, const CUtensorMap& r2, const CUtensorMap& t1, const CUtensorMap& t2, dim3 grid, const BwdArgs& p,
                       cudaStream_t s) {
    using C = BwdConfig<D, DKDV, TILE>;
    if (first_use_on_device((const void*)attention_bwd_kernel<D, DKDV, TILE>))
        LB_CUDA(cudaFuncSetAttribute(attention_bwd_kernel<D, DKDV, TILE>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kBytes));
    launch_overlapped(attention_bwd_kernel<D, DKDV, TILE>, grid, dim3(C::kThreads), C::kBytes, s, 0, r1, r2, t1, t2, p);
}

// Of the dS that is left in memory at a time, and the fewest dK/dV CTAs of each of several rounds, whose ends leave SMs idle: batch 8, 32
// heads, sequence 4096, causal, us, dS computed twice 3230, in rounds of 1000 CTAs 3590, of 2000 3400, of 4000 3080, at once 3030; batch 4, 32
// heads, 8192 in two rounds of 4096 0.93 of the time, not causal in four of 2048 1.00.
constexpr size_t kMostScores = (size_t)4608 << 20;
constexpr long long kLeastRound = 3000;

// Whether 128-row tiles are streamed at head dim 128 (see launch_bwd_pair)
bool tall_tiles(long long streamed) { return (streamed + 63) / 64 % 2 == 0 || streamed > 5 * 64; }

// Whether the backward may take dQ from the dS that its dK/dV kernel leaves, and how that lies: head dim 128 with 128-row tiles of queries
// that all start at a multiple of 128.
bool hands_scores(const lb_attn_desc& desc, long long Sq, long long Sk, long long D, DsLayout& ds) {
    if (D != 128 || Sq <= 0 || Sk <= 0 || !tall_tiles(Sq) || Sq > (1 << 24) || Sk > (1 << 24)) return false;
    if (desc.causal && (desc.causal_offset % 128 != 0 || std::abs(desc.causal_offset) > (1 << 24))) return false;
    ds.query_blocks = (int)((Sq + 127) / 128) * 2, ds.key_tiles = (int)((Sk + 127) / 128);
    ds.causal = desc.causal != 0, ds.offset = desc.causal ? (int)(desc.causal_offset / 64) : 0;
    return ds.head_bytes() > 0;
}

// The heads a launch of both kernels takes at once: batch entries whole, or (0) kv heads of one entry; nothing where the rounds would be small.
struct HandedHeads {
    long long batches = 0, kv_heads = 0;
    size_t bytes = 0;
};
HandedHeads handed_heads(const DsLayout& ds, long long B, long long N, long long Nkv, size_t most) {
    const long long kv_head = N / Nkv * ds.head_bytes(), entry = Nkv * kv_head;
    auto even = [](long long all, long long at_once) { return (all + (all + at_once - 1) / at_once - 1) / ((all + at_once - 1) / at_once); };
    HandedHeads h;
    if (entry <= (long long)most) h.batches = even(B, std::min<long long>(B, (long long)most / entry)), h.kv_heads = Nkv, h.bytes = (size_t)(h.batches * entry);
    else if (kv_head <= (long long)most) h.kv_heads = even(Nkv, (long long)most / kv_head), h.bytes = (size_t)(h.kv_heads * kv_head);
    const bool rounds = h.batches < B || h.kv_heads < Nkv;
    return rounds && std::max<long long>(1, h.batches) * h.kv_heads * ds.key_tiles < kLeastRound ? HandedHeads{} : h;
}

// The two kernels; `rows` makes the map of an operand's tiles, 128 or 64 rows high. Head dim 64 streams 64 rows a tile. Head dim 128
// streams 128, but 64 where the streamed rows are one, three or five blocks of 64: the last 128-row tile would be half empty, which
// shows while tiles are few. Measured (us, 128 rows a tile -> 64 for dK/dV and dQ together), 64 x 4 heads: 16 rows 23.4 -> 17.4 and,
// one head to a key head, 16.9 -> 13.7; 160 rows 32.8 -> 28.9, 21.3 -> 19.0; 320 rows 49.0 -> 45.6; two and four blocks are as fast or
// faster with 128 (128 rows 21.6 -> 22.0, 256 30.7 -> 33.5). The 64-row form also stands in where the compiler did not assign the
// registers that the budgets of the 128-row form (setmaxnreg) are drawn from.
// With `scratch` for the dS of some heads (handed_heads), dK/dV leaves it there and attention_dq takes dQ from it, those heads at a time.
template <int D, class Rows>
void launch_bwd_pair(const Rows& rows, const lb_tensor& q, const lb_tensor& d_o, const lb_tensor& k, const lb_tensor& v, const BwdArgs& dkdv,
                     const BwdArgs& dq, void* scratch, const DsLayout& ds, const HandedHeads& handed, cudaStream_t s) {
    const CUtensorMap mq = rows(q, "query", 128), mdo = rows(d_o, "dO", 128), mk = rows(k, "key", 128), mv = rows(v, "value", 128);
    const dim3 grid_kv((unsigned)((dkdv.Sk + BR - 1) / BR), (unsigned)dkdv.Nkv, (unsigned)dkdv.B);
    const dim3 grid_q((unsigned)((dq.Sq + BR - 1) / BR), (unsigned)dq.N, (unsigned)dq.B);
    bool tall_kv = false, tall_q = false;  // 128 streamed rows a tile
    if constexpr (D == 128) {
        static const bool budgets = launch_regs((const void*)attention_bwd_kernel<128, true, 128>) >= BwdConfig<128, true, 128>::kLaunchRegs &&
                                    launch_regs((const void*)attention_bwd_kernel<128, false, 128>) >= BwdConfig<128, false, 128>::kLaunchRegs;
        static const bool hands = launch_regs((const void*)attention_bwd_kernel<128, true, 128 + kHands>) >= BwdConfig<128, true, 128 + kHands>::kLaunchRegs;
        tall_kv = budgets && tall_tiles(dkdv.Sq), tall_q = budgets && tall_tiles(dq.Sk);
        if (hands && tall_kv && scratch && handed.kv_heads) {
            const CUtensorMap keys = rows(k, "key", 64);
            const int group = dq.N / dq.Nkv;
            BwdArgs a = dkdv;
            a.scores = (uint8_t*)scratch, a.ds = ds;
            DqArgs d{};
            d.ds = ds, d.scores = a.scores, d.N = dq.N, d.Nkv = dq.Nkv, d.Sq = dq.Sq, d.Sk = dq.Sk;
            d.dq = dq.out_a, d.sb = dq.a_sb, d.ss = dq.a_ss, d.sn = dq.a_sn, d.status = dq.status;
            const int batches = (int)std::max<long long>(1, handed.batches), heads = (int)handed.kv_heads;
            for (int b = 0; b < dkdv.B; b += batches)
                for (int h = 0; h < dkdv.Nkv; h += heads) {
                    const int nb = std::min(batches, dkdv.B - b), nh = std::min(heads, dkdv.Nkv - h);
                    a.batch0 = d.batch0 = b, a.head0 = h, d.head0 = h * group, d.heads = nh * group;
                    launch_bwd_kernel<128, true, 128 + kHands>(mk, mv, mq, mdo, dim3(grid_kv.x, (unsigned)nh, (unsigned)nb), a, s);
                    attention_dq_launch(keys, nb, d, s);
                }
            return;
        }
        if (tall_kv) launch_bwd_kernel<128, true, 128>(mk, mv, mq, mdo, grid_kv, dkdv, s);
    }
    if (!tall_kv) launch_bwd_kernel<D, true, 64>(mk, mv, rows(q, "query", 64), rows(d_o, "dO", 64), grid_kv, dkdv, s);
    if constexpr (D == 128)
        if (tall_q) launch_bwd_kernel<128, false, 128>(mq, mdo, mk, mv, grid_q, dq, s);
    if (!tall_q) launch_bwd_kernel<D, false, 64>(mq, mdo, rows(k, "key", 64), rows(v, "value", 64), grid_q, dq, s);
}
template <class Rows>
void launch_bwd(long long D, const Rows& rows, const lb_tensor& q, const lb_tensor& d_o, const lb_tensor& k, const lb_tensor& v, const BwdArgs& dkdv,
                const BwdArgs& dq, cudaStream_t s, void* scratch = nullptr, const DsLayout& ds = {}, const HandedHeads& handed = {}) {
    if (D == 128) launch_bwd_pair<128>(rows, q, d_o, k, v, dkdv, dq, scratch, ds, handed, s);
    else launch_bwd_pair<64>(rows, q, d_o, k, v, dkdv, dq, nullptr, ds, handed, s);
}

}  // namespace

// `dq_acc` (optional): a dense float32 [B, Sq, N, H] accumulator. With it, and where the single-kernel form applies
// (head dim 64), dQ is summed there atomically over the key blocks - in no fixed order, as the reference's backend does
// unless `deterministic` (lumen/codegen/attention/triton/mod.rs:458-466) - and rounded to dq afterwards.
void attention_bwd(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o,
                   const lb_tensor& d_o, const lb_tensor& lse, const lb_tensor& delta, const lb_tensor& dq, const lb_tensor& dk,
                   const lb_tensor& dv, void* stream, const lb_tensor* dq_acc, void* scratch, size_t scratch_bytes) {
    const long long B = q.shape[0], Sq = q.shape[1], N = q.shape[2], D = q.shape[3];
    if (q.rank != 4 || k.rank != 4 || v.rank != 4) fail(LB_ERR_INVALID, "attention backward: operands must be [B, S, N, H] tensors");
    const long long Sk = k.shape[1], Nkv = k.shape[2];
    if (k.shape[0] != B || v.shape[0] != B || k.shape[3] != D || v.shape[1] != Sk || v.shape[2] != Nkv || v.shape[3] != D || Nkv == 0 || N % Nkv)
        fail(LB_ERR_INVALID, "attention backward: shapes are not [B,Sq,N,H], [B,Sk,Nkv,H], [B,Sk,Nkv,H] with N a multiple of Nkv");
    if (D != 64 && D != 128) fail(LB_ERR_UNSUPPORTED, "attention backward: head dims 64 and 128 have a tcgen05 kernel (the reference supports up to 128)");
    if (!(desc.scale > 0.0f)) fail(LB_ERR_UNSUPPORTED, "attention: the softmax scale must be positive");
    auto same = [&](const lb_tensor& t, const lb_tensor& like, const char* what) {
        if (t.rank != 4 || t.dtype != LB_BF16 || t.stride[3] != 1)
            fail(LB_ERR_INVALID, format("attention backward: %s must be a bfloat16 [B, S, N, H] view with a unit head-dim stride", what));
        for (int d = 0; d < 4; d++)
            if (t.shape[d] != like.shape[d]) fail(LB_ERR_INVALID, format("attention backward: %s has the wrong shape", what));
    };
    same(o, q, "o"), same(d_o, q, "dO"), same(dq, q, "dQ"), same(dk, k, "dK"), same(dv, v, "dV");
    if (B == 0 || N == 0) return;  // nothing to compute: no launch
    check_dense(lse, LB_F32, {B, N, Sq}, "attention log-sum-exp");
    check_dense(delta, LB_F32, {B, N, Sq}, "attention delta");
    driver();
    cudaStream_t s = (cudaStream_t)stream;
    const bool atomic = dq_acc && attention_bwd_atomic_supported(q, dq);
    if (atomic) {
        check_dense(*dq_acc, LB_F32, {B, Sq, N, D}, "attention dQ accumulator");
        if (((uintptr_t)dq_acc->ptr & 15) != 0) fail(LB_ERR_UNSUPPORTED, "attention backward: the dQ accumulator must be 16-byte aligned");
    }
    if (Sq > 0) {
        if (o.stride[0] % 8 || o.stride[1] % 8 || o.stride[2] % 8 || d_o.stride[0] % 8 || d_o.stride[1] % 8 || d_o.stride[2] % 8 ||
            ((uintptr_t)o.ptr & 15) || ((uintptr_t)d_o.ptr & 15))
            fail(LB_ERR_UNSUPPORTED, "attention backward: o and dO rows must be 16-byte aligned");
        launch_delta(o, d_o, (float*)delta.ptr, atomic ? (float*)dq_acc->ptr : nullptr, s);
    }
    BwdArgs a{};
    a.B = (int)B, a.N = (int)N, a.Nkv = (int)Nkv, a.Sq = (int)Sq, a.Sk = (int)Sk;
    a.causal = desc.causal, a.causal_offset = desc.causal_offset;
    a.scale = desc.scale, a.scale_log2 = desc.scale * 1.4426950408889634f;
    a.lse = (const float*)lse.ptr, a.delta = (const float*)delta.ptr;
    a.status = status_word();
    BwdArgs kv = a, qq = a;
    kv.out_a = dk.ptr, kv.a_sb = dk.stride[0], kv.a_ss = dk.stride[1], kv.a_sn = dk.stride[2];
    kv.out_b = dv.ptr, kv.b_sb = dv.stride[0], kv.b_ss = dv.stride[1], kv.b_sn = dv.stride[2];
    qq.out_a = dq.ptr, qq.a_sb = dq.stride[0], qq.a_ss = dq.stride[1], qq.a_sn = dq.stride[2];
    if (Sk == 0 || Sq == 0) fail(LB_ERR_UNSUPPORTED, "attention backward: empty sequences");
    if (atomic) {
        attention_bwd_atomic_launch(desc, attention_map_rows(k, "key", 128), attention_map_rows(v, "value", 128),
                                    attention_map_rows(q, "query", 128), attention_map_rows(d_o, "dO", 128), q, k, a.lse, a.delta, (float*)dq_acc->ptr, dq, dk, dv, s);
        return;
    }
    // dQ rows leave in whole lines there
    DsLayout ds;
    HandedHeads handed;
    const bool aligned = dq.stride[0] % 8 == 0 && dq.stride[1] % 8 == 0 && dq.stride[2] % 8 == 0 && ((uintptr_t)dq.ptr & 15) == 0;
    if (scratch && ((uintptr_t)scratch & 15) == 0 && aligned && hands_scores(desc, Sq, Sk, D, ds)) handed = handed_heads(ds, B, N, Nkv, scratch_bytes);
    launch_bwd(D, attention_map_rows, q, d_o, k, v, kv, qq, s, scratch, ds, handed);
}

// Scratch with which the backward hands dS on: that of as many heads as kMostScores holds, 0 where it does not.
size_t attention_bwd_scratch_bytes(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k) {
    DsLayout ds;
    if (q.rank != 4 || k.rank != 4 || q.dtype != LB_BF16 || q.shape[0] <= 0 || k.shape[2] <= 0 || q.shape[2] < k.shape[2] || q.shape[2] % k.shape[2]) return 0;
    if (!hands_scores(desc, q.shape[1], k.shape[1], q.shape[3], ds)) return 0;
    return handed_heads(ds, q.shape[0], q.shape[2], k.shape[2], kMostScores).bytes;
}

}  // namespace lb

namespace lb {
bool attention_on_tensor_cores(const lb_tensor& q, const lb_tensor& k, const lb_tensor& v);
void attention_simt_bwd(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o,
                        const lb_tensor& g, const lb_tensor& lse, const lb_tensor& delta, const lb_tensor& dq, const lb_tensor& dk,
                        const lb_tensor& dv, void* stream);
// The same tensor with strides that any kernel takes where a dimension has one element: one batch entry of a plan has a stride of one, which
// sent its backward to the CUDA cores. Those round P and dS to the operands' 16 bits like the tensor-core kernels, and sum in float32 like them
// (the forward does not round its probabilities there, and stays). us, 704 tokens x 16 heads x 64 452 -> 39, 2048 3074 -> 89, 300 x 4 x 128 109 ->
// 38, 440 x 8 x 64 155 -> 37, 64 x 4 x 64 31 -> 32; errors against float64 of dq, dk and dv at eight shapes equal to five digits (0.0023 - 0.0027).
static lb_tensor any_unit_strides(lb_tensor t) {
    for (int d = 0; d < t.rank - 1; d++)
        if (t.shape[d] == 1) t.stride[d] = 0;
    return t;
}
void attention_backward(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o,
                        const lb_tensor& d_o, const lb_tensor& lse, const lb_tensor& delta, const lb_tensor& dq, const lb_tensor& dk,
                        const lb_tensor& dv, void* stream, const lb_tensor* dq_acc, void* scratch, size_t scratch_bytes) {
    auto on_tensor_cores = [&](const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o, const lb_tensor& g) {
        return attention_on_tensor_cores(q, k, v) && attention_on_tensor_cores(g, k, v) && attention_on_tensor_cores(o, k, v) && q.shape[1] > 0 && k.shape[1] > 0;
    };
    const lb_tensor tq = any_unit_strides(q), tk = any_unit_strides(k), tv = any_unit_strides(v), to = any_unit_strides(o), tg = any_unit_strides(d_o);
    if (on_tensor_cores(q, k, v, o, d_o))
        attention_bwd(desc, q, k, v, o, d_o, lse, delta, dq, dk, dv, stream, dq_acc, scratch, scratch_bytes);
    // (what attention_bwd refuses stays on the CUDA cores with such strides: scales that are not positive, accumulators that are not aligned,
    // more entries or heads than a grid's second and third axes take)
    else if (desc.scale > 0.0f && (!dq_acc || ((uintptr_t)dq_acc->ptr & 15) == 0) && tq.shape[0] <= 65535 && tq.shape[2] <= 65535 && on_tensor_cores(tq, tk, tv, to, tg))
        attention_bwd(desc, tq, tk, tv, to, tg, lse, delta, any_unit_strides(dq), any_unit_strides(dk), any_unit_strides(dv), stream, dq_acc, scratch, scratch_bytes);
    else
        attention_simt_bwd(desc, q, k, v, o, d_o, lse, delta, dq, dk, dv, stream);
}
}  // namespace lb

extern "C" int lb_attention_bwd(const lb_attn_desc* desc, const lb_tensor* q, const lb_tensor* k, const lb_tensor* v,
                                const lb_tensor* o, const lb_tensor* d_o, const lb_tensor* lse, const lb_tensor* delta,
                                const lb_tensor* dq, const lb_tensor* dk, const lb_tensor* dv, void* stream) {
    return lb::guarded([&] {
        if (!desc || !q || !k || !v || !o || !d_o || !lse || !delta || !dq || !dk || !dv)
            lb::fail(LB_ERR_INVALID, "lb_attention_bwd: null argument");
        lb::attention_backward(*desc, *q, *k, *v, *o, *d_o, *lse, *delta, *dq, *dk, *dv, stream, nullptr, nullptr, 0);
    });
}

// lb_attention_bwd with scratch for the dS of some of the heads (lb_attention_bwd_scratch_bytes, 16-byte aligned), where it is faster for it
// (attention_dq.cu); without, or with less than one kv head's, lb_attention_bwd.
extern "C" size_t lb_attention_bwd_scratch_bytes(const lb_attn_desc* desc, const lb_tensor* q, const lb_tensor* k) {
    return desc && q && k ? lb::attention_bwd_scratch_bytes(*desc, *q, *k) : 0;
}
extern "C" int lb_attention_bwd_scratch(const lb_attn_desc* desc, const lb_tensor* q, const lb_tensor* k, const lb_tensor* v, const lb_tensor* o,
                                        const lb_tensor* d_o, const lb_tensor* lse, const lb_tensor* delta, const lb_tensor* dq, const lb_tensor* dk,
                                        const lb_tensor* dv, void* scratch, size_t scratch_bytes, void* stream) {
    return lb::guarded([&] {
        if (!desc || !q || !k || !v || !o || !d_o || !lse || !delta || !dq || !dk || !dv)
            lb::fail(LB_ERR_INVALID, "lb_attention_bwd_scratch: null argument");
        lb::attention_backward(*desc, *q, *k, *v, *o, *d_o, *lse, *delta, *dq, *dk, *dv, stream, nullptr, scratch, scratch_bytes);
    });
}

// lb_attention_bwd in the reference backend's default (non-deterministic) mode: with bfloat16 operands of head dim 64
// the backward runs as ONE kernel that adds each key block's dS K into `dq_accum` (dense float32 [B, Sq, N, H], zeroed
// by the call) in no fixed order and rounds it to dq at the end; other operands run exactly as lb_attention_bwd does.
extern "C" int lb_attention_bwd_atomic(const lb_attn_desc* desc, const lb_tensor* q, const lb_tensor* k, const lb_tensor* v,
                                       const lb_tensor* o, const lb_tensor* d_o, const lb_tensor* lse, const lb_tensor* delta,
                                       const lb_tensor* dq_accum, const lb_tensor* dq, const lb_tensor* dk, const lb_tensor* dv, void* stream) {
    return lb::guarded([&] {
        if (!desc || !q || !k || !v || !o || !d_o || !lse || !delta || !dq_accum || !dq || !dk || !dv)
            lb::fail(LB_ERR_INVALID, "lb_attention_bwd_atomic: null argument");
        lb::attention_backward(*desc, *q, *k, *v, *o, *d_o, *lse, *delta, *dq, *dk, *dv, stream, dq_accum, nullptr, 0);
    });
}

// ---- allocation-free variant ---------------------------------------------------------------------------------
// For callers that must not allocate device memory when they call in: code running inside a memory pool that
// forbids cudaMalloc after start-up, inside a region where the allocator is locked, or under a real-time budget
// where an allocation's latency and possible failure are unacceptable. The backward's one piece of scratch, the
// per-row delta = rowsum(dO * O), lives in a fixed array in the library's device image instead of caller memory.
namespace lb {
namespace {

constexpr long long kStaticDeltaFloats = 1LL << 20;  // 4 MiB per GPU that loads the library, held until exit
static __device__ __align__(256) float g_static_delta[kStaticDeltaFloats];
static __device__ __align__(256) int g_static_status[64];

struct StaticSetup {
    bool ready = false;
    float* delta = nullptr;  // DEVICE address of g_static_delta (the symbol's name is only a host-side stand-in)
    int* status = nullptr;
    decltype(Driver::cuTensorMapEncodeTiled) encode = nullptr;
};
StaticSetup g_static[64];
std::mutex g_static_mutex;

// Once per device, with that device current: resolve the device addresses of the static arrays and the tensor-map
// encoder. Nothing here allocates.
const StaticSetup& static_setup() {
    int dev = 0;
    LB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) fail(LB_ERR_UNSUPPORTED, "lb_attention_bwd_static: device index beyond 63");
    std::lock_guard<std::mutex> lock(g_static_mutex);
    StaticSetup& s = g_static[dev];
    if (s.ready) return s;
    cudaError_t err = cudaGetSymbolAddress((void**)&s.delta, g_static_delta);
    if (err != cudaSuccess) fail(LB_ERR_CUDA, format("cudaGetSymbolAddress(delta scratch): %s", cudaGetErrorString(err)));
    err = cudaGetSymbolAddress((void**)&s.status, g_static_status);
    if (err != cudaSuccess) fail(LB_ERR_CUDA, format("cudaGetSymbolAddress(status word): %s", cudaGetErrorString(err)));
    cudaDriverEntryPointQueryResult found;
    void* fn = nullptr;
    err = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found);
    if (err != cudaSuccess || found != cudaDriverEntryPointSuccess || !fn)
        fail(LB_ERR_CUDA, "lb_attention_bwd_static: cuTensorMapEncodeTiled is unavailable");
    s.encode = (decltype(s.encode))fn;
    LB_CUDA(cudaMemset(s.status, 0, sizeof(int)));  // the status word must start at zero
    register_status_word(s.status);                 // lb_device_status() reads (and clears) it with the library's other words
    s.ready = true;
    return s;
}

CUtensorMap static_map(const StaticSetup& s, const lb_tensor& t, const char* what, int box_rows) {
    if (t.rank != 4 || t.dtype != LB_BF16 || t.stride[3] != 1 || ((uintptr_t)t.ptr & 15) || t.stride[0] % 8 || t.stride[1] % 8 || t.stride[2] % 8)
        fail(LB_ERR_UNSUPPORTED, format("lb_attention_bwd_static: %s must be a bfloat16 [B, S, N, H] view with a unit head-dim stride and 16-byte aligned rows", what));
    cuuint64_t dims[4] = {(cuuint64_t)t.shape[3], (cuuint64_t)t.shape[2], (cuuint64_t)t.shape[1], (cuuint64_t)t.shape[0]};
    cuuint64_t strides[3] = {(cuuint64_t)t.stride[2] * 2, (cuuint64_t)t.stride[1] * 2, (cuuint64_t)t.stride[0] * 2};
    if (t.shape[2] == 1) strides[0] = (cuuint64_t)t.shape[3] * 2;
    if (t.shape[1] == 1) strides[1] = strides[0] * t.shape[2];
    if (t.shape[0] == 1) strides[2] = strides[1] * t.shape[1];
    cuuint32_t box[4] = {64, 1, (cuuint32_t)box_rows, 1};
    cuuint32_t elem[4] = {1, 1, 1, 1};
    CUtensorMap map;
    CUresult rc = s.encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, t.ptr, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) fail(LB_ERR_CUDA, format("cuTensorMapEncodeTiled(%s) failed with CUresult %d", what, (int)rc));
    return map;
}

void attention_bwd_static(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o,
                          const lb_tensor& d_o, const lb_tensor& lse, const lb_tensor& dq, const lb_tensor& dk, const lb_tensor& dv,
                          void* stream) {
    if (q.rank != 4 || k.rank != 4 || v.rank != 4) fail(LB_ERR_INVALID, "lb_attention_bwd_static: operands must be [B, S, N, H] tensors");
    const long long B = q.shape[0], Sq = q.shape[1], N = q.shape[2], D = q.shape[3], Sk = k.shape[1], Nkv = k.shape[2];
    if (k.shape[0] != B || v.shape[0] != B || k.shape[3] != D || v.shape[1] != Sk || v.shape[2] != Nkv || v.shape[3] != D || Nkv == 0 || N % Nkv)
        fail(LB_ERR_INVALID, "lb_attention_bwd_static: shapes are not [B,Sq,N,H], [B,Sk,Nkv,H], [B,Sk,Nkv,H] with N a multiple of Nkv");
    if (D != 64 && D != 128) fail(LB_ERR_UNSUPPORTED, "lb_attention_bwd_static: head dims 64 and 128 only");
    if (!(desc.scale > 0.0f)) fail(LB_ERR_UNSUPPORTED, "lb_attention_bwd_static: the softmax scale must be positive");
    if (B <= 0 || N <= 0 || Sq <= 0 || Sk <= 0) fail(LB_ERR_UNSUPPORTED, "lb_attention_bwd_static: empty operands");
    if (B * N * Sq > kStaticDeltaFloats)
        fail(LB_ERR_INVALID, format("lb_attention_bwd_static: batch * heads * query length = %lld exceeds the built-in scratch of %lld rows; "
                                    "use lb_attention_bwd with caller-provided scratch", B * N * Sq, kStaticDeltaFloats));
    auto same = [&](const lb_tensor& t, const lb_tensor& like, const char* what) {
        if (t.rank != 4 || t.dtype != LB_BF16 || t.stride[3] != 1) fail(LB_ERR_INVALID, format("lb_attention_bwd_static: %s must be a bfloat16 [B, S, N, H] view", what));
        for (int d = 0; d < 4; d++)
            if (t.shape[d] != like.shape[d]) fail(LB_ERR_INVALID, format("lb_attention_bwd_static: %s has the wrong shape", what));
    };
    same(o, q, "o"), same(d_o, q, "dO"), same(dq, q, "dQ"), same(dk, k, "dK"), same(dv, v, "dV");
    check_dense(lse, LB_F32, {B, N, Sq}, "attention log-sum-exp");
    if (o.stride[0] % 8 || o.stride[1] % 8 || o.stride[2] % 8 || d_o.stride[0] % 8 || d_o.stride[1] % 8 || d_o.stride[2] % 8 ||
            ((uintptr_t)o.ptr & 15) || ((uintptr_t)d_o.ptr & 15))
        fail(LB_ERR_UNSUPPORTED, "lb_attention_bwd_static: o and dO rows must be 16-byte aligned");
    const StaticSetup& st = static_setup();
    cudaStream_t s = (cudaStream_t)stream;
    launch_delta(o, d_o, st.delta, nullptr, s);
    BwdArgs a{};
    a.B = (int)B, a.N = (int)N, a.Nkv = (int)Nkv, a.Sq = (int)Sq, a.Sk = (int)Sk;
    a.causal = desc.causal, a.causal_offset = desc.causal_offset;
    a.scale = desc.scale, a.scale_log2 = desc.scale * 1.4426950408889634f;
    a.lse = (const float*)lse.ptr, a.delta = st.delta, a.status = st.status;
    BwdArgs kv = a, qq = a;
    kv.out_a = dk.ptr, kv.a_sb = dk.stride[0], kv.a_ss = dk.stride[1], kv.a_sn = dk.stride[2];
    kv.out_b = dv.ptr, kv.b_sb = dv.stride[0], kv.b_ss = dv.stride[1], kv.b_sn = dv.stride[2];
    qq.out_a = dq.ptr, qq.a_sb = dq.stride[0], qq.a_ss = dq.stride[1], qq.a_sn = dq.stride[2];
    launch_bwd(D, [&](const lb_tensor& t, const char* what, int box_rows) { return static_map(st, t, what, box_rows); }, q, d_o, k, v, kv, qq, s);
}

}  // namespace

// The status word of lb_attention_bwd_static on the current device (sets the entry up on first use; allocates nothing).
int* static_status_word() { return static_setup().status; }
}  // namespace lb

// lb_attention_bwd without any device allocation. The scratch the backward needs (one float per query row and
// head) is a 4 MiB array built into the library; it is shared by every call, so two calls whose kernels can overlap
// on the GPU (different streams, or different host threads) race on it: serialise them. The array keeps whatever
// the previous call left there; each call overwrites the part it reads before reading it, so nothing needs
// clearing. The first call on a device resolves the array's device address (cudaGetSymbolAddress) and the
// tensor-map encoder; make that first call before starting any stream capture. Limit: batch * heads * query
// length <= 1,048,576, bfloat16 operands, head dim 64 or 128; beyond that the call fails with a message and
// lb_attention_bwd (caller-provided scratch) is the entry to use.
extern "C" int lb_attention_bwd_static(const lb_attn_desc* desc, const lb_tensor* q, const lb_tensor* k, const lb_tensor* v,
                                       const lb_tensor* o, const lb_tensor* d_o, const lb_tensor* lse, const lb_tensor* dq,
                                       const lb_tensor* dk, const lb_tensor* dv, void* stream) {
    return lb::guarded([&] {
        if (!desc || !q || !k || !v || !o || !d_o || !lse || !dq || !dk || !dv) lb::fail(LB_ERR_INVALID, "lb_attention_bwd_static: null argument");
        lb::attention_bwd_static(*desc, *q, *k, *v, *o, *d_o, *lse, *dq, *dk, *dv, stream);
    });
}

