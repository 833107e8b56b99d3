// Row gather/scatter and a CUDA-core attention for the shapes the tensor-core kernels do not take.
//
//  * scatter_add_rows: out[clamp(ids[t]), :] += updates[t, :] (the embedding gradient; lumen/reference/mod.rs:765-808),
//    in the two forms of the reference's backends (lumen/codegen/scatter_add/README.md:23-39). The DETERMINISTIC form
//    (count, starts, place, sort, rows) adds a row's updates in update order, rounding to the operand's dtype after
//    every add exactly like the interpreter: bit-identical to it and from run to run. The ATOMIC form adds in float32
//    atomics in arrival order and rounds once: results vary in the last bits when a row is hit more than once.
//  * attention_simt_fwd / attention_simt_bwd: float32 or bfloat16, any head dim up to 256, one or two query rows a warp,
//    scores and sums in float32. Used for float32 graphs (no hidden narrowing to bf16 tensor cores)
//    and head dims other than 64/128.
#include "launch.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

namespace lb {
namespace {

template <class T> __device__ __forceinline__ float to_f(T x);
template <> __device__ __forceinline__ float to_f<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <class T> __device__ __forceinline__ T from_f(float x);
template <> __device__ __forceinline__ float from_f<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// Four consecutive elements as floats, and back; the address is a multiple of four elements.
__device__ __forceinline__ float4 load4(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 w = *(const uint2*)p;
    return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
}
__device__ __forceinline__ void store4(float* p, float4 v) { *(float4*)p = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *(uint2*)p = make_uint2(*(const uint32_t*)&lo, *(const uint32_t*)&hi);
}

// The atomic form: bound by the number of atomics, then by the bytes of the float32 sums on their way to the result. VEC: four columns a
// thread and atomic, four elements a thread of the conversion (width a multiple of four, rows aligned). 16384 updates of 1024 bfloat16
// into 32768 rows, with the memset of the sums 162 -> 86 us; 1000 updates of 256 into 4096 rows 6.7 -> 5.1.
template <class T, class I, bool VEC>
__global__ void scatter_add_rows_kernel(float* __restrict__ acc, const I* __restrict__ ids, const T* __restrict__ updates,
                                        long long tokens, long long rows, int width) {
    grid_wait(ids, updates);
    const long long t = blockIdx.x;
    if (t >= tokens) return;
    long long r = (long long)ids[t];
    r = r < 0 ? 0 : (r > rows - 1 ? rows - 1 : r);
    if constexpr (VEC) {
        for (int d = threadIdx.x * 4; d < width; d += blockDim.x * 4) {
            const float4 v = load4(updates + t * width + d);
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(__cvta_generic_to_global(acc + r * width + d)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                         : "memory");
        }
    } else {
        for (int d = threadIdx.x; d < width; d += blockDim.x) atomicAdd(acc + r * width + d, to_f(updates[t * width + d]));
    }
}

// out = x + sum(updates): one rounding of the float32 sum into the operand dtype
template <class T, bool VEC>
__global__ void add_convert_kernel(T* __restrict__ out, const T* __restrict__ x, const float* __restrict__ acc, long long n, int has_x) {
    grid_wait(x, acc);
    const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * (VEC ? 4 : 1);
    if (i >= n) return;
    if constexpr (VEC) {
        float4 v = load4(acc + i);
        if (has_x) {
            const float4 u = load4(x + i);
            v = make_float4(__fadd_rn(u.x, v.x), __fadd_rn(u.y, v.y), __fadd_rn(u.z, v.z), __fadd_rn(u.w, v.w));
        }
        store4(out + i, v);
    } else {
        out[i] = from_f<T>(has_x ? __fadd_rn(to_f(x[i]), acc[i]) : acc[i]);
    }
}

// ---- deterministic scatter-add: a counting sort of the picks by destination row, then one block per row -----------
template <class I>
__device__ __forceinline__ int clamped_row(const I* ids, long long t, long long rows) {
    long long r = (long long)ids[t];
    return (int)(r < 0 ? 0 : (r > rows - 1 ? rows - 1 : r));
}

template <class I>
__global__ void scatter_count_kernel(int* __restrict__ counts, const I* __restrict__ ids, long long tokens, long long rows) {
    grid_wait(ids);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < tokens) atomicAdd(counts + clamped_row(ids, t, rows), 1);  // integer atomics: the counts do not depend on order
}

// starts[r] = sum of counts[0 .. r), starts[rows] = tokens; one block walks the rows in chunks of its size.
__global__ void scatter_starts_kernel(int* __restrict__ starts, const int* __restrict__ counts, long long rows) {
    grid_wait(counts);
    __shared__ int warp_sums[32];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long base = 0; base < rows; base += blockDim.x) {
        const long long r = base + threadIdx.x;
        const int c = r < rows ? counts[r] : 0;
        int incl = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            int up = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += up;
        }
        if (lane == 31) warp_sums[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            int w = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                int up = __shfl_up_sync(0xffffffffu, w, d);
                if (lane >= d) w += up;
            }
            warp_sums[lane] = w;  // inclusive over warps
        }
        __syncthreads();
        const int before = carry + (warp ? warp_sums[warp - 1] : 0) + incl - c;
        if (r < rows) starts[r] = before;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = before + c;
        __syncthreads();
    }
    if (threadIdx.x == 0) starts[rows] = carry;
}

template <class I>
__global__ void scatter_place_kernel(int* __restrict__ order, int* __restrict__ cursor, const int* __restrict__ starts,
                                     const I* __restrict__ ids, long long tokens, long long rows) {
    grid_wait(starts, ids);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= tokens) return;
    const int r = clamped_row(ids, t, rows);
    order[starts[r] + atomicAdd(cursor + r, 1)] = (int)t;  // arrival order within the row's segment; sorted next
}

// One block per destination row: sorts the row's picks into update order (ascending update number), then every thread
// owns columns and adds the row's updates one after the other, rounding to T after each add as the interpreter does.
// Short segments are sorted in shared memory (bitonic); longer ones by rank (every pick counts the smaller ones) into
// `sorted`, a second array of `tokens` ints.
constexpr int kSortSmem = 2048;
template <class T>
__global__ void scatter_rows_kernel(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ updates, const int* __restrict__ starts,
                                    const int* __restrict__ order, int* __restrict__ sorted, int width, int has_x) {
    __shared__ int picks[kSortSmem];
    grid_wait(x, updates, starts, order);
    const long long r = blockIdx.x;
    const int begin = starts[r], n = starts[r + 1] - begin;
    const int* list = picks;
    if (n <= kSortSmem) {
        int padded = 1;
        while (padded < n) padded <<= 1;
        for (int i = threadIdx.x; i < padded; i += blockDim.x) picks[i] = i < n ? order[begin + i] : 0x7fffffff;
        __syncthreads();
        for (int k = 2; k <= padded; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = threadIdx.x; i < padded; i += blockDim.x) {
                    const int partner = i ^ j;
                    if (partner > i) {
                        const int a = picks[i], b = picks[partner];
                        const bool up = (i & k) == 0;
                        if ((a > b) == up) picks[i] = b, picks[partner] = a;
                    }
                }
                __syncthreads();
            }
    } else {
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int mine = order[begin + i];
            int rank = 0;
            for (int j = 0; j < n; j++) rank += order[begin + j] < mine;
            sorted[begin + rank] = mine;  // update numbers are distinct: ranks are a permutation
        }
        __syncthreads();
        list = sorted + begin;
    }
    for (int d = threadIdx.x; d < width; d += blockDim.x) {
        float acc = has_x ? to_f(x[r * width + d]) : 0.0f;
        for (int i = 0; i < n; i++) acc = to_f(from_f<T>(__fadd_rn(acc, to_f(updates[(long long)list[i] * width + d]))));
        out[r * width + d] = from_f<T>(acc);
    }
}

// The same in one kernel for few updates: every block looks through all destinations and keeps the updates of its row, in update
// order: each of its eight warps those of a stretch, found by ballots. What bounds it is latency, one pass over the destinations
// and one over the row's updates, where the counting sort is a memset and four kernels in a chain; the destinations are read by every
// row, so the rule keeps rows, updates and their product small. us: 512 updates of 128 float32 into 256 rows 10.5 -> 2.9, 1024 into
// 512 rows 10.5 -> 4.2, 336 of 256 bfloat16 into 1280 rows 8.4 -> 7.1, 4096 of 512 into 1024 rows 11.9 -> 9.7; beyond it 512 of 1024
// into 8192 rows 26 -> 40.
constexpr int kFewUpdates = 4096, kFewRows = 2048;
constexpr long long kFewReads = 1LL << 22;
template <class T, class I>
__global__ void __launch_bounds__(256) scatter_rows_few_kernel(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ updates, const I* __restrict__ ids,
                                                               int tokens, long long rows, int width, int has_x) {
    constexpr int kWarps = 8, kBallots = kFewUpdates / (32 * kWarps);
    __shared__ int picks[kFewUpdates], counts[kWarps];
    grid_wait(x, updates, ids);
    const int r = (int)blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int stretch = (tokens + 32 * kWarps - 1) / (32 * kWarps) * 32, first = warp * stretch;
    unsigned hits[kBallots];
    int mine = 0;
#pragma unroll
    for (int i = 0; i < kBallots; i++) {
        const int t = first + i * 32 + lane;
        const bool hit = i * 32 < stretch && t < tokens && clamped_row(ids, t, rows) == r;
        hits[i] = __ballot_sync(0xffffffffu, hit);
        mine += __popc(hits[i]);
    }
    if (lane == 0) counts[warp] = mine;
    __syncthreads();
    int at = 0, n = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        if (w == warp) at = n;
        n += counts[w];
    }
#pragma unroll
    for (int i = 0; i < kBallots; i++) {
        if (hits[i] >> lane & 1) picks[at + __popc(hits[i] & ((1u << lane) - 1))] = first + i * 32 + lane;
        at += __popc(hits[i]);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < width; d += blockDim.x) {
        float acc = has_x ? to_f(x[(long long)r * width + d]) : 0.0f;
#pragma unroll 4
        for (int i = 0; i < n; i++) acc = to_f(from_f<T>(__fadd_rn(acc, to_f(updates[(long long)picks[i] * width + d]))));
        out[(long long)r * width + d] = from_f<T>(acc);
    }
}

struct AttnShape {
    int B, Sq, Sk, N, Nkv, D;
    long long q_s[3], k_s[3], v_s[3], o_s[3], g_s[3], dq_s[3], dk_s[3], dv_s[3];  // strides of dims B, S, N (head dim is dense)
    int causal;
    long long offset;
    float scale;
    int tile_rows;  // CUDA-core attention: rows of the streamed tiles in shared memory (launch_attn)
};

// CUDA-core attention: a warp for one row or two (queries of the forward and dQ kernels, keys of the dK/dV kernel), eight warps of
// neighbouring rows of one head per CTA. The rows they attend to stream through shared memory 32 at a time, as float32.
// Within a chunk a lane first owns one streamed row (its dot products run over the head dimension without any exchange
// between lanes), then head-dim elements l, l + 32, ... (the weighted sum over the chunk). A warp-wide sum per streamed
// row, as one row at a time would need, is a chain of five shuffles: at 64 keys of 32 elements those chains were nine
// tenths of the 48 us that the forward took.
constexpr int kAttnWarps = 8, kChunk = 32;

// DU: head-dim elements per lane. Row pitch: a multiple of four floats whose 16-byte groups fall in different banks for
// eight neighbouring rows. The streamed tiles have as many rows as there are to stream, at most a chunk: with full tiles of
// zeros, which left room for two blocks an SM, 1024 heads of one query and one key of 256 elements took 34 us (now 12; one row at a time,
// without shared memory, 3.6: seven of a block's eight warps idle there), of eight 43 us (now 26), of 16 89 us (now 62).
template <int DU, int RW = 1>
struct AttnSmem {
    static constexpr int kD = DU * 32, kPitch = kD + 4, kRows = kAttnWarps * RW;
    float (*weight)[kRows][kChunk];  // [2]
    float* own[2];                   // the warps' rows, kD apart
    float* tile[2];                  // streamed rows, kPitch apart
    __device__ __forceinline__ AttnSmem(uint8_t* raw, int tile_rows) {
        weight = (float(*)[kRows][kChunk])raw;
        own[0] = (float*)raw + 2 * kRows * kChunk, own[1] = own[0] + kRows * kD;
        tile[0] = own[1] + kRows * kD, tile[1] = tile[0] + tile_rows * kPitch;
    }
    static int bytes(int tile_rows) { return (2 * kRows * (kChunk + kD) + 2 * tile_rows * kPitch) * (int)sizeof(float); }
};

// Rows [row0, row0 + kChunk) of those before `end`; nothing is stored for the others, which no lane may then read. Unrolled to eight
// elements at most: a whole chunk of 256-wide rows held 32, and with 170 to 210 registers a thread one block an SM (head dim 256, 8 heads x
// 1024: 900 -> 669 us forward, 2238 -> 1824 backward).
template <class T, int DU>
__device__ __forceinline__ void load_chunk(float* dst, const T* base, long long stride, long long row0, long long end, int D) {
    constexpr int kD = AttnSmem<DU>::kD;
    auto element = [&](int i) {
        const int r = i / kD, d = i % kD;
        dst[r * AttnSmem<DU>::kPitch + d] = d < D ? to_f(base[(row0 + r) * stride + d]) : 0.0f;
    };
    if (end - row0 >= kChunk) {
#pragma unroll (DU > 2 ? 8 : 4 * DU)
        for (int i = threadIdx.x; i < kChunk * kD; i += kAttnWarps * 32) element(i);
    } else {
#pragma unroll 2
        for (int i = threadIdx.x; i < (int)(end - row0) * kD; i += kAttnWarps * 32) element(i);
    }
}
template <class T, int DU>
__device__ __forceinline__ void load_own(float* dst, const T* row, bool live, int D, int lane) {  // this warp's row
#pragma unroll
    for (int u = 0; u < DU; u++) dst[lane + 32 * u] = live && lane + 32 * u < D ? to_f(row[lane + 32 * u]) : 0.0f;
}
// The warp's own rows times the chunk row this lane owns: 64 elements at a time (32 at head dims up to 64) in sixteen (eight)
// sums that are added as a tree. The error of a score then is that of a warp-wide sum - a lane's few terms, then a tree of
// five - which one row at a time had, or a little below; in two running sums it is 1.2 times that at 32 elements and 2.5 times at 256.
template <int DU, int RW>
__device__ __forceinline__ void dot_rows(float* total, const float* own, const float* tile, int lane) {
    constexpr int kBlock = DU <= 2 ? 32 : 64, kSums = kBlock / 4;
    const float4* b = (const float4*)(tile + lane * AttnSmem<DU>::kPitch);
#pragma unroll (DU > 2 ? 1 : 2)
    for (int d0 = 0; d0 < DU * 32; d0 += kBlock) {
        float s[RW][kSums] = {};
#pragma unroll
        for (int d = 0; d < kBlock; d += 4) {
            const float4 y = b[(d0 + d) / 4];
#pragma unroll
            for (int r = 0; r < RW; r++) {
                const float4 x = ((const float4*)(own + r * AttnSmem<DU>::kD))[(d0 + d) / 4];
                float* t = s[r] + d % kSums;
                t[0] = fmaf(x.x, y.x, t[0]), t[1] = fmaf(x.y, y.y, t[1]), t[2] = fmaf(x.z, y.z, t[2]), t[3] = fmaf(x.w, y.w, t[3]);
            }
        }
#pragma unroll
        for (int r = 0; r < RW; r++) {
#pragma unroll
            for (int h = kSums / 2; h >= 1; h /= 2)
#pragma unroll
                for (int i = 0; i < h; i++) s[r][i] += s[r][i + h];
            total[r] = d0 ? total[r] + s[r][0] : s[r][0];
        }
    }
}
// acc[u] += sum over the chunk's rows [lo, hi) of weight[row] * tile[row][lane + 32 u], in row order. The other rows are not
// read: their weights are 0, but a value behind the mask may be infinite or NaN, and 0 times that is NaN.
template <int DU>
__device__ __forceinline__ void add_weighted(float* acc, const float* weight, const float* tile, int lane, int lo, int hi) {
    if (lo > 0 || hi < kChunk) {  // warp-uniform
#pragma unroll 1
        for (int j = lo & ~3; j < hi; j += 4) {
            const float4 w = *(const float4*)(weight + j);
            const float* t = tile + j * AttnSmem<DU>::kPitch + lane;
#pragma unroll
            for (int u = 0; u < DU; u++, t += 32) {
                acc[u] = fmaf(w.x, j >= lo ? t[0] : 0.0f, acc[u]);
                acc[u] = fmaf(w.y, j + 1 >= lo && j + 1 < hi ? t[AttnSmem<DU>::kPitch] : 0.0f, acc[u]);
                acc[u] = fmaf(w.z, j + 2 >= lo && j + 2 < hi ? t[2 * AttnSmem<DU>::kPitch] : 0.0f, acc[u]);
                acc[u] = fmaf(w.w, j + 3 >= lo && j + 3 < hi ? t[3 * AttnSmem<DU>::kPitch] : 0.0f, acc[u]);
            }
        }
        return;
    }
#pragma unroll (DU > 2 ? 2 : 8)
    for (int j = 0; j < kChunk; j += 4) {
        const float4 w = *(const float4*)(weight + j);
#pragma unroll
        for (int u = 0; u < DU; u++) {
            const float* t = tile + j * AttnSmem<DU>::kPitch + lane + 32 * u;
            acc[u] = fmaf(w.x, t[0], acc[u]);
            acc[u] = fmaf(w.y, t[AttnSmem<DU>::kPitch], acc[u]);
            acc[u] = fmaf(w.z, t[2 * AttnSmem<DU>::kPitch], acc[u]);
            acc[u] = fmaf(w.w, t[3 * AttnSmem<DU>::kPitch], acc[u]);
        }
    }
}
// The same for the warp's RW rows, weights kChunk apart, whose ranges are [lo[r], hi[r]): a streamed element is fetched once for all of
// them where they see the whole chunk.
template <int DU, int RW>
__device__ __forceinline__ void add_weighted_rows(float (*acc)[DU], const float* weight, const float* tile, int lane, const int* lo, const int* hi) {
    bool whole = true;  // warp-uniform
#pragma unroll
    for (int r = 0; r < RW; r++) whole &= lo[r] <= 0 && hi[r] >= kChunk;
    if (RW == 1 || !whole) {
#pragma unroll
        for (int r = 0; r < RW; r++) add_weighted<DU>(acc[r], weight + r * kChunk, tile, lane, lo[r], hi[r]);
        return;
    }
#pragma unroll (DU > 2 ? 1 : 2)
    for (int j = 0; j < kChunk; j += 4) {
        float4 w[RW];
#pragma unroll
        for (int r = 0; r < RW; r++) w[r] = *(const float4*)(weight + r * kChunk + j);
#pragma unroll
        for (int u = 0; u < DU; u++) {
            const float* t = tile + j * AttnSmem<DU>::kPitch + lane + 32 * u;
            const float t0 = t[0], t1 = t[AttnSmem<DU>::kPitch], t2 = t[2 * AttnSmem<DU>::kPitch], t3 = t[3 * AttnSmem<DU>::kPitch];
#pragma unroll
            for (int r = 0; r < RW; r++) {
                acc[r][u] = fmaf(w[r].x, t0, acc[r][u]);
                acc[r][u] = fmaf(w[r].y, t1, acc[r][u]);
                acc[r][u] = fmaf(w[r].z, t2, acc[r][u]);
                acc[r][u] = fmaf(w[r].w, t3, acc[r][u]);
            }
        }
    }
}
// the CTA's rows: kAttnWarps * RW neighbours of one (batch, head)
template <int RW>
__device__ __forceinline__ void block_rows(int rows, int heads, int& r0, int& n, int& b) {
    constexpr int kRows = kAttnWarps * RW;
    const int per = (rows + kRows - 1) / kRows;
    r0 = (int)(blockIdx.x % per) * kRows, n = (int)(blockIdx.x / per % heads), b = (int)(blockIdx.x / per / heads);
}

template <class T, int DU, int RW>
__global__ void __launch_bounds__(kAttnWarps * 32)
attention_simt_fwd_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, T* __restrict__ o,
                          float* __restrict__ lse, AttnShape s) {
    extern __shared__ __align__(16) uint8_t raw[];
    AttnSmem<DU, RW> sm(raw, s.tile_rows);
    grid_wait(q, k, v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int i0, n, b;
    block_rows<RW>(s.Sq, s.N, i0, n, b);
    const int i = i0 + warp * RW, nk = n / (s.N / s.Nkv);  // the warp's first row
    float* own = sm.own[0] + warp * RW * AttnSmem<DU>::kD;
    long long last[RW];  // a row's last key, -1: none
#pragma unroll
    for (int r = 0; r < RW; r++) {
        const bool live = i + r < s.Sq;
        load_own<T, DU>(own + r * AttnSmem<DU>::kD, q + b * s.q_s[0] + (long long)(i + r) * s.q_s[1] + n * s.q_s[2], live, s.D, lane);
        last[r] = !live ? -1 : s.causal ? min((long long)s.Sk - 1, (long long)i + r + s.offset) : (long long)s.Sk - 1;
    }
    const long long end = s.causal ? min((long long)s.Sk, (long long)i0 + kAttnWarps * RW + s.offset) : (long long)s.Sk;  // past the CTA's last key
    float acc[RW][DU] = {}, m[RW], l[RW];
#pragma unroll
    for (int r = 0; r < RW; r++) m[r] = -INFINITY, l[r] = 0.0f;
    for (long long j0 = 0; j0 < end; j0 += kChunk) {
        __syncthreads();
        load_chunk<T, DU>(sm.tile[0], k + b * s.k_s[0] + nk * s.k_s[2], s.k_s[1], j0, end, s.D);
        load_chunk<T, DU>(sm.tile[1], v + b * s.v_s[0] + nk * s.v_s[2], s.v_s[1], j0, end, s.D);
        __syncthreads();
        bool any = false;  // warp-uniform: rows that see something of the chunk
        int hi[RW], lo[RW];
#pragma unroll
        for (int r = 0; r < RW; r++) lo[r] = 0, hi[r] = (int)max(0LL, min((long long)kChunk, last[r] + 1 - j0)), any |= hi[r] > 0;
        if (!any) continue;
        float dots[RW];
        bool seen = false;
#pragma unroll
        for (int r = 0; r < RW; r++) seen |= lane < hi[r];
        if (seen) dot_rows<DU, RW>(dots, own, sm.tile[0], lane);
#pragma unroll
        for (int r = 0; r < RW; r++) {
            if (hi[r] == 0) continue;
            const float sc = lane < hi[r] ? dots[r] * s.scale : -INFINITY;
            float top = sc;
#pragma unroll
            for (int x = 16; x >= 1; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
            const float m_new = fmaxf(m[r], top);
            const float alpha = __expf(m[r] - m_new), p = lane < hi[r] ? __expf(sc - m_new) : 0.0f;
            sm.weight[0][warp * RW + r][lane] = p;
            float sum = p;
#pragma unroll
            for (int x = 16; x >= 1; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
            l[r] = l[r] * alpha + sum;
#pragma unroll
            for (int u = 0; u < DU; u++) acc[r][u] *= alpha;
            m[r] = m_new;
        }
        __syncwarp();
        // the normaliser is applied at the end
        add_weighted_rows<DU, RW>(acc, sm.weight[0][warp * RW], sm.tile[1], lane, lo, hi);
        __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < RW; r++) {
        if (i + r >= s.Sq) break;
        T* op = o + b * s.o_s[0] + (long long)(i + r) * s.o_s[1] + n * s.o_s[2];
#pragma unroll
        for (int u = 0; u < DU; u++)
            if (lane + 32 * u < s.D) op[lane + 32 * u] = from_f<T>(acc[r][u] / l[r]);
        if (lse && lane == 0) lse[((long long)b * s.N + n) * s.Sq + i + r] = m[r] + logf(l[r]);
    }
}

// dQ: RW query rows a warp.
template <class T, int DU, int RW>
__global__ void __launch_bounds__(kAttnWarps * 32)
attention_simt_dq_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, const T* __restrict__ g,
                         const float* __restrict__ lse, const float* __restrict__ delta, T* __restrict__ dq, AttnShape s) {
    extern __shared__ __align__(16) uint8_t raw[];
    AttnSmem<DU, RW> sm(raw, s.tile_rows);
    grid_wait(q, k, v, g, lse, delta);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int i0, n, b;
    block_rows<RW>(s.Sq, s.N, i0, n, b);
    const int i = i0 + warp * RW, nk = n / (s.N / s.Nkv);
    float *own_q = sm.own[0] + warp * RW * AttnSmem<DU>::kD, *own_g = sm.own[1] + warp * RW * AttnSmem<DU>::kD;
    long long last[RW];
    float L[RW], dl[RW];
#pragma unroll
    for (int r = 0; r < RW; r++) {
        const bool live = i + r < s.Sq;
        load_own<T, DU>(own_q + r * AttnSmem<DU>::kD, q + b * s.q_s[0] + (long long)(i + r) * s.q_s[1] + n * s.q_s[2], live, s.D, lane);
        load_own<T, DU>(own_g + r * AttnSmem<DU>::kD, g + b * s.g_s[0] + (long long)(i + r) * s.g_s[1] + n * s.g_s[2], live, s.D, lane);
        const long long at = ((long long)b * s.N + n) * s.Sq + i + r;
        L[r] = live ? lse[at] : 0.0f, dl[r] = live ? delta[at] : 0.0f;
        last[r] = !live ? -1 : s.causal ? min((long long)s.Sk - 1, (long long)i + r + s.offset) : (long long)s.Sk - 1;
    }
    const long long end = s.causal ? min((long long)s.Sk, (long long)i0 + kAttnWarps * RW + s.offset) : (long long)s.Sk;
    float acc[RW][DU] = {};
    for (long long j0 = 0; j0 < end; j0 += kChunk) {
        __syncthreads();
        load_chunk<T, DU>(sm.tile[0], k + b * s.k_s[0] + nk * s.k_s[2], s.k_s[1], j0, end, s.D);
        load_chunk<T, DU>(sm.tile[1], v + b * s.v_s[0] + nk * s.v_s[2], s.v_s[1], j0, end, s.D);
        __syncthreads();
        bool any = false, seen = false;
        int hi[RW], lo[RW];
#pragma unroll
        for (int r = 0; r < RW; r++) lo[r] = 0, hi[r] = (int)max(0LL, min((long long)kChunk, last[r] + 1 - j0)), any |= hi[r] > 0, seen |= lane < hi[r];
        if (!any) continue;
        float ds[RW] = {};
        if (seen) {
            float dots[RW], dp[RW];
            dot_rows<DU, RW>(dots, own_q, sm.tile[0], lane);
            dot_rows<DU, RW>(dp, own_g, sm.tile[1], lane);
#pragma unroll
            for (int r = 0; r < RW; r++) {
                const float p = __expf(dots[r] * s.scale - L[r]);
                if (lane < hi[r]) ds[r] = to_f(from_f<T>(p * (dp[r] - dl[r]) * s.scale));  // dS is rounded to the operands' dtype (flash.py:71)
            }
        }
#pragma unroll
        for (int r = 0; r < RW; r++) sm.weight[0][warp * RW + r][lane] = ds[r];
        __syncwarp();
        add_weighted_rows<DU, RW>(acc, sm.weight[0][warp * RW], sm.tile[0], lane, lo, hi);
        __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < RW; r++) {
        if (i + r >= s.Sq) break;
        T* out = dq + b * s.dq_s[0] + (long long)(i + r) * s.dq_s[1] + n * s.dq_s[2];
#pragma unroll
        for (int u = 0; u < DU; u++)
            if (lane + 32 * u < s.D) out[lane + 32 * u] = from_f<T>(acc[r][u]);
    }
}

// dK/dV: RW keys of a (batch, kv head) a warp, looping over the group's heads and the queries that see them.
template <class T, int DU, int RW>
__global__ void __launch_bounds__(kAttnWarps * 32)
attention_simt_dkdv_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, const T* __restrict__ g,
                           const float* __restrict__ lse, const float* __restrict__ delta, T* __restrict__ dk, T* __restrict__ dv, AttnShape s) {
    extern __shared__ __align__(16) uint8_t raw[];
    AttnSmem<DU, RW> sm(raw, s.tile_rows);
    grid_wait(q, k, v, g, lse, delta);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int k0, nk, b;
    block_rows<RW>(s.Sk, s.Nkv, k0, nk, b);
    const int j = k0 + warp * RW, group = s.N / s.Nkv;
    float *own_k = sm.own[0] + warp * RW * AttnSmem<DU>::kD, *own_v = sm.own[1] + warp * RW * AttnSmem<DU>::kD;
    long long first[RW];  // the first query that sees the key
#pragma unroll
    for (int r = 0; r < RW; r++) {
        const bool live = j + r < s.Sk;
        load_own<T, DU>(own_k + r * AttnSmem<DU>::kD, k + b * s.k_s[0] + (long long)(j + r) * s.k_s[1] + nk * s.k_s[2], live, s.D, lane);
        load_own<T, DU>(own_v + r * AttnSmem<DU>::kD, v + b * s.v_s[0] + (long long)(j + r) * s.v_s[1] + nk * s.v_s[2], live, s.D, lane);
        first[r] = !live ? (long long)s.Sq : s.causal ? max(0LL, (long long)j + r - s.offset) : 0LL;
    }
    float ak[RW][DU] = {}, av[RW][DU] = {};
    const long long begin = s.causal ? max(0LL, (long long)k0 - s.offset) : 0LL;  // the first query that sees the CTA's first key
    for (int h = 0; h < group; h++) {
        const int n = nk * group + h;
        for (long long i0 = begin; i0 < s.Sq; i0 += kChunk) {
            __syncthreads();
            load_chunk<T, DU>(sm.tile[0], q + b * s.q_s[0] + n * s.q_s[2], s.q_s[1], i0, s.Sq, s.D);
            load_chunk<T, DU>(sm.tile[1], g + b * s.g_s[0] + n * s.g_s[2], s.g_s[1], i0, s.Sq, s.D);
            __syncthreads();
            const int rows = (int)min((long long)kChunk, s.Sq - i0);
            bool any = false, seen = false;
            int hi[RW], lo[RW];
#pragma unroll
            for (int r = 0; r < RW; r++)
                lo[r] = (int)max(0LL, min((long long)kChunk, first[r] - i0)), hi[r] = lo[r] < rows ? rows : 0, any |= hi[r] > 0, seen |= lane >= lo[r] && lane < hi[r];
            if (!any) continue;
            float ds[RW] = {}, pr[RW] = {};
            if (seen) {
                const long long at = ((long long)b * s.N + n) * s.Sq + i0 + lane;
                const float L = lse[at], dl = delta[at];
                float dots[RW], dp[RW];
                dot_rows<DU, RW>(dots, own_k, sm.tile[0], lane);
                dot_rows<DU, RW>(dp, own_v, sm.tile[1], lane);
#pragma unroll
                for (int r = 0; r < RW; r++) {
                    const float p = __expf(dots[r] * s.scale - L);
                    if (lane >= lo[r] && lane < hi[r]) ds[r] = to_f(from_f<T>(p * (dp[r] - dl) * s.scale)), pr[r] = to_f(from_f<T>(p));
                }
            }
#pragma unroll
            for (int r = 0; r < RW; r++) sm.weight[0][warp * RW + r][lane] = ds[r], sm.weight[1][warp * RW + r][lane] = pr[r];
            __syncwarp();
            add_weighted_rows<DU, RW>(ak, sm.weight[0][warp * RW], sm.tile[0], lane, lo, hi);
            add_weighted_rows<DU, RW>(av, sm.weight[1][warp * RW], sm.tile[1], lane, lo, hi);
            __syncwarp();
        }
    }
#pragma unroll
    for (int r = 0; r < RW; r++) {
        if (j + r >= s.Sk) break;
        T* ok = dk + b * s.dk_s[0] + (long long)(j + r) * s.dk_s[1] + nk * s.dk_s[2];
        T* ov = dv + b * s.dv_s[0] + (long long)(j + r) * s.dv_s[1] + nk * s.dv_s[2];
#pragma unroll
        for (int u = 0; u < DU; u++)
            if (lane + 32 * u < s.D) ok[lane + 32 * u] = from_f<T>(ak[r][u]), ov[lane + 32 * u] = from_f<T>(av[r][u]);
    }
}

template <class T>
__global__ void attention_delta_simt(const T* __restrict__ o, const T* __restrict__ g, float* __restrict__ delta, AttnShape s) {
    grid_wait(o, g);
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= (long long)s.B * s.N * s.Sq) return;
    const int i = (int)(w % s.Sq), n = (int)((w / s.Sq) % s.N), b = (int)(w / ((long long)s.Sq * s.N));
    const T* op = o + b * s.o_s[0] + (long long)i * s.o_s[1] + n * s.o_s[2];
    const T* gp = g + b * s.g_s[0] + (long long)i * s.g_s[1] + n * s.g_s[2];
    float acc = 0.0f;
    for (int d = lane; d < s.D; d += 32) acc = fmaf(to_f(op[d]), to_f(gp[d]), acc);
#pragma unroll
    for (int x = 16; x >= 1; x >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, x);
    if (lane == 0) delta[((long long)b * s.N + n) * s.Sq + i] = acc;
}

// out[c, r] = in[r, c] for dense row-major 2-byte or 4-byte elements: 32 x 32 tiles through shared memory, both sides
// coalesced. Used by plans to give a GEMM a K-major copy of a weight whose rows are 8 KB or more apart.
template <class T>
__global__ void __launch_bounds__(256) transpose_kernel(const T* __restrict__ in, T* __restrict__ out, int rows, int cols) {
    __shared__ T tile[32][33];
    grid_wait(in);
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
#pragma unroll
    for (int k = 0; k < 32; k += 8) {
        const int r = r0 + ty + k, c = c0 + tx;
        if (r < rows && c < cols) tile[ty + k][tx] = in[(long long)r * cols + c];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 32; k += 8) {
        const int c = c0 + ty + k, r = r0 + tx;
        if (r < rows && c < cols) out[(long long)c * rows + r] = tile[tx][ty + k];
    }
}

void fill_strides(long long* dst, const lb_tensor& t) {
    for (int d = 0; d < 3; d++) dst[d] = t.stride[d];
    if (t.stride[3] != 1 && t.shape[3] > 1) fail(LB_ERR_UNSUPPORTED, "attention: the head dimension must be dense");
}

}  // namespace

// bfloat16 noise in [-1, 1) from a linear congruential generator, over a whole buffer: what an autotuner times its
// candidates on (a GPU's clocks under all-zero operands differ from those under real data).
__global__ void fill_noise_kernel(uint16_t* __restrict__ out, size_t n) {
    grid_wait();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        uint32_t x = (uint32_t)i * 1664525u + 1013904223u;
        x = x * 1664525u + 1013904223u;
        const float f = (float)(x >> 8) * (2.0f / 16777216.0f) - 1.0f;
        out[i] = __bfloat16_as_ushort(__float2bfloat16_rn(f));
    }
}

void fill_noise(void* ptr, size_t bytes, void* stream) {
    const size_t n = bytes / 2;
    if (n == 0) return;
    driver();
    launch_overlapped(fill_noise_kernel, dim3((unsigned)std::min<size_t>((n + 255) / 256, 148 * 16)), dim3(256), 0, (cudaStream_t)stream, 0, (uint16_t*)ptr, n);
    LB_CUDA(cudaGetLastError());
}

size_t scatter_add_scratch_bytes(long long rows, long long width, long long tokens, bool deterministic) {
    // deterministic: counts[rows], cursor[rows], starts[rows + 1], order[tokens], sorted[tokens]; atomic: float32 rows
    return deterministic ? (size_t)(3 * rows + 1 + 2 * tokens) * 4 : (size_t)rows * width * 4;
}

// Kernels that scatter_add_rows launches.
int scatter_add_launches(long long rows, long long tokens, bool deterministic) {
    return !deterministic ? 2 : tokens <= kFewUpdates && rows <= kFewRows && rows * tokens <= kFewReads ? 1 : 4;
}

void scatter_add_rows(const lb_tensor& x, const lb_tensor& ids, const lb_tensor& updates, const lb_tensor& out, void* scratch,
                      bool x_is_zero, bool deterministic, void* stream) {
    if (x.rank != 2) fail(LB_ERR_UNSUPPORTED, "scatter_add: a [rows, width] operand scattered along axis 0");
    const long long rows = x.shape[0], width = x.shape[1];
    long long tokens = 1;
    for (int d = 0; d < ids.rank; d++) tokens *= ids.shape[d];
    check_dense(x, x.dtype, {rows, width}, "scatter_add operand");
    check_dense(out, x.dtype, {rows, width}, "scatter_add result");
    if (updates.dtype != x.dtype) fail(LB_ERR_INVALID, "scatter_add: updates must have the operand's dtype");
    if (x.dtype != LB_F32 && x.dtype != LB_BF16) fail(LB_ERR_UNSUPPORTED, "scatter_add: float32 or bfloat16 rows");
    if (ids.dtype != LB_I64 && ids.dtype != LB_I32) fail(LB_ERR_INVALID, "scatter_add: int32 or int64 indices");
    if (!scratch || ((uintptr_t)scratch & 3)) fail(LB_ERR_INVALID, "scatter_add: needs scratch memory (scatter_add_scratch_bytes), 4-byte aligned");
    if (rows > INT32_MAX || tokens > INT32_MAX || width > INT32_MAX) fail(LB_ERR_UNSUPPORTED, "scatter_add: more than 2^31 rows, updates or columns");
    driver();
    cudaStream_t s = (cudaStream_t)stream;
    if (rows == 0 || width == 0) return;
    if (scatter_add_launches(rows, tokens, deterministic) == 1) {
        auto launch = [&](auto* o, auto* i) {
            using T = std::remove_pointer_t<decltype(o)>;
            using I = std::remove_const_t<std::remove_pointer_t<decltype(i)>>;
            launch_overlapped(scatter_rows_few_kernel<T, I>, dim3((unsigned)rows), dim3(256), 0, s, 0, o, (const T*)x.ptr, (const T*)updates.ptr, i, (int)tokens, rows, (int)width, !x_is_zero);
        };
        auto by_ids = [&](auto* o) {
            if (ids.dtype == LB_I64) launch(o, (const long long*)ids.ptr);
            else launch(o, (const int*)ids.ptr);
        };
        if (x.dtype == LB_F32) by_ids((float*)out.ptr);
        else by_ids((__nv_bfloat16*)out.ptr);
        return;
    }
    if (deterministic) {
        int* counts = (int*)scratch;
        int* cursor = counts + rows;
        int* starts = cursor + rows;
        int* order = starts + rows + 1;
        int* sorted = order + tokens;
        LB_CUDA(cudaMemsetAsync(counts, 0, (size_t)rows * 2 * 4, s));  // counts and cursor start at zero
        if (tokens > 0) {
            const unsigned blocks = (unsigned)((tokens + 255) / 256);
            if (ids.dtype == LB_I64) launch_overlapped(scatter_count_kernel<long long>, dim3(blocks), dim3(256), 0, s, 0, counts, (const long long*)ids.ptr, tokens, rows);
            else launch_overlapped(scatter_count_kernel<int>, dim3(blocks), dim3(256), 0, s, 0, counts, (const int*)ids.ptr, tokens, rows);
        }
        launch_overlapped(scatter_starts_kernel, dim3(1), dim3(1024), 0, s, 0, starts, counts, rows);
        if (tokens > 0) {
            const unsigned blocks = (unsigned)((tokens + 255) / 256);
            if (ids.dtype == LB_I64) launch_overlapped(scatter_place_kernel<long long>, dim3(blocks), dim3(256), 0, s, 0, order, cursor, starts, (const long long*)ids.ptr, tokens, rows);
            else launch_overlapped(scatter_place_kernel<int>, dim3(blocks), dim3(256), 0, s, 0, order, cursor, starts, (const int*)ids.ptr, tokens, rows);
        }
        const int threads = (int)std::min<long long>(256, ((width + 31) / 32) * 32);
        if (x.dtype == LB_F32)
            launch_overlapped(scatter_rows_kernel<float>, dim3((unsigned)rows), dim3(threads), 0, s, 0, (float*)out.ptr, (const float*)x.ptr, (const float*)updates.ptr, starts, order, sorted, (int)width, !x_is_zero);
        else
            launch_overlapped(scatter_rows_kernel<__nv_bfloat16>, dim3((unsigned)rows), dim3(threads), 0, s, 0, (__nv_bfloat16*)out.ptr, (const __nv_bfloat16*)x.ptr, (const __nv_bfloat16*)updates.ptr, starts, order, sorted, (int)width, !x_is_zero);
        LB_CUDA(cudaGetLastError());
        return;
    }
    float* acc = (float*)scratch;
    LB_CUDA(cudaMemsetAsync(acc, 0, (size_t)rows * width * 4, s));
    const size_t quad = 4 * dtype_size(x.dtype);  // bytes of four elements
    auto aligned = [&](const lb_tensor& t) { return (uintptr_t)t.ptr % quad == 0; };
    const bool sums_ok = width % 4 == 0 && (uintptr_t)acc % 16 == 0;
    auto launch = [&](auto* o, auto* i, auto add_vec, auto out_vec) {
        using T = std::remove_pointer_t<decltype(o)>;
        using I = std::remove_const_t<std::remove_pointer_t<decltype(i)>>;
        const long long cols = add_vec ? width / 4 : width, n = rows * width, items = out_vec ? n / 4 : n;
        if (tokens > 0)
            launch_overlapped(scatter_add_rows_kernel<T, I, add_vec>, dim3((unsigned)tokens), dim3((unsigned)std::min<long long>(256, (cols + 31) / 32 * 32)), 0, s, 0, acc, i,
                              (const T*)updates.ptr, tokens, rows, (int)width);
        launch_overlapped(add_convert_kernel<T, out_vec>, dim3((unsigned)((items + 255) / 256)), dim3(256), 0, s, 0, o, (const T*)x.ptr, (const float*)acc, n, !x_is_zero);
    };
    auto by_vec = [&](auto* o, auto* i) {
        const bool add_vec = sums_ok && aligned(updates), out_vec = sums_ok && aligned(out) && (x_is_zero || aligned(x));
        if (add_vec && out_vec) launch(o, i, std::true_type(), std::true_type());
        else if (add_vec) launch(o, i, std::true_type(), std::false_type());
        else if (out_vec) launch(o, i, std::false_type(), std::true_type());
        else launch(o, i, std::false_type(), std::false_type());
    };
    auto by_ids = [&](auto* o) {
        if (ids.dtype == LB_I64) by_vec(o, (const long long*)ids.ptr);
        else by_vec(o, (const int*)ids.ptr);
    };
    if (x.dtype == LB_F32) by_ids((float*)out.ptr);
    else by_ids((__nv_bfloat16*)out.ptr);
}

static AttnShape attn_shape(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v) {
    if (q.rank != 4 || k.rank != 4 || v.rank != 4) fail(LB_ERR_INVALID, "attention: operands must be [B, S, N, H] tensors");
    AttnShape s{};
    s.B = (int)q.shape[0], s.Sq = (int)q.shape[1], s.N = (int)q.shape[2], s.D = (int)q.shape[3];
    s.Sk = (int)k.shape[1], s.Nkv = (int)k.shape[2];
    if (s.D > 256 || v.shape[3] != s.D || s.Nkv == 0 || s.N % s.Nkv) fail(LB_ERR_UNSUPPORTED, "attention: head dim up to 256, equal for values, N a multiple of Nkv");
    fill_strides(s.q_s, q), fill_strides(s.k_s, k), fill_strides(s.v_s, v);
    s.causal = desc.causal, s.offset = desc.causal_offset, s.scale = desc.scale;
    return s;
}

void transpose_2d(const lb_tensor& in, const lb_tensor& out, void* stream) {
    if (in.rank != 2 || out.rank != 2 || in.dtype != out.dtype || in.shape[0] != out.shape[1] || in.shape[1] != out.shape[0] ||
        in.stride[1] != 1 || in.stride[0] != in.shape[1] || out.stride[1] != 1 || out.stride[0] != out.shape[1])
        fail(LB_ERR_INVALID, "transpose: dense row-major [R, C] in, [C, R] out of one dtype");
    const long long rows = in.shape[0], cols = in.shape[1];
    if (rows == 0 || cols == 0) return;
    if (rows > INT32_MAX || cols > INT32_MAX || (cols + 31) / 32 > INT32_MAX || (rows + 31) / 32 > 65535)
        fail(LB_ERR_UNSUPPORTED, "transpose: matrix too large for the kernel's grid");
    dim3 grid((unsigned)((cols + 31) / 32), (unsigned)((rows + 31) / 32));
    const int size = dtype_size(in.dtype);
    if (size == 2) launch_overlapped(transpose_kernel<uint16_t>, dim3(grid), dim3(256), 0, (cudaStream_t)stream, 0, (const uint16_t*)in.ptr, (uint16_t*)out.ptr, (int)rows, (int)cols);
    else if (size == 4) launch_overlapped(transpose_kernel<uint32_t>, dim3(grid), dim3(256), 0, (cudaStream_t)stream, 0, (const uint32_t*)in.ptr, (uint32_t*)out.ptr, (int)rows, (int)cols);
    else fail(LB_ERR_UNSUPPORTED, "transpose: 2-byte and 4-byte elements");
    LB_CUDA(cudaGetLastError());
}

// ---- a view copied element by element: any strides on either side ---------------------------------------------------
// The plan's copies of views that are neither dense nor rows of a wider matrix (a permuted or sliced tensor made dense
// for a kernel that reads dense operands, or written out as a graph output). Consecutive threads take consecutive
// elements of the destination's index order, so a dense destination is written in whole lines.
struct CopyDims {
    int rank;
    long long shape[LB_MAX_RANK], src[LB_MAX_RANK], dst[LB_MAX_RANK];
};

template <class T>
__global__ void strided_copy_kernel(const T* __restrict__ src, T* __restrict__ dst, CopyDims d, long long total) {
    grid_wait(src);
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
        long long rest = i, from = 0, to = 0;
        for (int k = d.rank - 1; k >= 0; k--) {
            const long long c = rest % d.shape[k];
            rest /= d.shape[k];
            from += c * d.src[k], to += c * d.dst[k];
        }
        dst[to] = src[from];
    }
}

// The same copy when the source is contiguous along one axis (a) and the destination along another (b): 32 x 32 tiles
// over those two axes go through shared memory, read along a and written along b, so both sides move whole lines. The
// other axes are enumerated by the block index.
template <class T>
__global__ void __launch_bounds__(256) tiled_copy_kernel(const T* __restrict__ src, T* __restrict__ dst, CopyDims d, int a, int b, long long tiles_a,
                                                         long long tiles_b) {
    __shared__ T tile[32][33];
    grid_wait(src);
    long long block = blockIdx.x;
    const long long ta = block % tiles_a;
    block /= tiles_a;
    const long long tb = block % tiles_b;
    block /= tiles_b;
    long long from = 0, to = 0;
    for (int k = d.rank - 1; k >= 0; k--) {
        if (k == a || k == b) continue;
        const long long c = block % d.shape[k];
        block /= d.shape[k];
        from += c * d.src[k], to += c * d.dst[k];
    }
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int j = ty; j < 32; j += 8) {
        const long long ia = ta * 32 + tx, ib = tb * 32 + j;
        if (ia < d.shape[a] && ib < d.shape[b]) tile[j][tx] = src[from + ia * d.src[a] + ib * d.src[b]];
    }
    __syncthreads();
    for (int j = ty; j < 32; j += 8) {
        const long long ia = ta * 32 + j, ib = tb * 32 + tx;
        if (ia < d.shape[a] && ib < d.shape[b]) dst[to + ia * d.dst[a] + ib * d.dst[b]] = tile[tx][j];
    }
}

void strided_copy(const lb_tensor& in, const lb_tensor& out, void* stream) {
    if (in.rank != out.rank || in.dtype != out.dtype) fail(LB_ERR_INVALID, "copy: views of one rank and dtype");
    CopyDims d{};
    long long total = 1;
    for (int k = 0; k < in.rank; k++) {
        if (in.shape[k] != out.shape[k]) fail(LB_ERR_INVALID, "copy: views of one shape");
        total *= in.shape[k];
        if (in.shape[k] == 1) continue;  // contributes no offset
        // an axis that continues the one before it on both sides is merged into it
        if (d.rank > 0 && d.src[d.rank - 1] == in.stride[k] * in.shape[k] && d.dst[d.rank - 1] == out.stride[k] * out.shape[k]) {
            d.shape[d.rank - 1] *= in.shape[k], d.src[d.rank - 1] = in.stride[k], d.dst[d.rank - 1] = out.stride[k];
            continue;
        }
        d.shape[d.rank] = in.shape[k], d.src[d.rank] = in.stride[k], d.dst[d.rank] = out.stride[k];
        d.rank++;
    }
    if (total == 0) return;
    cudaStream_t st = (cudaStream_t)stream;
    // contiguous along different axes on the two sides (a transposition of the last axis with another): tiles
    int a = -1, b = -1;
    for (int k = 0; k < d.rank; k++) {
        if (d.src[k] == 1 && a < 0) a = k;
        if (d.dst[k] == 1 && b < 0) b = k;
    }
    if (a >= 0 && b >= 0 && a != b && d.shape[a] >= 8 && d.shape[b] >= 8) {
        const long long tiles_a = (d.shape[a] + 31) / 32, tiles_b = (d.shape[b] + 31) / 32;
        const long long blocks = total / (d.shape[a] * d.shape[b]) * tiles_a * tiles_b;
        if (blocks <= 0x7fffffffLL) {
            switch (dtype_size(in.dtype)) {
                case 1: launch_overlapped(tiled_copy_kernel<uint8_t>, dim3((unsigned)blocks), dim3(256), 0, st, 0, (const uint8_t*)in.ptr, (uint8_t*)out.ptr, d, a, b, tiles_a, tiles_b); break;
                case 2: launch_overlapped(tiled_copy_kernel<uint16_t>, dim3((unsigned)blocks), dim3(256), 0, st, 0, (const uint16_t*)in.ptr, (uint16_t*)out.ptr, d, a, b, tiles_a, tiles_b); break;
                case 4: launch_overlapped(tiled_copy_kernel<uint32_t>, dim3((unsigned)blocks), dim3(256), 0, st, 0, (const uint32_t*)in.ptr, (uint32_t*)out.ptr, d, a, b, tiles_a, tiles_b); break;
                default: launch_overlapped(tiled_copy_kernel<uint64_t>, dim3((unsigned)blocks), dim3(256), 0, st, 0, (const uint64_t*)in.ptr, (uint64_t*)out.ptr, d, a, b, tiles_a, tiles_b); break;
            }
            LB_CUDA(cudaGetLastError());
            return;
        }
    }
    const unsigned blocks = (unsigned)std::min<long long>((total + 255) / 256, 148LL * 16);
    switch (dtype_size(in.dtype)) {
        case 1: launch_overlapped(strided_copy_kernel<uint8_t>, dim3(blocks), dim3(256), 0, st, 0, (const uint8_t*)in.ptr, (uint8_t*)out.ptr, d, total); break;
        case 2: launch_overlapped(strided_copy_kernel<uint16_t>, dim3(blocks), dim3(256), 0, st, 0, (const uint16_t*)in.ptr, (uint16_t*)out.ptr, d, total); break;
        case 4: launch_overlapped(strided_copy_kernel<uint32_t>, dim3(blocks), dim3(256), 0, st, 0, (const uint32_t*)in.ptr, (uint32_t*)out.ptr, d, total); break;
        default: launch_overlapped(strided_copy_kernel<uint64_t>, dim3(blocks), dim3(256), 0, st, 0, (const uint64_t*)in.ptr, (uint64_t*)out.ptr, d, total); break;
    }
    LB_CUDA(cudaGetLastError());
}

namespace {
// CTAs of kAttnWarps * RW rows over `rows` rows of every (batch, head)
unsigned attn_blocks(long long batch, long long heads, long long rows, int rw) {
    const long long blocks = batch * heads * ((rows + kAttnWarps * rw - 1) / (kAttnWarps * rw));
    if (blocks > INT32_MAX) fail(LB_ERR_UNSUPPORTED, "attention: too many rows for the CUDA-core kernels' grid");
    return (unsigned)blocks;
}
// `streamed`: the rows that the kernel walks per head
template <int DU, int RW, class Kernel, class... Args>
void launch_attn(Kernel kernel, unsigned blocks, int streamed, cudaStream_t st, AttnShape s, Args... args) {
    if (AttnSmem<DU, RW>::bytes(kChunk) > 48 * 1024 && first_use_on_device((const void*)kernel))
        LB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnSmem<DU, RW>::bytes(kChunk)));
    s.tile_rows = std::min(kChunk, (std::max(streamed, 1) + 3) / 4 * 4);
    launch_overlapped(kernel, dim3(blocks), dim3(kAttnWarps * 32), AttnSmem<DU, RW>::bytes(s.tile_rows), st, 0, args..., s);
}
// Two rows a warp fetch a streamed element for both (every bit the same): from 512 blocks of one row a warp on, which is where they win. us,
// one row -> two, forward, backward: 4 x 8 heads x 256 x 64 float32 48.9 -> 43.5, 140 -> 118; 2 x 8 x 300 x 128 109 -> 104, 317 -> 270; 2 x 4 x 500 x
// 256 202 -> 166, 567 -> 492; bfloat16 16 x 704 x 64 of one batch entry 160 -> 138; but fewer blocks 8 x 4 x 64 x 32 6.1 -> 6.3, 2 x 140 x 32 9.4 ->
// 11.0. Where head dims up to 32 are masked the line is at 768: 2 x 4 x 520 (520 blocks) 38.5 -> 40.2, 2 x 4 x 1000 106 -> 93, 277 -> 213. Over 14
// shapes of 512 to 4096 blocks, head dims of 32 to 256 in either type: 0.53 - 1.02 of the time; the six forms that spill up to 52 bytes 0.65 - 0.87.
// Four rows: 0.68 - 1.6 of the time.
bool two_rows(const AttnShape& s, long long heads, long long rows) {
    return s.B * heads * ((rows + kAttnWarps - 1) / kAttnWarps) >= (s.causal && s.D <= 32 ? 768 : 512);
}
template <class F>
void with_rows(bool two, F&& f) {
    if (two) f(std::integral_constant<int, 2>());
    else f(std::integral_constant<int, 1>());
}
// calls `f` with the head-dim elements per lane as a compile-time number: 1, 2, 4 or 8
template <class F>
void with_dims_per_lane(int D, F&& f) {
    if (D <= 32) f(std::integral_constant<int, 1>());
    else if (D <= 64) f(std::integral_constant<int, 2>());
    else if (D <= 128) f(std::integral_constant<int, 4>());
    else f(std::integral_constant<int, 8>());
}
template <class T>
void simt_fwd(const AttnShape& s, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o, float* lse, cudaStream_t st) {
    with_dims_per_lane(s.D, [&](auto du) {
        with_rows(two_rows(s, s.N, s.Sq), [&](auto rw) {
            launch_attn<du, rw>(attention_simt_fwd_kernel<T, du, rw>, attn_blocks(s.B, s.N, s.Sq, rw), s.Sk, st, s, (const T*)q.ptr, (const T*)k.ptr, (const T*)v.ptr,
                                (T*)o.ptr, lse);
        });
    });
}
template <class T>
void simt_bwd(const AttnShape& s, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o, const lb_tensor& g,
              const float* lse, float* delta, const lb_tensor& dq, const lb_tensor& dk, const lb_tensor& dv, cudaStream_t st) {
    const long long warps = (long long)s.B * s.N * s.Sq;
    launch_overlapped(attention_delta_simt<T>, dim3((unsigned)((warps * 32 + 255) / 256)), dim3(256), 0, st, 0, (const T*)o.ptr, (const T*)g.ptr, delta, s);
    with_dims_per_lane(s.D, [&](auto du) {
        with_rows(two_rows(s, s.N, s.Sq), [&](auto rw) {
            launch_attn<du, rw>(attention_simt_dq_kernel<T, du, rw>, attn_blocks(s.B, s.N, s.Sq, rw), s.Sk, st, s, (const T*)q.ptr, (const T*)k.ptr, (const T*)v.ptr,
                                (const T*)g.ptr, lse, (const float*)delta, (T*)dq.ptr);
        });
        with_rows(two_rows(s, s.Nkv, s.Sk), [&](auto rw) {
            launch_attn<du, rw>(attention_simt_dkdv_kernel<T, du, rw>, attn_blocks(s.B, s.Nkv, s.Sk, rw), s.Sq, st, s, (const T*)q.ptr, (const T*)k.ptr, (const T*)v.ptr,
                                (const T*)g.ptr, lse, (const float*)delta, (T*)dk.ptr, (T*)dv.ptr);
        });
    });
}
}  // namespace

void attention_simt_fwd(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o,
                        const lb_tensor* lse, void* stream) {
    AttnShape s = attn_shape(desc, q, k, v);
    fill_strides(s.o_s, o);
    driver();
    if ((long long)s.B * s.N * s.Sq == 0) return;
    cudaStream_t st = (cudaStream_t)stream;
    float* out_lse = lse ? (float*)lse->ptr : nullptr;
    if (q.dtype == LB_F32) simt_fwd<float>(s, q, k, v, o, out_lse, st);
    else if (q.dtype == LB_BF16) simt_fwd<__nv_bfloat16>(s, q, k, v, o, out_lse, st);
    else fail(LB_ERR_UNSUPPORTED, "attention: float32 or bfloat16 operands");
    LB_CUDA(cudaGetLastError());
}

void attention_simt_bwd(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o,
                        const lb_tensor& g, const lb_tensor& lse, const lb_tensor& delta, const lb_tensor& dq, const lb_tensor& dk,
                        const lb_tensor& dv, void* stream) {
    AttnShape s = attn_shape(desc, q, k, v);
    fill_strides(s.o_s, o), fill_strides(s.g_s, g), fill_strides(s.dq_s, dq), fill_strides(s.dk_s, dk), fill_strides(s.dv_s, dv);
    driver();
    cudaStream_t st = (cudaStream_t)stream;
    if ((long long)s.B * s.N * s.Sq == 0 || (long long)s.B * s.Nkv * s.Sk == 0) return;
    if (q.dtype == LB_F32) simt_bwd<float>(s, q, k, v, o, g, (const float*)lse.ptr, (float*)delta.ptr, dq, dk, dv, st);
    else if (q.dtype == LB_BF16) simt_bwd<__nv_bfloat16>(s, q, k, v, o, g, (const float*)lse.ptr, (float*)delta.ptr, dq, dk, dv, st);
    else fail(LB_ERR_UNSUPPORTED, "attention: float32 or bfloat16 operands");
    LB_CUDA(cudaGetLastError());
}

}  // namespace lb
