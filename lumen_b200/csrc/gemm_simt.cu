// The CUDA-core GEMM: exact float32 accumulation in contracting order (lumen/reference/mod.rs:958-970), for float32 operands
// and for layouts the tensor-core kernels do not take.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <vector>

#include "gemm.h"
#include "launch.cuh"

namespace lb {
namespace {

template <class T>
__device__ __forceinline__ float load_as_float(const T* p);
template <>
__device__ __forceinline__ float load_as_float<float>(const float* p) { return *p; }
template <>
__device__ __forceinline__ float load_as_float<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <>
__device__ __forceinline__ float load_as_float<__half>(const __half* p) { return __half2float(*p); }

// Four consecutive elements widened to float; the address is a multiple of four elements.
template <class T>
__device__ __forceinline__ float4 load4_as_float(const T* p) {
    if constexpr (sizeof(T) == 4) {
        return *(const float4*)p;
    } else {
        const uint2 w = *(const uint2*)p;
        const T* e = (const T*)&w;
        return make_float4(load_as_float(e), load_as_float(e + 1), load_as_float(e + 2), load_as_float(e + 3));
    }
}

// One operand's [TX rows x SK] slice of a tile on its way from global to shared memory: groups of four elements along
// the contiguous axis are fetched into registers one slice ahead of the arithmetic and then stored as s[k][row], rows
// permuted within a slice by an XOR with the k group: the four scalar stores of a group along k and the one vector store
// of a group along the rows then spread over the banks, and a thread still reads aligned vectors.
template <class T, int TX, int SK, int THREADS>
struct SimtSlice {
    static constexpr int kGroups = TX * SK / 4 / THREADS;
    static_assert(kGroups * 4 * THREADS == TX * SK && THREADS % (SK / 4) == 0 && THREADS % (TX / 4) == 0, "whole groups per thread");
    float4 held[kGroups];

    static __device__ __forceinline__ int slot(int k, int row) { return k * TX + (row ^ ((k & ~3) & (TX - 4) & 28)); }

    // `x` points at the operand's batch; rows [row0, row0 + TX), contracting indices [k0, k0 + SK); `whole`: all of them
    // exist and groups of four along the contiguous axis are aligned
    __device__ __forceinline__ void fetch(const T* x, int row0, int rows, int k0, int K, long long s_row, long long s_k, bool along_k, bool whole) {
        const int r0 = row0 + (along_k ? threadIdx.x / (SK / 4) : threadIdx.x % (TX / 4) * 4);
        const int kk = k0 + (along_k ? threadIdx.x % (SK / 4) * 4 : threadIdx.x / (TX / 4));
        const T* at = x + r0 * s_row + kk * s_k;
        const long long step = along_k ? THREADS / (SK / 4) * s_row : THREADS / (TX / 4) * s_k;
        if (whole) {
#pragma unroll
            for (int i = 0; i < kGroups; i++) held[i] = load4_as_float(at + i * step);
        } else {
#pragma unroll
            for (int i = 0; i < kGroups; i++) {
                const int r = r0 + (along_k ? i * (THREADS / (SK / 4)) : 0), k = kk + (along_k ? 0 : i * (THREADS / (TX / 4)));
                float e[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                    e[j] = (along_k ? r < rows && k + j < K : r + j < rows && k < K) ? load_as_float(at + i * step + j * (along_k ? s_k : s_row)) : 0.0f;
                held[i] = make_float4(e[0], e[1], e[2], e[3]);
            }
        }
    }
    __device__ __forceinline__ void put(float* s, bool along_k) const {
#pragma unroll
        for (int i = 0; i < kGroups; i++) {
            const int id = threadIdx.x + i * THREADS;
            if (along_k) {
                const int r = id / (SK / 4), k = id % (SK / 4) * 4;
                s[slot(k, r)] = held[i].x, s[slot(k + 1, r)] = held[i].y, s[slot(k + 2, r)] = held[i].z, s[slot(k + 3, r)] = held[i].w;
            } else {
                *(float4*)(s + slot(id / (TX / 4), id % (TX / 4) * 4)) = held[i];
            }
        }
    }
};

template <int N> struct SimtVec;
template <> struct SimtVec<1> { typedef float type; };
template <> struct SimtVec<2> { typedef float2 type; };
template <> struct SimtVec<4> { typedef float4 type; };

// A TM x TN output tile per CTA, RM x RN outputs per thread. Slices of SK contracting indices are double-buffered in shared
// memory and the next one is in flight to registers meanwhile. Products and sums are rounded one by one in contracting
// order. A last slice that K does not fill is summed index by index: with a whole slice of zeros instead, 4096 x 4096 with K = 1
// took 49 us against 20, 1024 x 1024 with K = 15 9.9 against 5.9.
template <class T, int TM, int TN, int RM, int RN, int SK>
__device__ __forceinline__ void simt_tile(const T* ab, const T* bb, const SimtArgs& p, int m0, int n0, int bz, float (*sa)[SK * TM], float (*sb)[SK * TN]) {
    constexpr int THREADS = TM / RM * (TN / RN);
    typedef SimtSlice<T, TM, SK, THREADS> SliceA;
    typedef SimtSlice<T, TN, SK, THREADS> SliceB;
    typedef typename SimtVec<RM>::type VecA;
    typedef typename SimtVec<RN>::type VecB;
    const int tx = threadIdx.x % (TN / RN), ty = threadIdx.x / (TN / RN);
    const bool a_k = p.a_sk == 1, b_k = p.b_sn != 1;  // fetch along whichever axis is contiguous
    const bool a_whole = p.a_vec && m0 + TM <= p.M, b_whole = p.b_vec && n0 + TN <= p.N;
    float acc[RM][RN] = {};
    SliceA fa;
    SliceB fb;
    fa.fetch(ab, m0, p.M, 0, p.K, p.a_sm, p.a_sk, a_k, a_whole && SK <= p.K);
    fb.fetch(bb, n0, p.N, 0, p.K, p.b_sn, p.b_sk, b_k, b_whole && SK <= p.K);
    int buf = 0;
    for (int k0 = 0; k0 < p.K; k0 += SK, buf ^= 1) {
        fa.put(sa[buf], a_k);
        fb.put(sb[buf], b_k);
        __syncthreads();  // the other buffer's readers are two slices back: one barrier per slice is enough
        if (k0 + SK < p.K) {
            fa.fetch(ab, m0, p.M, k0 + SK, p.K, p.a_sm, p.a_sk, a_k, a_whole && k0 + 2 * SK <= p.K);
            fb.fetch(bb, n0, p.N, k0 + SK, p.K, p.b_sn, p.b_sk, b_k, b_whole && k0 + 2 * SK <= p.K);
        }
        if (p.K - k0 < SK) {  // the last slice of a K that is no multiple: only its indices
#pragma unroll 4
            for (int k = 0; k < p.K - k0; k++) {
                const VecA a1 = *(const VecA*)(sa[buf] + SliceA::slot(k, ty * RM));
                const VecB b1 = *(const VecB*)(sb[buf] + SliceB::slot(k, tx * RN));
#pragma unroll
                for (int i = 0; i < RM; i++)
#pragma unroll
                    for (int j = 0; j < RN; j++) acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(((const float*)&a1)[i], ((const float*)&b1)[j]));
            }
            break;
        }
        // 32 indices unrolled: the row permutation has that period, so its XORs become eight precomputed addresses per
        // operand. Values are read from shared memory a group of four indices ahead of their use.
        VecA av[2][4];
        VecB bv[2][4];
        auto read = [&](int to, const float* pa, const float* pb, int k) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                av[to][u] = *(const VecA*)(pa + SliceA::slot(k + u, ty * RM));
                bv[to][u] = *(const VecB*)(pb + SliceB::slot(k + u, tx * RN));
            }
        };
        read(0, sa[buf], sb[buf], 0);
#pragma unroll 1
        for (int k32 = 0; k32 < SK; k32 += 32) {
            const float *pa = sa[buf] + k32 * TM, *pb = sb[buf] + k32 * TN;
#pragma unroll
            for (int k = 0; k < 32; k += 4) {
                const int now = (k / 4) & 1;
                if (k + 4 < 32) read(now ^ 1, pa, pb, k + 4);
                else if (k32 + 32 < SK) read(now ^ 1, pa + 32 * TM, pb + 32 * TN, 0);
#pragma unroll
                for (int u = 0; u < 4; u++)
#pragma unroll
                    for (int i = 0; i < RM; i++)
#pragma unroll
                        for (int j = 0; j < RN; j++)
                            acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(((const float*)&av[now][u])[i], ((const float*)&bv[now][u])[j]));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RM; i++)
#pragma unroll
        for (int j = 0; j < RN; j++) {
            const int gm = m0 + ty * RM + i, gn = n0 + tx * RN + j;
            if (gm >= p.M || gn >= p.N) continue;
            float x = acc[i][j];
            if (p.epilogue == EPI_RELU) x = fmaxf(x, 0.0f);
            if (p.epilogue >= EPI_ADD) {  // the rounded product, then the second primitive on it (as the tensor-core kernels do)
                const long long from = (long long)bz * p.aux_sb + (long long)gm * p.ld_aux + gn;
                float prod = x, other;
                if (p.d_dtype == LB_F32) {
                    other = ((const float*)p.aux)[from];
                } else {
                    const uint16_t a16 = ((const uint16_t*)p.aux)[from];
                    if (p.d_dtype == LB_BF16) prod = __bfloat162float(__float2bfloat16_rn(x)), other = __uint_as_float((uint32_t)a16 << 16);
                    else prod = __half2float(__float2half_rn(x)), other = __half2float(__ushort_as_half(a16));
                }
                x = p.epilogue == EPI_ADD ? __fadd_rn(other, prod) : (other > 0.0f ? prod : 0.0f);
            }
            long long at = (long long)bz * p.d_sb + (long long)gm * p.ldd + gn;
            if (p.d_dtype == LB_F32) ((float*)p.d)[at] = x;
            else if (p.d_dtype == LB_BF16) ((__nv_bfloat16*)p.d)[at] = __float2bfloat16_rn(x);
            else ((__half*)p.d)[at] = __float2half_rn(x);
        }
}

template <class T, int TM, int TN, int RM, int RN, int SK>
__global__ void __launch_bounds__(TM / RM * (TN / RN)) gemm_simt_kernel(const T* __restrict__ a, const T* __restrict__ b, const SimtArgs p) {
    __shared__ __align__(16) float sa[2][SK * TM], sb[2][SK * TN];
    const T* ab = a + (long long)blockIdx.z * p.a_sb;
    const T* bb = b + (long long)blockIdx.z * p.b_sb;
    grid_wait(ab, bb);
    simt_tile<T, TM, TN, RM, RN, SK>(ab, bb, p, blockIdx.y * TM, blockIdx.x * TN, blockIdx.z, sa, sb);
}

// Several products that do not depend on one another in one launch: each with its blocks' first place in the grid, on the tiles, and so
// with the bits, that it would have alone. What bounds such a product is the chain of one sum of K terms: alone it gives an SM one or
// two blocks of four warps, which leave most of its cycles empty, and the next product waits for the last of them. The nine pairs of gradients
// of linear layers in a training step of two layers of width 128 (vocabulary 256, 256 tokens) took 9 launches less: 139.5 -> 130.7 us a step
// queued ahead, 276 -> 265.6 alone; of width 64 and 140 tokens 63.3 -> 57.4 and 183 -> 161.
struct SimtGroup {
    int n;
    unsigned first[kSimtGroup + 1], tiles_n[kSimtGroup], tiles_m[kSimtGroup];
    int wide[kSimtGroup];
    const float* a[kSimtGroup];
    const float* b[kSimtGroup];
    SimtArgs p[kSimtGroup];
};
__global__ void __launch_bounds__(128) gemm_simt_group_kernel(const __grid_constant__ SimtGroup g) {
    __shared__ __align__(16) float sa[2][64 * 32], sb[2][64 * 32];
    int i = 0;
    while (i + 1 < g.n && g.first[i + 1] <= blockIdx.x) i++;
    const unsigned t = blockIdx.x - g.first[i], x = t % g.tiles_n[i], y = t / g.tiles_n[i] % g.tiles_m[i], z = t / g.tiles_n[i] / g.tiles_m[i];
    grid_wait();
    const SimtArgs& p = g.p[i];
    const float* ab = g.a[i] + (long long)z * p.a_sb;
    const float* bb = g.b[i] + (long long)z * p.b_sb;
    if (g.wide[i]) simt_tile<float, 32, 32, 2, 4, 64>(ab, bb, p, y * 32, x * 32, z, sa, sb);
    else simt_tile<float, 16, 32, 2, 2, 64>(ab, bb, p, y * 16, x * 32, z, (float(*)[64 * 16])sa, sb);
}

// The largest tile of which there are enough to give every SM one: a sum runs in contracting order, so the only
// parallelism is over outputs. A product too small to fill the SMs with 64 x 64 tiles is bound by the instructions and
// latencies between one contracting index and the next, which smaller tiles shorten. Alone on a B200, float32:
// 512 x 128 x 512 8.6 us with 16 x 32 tiles against 11.8 (32 x 32) and 30 (64 x 64), 512 x 512 x 128 6.1 us with 32 x 32
// against 7.0 and 9.9, 2048^3 0.66 ms with 64 x 64 against 0.80 and 1.01; a single 64 x 64 kernel that fetched its slices
// between two barriers took 57 us a product at the first two shapes.
enum SimtTile { TILE_64, TILE_32, TILE_16 };  // 64 x 64, 32 x 32, 16 x 32
dim3 simt_grid(const SimtArgs& p, SimtTile t) {
    const int tm = t == TILE_64 ? 64 : t == TILE_32 ? 32 : 16, tn = t == TILE_64 ? 64 : 32;
    return dim3((unsigned)((p.N + tn - 1) / tn), (unsigned)((p.M + tm - 1) / tm), (unsigned)p.batch);
}
SimtTile simt_tile_for(const SimtArgs& p, int sms) {
    auto tiles = [&](SimtTile t) { const dim3 g = simt_grid(p, t); return (long long)g.x * g.y * g.z; };
    return tiles(TILE_64) >= 2LL * sms ? TILE_64 : tiles(TILE_32) >= sms ? TILE_32 : TILE_16;
}
template <class T>
void launch_simt(const T* a, const T* b, const SimtArgs& p, int sms, cudaStream_t s) {
    const SimtTile t = simt_tile_for(p, sms);
    const dim3 grid = simt_grid(p, t);
    if (t == TILE_64) launch_overlapped(gemm_simt_kernel<T, 64, 64, 4, 4, 32>, grid, dim3(256), 0, s, 0, a, b, p);
    else if (t == TILE_32) launch_overlapped(gemm_simt_kernel<T, 32, 32, 2, 4, 64>, grid, dim3(128), 0, s, 0, a, b, p);
    else launch_overlapped(gemm_simt_kernel<T, 16, 32, 2, 2, 64>, grid, dim3(128), 0, s, 0, a, b, p);
}

}  // namespace

void gemm_simt(const void* a, const void* b, int dtype, const SimtArgs& p, int sms, cudaStream_t s) {
    if (dtype == LB_F32) launch_simt<float>((const float*)a, (const float*)b, p, sms, s);
    else if (dtype == LB_BF16) launch_simt<__nv_bfloat16>((const __nv_bfloat16*)a, (const __nv_bfloat16*)b, p, sms, s);
    else launch_simt<__half>((const __half*)a, (const __half*)b, p, sms, s);
}

// Products of float32 operands that do not depend on one another: those on tiles of 64 x 64 fill the GPU by themselves, of the others up to
// kSimtGroup share a launch, the ones with the longest sums first. Returns how many launches that takes; `launch` false only counts them.
int gemm_simt_many(const SimtProblem* problems, int n, int sms, bool launch, cudaStream_t s) {
    std::vector<const SimtProblem*> small;
    int launches = 0;
    for (int i = 0; i < n; i++) {
        if (simt_tile_for(problems[i].p, sms) != TILE_64) {
            small.push_back(&problems[i]);
            continue;
        }
        launches++;
        if (launch) launch_simt<float>((const float*)problems[i].a, (const float*)problems[i].b, problems[i].p, sms, s);
    }
    std::stable_sort(small.begin(), small.end(), [](const SimtProblem* x, const SimtProblem* y) { return x->p.K > y->p.K; });
    for (size_t at = 0; at < small.size(); at += kSimtGroup) {
        const int count = (int)std::min<size_t>(kSimtGroup, small.size() - at);
        launches++;
        if (!launch) continue;
        if (count == 1) {
            launch_simt<float>((const float*)small[at]->a, (const float*)small[at]->b, small[at]->p, sms, s);
            continue;
        }
        SimtGroup g{};
        g.n = count;
        for (int i = 0; i < count; i++) {
            const SimtProblem& q = *small[at + i];
            const SimtTile t = simt_tile_for(q.p, sms);
            const dim3 grid = simt_grid(q.p, t);
            g.tiles_n[i] = grid.x, g.tiles_m[i] = grid.y, g.wide[i] = t == TILE_32;
            g.first[i + 1] = g.first[i] + grid.x * grid.y * grid.z;
            g.a[i] = (const float*)q.a, g.b[i] = (const float*)q.b, g.p[i] = q.p;
        }
        launch_overlapped(gemm_simt_group_kernel, dim3(g.first[count]), dim3(128), 0, s, 0, g);
    }
    return launches;
}

}  // namespace lb
