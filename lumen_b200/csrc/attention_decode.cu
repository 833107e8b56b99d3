// Flash-attention forward for few query rows per key head (decoding against a cache): at most 32 rows share a key head's
// keys, so the keys and values are read once and everything else is small. What bounds it is HBM bandwidth, provided
// that enough loads are in flight on every SM - the tile kernel (attention_fwd.cu) gave a CTA per query head a 128-row
// tile of which one row was live and walked the whole cache in series: 158 us for 16 x 32 heads (8 key heads) against
// 4097 keys of 128, 269 MB, which this kernel does in 45 us (5.9 TB/s).
//
// Grid: (splits, key heads, batch), the splits of one key head a thread-block cluster. The query heads of the group and
// the query positions are the rows of one or two 16-row tiles, so grouped heads share what is read. Each of the CTA's
// four warps walks a range of keys of its own, 16 at a time: its rows of K and V come through a private ring of
// shared memory (cp.async, no barrier between warps), scores and values by mma.sync m16n8k16 - 16-row tiles are what
// this shape needs; a tcgen05 product has at least 64 rows and the tensor pipe is idle either way. Every warp keeps its
// own running maximum, sum and output; they are merged in shared memory, across the cluster through distributed shared
// memory (no scratch memory, no second kernel), and rounded once.
#include <cuda_bf16.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "attention.h"
#include "launch.cuh"
#include "sm100.cuh"

namespace lb {
namespace {

using namespace sm100;

constexpr int kWarps = 4, kSlice = 16, kStages = 3, kMaxRows = 32, kMaxSplits = 16;

struct DecodeArgs {
    const __nv_bfloat16 *q, *k, *v;
    __nv_bfloat16* o;
    float* lse;
    long long q_sb, q_ss, q_sn, k_sb, k_ss, k_sn, v_sb, v_ss, v_sn, o_sb, o_ss, o_sn;
    int N, Nkv, Sq, Sk, causal;
    long long causal_offset;
    float scale_log2;
    int pair_stores;  // the output's rows are 4-byte aligned
};

__device__ __forceinline__ void copy_16(uint32_t dst, const void* src, bool live) {  // zeros where there is no row
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void ldmatrix_x4(uint32_t* r, uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t* r, uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void mma_16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *(const uint32_t*)&h;
}
// byte offset of 16-byte chunk `c` of row `r` in a tile of rows of D elements: chunks permuted so that eight rows' equal
// chunks fall in different banks
template <int D> __device__ __forceinline__ uint32_t chunk_at(int r, int c) { return (uint32_t)(r * D * 2 + ((c ^ (r & 7)) << 4)); }

template <int D, int MT>
struct DecodeSmem {
    static constexpr int kRows = MT * 16;
    static constexpr int kQ = kRows * D * 2, kTile = kSlice * D * 2;
    static constexpr int kRing = kWarps * kStages * 2 * kTile;
    static constexpr int kMerge = kWarps * kRows * D * 4;  // the warps' outputs, over the ring once it is drained
    static constexpr int kWork = kRing > kMerge ? kRing : kMerge;
    static constexpr int kBytes = kQ + kWork + kRows * D * 4 /* the CTA's output */ + (kWarps + 1) * kRows * 2 * 4 /* maxima, sums */;
};

template <int D, int MT>
__global__ void __launch_bounds__(kWarps * 32, 2) attention_decode_kernel(const DecodeArgs p) {
    typedef DecodeSmem<D, MT> L;
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* sq = smem;
    uint8_t* ring = smem + L::kQ;
    float* out_cta = (float*)(ring + L::kWork);           // [rows][D], merged over the CTA's warps
    float* max_w = out_cta + L::kRows * D;                // [warps + 1][rows]; the last row set is the CTA's
    float* sum_w = max_w + (kWarps + 1) * L::kRows;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split = blockIdx.x, splits = gridDim.x, kv = blockIdx.y, b = blockIdx.z;
    const int group = p.N / p.Nkv, rows = group * p.Sq;  // row r: query head kv * group + r % group, position r / group
    grid_wait();

    for (int i = threadIdx.x; i < L::kRows * (D / 8); i += kWarps * 32) {
        const int r = i / (D / 8), c = i % (D / 8);
        uint4 x = make_uint4(0, 0, 0, 0);
        if (r < rows) x = *(const uint4*)(p.q + b * p.q_sb + (long long)(r / group) * p.q_ss + (long long)(kv * group + r % group) * p.q_sn + c * 8);
        *(uint4*)(sq + chunk_at<D>(r, c)) = x;
    }
    // this warp's slices of 16 keys: a contiguous range
    const long long keys = p.causal ? max(0LL, min((long long)p.Sk, (long long)p.Sq + p.causal_offset)) : (long long)p.Sk;
    const long long slices = (keys + kSlice - 1) / kSlice;
    const int worker = split * kWarps + warp, workers = splits * kWarps;
    const int first = (int)(slices * worker / workers), last = (int)(slices * (worker + 1) / workers);
    const __nv_bfloat16 *kb = p.k + b * p.k_sb + kv * p.k_sn, *vb = p.v + b * p.v_sb + kv * p.v_sn;
    uint8_t* mine = ring + warp * (kStages * 2 * L::kTile);
    auto fetch = [&](int slice) {
        if (slice < last) {
            const uint32_t at = smem_u32(mine + (slice - first) % kStages * (2 * L::kTile));
#pragma unroll
            for (int i = 0; i < kSlice * (D / 8) / 32; i++) {
                const int r = (i * 32 + lane) / (D / 8), c = (i * 32 + lane) % (D / 8);
                const long long j = (long long)slice * kSlice + r;
                const long long row = j < p.Sk ? j : 0;
                copy_16(at + chunk_at<D>(r, c), kb + row * p.k_ss + c * 8, j < p.Sk);
                copy_16(at + L::kTile + chunk_at<D>(r, c), vb + row * p.v_ss + c * 8, j < p.Sk);
            }
        }
        copies_commit();  // an empty group where there is nothing left: the counts below stay the same
    };
#pragma unroll
    for (int s = 0; s < kStages - 1; s++) fetch(first + s);
    __syncthreads();  // the queries are in place

    uint32_t qf[MT][D / 16][4];
#pragma unroll
    for (int t = 0; t < MT; t++)
#pragma unroll
        for (int k = 0; k < D / 16; k++) ldmatrix_x4(qf[t][k], smem_u32(sq) + chunk_at<D>(t * 16 + (lane & 15), k * 2 + (lane >> 4)));
    float acc[MT][D / 8][4] = {}, m[MT][2], l[MT][2];
    long long limit[MT][2];  // last visible key of this thread's two rows per tile
#pragma unroll
    for (int t = 0; t < MT; t++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = t * 16 + h * 8 + (lane >> 2);
            m[t][h] = -INFINITY, l[t][h] = 0.0f;
            limit[t][h] = p.causal ? min((long long)p.Sk - 1, (long long)(r / group) + p.causal_offset) : (long long)p.Sk - 1;
        }
    for (int slice = first; slice < last; slice++) {
        copies_wait<kStages - 2>();
        __syncwarp();
        fetch(slice + kStages - 1);  // into the stage read in the last round
        const uint32_t at = smem_u32(mine + (slice - first) % kStages * (2 * L::kTile));
        float s[MT][2][4] = {};
#pragma unroll
        for (int k = 0; k < D / 16; k++) {
            uint32_t kf[4];  // keys 0-7 and 8-15 of head-dim elements 16 k .. 16 k + 15
            ldmatrix_x4(kf, at + chunk_at<D>((lane & 7) + ((lane >> 4) << 3), k * 2 + ((lane >> 3) & 1)));
#pragma unroll
            for (int t = 0; t < MT; t++) mma_16816(s[t][0], qf[t][k], kf[0], kf[1]), mma_16816(s[t][1], qf[t][k], kf[2], kf[3]);
        }
        uint32_t pf[MT][4];
#pragma unroll
        for (int t = 0; t < MT; t++) {
            const long long key0 = (long long)slice * kSlice + (lane & 3) * 2;
#pragma unroll
            for (int h = 0; h < 2; h++) {  // rows lane / 4 and lane / 4 + 8
                float x[4] = {s[t][0][2 * h], s[t][0][2 * h + 1], s[t][1][2 * h], s[t][1][2 * h + 1]};
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (key0 + (i & 1) + (i >> 1) * 8 > limit[t][h]) x[i] = -INFINITY;
                float top = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
                const float m_new = fmaxf(m[t][h], top * p.scale_log2), shift = m_new == -INFINITY ? 0.0f : m_new;
                const float alpha = fast_exp2(m[t][h] - shift);
#pragma unroll
                for (int i = 0; i < 4; i++) x[i] = fast_exp2(fmaf(x[i], p.scale_log2, -shift));  // rounded once, as in the tile kernel
                l[t][h] = l[t][h] * alpha + ((x[0] + x[1]) + (x[2] + x[3]));  // this thread's keys; the quad is added up at the end
                pf[t][h] = pack(x[0], x[1]), pf[t][2 + h] = pack(x[2], x[3]);
                m[t][h] = m_new;
                if (__any_sync(0xffffffffu, alpha != 1.0f)) {
#pragma unroll
                    for (int d = 0; d < D / 8; d++) acc[t][d][2 * h] *= alpha, acc[t][d][2 * h + 1] *= alpha;
                }
            }
        }
#pragma unroll
        for (int d = 0; d < D / 16; d++) {
            uint32_t vf[4];  // 16 keys of head-dim elements 16 d .. 16 d + 15, transposed on the way
            ldmatrix_x4_trans(vf, at + L::kTile + chunk_at<D>(lane & 15, d * 2 + (lane >> 4)));
#pragma unroll
            for (int t = 0; t < MT; t++) mma_16816(acc[t][2 * d], pf[t], vf[0], vf[1]), mma_16816(acc[t][2 * d + 1], pf[t], vf[2], vf[3]);
        }
    }
    copies_wait<0>();
    __syncthreads();  // every warp is done with its ring

    // ---- the CTA's four warps into one ----
    float* merge = (float*)ring;
#pragma unroll
    for (int t = 0; t < MT; t++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = t * 16 + h * 8 + (lane >> 2);
            float sum = l[t][h];
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            if ((lane & 3) == 0) max_w[warp * L::kRows + r] = m[t][h], sum_w[warp * L::kRows + r] = sum;
#pragma unroll
            for (int d = 0; d < D / 8; d++)
                *(float2*)(merge + (warp * L::kRows + r) * D + d * 8 + (lane & 3) * 2) = make_float2(acc[t][d][2 * h], acc[t][d][2 * h + 1]);
        }
    __syncthreads();
    auto weight = [](float part, float whole) { return part == -INFINITY ? 0.0f : fast_exp2(part - whole); };
    for (int i = threadIdx.x; i < rows * D; i += kWarps * 32) {
        const int r = i / D, d = i % D;
        float whole = -INFINITY, sum = 0.0f, o = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; w++) whole = fmaxf(whole, max_w[w * L::kRows + r]);
#pragma unroll
        for (int w = 0; w < kWarps; w++) {
            const float a = weight(max_w[w * L::kRows + r], whole);
            o += a * merge[(w * L::kRows + r) * D + d], sum += a * sum_w[w * L::kRows + r];
        }
        out_cta[i] = o;
        if (d == 0) max_w[kWarps * L::kRows + r] = whole, sum_w[kWarps * L::kRows + r] = sum;
    }
    // ---- the cluster's CTAs into one: each writes its share of the outputs ----
    cluster_sync();
    auto remote = [](const float* at, int rank) {
        uint32_t there;
        float x;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(smem_u32(at)), "r"(rank));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(there) : "memory");
        return x;
    };
    for (int i = split * kWarps * 32 + threadIdx.x; i < rows * (D / 2); i += splits * kWarps * 32) {
        const int r = i / (D / 2), d = i % (D / 2) * 2;
        float whole = -INFINITY, sum = 0.0f, x = 0.0f, y = 0.0f;
        for (int c = 0; c < splits; c++) whole = fmaxf(whole, remote(max_w + kWarps * L::kRows + r, c));
        for (int c = 0; c < splits; c++) {
            const float a = weight(remote(max_w + kWarps * L::kRows + r, c), whole);
            sum += a * remote(sum_w + kWarps * L::kRows + r, c);
            x += a * remote(out_cta + r * D + d, c), y += a * remote(out_cta + r * D + d + 1, c);
        }
        const float inv = 1.0f / sum;  // a row that sees no key is 0 / 0 in the traced program: NaN
        const int head = kv * group + r % group, position = r / group;
        __nv_bfloat16* o = p.o + b * p.o_sb + (long long)position * p.o_ss + (long long)head * p.o_sn + d;
        if (p.pair_stores) *(__nv_bfloat162*)o = __floats2bfloat162_rn(x * inv, y * inv);
        else o[0] = __float2bfloat16_rn(x * inv), o[1] = __float2bfloat16_rn(y * inv);
        // one rounding at the size of the result: (whole + log2f(sum)) * ln 2 has two, one of them at 1.44 times the size
        if (d == 0 && p.lse) p.lse[((long long)b * p.N + head) * p.Sq + position] = fmaf(whole, 0.6931471805599453f, logf(sum));
    }
    cluster_sync();  // nobody leaves while it is read
}

// How the kernel does on a problem, in microseconds of a B200: a CTA costs `base + per_row * rows` (prologue, merge, the way out)
// and `per_slice` per slice that a warp walks, and the keys and values cross HBM at most at `gb` GB/s. Fitted to 1373 timings of
// 1 to 32 rows, 4 to 4096 (batch, key head)s and 32 to 8192 keys (root mean square of the error 15 to 20 %).
struct DecodeCost {
    int resident;  // CTAs per SM: shared memory at head dim 128, registers at 64
    double base, per_row, per_slice, gb;
};
constexpr DecodeCost decode_cost(int D, int MT) {
    return D == 64 ? (MT == 1 ? DecodeCost{4, 3.4, 0.14, 1.37, 6100} : DecodeCost{2, 4.9, 0.11, 1.01, 4400})
                   : (MT == 1 ? DecodeCost{2, 3.8, 0.26, 1.31, 6600} : DecodeCost{1, 5.5, 0.245, 1.2, 3500});
}
// CTAs that share one key head's keys: the number that spreads the slices most evenly over the CTAs that fit the SMs, in
// units of slices per warp; a CTA counts as six slices besides (the costs above: 3 to 6 with one tile of rows, 7 to 11 with two).
int pick_splits(const DecodeCost& cost, long long pairs, long long keys, int sms) {
    const long long slices = (keys + kSlice - 1) / kSlice, slots = (long long)cost.resident * sms;
    int best = 1;
    double best_cost = 1e30;
    for (int s = 1; s <= kMaxSplits; s++) {
        if (s > 1 && (long long)s * kWarps > slices) break;
        const double waves = (double)((pairs * s + slots - 1) / slots);
        const double units = waves * ((double)((slices + s * kWarps - 1) / (s * kWarps)) + 6.0);
        if (units < best_cost * 0.98) best = s, best_cost = units;
    }
    return best;
}
// Clusters of more than eight CTAs (a size not every part has) only where the runtime says that they can be resident.
template <int D, int MT>
int resident_splits(int splits) {
    if (splits <= 8) return splits;
    auto kernel = attention_decode_kernel<D, MT>;
    static std::map<int, bool> fits;  // by device
    static std::mutex mutex;
    int dev = 0;
    LB_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mutex);
    auto it = fits.find(dev);
    if (it == fits.end()) {
        int clusters = 0;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kMaxSplits, attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(kMaxSplits), cfg.blockDim = dim3(kWarps * 32), cfg.dynamicSmemBytes = DecodeSmem<D, MT>::kBytes;
        cfg.attrs = &attr, cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) cudaGetLastError(), clusters = 0;
        it = fits.emplace(dev, clusters > 0).first;
    }
    return it->second ? splits : 8;
}

template <int D, int MT>
void launch(const DecodeArgs& p, int batch, long long keys, cudaStream_t s) {
    auto kernel = attention_decode_kernel<D, MT>;
    constexpr int bytes = DecodeSmem<D, MT>::kBytes;
    if (first_use_on_device((const void*)kernel)) {
        LB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        LB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    }
    const int splits = resident_splits<D, MT>(pick_splits(decode_cost(D, MT), (long long)batch * p.Nkv, keys, device_info().sms));
    launch_overlapped(kernel, dim3((unsigned)splits, (unsigned)p.Nkv, (unsigned)batch), dim3(kWarps * 32), bytes, s, (unsigned)splits, p);
}

}  // namespace

// Whether attention_decode takes the problem: all rows of a key head's group in two 16-row tiles. (Operands as the
// tensor-core kernels need them: bfloat16, head dim 64 or 128, unit head-dim stride, 16-byte aligned rows.)
bool attention_decodes(const lb_tensor& q, const lb_tensor& k) {
    return q.shape[0] > 0 && k.shape[1] > 0 && k.shape[2] > 0 && q.shape[2] % k.shape[2] == 0 && q.shape[0] <= 65535 && k.shape[2] <= 65535 &&
           q.shape[1] > 0 && q.shape[2] / k.shape[2] * q.shape[1] <= kMaxRows;
}

double attention_decode_us(const lb_tensor& q, const lb_tensor& k, int sms) {
    const long long pairs = q.shape[0] * k.shape[2], rows = q.shape[2] / k.shape[2] * q.shape[1], keys = k.shape[1], D = q.shape[3];
    const DecodeCost cost = decode_cost((int)D, rows <= 16 ? 1 : 2);
    const long long splits = pick_splits(cost, pairs, keys, sms), slots = (long long)cost.resident * sms;
    const long long waves = (pairs * splits + slots - 1) / slots, slices = ((keys + kSlice - 1) / kSlice + splits * kWarps - 1) / (splits * kWarps);
    const double bytes = (double)pairs * keys * D * 4;
    return std::max(waves * (cost.base + cost.per_row * rows + cost.per_slice * slices), bytes / (cost.gb * 1e3));
}

void attention_decode(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o,
                      const lb_tensor* lse, void* stream) {
    DecodeArgs p{};
    p.q = (const __nv_bfloat16*)q.ptr, p.k = (const __nv_bfloat16*)k.ptr, p.v = (const __nv_bfloat16*)v.ptr, p.o = (__nv_bfloat16*)o.ptr;
    p.lse = lse ? (float*)lse->ptr : nullptr;
    p.q_sb = q.stride[0], p.q_ss = q.stride[1], p.q_sn = q.stride[2];
    p.k_sb = k.stride[0], p.k_ss = k.stride[1], p.k_sn = k.stride[2];
    p.v_sb = v.stride[0], p.v_ss = v.stride[1], p.v_sn = v.stride[2];
    p.o_sb = o.stride[0], p.o_ss = o.stride[1], p.o_sn = o.stride[2];
    p.N = (int)q.shape[2], p.Nkv = (int)k.shape[2], p.Sq = (int)q.shape[1], p.Sk = (int)k.shape[1];
    p.causal = desc.causal, p.causal_offset = desc.causal_offset, p.scale_log2 = desc.scale * 1.4426950408889634f;
    p.pair_stores = o.stride[0] % 2 == 0 && o.stride[1] % 2 == 0 && o.stride[2] % 2 == 0 && ((uintptr_t)o.ptr & 3) == 0;
    const int rows = p.N / p.Nkv * p.Sq, batch = (int)q.shape[0];
    cudaStream_t s = (cudaStream_t)stream;
    if (q.shape[3] == 128) rows <= 16 ? launch<128, 1>(p, batch, p.Sk, s) : launch<128, 2>(p, batch, p.Sk, s);
    else rows <= 16 ? launch<64, 1>(p, batch, p.Sk, s) : launch<64, 2>(p, batch, p.Sk, s);
}

}  // namespace lb
