// What the GEMM kernels' files share.
#pragma once
#include <cuda.h>
#ifdef __CUDACC__
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#endif

#include "device.h"

namespace lb {

// EPI_ADD: out = round(round(acc) + aux); EPI_MASK: out = aux > 0 ? round(acc) : 0 - each exactly the two primitives
// of the traced program (a rounded product followed by an add / a select), with `aux` a tensor shaped like the output
enum Epilogue : int { EPI_NONE = 0, EPI_RELU = 1, EPI_ADD = 2, EPI_MASK = 3 };

#ifdef __CUDACC__
// Two products rounded to 16 bits and the tail's operand beside them: their sums, or the products where the operand is positive. The packed
// add rounds the exact sum once; a float32 add and a rounding to 16 bits give the same, since what float32 drops lies 2^-24 below the larger
// term, and no 16-bit rounding boundary is as near to a 16-bit value.
__device__ __forceinline__ uint32_t tail_pair(uint32_t product, uint32_t other, bool adds, bool bf16) {
    if (bf16) {
        const __nv_bfloat162 x = *(const __nv_bfloat162*)&other, y = *(const __nv_bfloat162*)&product;
        const __nv_bfloat162 sum = __hadd2_rn(x, y);
        return adds ? *(const uint32_t*)&sum : product & __hgt2_mask(x, __floats2bfloat162_rn(0.0f, 0.0f));
    }
    const __half2 x = *(const __half2*)&other, y = *(const __half2*)&product;
    const __half2 sum = __hadd2_rn(x, y);
    return adds ? *(const uint32_t*)&sum : product & __hgt2_mask(x, __floats2half2_rn(0.0f, 0.0f));
}
#endif

// The CUDA-core GEMM (gemm_simt.cu): any strides, element strides of the M, N and K axes.
struct SimtArgs {
    int M, N, K, batch;
    long long a_sm, a_sk, a_sb, b_sk, b_sn, b_sb, ldd, d_sb;
    void* d;
    int d_dtype;
    int epilogue;
    const void* aux;  // EPI_ADD / EPI_MASK operand (the output's dtype), rows ld_aux apart, batches aux_sb apart
    long long ld_aux, aux_sb;
    int a_vec, b_vec;  // groups of four elements along the operand's contiguous axis are aligned
};

void gemm_simt(const void* a, const void* b, int dtype, const SimtArgs& p, int sms, cudaStream_t s);

struct SimtProblem {
    const void* a;
    const void* b;
    SimtArgs p;
};
constexpr int kSimtGroup = 4;
int gemm_simt_many(const SimtProblem* problems, int n, int sms, bool launch, cudaStream_t s);

// 128 x 64 tiles with the K range of a tile over a cluster (gemm_small.cu): 16-bit operands, maps with boxes of 64
// elements along the contiguous axis by 128 rows of A, 64 of B (K-major) or 64 (M- / N-major).
struct SmallGemmArgs {
    int M, N, K;
    int a_mn_major, b_mn_major, in_bf16;
    void* d;
    int d_bf16, d_f16;  // else float32
    long long ldd, d_batch_stride;
    int epilogue;
    const void* aux;
    long long ld_aux, aux_batch_stride;
    int splits;  // CTAs of a cluster: 1, 2, 4 or 8, no more than the 64-wide blocks of K
    int* status;
    int tiles_m, tiles_n, vec, aux_vec;  // set by gemm_small
};

void gemm_small(const CUtensorMap& map_a, const CUtensorMap& map_b, SmallGemmArgs p, int batch, int sms, cudaStream_t s);

}  // namespace lb
