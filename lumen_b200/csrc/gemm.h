// What the GEMM kernels' files share.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "device.h"

namespace lb {

// EPI_ADD: out = round(round(acc) + aux); EPI_MASK: out = aux > 0 ? round(acc) : 0 - each exactly the two primitives
// of the traced program (a rounded product followed by an add / a select), with `aux` a tensor shaped like the output
enum Epilogue : int { EPI_PARTIAL = -1 /* of a kernel: sums of a range of K */, EPI_NONE = 0, EPI_RELU = 1, EPI_ADD = 2, EPI_MASK = 3 };
#ifdef __CUDACC__
__host__ __device__ constexpr bool reads_aux(int epilogue) { return epilogue >= EPI_ADD; }
// The second primitive on the rounded product.
__device__ __forceinline__ float second_primitive(int epilogue, float product, float other) {
    return epilogue == EPI_ADD ? __fadd_rn(other, product) : (other > 0.0f ? product : 0.0f);
}
// A 16-bit element's bits from and to float32.
template <int DT>
__device__ __forceinline__ uint16_t to16(float x) {
    return DT == LB_BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(x)) : __half_as_ushort(__float2half_rn(x));
}
template <int DT>
__device__ __forceinline__ float from16(uint16_t x) {
    return DT == LB_BF16 ? __uint_as_float((uint32_t)x << 16) : __half2float(__ushort_as_half(x));
}
template <int DT>
__device__ __forceinline__ uint32_t pair16(float lo, float hi) {
    if constexpr (DT == LB_BF16) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *(const uint32_t*)&h;
    } else {
        const __half2 h = __floats2half2_rn(lo, hi);
        return *(const uint32_t*)&h;
    }
}

// Calls `launch` with the kernel's epilogue and type of the result as constants.
template <class Launch>
void with_epilogue(int epilogue, int dtype, Launch launch) {
    auto go = [&](auto dt) {
        switch (epilogue) {
            case EPI_NONE: return launch(std::integral_constant<int, EPI_NONE>{}, dt);
            case EPI_RELU: return launch(std::integral_constant<int, EPI_RELU>{}, dt);
        }
        if constexpr (decltype(dt)::value != LB_F32) {
            switch (epilogue) {
                case EPI_ADD: return launch(std::integral_constant<int, EPI_ADD>{}, dt);
                case EPI_MASK: return launch(std::integral_constant<int, EPI_MASK>{}, dt);
            }
        }
        fail(LB_ERR_INVALID, "gemm: unknown epilogue");
    };
    if (dtype == LB_BF16) go(std::integral_constant<int, LB_BF16>{});
    else if (dtype == LB_F16) go(std::integral_constant<int, LB_F16>{});
    else go(std::integral_constant<int, LB_F32>{});
}
#endif

// The CUDA-core GEMM (gemm_simt.cu): any strides, element strides of the M, N and K axes.
struct SimtArgs {
    int M, N, K, batch;
    long long a_sm, a_sk, a_sb, b_sk, b_sn, b_sb, ldd, d_sb;
    void* d;
    int d_dtype;
    int epilogue;
    const void* aux;  // EPI_ADD / EPI_MASK operand (16-bit, the output's dtype), rows ld_aux apart, batches aux_sb apart
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
    int tiles_m, tiles_n, whole;  // set by gemm_small
};

void gemm_small(const CUtensorMap& map_a, const CUtensorMap& map_b, SmallGemmArgs p, int batch, int sms, cudaStream_t s);

}  // namespace lb
