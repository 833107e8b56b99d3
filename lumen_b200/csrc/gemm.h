// What the tensor-core and the CUDA-core GEMM share.
#pragma once
#include "device.h"

namespace lb {

// EPI_ADD: out = round(round(acc) + aux); EPI_MASK: out = aux > 0 ? round(acc) : 0 - each exactly the two primitives
// of the traced program (a rounded product followed by an add / a select), with `aux` a tensor shaped like the output
enum Epilogue : int { EPI_NONE = 0, EPI_RELU = 1, EPI_ADD = 2, EPI_MASK = 3 };

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

}  // namespace lb
