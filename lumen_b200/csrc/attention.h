// What the files of the attention forward share.
#pragma once
#include "device.h"

namespace lb {

// The kernels behind lb_attention_fwd (its codes are those of lb_attention_fwd_kernel).
enum AttentionKernel { ATTN_CUDA_CORES = 0, ATTN_ONE_TILE = 1, ATTN_TWO_TILES = 2, ATTN_FEW_ROWS = 3 };

// Few query rows per key head (attention_decode.cu): whether that kernel takes the problem at all, and the microseconds a
// B200 takes for it. Operands are as the tensor-core kernels need them.
bool attention_decodes(const lb_tensor& q, const lb_tensor& k);
double attention_decode_us(const lb_tensor& q, const lb_tensor& k, int sms);
void attention_decode(const lb_attn_desc& desc, const lb_tensor& q, const lb_tensor& k, const lb_tensor& v, const lb_tensor& o,
                      const lb_tensor* lse, void* stream);

}  // namespace lb
