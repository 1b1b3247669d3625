// Parameters and launcher of the query / key norm + rotary kernel (norm_rope.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace dtb {

struct NormRopeParams {
  const uint16_t* src[2];        // query and key projections, [tokens, num_heads, D] bf16
  uint16_t* dst[2];
  const uint16_t* weight[2];     // [D] bf16
  const uint16_t* bias[2];
  const float* cos;              // [seq - text_len, D] fp32
  const float* sin;
  float eps[2];
  int64_t tokens;                // batch * seq
  int seq;
  int text_len;                  // the first text_len tokens of a sequence are normalised only
  int num_heads;
};

cudaError_t launch_norm_rope(const NormRopeParams& p, int head_dim, int sm_count, cudaStream_t stream);

}  // namespace dtb
