// Parameters and launchers of the transformer block's elementwise kernels (norm_mod.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace dtb {

constexpr int kModMaxDim = 3072;     // a row is held in registers: 12 x 16 bytes per lane

// `mod` is the [batch, 6 dim] bf16 modulation (shift, scale, gate of the video stream, then of the text stream), rows
// mod_stride elements apart.
struct LnModulateParams {
  const uint16_t* video;             // [batch, video_len, dim] bf16
  const uint16_t* text;              // [batch, text_len, dim]
  const uint16_t* weight;            // [dim]
  const uint16_t* bias;
  const uint16_t* mod;
  uint16_t* out;                     // [batch, text_len + video_len, dim], text first
  int64_t mod_stride;
  float eps;
  int video_len, text_len, dim;
};

struct GateAddParams {
  const uint16_t* video;
  const uint16_t* text;
  const uint16_t* a;                 // [batch, text_len + video_len, dim]
  const uint16_t* mod;
  uint16_t* video_out;
  uint16_t* text_out;
  int64_t mod_stride;
  int video_len, text_len, dim;
};

cudaError_t launch_ln_modulate(const LnModulateParams& p, int batch, int sm_count, cudaStream_t stream);
cudaError_t launch_gate_add(const GateAddParams& p, int batch, int sm_count, cudaStream_t stream);

}  // namespace dtb
