// Elementwise passes of a transformer block over the joint [text, video] sequence.
//
//   ln_modulate   x_out = LayerNorm(x) * weight' + bias' of both streams, written side by side: what the block ran as a
//                 layer norm, a product, a sum and a concatenation, each over the whole activation
//   gate_add      x += gate * a for both streams, a being the joint tensor: a product and a sum over slices
//
// Bound by HBM: each activation value is read once and written once (bf16).  In ln_modulate a warp owns a row (16 bytes
// per lane and access, all of a row's loads in flight together, the reductions in shuffles), which holds rows of up to
// 3072 values in registers; wider models keep the separate passes.  The row-independent factors weight * (1 + scale) and
// bias * (1 + scale) + shift of a sequence are formed once per CTA in shared memory (fp32) and serve all its rows.
// Measured at 2 x 17776 tokens x 3072, L2 flushed before each launch: ln_modulate 104 us (437 MB, 4.2 TB/s), gate_add 113 us
// (655 MB, 5.8 TB/s); the chains they replace took about 400 and 250 us.  At 11 and 12 pieces per lane ln_modulate takes 130
// registers, so that one CTA fits an SM, with 8 of its 64 warps: what holds it below gate_add's rate.
#include "norm_mod.cuh"

#include "ptx_sm100.cuh"

namespace dtb {

namespace {

constexpr int kWarps = 8;

__device__ __forceinline__ void unpack8(uint4 v, float (&x)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[2 * i] = __uint_as_float(w[i] << 16);
    x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint4 pack8(const float (&x)[8]) {
  return make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7]));
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace

// grid: (CTAs per sequence, batch, stream).  kVec = dim / 256.
template <int kVec>
__global__ void __launch_bounds__(kWarps * 32) ln_modulate_kernel(const LnModulateParams p) {
  extern __shared__ float4 s_fac[];              // [dim / 4] factors, then [dim / 4] offsets
  const bool video = blockIdx.z != 0;
  const int b = blockIdx.y;
  const int len = video ? p.video_len : p.text_len;
  const uint16_t* x = (video ? p.video : p.text) + static_cast<int64_t>(b) * len * p.dim;
  uint16_t* out = p.out + (static_cast<int64_t>(b) * (p.text_len + p.video_len) + (video ? p.text_len : 0)) * p.dim;
  const uint16_t* mod = p.mod + b * p.mod_stride + (video ? 0 : 3 * p.dim);      // shift, scale of the stream
  for (int i = threadIdx.x * 8; i < p.dim; i += kWarps * 32 * 8) {
    float w[8], o[8], sh[8], sc[8];
    unpack8(*reinterpret_cast<const uint4*>(p.weight + i), w);
    unpack8(*reinterpret_cast<const uint4*>(p.bias + i), o);
    unpack8(*reinterpret_cast<const uint4*>(mod + i), sh);
    unpack8(*reinterpret_cast<const uint4*>(mod + p.dim + i), sc);
    float* f = reinterpret_cast<float*>(s_fac) + i;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      f[k] = w[k] * (1.f + sc[k]);
      f[p.dim + k] = fmaf(o[k], 1.f + sc[k], sh[k]);
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const float inv = 1.f / p.dim;
  for (int row = blockIdx.x * kWarps + (threadIdx.x >> 5); row < len; row += gridDim.x * kWarps) {
    const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<int64_t>(row) * p.dim) + lane;
    uint4 v[kVec];
#pragma unroll
    for (int i = 0; i < kVec; ++i) v[i] = __ldg(src + i * 32);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      float e[8];
      unpack8(v[i], e);
      sum += ((e[0] + e[1]) + (e[2] + e[3])) + ((e[4] + e[5]) + (e[6] + e[7]));
    }
    const float mean = warp_sum(sum) * inv;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      float e[8];
      unpack8(v[i], e);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float d = e[k] - mean;
        sq = fmaf(d, d, sq);
      }
    }
    const float rstd = rsqrtf(warp_sum(sq) * inv + p.eps);
    uint4* dst = reinterpret_cast<uint4*>(out + static_cast<int64_t>(row) * p.dim) + lane;
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      float e[8];
      unpack8(v[i], e);
      const int c = (i * 32 + lane) * 2;
      const float4 f0 = s_fac[c], f1 = s_fac[c + 1], o0 = s_fac[p.dim / 4 + c], o1 = s_fac[p.dim / 4 + c + 1];
      e[0] = fmaf((e[0] - mean) * rstd, f0.x, o0.x);
      e[1] = fmaf((e[1] - mean) * rstd, f0.y, o0.y);
      e[2] = fmaf((e[2] - mean) * rstd, f0.z, o0.z);
      e[3] = fmaf((e[3] - mean) * rstd, f0.w, o0.w);
      e[4] = fmaf((e[4] - mean) * rstd, f1.x, o1.x);
      e[5] = fmaf((e[5] - mean) * rstd, f1.y, o1.y);
      e[6] = fmaf((e[6] - mean) * rstd, f1.z, o1.z);
      e[7] = fmaf((e[7] - mean) * rstd, f1.w, o1.w);
      dst[i * 32] = pack8(e);
    }
  }
}

// grid: (CTAs, batch, stream); one 16-byte piece per thread and step.
__global__ void __launch_bounds__(256) gate_add_kernel(const GateAddParams p) {
  const bool video = blockIdx.z != 0;
  const int b = blockIdx.y;
  const int len = video ? p.video_len : p.text_len;
  const int vecs = p.dim / 8;
  const uint4* x = reinterpret_cast<const uint4*>(video ? p.video : p.text) + static_cast<int64_t>(b) * len * vecs;
  uint4* out = reinterpret_cast<uint4*>(video ? p.video_out : p.text_out) + static_cast<int64_t>(b) * len * vecs;
  const uint4* a = reinterpret_cast<const uint4*>(p.a) +
                   (static_cast<int64_t>(b) * (p.text_len + p.video_len) + (video ? p.text_len : 0)) * vecs;
  const uint4* gate = reinterpret_cast<const uint4*>(p.mod + b * p.mod_stride + (video ? 2 : 5) * p.dim);
  const int64_t total = static_cast<int64_t>(len) * vecs;
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < total; i0 += 4 * step) {
    uint4 xv[4], av[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + u * step < total) {
        xv[u] = __ldcs(x + i0 + u * step);
        av[u] = __ldcs(a + i0 + u * step);
      }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t i = i0 + u * step;
      if (i < total) {
        float e[8], f[8], g[8];
        unpack8(xv[u], e);
        unpack8(av[u], f);
        unpack8(__ldg(gate + static_cast<int>(i % vecs)), g);
#pragma unroll
        for (int k = 0; k < 8; ++k) e[k] = fmaf(g[k], f[k], e[k]);
        out[i] = pack8(e);
      }
    }
  }
}

template <int kVec>
static cudaError_t launch_ln(const LnModulateParams& p, dim3 grid, cudaStream_t stream) {
  ln_modulate_kernel<kVec><<<grid, kWarps * 32, static_cast<size_t>(p.dim) * 8, stream>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_ln_modulate(const LnModulateParams& p, int batch, int sm_count, cudaStream_t stream) {
  // about four CTAs per SM in all per stream, so that the factors are formed rarely next to the rows they serve (how many
  // of them run at a time is up to the registers: one at 11 and 12 pieces per lane)
  const int longest = p.text_len > p.video_len ? p.text_len : p.video_len;
  const int cap = (4 * sm_count + batch - 1) / batch;
  const int need = (longest + kWarps - 1) / kWarps;
  const dim3 grid(need < cap ? need : cap, batch, 2);
  switch (p.dim / 256) {
    case 1: return launch_ln<1>(p, grid, stream);
    case 2: return launch_ln<2>(p, grid, stream);
    case 3: return launch_ln<3>(p, grid, stream);
    case 4: return launch_ln<4>(p, grid, stream);
    case 5: return launch_ln<5>(p, grid, stream);
    case 6: return launch_ln<6>(p, grid, stream);
    case 7: return launch_ln<7>(p, grid, stream);
    case 8: return launch_ln<8>(p, grid, stream);
    case 9: return launch_ln<9>(p, grid, stream);
    case 10: return launch_ln<10>(p, grid, stream);
    case 11: return launch_ln<11>(p, grid, stream);
    case 12: return launch_ln<12>(p, grid, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_gate_add(const GateAddParams& p, int batch, int sm_count, cudaStream_t stream) {
  const int64_t longest = static_cast<int64_t>(p.text_len > p.video_len ? p.text_len : p.video_len) * (p.dim / 8);
  const int64_t need = (longest + 1023) / 1024, cap = (8ll * sm_count + batch - 1) / batch;
  const dim3 grid(static_cast<unsigned>(need < cap ? need : cap), batch, 2);
  gate_add_kernel<<<grid, 256, 0, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace dtb
