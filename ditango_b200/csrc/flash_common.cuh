// Pieces of the partial-attention forward kernels (flash_fwd_sm100.cu, flash_fwd_persistent_sm100.cu) that are not their schedule:
// tile geometry, the bounded barrier waits, the status word, packed fp32 arithmetic, the two exponentials, the lse layouts, the
// epilogue.
#pragma once
#include "flash_fwd_sm100.cuh"
#include "ptx_sm100.cuh"

#include <math.h>

namespace dtb {
namespace flash {

constexpr int kBM = 128;                  // query rows per tile
constexpr int kQT = 2;                    // query tiles per CTA
constexpr int kBN = 128;                  // key rows per tile
constexpr int kSlabBytes = 128 * 128;     // one TMA box: 128 rows x 64 bf16, 128-byte swizzled
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleThreshold = 8.0f; // log2 units: the running reference follows the maximum this lazily

__device__ __forceinline__ void report(int* status, int code) { atomicCAS(status, 0, code); }

// Bounded wait that also gives up as soon as any CTA has reported a failure.  The clock is read right after the first
// failed attempt and not only when it is needed: the pause keeps the waiting warps out of the softmax warps' issue slots
// (reading it only after 64 attempts: 119056 tokens at D = 128 150.3 ms against 142.7, a four-chunk ring of 7201 3 % slower,
// 2 x 17776 tokens at D = 64 1.7 %; a suspended try_wait or nanosleep in the loop was slower than this too, by up to 6 %).
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, int* status, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (((++spins) & 0xff) == 0) {
      if (*reinterpret_cast<volatile int*>(status) != 0) return false;
      if (globaltimer_ns() - t0 > 1000000000ull) {
        report(status, code);
        return false;
      }
    }
  }
  return true;
}

// The same by a whole warp: all of its lanes go on or all of them give up.  (Waiting each for itself, lanes of one warp can see the
// phase, the status word and the limit at different moments; those that went on would then wait without a limit, at the next
// operation of the whole warp, for those that had left.)  wait_or_abort is for a single thread.
// The vote costs up to 0.5 % with a CTA per block at D = 64 (74 heads x 512 x 8192: 106.0 -> 106.6 us) and nothing measurable at
// D = 128.  Asked as "any that failed", as here, the first attempt goes on faster than as "all that passed" (108.7 us there); a vote
// further down the tile, under the loads of the scores or with that on the rescale, 107.6 and 106.6 us, and 1.2 and 0.1 % at D = 128.
__device__ __forceinline__ bool warp_wait_or_abort(uint64_t* bar, uint32_t parity, int* status, int code) {
  if (!__any_sync(0xffffffffu, !mbar_try_wait(bar, parity))) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
    if (((++spins) & 0xff) == 0) {
      const bool late = globaltimer_ns() - t0 > 1000000000ull;
      if (late) report(status, code);
      if (__any_sync(0xffffffffu, late || *reinterpret_cast<volatile int*>(status) != 0)) return false;
    }
  }
  return true;
}

// ---------------------------------------------------------------------------- packed fp32 pairs
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// 2^x for a pair of exponents, on the ex2 unit ...
__device__ __forceinline__ uint64_t exp2_mufu2(uint64_t x) {
  float x0, x1;
  unpack2(x, x0, x1);
  return pack2(ex2(x0), ex2(x1));
}

// ... and on the FMA units, for x <= 127: x = n + f with n = round(x), 2^f on [-1/2, 1/2] by a degree-5 polynomial
// (p(0) = 1, weighted least squares iterated to equal ripple; with these coefficients the largest relative error is
// 1.1e-7, and 1.7e-7 as evaluated here in fp32), 2^n by
// placing n + 127 in the exponent field.  Below -127 the result is 0; a NaN stays a NaN.
__device__ __forceinline__ uint64_t exp2_poly2(uint64_t x) {
  float x0, x1;
  unpack2(x, x0, x1);
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x0) : "f"(-127.f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x1) : "f"(-127.f));
  x = pack2(x0, x1);
  constexpr float kMagic = 12582912.f + 127.f;       // 1.5 * 2^23: the sum's low bits hold n + 127
  const uint64_t t = add2(x, pack2(kMagic, kMagic));
  const uint64_t n = add2(t, pack2(-kMagic, -kMagic));
  const uint64_t f = fma2(n, pack2(-1.f, -1.f), x);
  uint64_t h = fma2(f, pack2(1.32646751e-3f, 1.32646751e-3f), pack2(9.67151e-3f, 9.67151e-3f));
  h = fma2(h, f, pack2(5.550734e-2f, 5.550734e-2f));
  h = fma2(h, f, pack2(2.4022242e-1f, 2.4022242e-1f));
  h = fma2(h, f, pack2(6.9314698e-1f, 6.9314698e-1f));
  h = fma2(h, f, pack2(1.f, 1.f));
  float t0, t1;
  unpack2(t, t0, t1);
  const uint64_t scale = pack2(__uint_as_float(__float_as_uint(t0) << 23), __uint_as_float(__float_as_uint(t1) << 23));
  return mul2(h, scale);
}

__device__ __forceinline__ int64_t lse_index(const FlashParams& p, int seg, int head, int q_pos, int64_t tok) {
  if (p.lse_layout == 1) return tok * p.num_heads + head;                        // [B,S,H]
  if (p.cu_q != nullptr) return static_cast<int64_t>(head) * p.total_q + tok;    // [H,T]
  return (static_cast<int64_t>(seg) * p.num_heads + head) * p.seqlen_q + q_pos;  // [B,H,S]
}

// A row of a (segment, head) that has no keys at all: an empty state (out = 0, lse = -inf).  Not for a launch that folds into a
// state (callers see to that): merging an empty state changes nothing.
template <int D>
__device__ __forceinline__ void write_empty_row(const FlashParams& p, int seg, int head, int q_begin, int q_len, int q_pos) {
  if (q_pos >= q_len) return;
  const int64_t tok = static_cast<int64_t>(q_begin) + q_pos;
  p.lse[lse_index(p, seg, head, q_pos, tok)] = -INFINITY;
  if (p.out_dtype == 0) {
    float4* o = reinterpret_cast<float4*>(static_cast<float*>(p.out) + tok * p.out_tok_stride + head * D);
    for (int c = 0; c < D / 4; ++c) o[c] = make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    uint4* o = reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.out) + tok * p.out_tok_stride + head * D);
    for (int c = 0; c < D / 8; ++c) o[c] = make_uint4(0u, 0u, 0u, 0u);
  }
}
// ... for a CTA's 256 query rows, by its first 256 threads.
template <int D>
__device__ __forceinline__ void write_empty_rows(const FlashParams& p, int seg, int head, int q_begin, int q_len, int q0) {
  if (p.accumulate || threadIdx.x >= kQT * kBM) return;
  grid_dependency_wait();      // the launch before this one may still be writing the same buffers
  write_empty_row<D>(p, seg, head, q_begin, q_len, q0 + static_cast<int>(threadIdx.x));
}

// The state in global memory that 32 consecutive columns of a warp's 32 output rows are merged with: lane i holds 16 bytes
// of each of the rows i / 8, i / 8 + 4, ... (see store_rows32).  Read whatever its weight turns out to be, so that the loads do
// not queue behind that of the lse; a state of weight 0 is not used.  (Reads behind the weight -> as here, a launch with
// a CTA per block folded into a state, overlapping the one before: 1024 x 24 x 128 20.9 -> 20.5 us, 2 x 1111 x 24 x 128 44.7 -> 44.0,
// 2 x 2222 x 48 x 64 192.7 -> 191.9.)
struct OldRows {
  float4 v[8];
};
__device__ __forceinline__ void load_old_rows32(const FlashParams& p, int64_t tok0, int rows, int64_t col, OldRows& old) {
  const int lane = threadIdx.x & 31;
  const int r0 = lane >> 3, piece = lane & 7;
  const float* src = static_cast<const float*>(p.out) + (tok0 + r0) * p.out_tok_stride + col + piece * 4;
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    old.v[it] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (it * 4 + r0 < rows) old.v[it] = *reinterpret_cast<const float4*>(src + it * 4 * p.out_tok_stride);
  }
}

// Final step for 32 consecutive columns of a warp's 32 output rows, executed by the whole warp: lane i holds row i
// (un-normalised fp32 accumulators `acc`) and its weights.  Scale by w_new, blend with the state already in global memory
// when accumulating (`old`, used where w_old != 0), store as fp32 or bf16.  `tok0` is the token of the warp's first row, `rows` how
// many of its rows exist, `col` the element offset of the columns inside a token; `stage` is 4 KB of shared memory of the warp.
//
// The rows go through shared memory so that 8 lanes write (and read) the 128 contiguous bytes of a row: a lane that
// stores its own row touches 32 cache lines per warp instruction, half a sector of each, and the load / store unit then
// spends a clock per line (32 x 16 instructions x 8 warps for 256 rows of 64 columns, twice that with a state to read).
// CogVideoX ring on rank 3 of 8 3.91 -> 3.70 ms, its whole sequence 9.65 -> 9.41 ms.  The 16-byte pieces are XOR-swizzled
// by row, so that neither side has bank conflicts.
__device__ __forceinline__ void store_rows32(const FlashParams& p, uint8_t* stage, int64_t tok0, int rows, int64_t col,
                                             const uint32_t (&acc)[32], const OldRows& old, float w_new, float w_old) {
  const int lane = threadIdx.x & 31;
  const bool f32 = p.out_dtype == 0;
  const int r0 = lane >> 3, piece = lane & 7;
  float* dst = static_cast<float*>(p.out) + (tok0 + r0) * p.out_tok_stride + col + piece * 4;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    *reinterpret_cast<float4*>(stage + lane * 128 + ((i ^ (lane & 7)) << 4)) =
        make_float4(__uint_as_float(acc[4 * i]) * w_new, __uint_as_float(acc[4 * i + 1]) * w_new,
                    __uint_as_float(acc[4 * i + 2]) * w_new, __uint_as_float(acc[4 * i + 3]) * w_new);
  __syncwarp();
  auto staged = [&](int r, int i) { return *reinterpret_cast<const float4*>(stage + r * 128 + ((i ^ (r & 7)) << 4)); };
  if (f32) {
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const int r = it * 4 + r0;
      float4 v = staged(r, piece);
      if (p.accumulate) {
        const float wo = __shfl_sync(0xffffffffu, w_old, r);
        if (wo != 0.f) {
          v.x = fmaf(old.v[it].x, wo, v.x);
          v.y = fmaf(old.v[it].y, wo, v.y);
          v.z = fmaf(old.v[it].z, wo, v.z);
          v.w = fmaf(old.v[it].w, wo, v.w);
        }
      }
      if (r < rows) *reinterpret_cast<float4*>(dst + it * 4 * p.out_tok_stride) = v;
    }
  } else {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int r = it * 8 + (lane >> 2), i = (lane & 3) * 2;
      const float4 a = staged(r, i), b = staged(r, i + 1);
      if (r < rows)
        *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.out) + (tok0 + r) * p.out_tok_stride + col + i * 4) =
            make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
    }
  }
  __syncwarp();        // the stage is written again for the next columns
}

// Weights of the final normalisation: a row whose un-normalised accumulator has row sum l_row and log-sum-exp
// lse_new is either written as is (w_new = 1 / l_row) or merged with the state (lse_old) already in memory.
__device__ __forceinline__ void merge_weights(bool accumulate, float lse_old, float lse_new, float l_row, float& w_new,
                                              float& w_old, float& lse_out) {
  w_new = 1.f / l_row;
  w_old = 0.f;
  lse_out = lse_new;
  if (accumulate && lse_old != -INFINITY) {
    const float mx = fmaxf(lse_old, lse_new);
    const float e_old = __expf(lse_old - mx), e_new = __expf(lse_new - mx);
    const float tot = e_old + e_new;
    lse_out = mx + __logf(tot);
    w_old = e_old / tot;
    w_new = (e_new / tot) / l_row;
  }
}

// Host: one launch of an attention kernel, with the programmatic-stream-serialization attribute when the caller
// allows the launch to overlap the end of the one before it.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_attention_kernel(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem_bytes,
                                           cudaStream_t stream, bool overlap_previous, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap_previous ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Args&&>(args)...);
}

}  // namespace flash

}  // namespace dtb
