// N-way merge of partial softmax-attention states in one pass over HBM.
//
// A "row" is one (token, head) pair: D values per state plus one log-sum-exp per state.  A group of
// D/8 lanes owns a row (8 values per lane: two 128-bit accesses in fp32, one in bf16); lane i of the
// group fetches lse_i (and lse_{i + D/8}), the group reduces max and sum with shuffles, and every lane
// then pulls the weight of state i from the lane that holds it.
// Traffic per row: reads sum_i (D * sizeof(state i) + 4) bytes, writes 4*D + 4 (+ 2*D) bytes.
//
// A state is kept as loaded (raw bits) until its weight is known.  Its type is only known at run time, so the
// fp32 and the bf16 load sit in different branches; converting there would make each branch wait for its own load,
// and the loads of several states would queue behind one another instead of being in flight together (4 values per lane
// with the conversion at the load: fp32 + bf16 at 14882 x 24 x 128 141 us, seven bf16 states and one fp32 into a bf16 result
// at 2 x 6851 x 48 x 128 726 us; as it stands 81 us and 306 us; L2 flushed before each launch).
#include "merge_states.cuh"

#include <math.h>

namespace dtb {

namespace {

// 8 consecutive values of one state: fp32 in a and b, or bf16 in a.
struct Raw8 {
  uint4 a, b;
};

__device__ __forceinline__ uint4 ld_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void st_stream(void* p, uint4 v) {
  asm volatile("st.global.cs.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint4 as_bits(const float* v) {
  return make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
}
// acc += w * state
__device__ __forceinline__ void add_weighted(float (&acc)[8], float w, const Raw8& r, bool f32) {
  const uint32_t a[4] = {r.a.x, r.a.y, r.a.z, r.a.w}, b[4] = {r.b.x, r.b.y, r.b.z, r.b.w};
  if (f32) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[i] = fmaf(w, __uint_as_float(a[i]), acc[i]);
      acc[4 + i] = fmaf(w, __uint_as_float(b[i]), acc[4 + i]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[2 * i] = fmaf(w, __uint_as_float(a[i] << 16), acc[2 * i]);
      acc[2 * i + 1] = fmaf(w, __uint_as_float(a[i] & 0xffff0000u), acc[2 * i + 1]);
    }
  }
}

// Offset of row = (b*S + s)*H + h in an lse tensor.  Rows fit 32 bits (checked by the launcher), so
// the two divisions are 32-bit.
__device__ __forceinline__ uint32_t lse_offset(int layout, uint32_t row, uint32_t H, uint32_t S) {
  if (layout == 1) return row;                    // [B,S,H]
  const uint32_t tok = row / H;
  const uint32_t h = row - tok * H;
  const uint32_t b = tok / S;
  const uint32_t s = tok - b * S;
  return (b * H + h) * S + s;                     // [B,H,S]
}

}  // namespace

// G = lanes per row = D/8.  U rows per group in flight, states fetched CH at a time: every thread
// has the loads of CH*U row pieces outstanding and issues them before it touches the weights, so the lse
// round trip and the value round trips overlap instead of queueing behind one another.
template <int G, int U, int CH>
__global__ void __launch_bounds__(128) merge_states_kernel(const MergeParams p) {
  constexpr int D = G * 8;
  constexpr int kGroupsPerWarp = 32 / G;
  constexpr int kPerLane = kMergeMaxStates / G;        // states whose lse a lane holds: lane, lane + G
  const int lane_in_group = threadIdx.x % G;
  const int64_t warp_id = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / 32;
  const int64_t n_warps = static_cast<int64_t>(gridDim.x) * blockDim.x / 32;
  const int group_in_warp = (threadIdx.x % 32) / G;
  const unsigned full = 0xffffffffu;
  const int n = p.nstates;

  auto load_chunk = [&](int c0, int64_t base, Raw8 (&v)[CH][U]) {
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      if (c0 + k < n) {
        if (p.out_dtype[c0 + k] == 0) {
          const float* src = static_cast<const float*>(p.outs[c0 + k]) + lane_in_group * 8;
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (base + u < p.rows) {
              v[k][u].a = ld_stream(src + (base + u) * D);
              v[k][u].b = ld_stream(src + (base + u) * D + 4);
            }
        } else {
          const uint16_t* src = static_cast<const uint16_t*>(p.outs[c0 + k]) + lane_in_group * 8;
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (base + u < p.rows) v[k][u].a = ld_stream(src + (base + u) * D);
        }
      }
    }
  };

  // The loop bound is the same for every lane of a warp (shuffles below use the full mask); rows
  // past the end are guarded individually.
  for (int64_t wbase = warp_id * kGroupsPerWarp * U; wbase < p.rows; wbase += n_warps * kGroupsPerWarp * U) {
    const int64_t base = wbase + group_in_warp * U;
    float my[U][kPerLane];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int t = 0; t < kPerLane; ++t) {
        const int st = lane_in_group + t * G;
        my[u][t] = -INFINITY;
        if (base + u < p.rows && st < n)
          my[u][t] = p.lse[st][lse_offset(p.lse_layout[st], static_cast<uint32_t>(base + u), p.H, p.S)];
      }
    Raw8 v[CH][U];
#pragma unroll
    for (int k = 0; k < CH; ++k)
#pragma unroll
      for (int u = 0; u < U; ++u) v[k][u].a = v[k][u].b = make_uint4(0u, 0u, 0u, 0u);
    load_chunk(0, base, v);

    float w[U][kPerLane];        // weights of the states this lane holds the lse of
    float lse_out[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float mx = my[u][0];
#pragma unroll
      for (int t = 1; t < kPerLane; ++t) mx = fmaxf(mx, my[u][t]);
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(full, mx, o, G));
      float e[kPerLane], sum = 0.f;
#pragma unroll
      for (int t = 0; t < kPerLane; ++t) {
        e[t] = (my[u][t] == -INFINITY) ? 0.f : __expf(my[u][t] - mx);
        sum += e[t];
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(full, sum, o, G);
#pragma unroll
      for (int t = 0; t < kPerLane; ++t) w[u][t] = (sum > 0.f) ? e[t] / sum : 0.f;
      lse_out[u] = (sum > 0.f) ? mx + __logf(sum) : -INFINITY;
    }
    float acc[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[u][i] = 0.f;
    for (int c0 = 0; c0 < n; c0 += CH) {
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        const int st = c0 + k;
        if (st < n) {
          const bool f32 = p.out_dtype[st] == 0;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const float mine = (kPerLane == 1 || st < G) ? w[u][0] : w[u][kPerLane - 1];
            const float wi = __shfl_sync(full, mine, st % G, G);
            // a state with weight 0 may hold anything (even inf/nan): it must not reach the sum
            if (wi != 0.f) add_weighted(acc[u], wi, v[k][u], f32);
          }
        }
      }
      if (c0 + CH < n) load_chunk(c0 + CH, base, v);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t row = base + u;
      if (row < p.rows) {
        const int64_t off = row * D + lane_in_group * 8;
        if (p.out != nullptr) {
          st_stream(p.out + off, as_bits(acc[u]));
          st_stream(p.out + off + 4, as_bits(acc[u] + 4));
        }
        if (p.out_bf16 != nullptr)
          st_stream(p.out_bf16 + off, make_uint4(pack_bf16(acc[u][0], acc[u][1]), pack_bf16(acc[u][2], acc[u][3]),
                                                 pack_bf16(acc[u][4], acc[u][5]), pack_bf16(acc[u][6], acc[u][7])));
        if (p.lse_out != nullptr && lane_in_group == 0)
          p.lse_out[lse_offset(p.lse_out_layout, static_cast<uint32_t>(row), p.H, p.S)] = lse_out[u];
      }
    }
  }
}

template <int U, int CH>
static cudaError_t launch_merge_cfg(const MergeParams& p, int G, int sm_count, cudaStream_t stream) {
  constexpr int kThreads = 128;
  const int64_t groups_needed = (p.rows + U - 1) / U;
  const int64_t blocks_needed = (groups_needed * G + kThreads - 1) / kThreads + 1;
  // one resident wave: CTAs per SM as the occupancy calculator reports them for this instantiation
  int per_sm = 0;
  cudaError_t oe = (G == 8)
      ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, merge_states_kernel<8, U, CH>, kThreads, 0)
      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, merge_states_kernel<16, U, CH>, kThreads, 0);
  if (oe != cudaSuccess || per_sm < 1) per_sm = 6;
  const int64_t cap = static_cast<int64_t>(sm_count) * per_sm;
  int blocks = static_cast<int>(blocks_needed < cap ? blocks_needed : cap);
  if (blocks < 1) blocks = 1;
  if (G == 8)
    merge_states_kernel<8, U, CH><<<blocks, kThreads, 0, stream>>>(p);
  else
    merge_states_kernel<16, U, CH><<<blocks, kThreads, 0, stream>>>(p);
  return cudaGetLastError();
}

// Rows per thread x states per fetch are chosen so that eight or nine row pieces are outstanding per thread whatever the
// number of states: 4 rows x 2 states, 3 x 3, or 2 x 4 (a piece is one 16-byte load in bf16 and two in fp32).  The registers
// that takes (128) leave four CTAs per SM.
cudaError_t launch_merge(const MergeParams& p, int head_dim, int sm_count, cudaStream_t stream) {
  const int G = head_dim / 8;
  if (p.rows >= (1ll << 31)) return cudaErrorInvalidValue;
#ifndef DTB_MERGE_FIXED_CFG
  if (p.nstates <= 2) return launch_merge_cfg<4, 2>(p, G, sm_count, stream);
  if (p.nstates == 3) return launch_merge_cfg<3, 3>(p, G, sm_count, stream);
#endif
  return launch_merge_cfg<2, 4>(p, G, sm_count, stream);
}

// ------------------------------------------------------------------------------------------------
// Strided chunk copy (head <-> sequence re-layouts around the Ulysses all-to-all).
// The 16-byte vectors of all chunks are numbered through; a thread copies Unroll of them, a block apart, whose loads are all in
// flight before the first store (one for small copies: see launch_copy_chunks).  Bound by HBM once the index arithmetic is out of the way: Index is 32 bits where the vectors can
// be counted in it, since three 64-bit divisions per vector, with one load in flight per thread, took longer than the copy.  The
// stores are ordinary ones: what reads the result (the exchange, the attention kernel) comes next and finds part of it in L2.
// us (bytes moved per time), L2 flushed before each launch: the re-layouts of a CogVideoX Ulysses call of one rank of 8, 164 MB
// 38.9 (4.2 TB/s) -> 32.8 (5.0) and 55 MB 18.5 (3.0) -> 16.4 (3.3); 437 MB 88.1 (5.0) -> 73.7 (5.9).
constexpr int kCopyThreads = 256;
constexpr int kCopyUnroll = 4;

template <typename Index, int Unroll>
__global__ void __launch_bounds__(kCopyThreads) copy_chunks_kernel(const CopyParams p) {
  const int pair = blockIdx.y;
  const uint8_t* src = static_cast<const uint8_t*>(p.src[pair]);
  uint8_t* dst = static_cast<uint8_t*>(p.dst[pair]);
  const Index vec_per_chunk = static_cast<Index>(p.chunk_bytes >> 4);
  const Index n1 = static_cast<Index>(p.n1), n2 = static_cast<Index>(p.n2);
  const Index total = static_cast<Index>(p.n0) * n1 * n2 * vec_per_chunk;
  constexpr Index kTile = kCopyThreads * Unroll;
  for (Index tile = static_cast<Index>(blockIdx.x); tile < (total + (kTile - 1)) / kTile; tile += gridDim.x) {
    uint4 val[Unroll];
    uint8_t* to[Unroll];
#pragma unroll
    for (int u = 0; u < Unroll; ++u) {
      const Index i = tile * kTile + static_cast<Index>(u * kCopyThreads + threadIdx.x);
      to[u] = nullptr;
      if (i < total) {
        const Index chunk = i / vec_per_chunk;
        const Index v = i - chunk * vec_per_chunk;
        const Index t = chunk / n2;
        const Index i2 = chunk - t * n2;
        const Index i0 = t / n1;
        const Index i1 = t - i0 * n1;
        val[u] = ld_stream(src + static_cast<int64_t>(i0) * p.ss0 + static_cast<int64_t>(i1) * p.ss1 + static_cast<int64_t>(i2) * p.ss2 + static_cast<int64_t>(v) * 16);
        to[u] = dst + static_cast<int64_t>(i0) * p.ds0 + static_cast<int64_t>(i1) * p.ds1 + static_cast<int64_t>(i2) * p.ds2 + static_cast<int64_t>(v) * 16;
      }
    }
#pragma unroll
    for (int u = 0; u < Unroll; ++u)
      if (to[u] != nullptr) *reinterpret_cast<uint4*>(to[u]) = val[u];
  }
}

template <typename Index, int Unroll>
static cudaError_t launch_copy_chunks_cfg(const CopyParams& p, int npairs, int64_t tiles, cudaStream_t stream) {
  copy_chunks_kernel<Index, Unroll><<<dim3(static_cast<unsigned>(tiles), npairs), kCopyThreads, 0, stream>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_copy_chunks(const CopyParams& p, int npairs, int sm_count, cudaStream_t stream) {
  constexpr int64_t kTile = kCopyThreads * kCopyUnroll;
  const int64_t total = p.n0 * p.n1 * p.n2 * (p.chunk_bytes >> 4);
  // Up to four tiles for every SM, one vector per thread: more warps in flight count for more there.  us per launch, back to back,
  // four vectors -> one: 0.2 MB moved 2.6 -> 1.7, 3.2 MB 2.6 -> 2.0, 5.2 MB 3.2 -> 2.4, 12.6 MB 3.8 -> 3.6, 22.9 MB 4.9 -> 5.3,
  // 54.6 MB 9.0 -> 10.8.
  if (total <= 4 * sm_count * kTile)
    return launch_copy_chunks_cfg<uint32_t, 1>(p, npairs, (total + kCopyThreads - 1) / kCopyThreads, stream);
  const int64_t tiles = (total + kTile - 1) / kTile;
  const int64_t cap = static_cast<int64_t>(sm_count) * 64;
  const int64_t grid = tiles < cap ? tiles : cap;
  // (a thread's index goes one grid past the last vector before it stops)
  if (total + cap * kTile < (1ll << 31)) return launch_copy_chunks_cfg<uint32_t, kCopyUnroll>(p, npairs, grid, stream);
  return launch_copy_chunks_cfg<uint64_t, kCopyUnroll>(p, npairs, grid, stream);
}

}  // namespace dtb
