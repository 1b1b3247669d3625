// Partial-attention forward: one thread per query row, key tiles of 128 rows.
//
// CTA = 256 query rows of one (segment, head): two 128-row Q tiles share the tensor core.  Warp roles
// (384 threads, three warpgroups):
//   warps 0-3   softmax group 0: one thread per row of Q tile 0
//   warps 4-7   softmax group 1: one thread per row of Q tile 1
//   warp  8     TMA producer: Q tiles once, then K_j, V_j tiles (128 keys each) through a shared-memory ring
//   warp  9     MMA issuer (one elected thread): S_i = Q_i K_j^T and O_i += P_i V_j via tcgen05.mma
//   warps 10-11 no role; they complete the third warpgroup so that it can hand registers over
// The work is a sequence of units u = 2 j + i (key tile j, Q tile i).  Tensor memory (512 columns x 128 lanes of
// fp32): S buffers of 128 columns at [128 b, 128 b + 128), unit u in buffer u % NB, then the O accumulators of D
// columns each.  NB = 2 at D = 128 (tensor memory is full), 3 at D = 64.  P(u) (bf16) overwrites the first 64
// columns of its S buffer.  S(u + NB) is issued right behind PV(u) (the pipe runs MMAs in issue order, so P is
// read before it is overwritten):
//     S(0) .. S(NB-1) | PV(0) S(NB) | PV(1) S(NB+1) | ...
// P is handed over in two parts, so that PV(u) starts while the rest of the row is still being exponentiated.
//
// Why these sizes.  128 keys per tile and not 64: an S instruction of N = 64 reads as much of Q from shared memory as
// one of N = 128 for half the products (192 bytes per clock wanted, 128 there), so the tensor side alone was the bound
// at D = 128.  One thread per row and 128 scores per thread: the barrier waits, tensor-memory round trips and
// hand-overs of a tile are paid once per 128 scores, and the row maximum needs no exchange.  One pair of scores in
// eight is exponentiated on the FMA units, which takes an eighth of the work off the ex2 unit (16 results per clock and
// SM: 2048 clocks for the 256 x 128 scores of a step, as much as all MMAs of a step at D = 128).  TFLOP/s in short bursts,
// D = 64 / D = 128: none 857 / 1221, one pair of eight 888 / 1255, two 881 / 1226, four 685 / 1058 (the FMA and issue slots
// then being the bound).
//
// Launches at D = 64 with enough blocks go to flash_fwd_persistent_sm100.cu (the rule is in capi.cu), those of the following
// figures among them; they were taken before the waits of whole warps voted (up to 0.5 % at D = 64, nothing at D = 128).
//
// Measured on one B200, SM clocks per step of 128 keys x 256 rows (key loop of every CTA, clock register read in front of it
// and behind it): D = 64 2368, D = 128 2931; in builds with one side left out, the MMAs alone 1280 and 2103, the softmax
// alone 2357 and 2594.  TFLOP/s, with the two kernels of 64-key tiles that this one replaced in brackets, as a burst of
// three launches after a pause and back to back for 2.5 s:
//   D = 64,  2 x 17776 tokens x 48 heads   925 (771) at 1.83 GHz     826 (733) at 1.77 GHz, the board at its power cap
//   D = 128, 14882 tokens x 24 heads      1283 (1198) at 1.65 GHz   1112 (1034) at 1.59 GHz, power cap
//   D = 128, 119056 tokens x 24 heads     1225 (1147) on average    1189 (1116) at 1.54 GHz, power cap
//
// Running max is kept lazily: O is rescaled only when the max grew by more than 2^8, which bounds every
// probability by 2^8 and keeps bf16 P exact enough; the final normalisation undoes it.
#include "flash_common.cuh"

#include <mutex>

namespace dtb {

namespace {

using namespace flash;

constexpr int kThreads = 384;
constexpr int kRegsLaunch = 168;    // what __launch_bounds__(384, 1) allots; checked before the first launch
constexpr int kRegsSoftmax = 208;   // 2 x 128 x (208 - 168) registers taken ...
constexpr int kRegsOther = 88;      // ... are the 128 x (168 - 88) the third warpgroup gives up
static_assert(2 * kRegsSoftmax + kRegsOther == 3 * kRegsLaunch, "register split");
constexpr int kTmaWarp = 8;
constexpr int kMmaWarp = 9;
constexpr int kSplit = 64;          // keys of a tile whose probabilities are handed over first
constexpr int kPolyPairs = 1;       // pairs of every 8 pairs of scores, exponentiated on the FMA units

template <int D>
struct Cfg {
  static constexpr int kSlabs = D / 64;
  static constexpr int kTileBytes = kBM * D * 2;          // one Q tile
  static constexpr int kKvTileBytes = kBN * D * 2;      // one K or V tile
  static constexpr int kStages = (D == 128) ? 5 : 10;
  static constexpr int kSBufs = (512 - kQT * D) / kBN;
  // barriers: q_full[2], kv_full[S], kv_empty[S], s_full[NB], p_lo[NB], p_hi[NB], pv_done[2], o_final[2], v_tail[1]
  static constexpr int kBars = 2 + 2 * kStages + 3 * kSBufs + 2 + 2 + 1;
  static constexpr int kSmemBytes = 1024 + kQT * kTileBytes + kStages * kKvTileBytes + kBars * 8 + 16;
  static constexpr uint32_t kTmemCols = 512;
  static constexpr uint32_t kColS = 0;                    // + buffer * 128
  static constexpr uint32_t kColO = kSBufs * kBN;       // + tile * D
  static_assert(kColO + kQT * D <= 512, "tensor memory");
  static_assert(kSmemBytes <= 232448, "shared memory");
};

}  // namespace

template <int D>
__global__ void __launch_bounds__(kThreads, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const FlashParams p) {
  using C = Cfg<D>;
  constexpr int NB = C::kSBufs;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* s_q = smem;
  uint8_t* s_kv = smem + kQT * C::kTileBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_kv + C::kStages * C::kKvTileBytes);
  uint64_t* q_full = bars;                    // [tile]
  uint64_t* kv_full = q_full + 2;
  uint64_t* kv_empty = kv_full + C::kStages;
  uint64_t* s_full = kv_empty + C::kStages;   // [buffer]: S(u) is in tensor memory
  uint64_t* p_lo = s_full + NB;               // [buffer]: first part of P(u) written (one arrival per softmax warp)
  uint64_t* p_hi = p_lo + NB;                 // [buffer]: the rest of P(u) written
  uint64_t* pv_done = p_hi + NB;              // [tile]: PV(u) has completed
  uint64_t* o_final = pv_done + 2;            // [tile]: the last PV of the tile has completed
  uint64_t* v_tail = o_final + 2;             // the foreign rows of the last V tile's last K step have been cleared
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::kBars);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int seg = blockIdx.z;
  const int head = blockIdx.y;

  int q_begin, q_len, k_begin, k_len;
  if (p.cu_q != nullptr) {
    q_begin = p.cu_q[seg];
    q_len = p.cu_q[seg + 1] - q_begin;
    k_begin = p.cu_k[seg];
    k_len = p.cu_k[seg + 1] - k_begin;
  } else {
    q_begin = seg * p.seqlen_q;
    q_len = p.seqlen_q;
    k_begin = seg * p.seqlen_k;
    k_len = p.seqlen_k;
  }
  const int q0 = blockIdx.x * (kQT * kBM);
  if (q0 >= q_len) {
    // (see the tear-down; a grid whose sequences are all empty has no CTA that gets that far)
    if (blockIdx.x == 0) grid_dependency_wait();
    return;
  }
  const int n_tiles = (k_len + kBN - 1) / kBN;
  if (n_tiles <= 0) {
    grid_dependency_wait();      // (also when nothing is written: a grid must not complete before the one it overlaps)
    write_empty_rows<D>(p, seg, head, q_begin, q_len, q0);
    return;
  }
  const int n_units = kQT * n_tiles;

  // ------------------------------------------------------------------ set-up
  if (threadIdx.x == kTmaWarp * 32) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&pv_done[i], 1);
      mbar_init(&o_final[i], 1);
    }
    mbar_init(v_tail, 1);
    for (int i = 0; i < C::kStages; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    for (int i = 0; i < NB; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_lo[i], 4);
      mbar_init(&p_hi[i], 4);
    }
    fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  // CTA-uniform view of the status word: a CTA that starts after a failure elsewhere does no work.
  const int aborted = __syncthreads_or(*reinterpret_cast<volatile int*>(p.status) != 0);
  // From here on a launch queued behind this one with the overlap attribute may fill idle SMs (it takes effect
  // once every CTA of this grid has got this far); it waits for this grid's completion before it touches results.
  grid_launch_dependents();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp >= kTmaWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
    // The last key tile holds `tail` keys of this sequence; the rows behind them belong to whatever follows it in memory (or
    // are TMA's zeros past the end of the tensor).  Their scores are masked, but a weight of 0 does not keep an infinity or
    // a NaN of their V rows out of the product: PV of the last tile runs the K steps of 16 keys that hold a key, and the
    // foreign rows of the last of these are cleared in shared memory first.
    const int tail = k_len - (n_tiles - 1) * kBN;
    const int tail_steps = (tail + 15) >> 4;
    if (aborted || warp > kMmaWarp) {
      // fall through to the tear-down
    } else if (warp == kTmaWarp) {
      // ------------------------------------------------------------ TMA producer
      bool live = true;
      if (elect_one()) {
        prefetch_tmap(&tm_q);
        prefetch_tmap(&tm_k);
        prefetch_tmap(&tm_v);
        auto load_q = [&](int t) {
          mbar_expect_tx(&q_full[t], C::kTileBytes);
          for (int s = 0; s < C::kSlabs; ++s)
            tma_load_2d(s_q + t * C::kTileBytes + s * kSlabBytes, &tm_q, &q_full[t], head * D + s * 64, q_begin + q0 + t * kBM);
        };
        int it = 0;
        auto load_kv = [&](const CUtensorMap* tm, int j) {
          const int stage = it % C::kStages;
          const int round = it / C::kStages;
          ++it;
          if (round > 0 && !wait_or_abort(&kv_empty[stage], (round - 1) & 1, p.status, 11)) return false;
          mbar_expect_tx(&kv_full[stage], C::kKvTileBytes);
          for (int s = 0; s < C::kSlabs; ++s)
            tma_load_2d(s_kv + stage * C::kKvTileBytes + s * kSlabBytes, tm, &kv_full[stage], head * D + s * 64, k_begin + j * kBN);
          return true;
        };
        // in the order in which the issuer consumes them
        load_q(0);
        live = load_kv(&tm_k, 0);
        load_q(1);
        if (NB > 2 && live && n_tiles > 1) live = load_kv(&tm_k, 1);
        for (int u = 0; live && u < n_units; ++u) {
          if ((u & 1) == 0) live = load_kv(&tm_v, u >> 1);
          const int un = u + NB;
          if (live && un < n_units && (un & 1) == 0) live = load_kv(&tm_k, un >> 1);
        }
      }
      __syncwarp();
      if ((tail & 15) != 0 && __all_sync(0xffffffffu, live)) {
        const int it = 2 * n_tiles - 1;                 // V of the last tile is the last load
        const int stage = it % C::kStages;
        if (warp_wait_or_abort(&kv_full[stage], (it / C::kStages) & 1, p.status, 12)) {
          // whole rows of 128 bytes: the swizzle moves 16-byte pieces inside a row only
#pragma unroll 1
          for (int s = 0; s < C::kSlabs; ++s) {
            uint8_t* first = s_kv + stage * C::kKvTileBytes + s * kSlabBytes + tail * 128;
#pragma unroll 1
            for (int i = lane; i < (16 * tail_steps - tail) * 8; i += 32)
              *reinterpret_cast<uint4*>(first + i * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          fence_proxy_async_smem();                     // the MMA reads shared memory through the asynchronous proxy
          __syncwarp();
          if (lane == 0) mbar_arrive(v_tail);
        }
      }
    } else {
      // ------------------------------------------------------------ MMA issuer
      if (elect_one()) {
        constexpr uint32_t idesc_qk = idesc_bf16_f32(kBM, kBN, false, false);
        constexpr uint32_t idesc_pv = idesc_bf16_f32(kBM, D, false, true);
        const uint32_t kv_addr = smem_u32(s_kv);

        // Descriptors are built once; a tile, stage or K step only moves the start-address field (units
        // of 16 bytes, no carry out of the field: shared memory ends below 2^18).
        const uint64_t q_desc = smem_desc_sw128(smem_u32(s_q), 16, 1024);    // K-major
        const uint64_t k_desc = smem_desc_sw128(kv_addr, 16, 1024);          // K-major
        const uint64_t v_desc = smem_desc_sw128(kv_addr, kSlabBytes, 1024);  // MN-major, slab pitch leading
        // S = Q_tile K^T into S buffer `buf`
        auto issue_s = [&](int tile, int stage, int buf) {
          const uint64_t a0 = q_desc + static_cast<uint32_t>(tile * (C::kTileBytes >> 4));
          const uint64_t b0 = k_desc + static_cast<uint32_t>(stage * (C::kKvTileBytes >> 4));
          const uint32_t d = tmem_base + C::kColS + buf * kBN;
#pragma unroll
          for (int k16 = 0; k16 < D / 16; ++k16) {
            const uint32_t off = ((k16 >> 2) * kSlabBytes + (k16 & 3) * 32) >> 4;
            mma_ss(d, a0 + off, b0 + off, idesc_qk, k16 > 0);
          }
        };
        // O_tile (+)= P V over the K steps [k0, k1) of 16 keys, as far as the tile has `steps`; P (bf16 pairs) at the start
        // of S buffer `buf`
        auto issue_pv = [&](int tile, int stage, int buf, bool acc, int k0, int k1, int steps) {
          const uint64_t b0 = v_desc + static_cast<uint32_t>(stage * (C::kKvTileBytes >> 4));
          const uint32_t d = tmem_base + C::kColO + tile * D;
          const uint32_t a = tmem_base + C::kColS + buf * kBN;
#pragma unroll
          for (int kk = k0; kk < k1; ++kk)
            if (kk < steps) mma_ts(d, a + kk * 8, b0 + (kk * 2048 >> 4), idesc_pv, (acc || kk > 0) ? 1u : 0u);
        };
        int stage = 0;             // next ring slot to consume
        uint32_t round = 0;        // its parity
        auto next_kv = [&](int& held, int code) {
          if (!wait_or_abort(&kv_full[stage], round, p.status, code)) return false;
          tc_fence_after();
          held = stage;
          if (++stage == C::kStages) { stage = 0; round ^= 1; }
          return true;
        };
        int k_stage = 0, v_stage = 0;
        bool ok = true;
        // S(un) into buffer `buf`, K fetched for the first Q tile and released behind the second
        auto do_s = [&](int un, int buf) {
          if ((un & 1) == 0 && !next_kv(k_stage, 22)) return false;
          if (un < 2) {
            if (!wait_or_abort(&q_full[un], 0, p.status, 21)) return false;
            tc_fence_after();
          }
          issue_s(un & 1, k_stage, buf);
          mma_commit(&s_full[buf]);
          if (un & 1) mma_commit(&kv_empty[k_stage]);
          return true;
        };
        for (int u = 0; ok && u < NB && u < n_units; ++u) ok = do_s(u, u);
        int buf = 0;
        uint32_t use = 0;          // parity of the buffer's barriers
        int u = 0;
        for (; ok && u < n_units - 2; ++u) {
          const int tile = u & 1;
          if (tile == 0 && !next_kv(v_stage, 23)) { ok = false; break; }
          ok = wait_or_abort(&p_lo[buf], use, p.status, 24 + tile);
          if (!ok) break;
          tc_fence_after();
          issue_pv(tile, v_stage, buf, u > 1, 0, kSplit / 16, kBN / 16);
          ok = wait_or_abort(&p_hi[buf], use, p.status, 26 + tile);
          if (!ok) break;
          tc_fence_after();
          issue_pv(tile, v_stage, buf, true, kSplit / 16, kBN / 16, kBN / 16);
          if (NB > 2) mma_commit(&pv_done[tile]);
          if (tile == 1) mma_commit(&kv_empty[v_stage]);
          if (u + NB < n_units) ok = do_s(u + NB, buf);
          if (++buf == NB) { buf = 0; use ^= 1; }
        }
        // The last key tile, behind the loop so that the loop's PV has no limit to test (with one test per MMA in the loop the
        // kernel was 1-2 % slower, like this 0.3 %).  It commits to o_final alone: nothing waits for its pv_done or for the ring
        // slot, and an arrival that nothing waits for could still be under way when the CTA ends and its shared memory gets
        // a new owner.
        ok = ok && next_kv(v_stage, 23) && ((tail & 15) == 0 || wait_or_abort(v_tail, 0, p.status, 28));
#pragma unroll 1
        for (int tile = 0; ok && tile < kQT; ++tile) {
          ok = wait_or_abort(&p_lo[buf], use, p.status, 24 + tile);
          if (!ok) break;
          tc_fence_after();
          issue_pv(tile, v_stage, buf, n_tiles > 1, 0, kSplit / 16, tail_steps);
          ok = wait_or_abort(&p_hi[buf], use, p.status, 26 + tile);
          if (!ok) break;
          tc_fence_after();
          issue_pv(tile, v_stage, buf, true, kSplit / 16, kBN / 16, tail_steps);
          mma_commit(&o_final[tile]);
          if (++buf == NB) { buf = 0; use ^= 1; }
        }
      }
      __syncwarp();
    }
  } else {
    // -------------------------------------------------------------- softmax + epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
    const int tile = warp >> 2;
    const int quarter = warp & 3;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t o_taddr = lane_base + C::kColO + tile * D;
    const float c = p.scale_log2;
    float m = -INFINITY;   // running max of raw scores (lazily updated)
    float l = 0.f;         // running sum of exp2((s - m) * c)
    bool ok = !aborted;
    int buf = tile;
    uint32_t use = 0;

    for (int j = 0; ok && j < n_tiles; ++j) {
      const uint32_t s_taddr = lane_base + C::kColS + buf * kBN;   // S(u), then P(u) over its first half
      ok = warp_wait_or_abort(&s_full[buf], use, p.status, 31 + tile);
      if (!ok) break;
      tc_fence_after();
      uint32_t sr[kBN];
      tmem_ld32(s_taddr, sr);
      tmem_ld32(s_taddr + 32, sr + 32);
      tmem_wait_ld<64>(sr);
      tmem_ld32(s_taddr + 64, sr + 64);      // in flight while the first half is scanned
      tmem_ld32(s_taddr + 96, sr + 96);
      const bool ragged = (j == n_tiles - 1) && (k_len & (kBN - 1)) != 0;
      const int valid = k_len - j * kBN;
      if (ragged) {
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (i >= valid) sr[i] = 0xff800000u;   // -inf
      }
      float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
      auto scan = [&](int i0) {
#pragma unroll
        for (int i = i0; i < i0 + 64; i += 8) {
          mx0 = max3(mx0, __uint_as_float(sr[i]), __uint_as_float(sr[i + 1]));
          mx1 = max3(mx1, __uint_as_float(sr[i + 2]), __uint_as_float(sr[i + 3]));
          mx2 = max3(mx2, __uint_as_float(sr[i + 4]), __uint_as_float(sr[i + 5]));
          mx3 = max3(mx3, __uint_as_float(sr[i + 6]), __uint_as_float(sr[i + 7]));
        }
      };
      scan(0);
      tmem_wait_ld<64>(sr + 64);
      if (ragged) {
#pragma unroll
        for (int i = 64; i < kBN; ++i)
          if (i >= valid) sr[i] = 0xff800000u;
      }
      scan(64);
      const float m_new = fmaxf(max3(m, mx0, mx1), fmaxf(mx2, mx3));
      if (j == 0) {
        m = m_new;
      } else {
        const bool grow = (m_new - m) * c > kRescaleThreshold;
        if (__any_sync(0xffffffffu, grow)) {
          // O is rescaled in place: PV(u-2), the unit of this Q tile before this one, must have drained (PV(u) is not
          // issued before this group hands over P(u)).  With two buffers S(u) was issued behind PV(u-2), so it has.
          if (NB > 2) {
            ok = warp_wait_or_abort(&pv_done[tile], (j - 1) & 1, p.status, 33 + tile);
            if (!ok) break;
            tc_fence_after();
          }
          const float f = ex2((m - m_new) * c);
#pragma unroll
          for (int q = 0; q < D / 16; ++q) {
            uint32_t orow[16];
            tmem_ld16(o_taddr + q * 16, orow);
            tmem_wait_ld<16>(orow);
#pragma unroll
            for (int i = 0; i < 16; ++i) orow[i] = __float_as_uint(__uint_as_float(orow[i]) * f);
            tmem_st16(o_taddr + q * 16, orow);
          }
          tmem_wait_st();
          l *= f;
          m = m_new;
        }
      }
      // p = 2^(s*c - m*c), at most 2^8
      const uint64_t c2 = pack2(c, c), nmc2 = pack2(-m * c, -m * c);
      uint64_t sum0 = pack2(0.f, 0.f), sum1 = sum0;
      auto exp_part = [&](int i0, int i1) {
#pragma unroll
        for (int i = i0; i < i1; i += 2) {
          const uint64_t x = fma2(pack2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), c2, nmc2);
          const uint64_t pp = ((i >> 1) & 7) >= 8 - kPolyPairs ? exp2_poly2(x) : exp2_mufu2(x);
          if (i & 2) sum1 = add2(sum1, pp); else sum0 = add2(sum0, pp);
          float p0, p1;
          unpack2(pp, p0, p1);
          sr[i >> 1] = pack_bf16x2(p0, p1);
        }
      };
      exp_part(0, kSplit);
      tmem_st32(s_taddr, sr);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_lo[buf]);
      exp_part(kSplit, kBN);
      tmem_st32(s_taddr + 32, sr + 32);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_hi[buf]);
      float s0, s1, s2, s3;
      unpack2(sum0, s0, s1);
      unpack2(sum1, s2, s3);
      l += (s0 + s1) + (s2 + s3);
      buf += 2;
      if (buf >= NB) { buf -= NB; use ^= 1; }
    }

    if (ok) ok = warp_wait_or_abort(&o_final[tile], 0, p.status, 41);
    // Results: the launch before this one (which may still be running if this launch overlaps it) must have
    // completed before its state is read for accumulation or its buffers are written.
    grid_dependency_wait();
    if (ok) {
      tc_fence_after();
      const int warp_pos = q0 + tile * kBM + quarter * 32;      // position of the warp's first row
      const int rows = q_len - warp_pos;
      const int64_t tok0 = static_cast<int64_t>(q_begin) + warp_pos;
      const float lse_new = (m * c + log2f(l)) * kLn2;
      float w_new = 1.f / l, w_old = 0.f;
      if (lane < rows) {
        const int64_t li = lse_index(p, seg, head, warp_pos + lane, tok0 + lane);
        float lse_out;
        merge_weights(p.accumulate != 0, p.accumulate ? p.lse[li] : -INFINITY, lse_new, l, w_new, w_old, lse_out);
        p.lse[li] = lse_out;
      }
      // staged in this warp's part of its Q tile, which the last S instruction has read
      uint8_t* stage = s_q + tile * C::kTileBytes + quarter * (C::kTileBytes / 4);
      static_assert(C::kTileBytes / 4 >= 4096, "32 rows x 128 bytes");
#pragma unroll
      for (int q = 0; q < D / 32; ++q) {
        uint32_t orow[32];
        tmem_ld32(o_taddr + q * 32, orow);
        tmem_wait_ld<32>(orow);
        OldRows old;
        if (p.accumulate) load_old_rows32(p, tok0, rows, static_cast<int64_t>(head) * D + q * 32, old);
        if (rows > 0) store_rows32(p, stage, tok0, rows, static_cast<int64_t>(head) * D + q * 32, orow, old, w_new, w_old);
      }
    }
  }

  // ------------------------------------------------------------------ tear-down
  // No CTA leaves before the launch it may overlap has completed: a launch that overlaps THIS one waits for this
  // grid only, and relies on this grid's completion implying that of everything before it.
  grid_dependency_wait();
  if (*reinterpret_cast<volatile int*>(p.status) != 0) __nanosleep(1000000);   // let copies in flight land
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <int D>
cudaError_t launch_flash(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FlashParams& p,
                         cudaStream_t stream) {
  using C = Cfg<D>;
  static bool configured[64] = {};
  static std::mutex mu;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64) {
    std::lock_guard<std::mutex> lk(mu);
    if (!configured[dev]) {
      // the register hand-over below waits for good unless the kernel starts with what it was computed for
      cudaFuncAttributes fa;
      cudaError_t e = cudaFuncGetAttributes(&fa, flash_fwd_kernel<D>);
      if (e == cudaSuccess && fa.numRegs != kRegsLaunch) e = cudaErrorInvalidKernelImage;
      if (e == cudaSuccess) e = cudaFuncSetAttribute(flash_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
      if (e != cudaSuccess) return e;
      configured[dev] = true;
    }
  }
  dim3 grid((p.seqlen_q + kQT * kBM - 1) / (kQT * kBM), p.num_heads, p.nseg);
  return launch_attention_kernel(flash_fwd_kernel<D>, grid, kThreads, C::kSmemBytes, stream, p.overlap_previous != 0, tq, tk, tv, p);
}

int flash_kv_box_rows() { return kBN; }

template cudaError_t launch_flash<64>(const CUtensorMap&, const CUtensorMap&, const CUtensorMap&, const FlashParams&, cudaStream_t);
template cudaError_t launch_flash<128>(const CUtensorMap&, const CUtensorMap&, const CUtensorMap&, const FlashParams&, cudaStream_t);

}  // namespace dtb
