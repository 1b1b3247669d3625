// Partial-attention forward at D = 64 for grids larger than the GPU (the rule is in capi.cu): the tiles, units and arithmetic of
// flash_fwd_sm100.cu (256 query rows as two 128-row Q tiles, key tiles of 128, one softmax thread per row), by CTAs that stay
// and take one block of queries (one (segment, head, 256 rows): a work item) after another.
//
// Warp roles (512 threads, four warpgroups):
//   warps 0-7    softmax, a warpgroup per Q tile; a finished row leaves its reference and sum in shared memory
//   warps 8-11   results: O out of tensor memory, normalisation, merge with the state in global memory, stores
//   warp  12     work items and TMA loads
//   warp  13     MMA issuer
//   warp  14     clears the foreign rows of an item's last V tile
//   warp  15     no role
//
// Why.  With a CTA per block, 6 us of the 33 us that a block of 2222 keys takes pass in front of its key loop and behind it:
// launch, tensor-memory allocation, first loads, then the read of the state it is merged with and the stores, all with idle
// tensor and softmax units.  Here the next item's queries and first keys are loaded and its first scores computed while the
// softmax warps finish the item before it, and results leave by warps of their own.
// Per key tile the two are level (512 queries x 296 heads, four blocks per SM, 4096 -> 16384 keys: +640 us with a CTA per block, +639
// here), though the softmax warps have 176 registers here and 208 there; what is saved is 3 to 5 us a block.  At D = 128 O takes
// half of tensor memory and the board is at its power cap, where idle phases let the clock recover: a version of this kernel for it
// reached 1203 to 1255 TFLOP/s at 14882 rows x 24 heads against 1273 to 1287.  Which launches come here: see the rule in capi.cu.
//
// Work items.  The grid has one block per item, as if every block were to run.  A CTA claims further blocks by cluster launch
// control, which hands out blocks that have not started: items go to whichever CTA is free (a static share would wait for SMs
// that other streams' kernels hold), nothing is counted in memory, and a launch that overlaps this one starts when the last
// block has started or been claimed.
//
// Every phase of a barrier is over for all that look at it before the next one can complete.  Most have a role that waits for each
// phase.  pv_done is only waited for when a reference moves, but PV(u) needs P(u), which the warps that look at it hand over behind
// that: it is never a phase ahead of them.  What a slow role could fall behind on (v_tail, tail_go) has a barrier per work slot, and
// slots are reused only when every role has given them back.
//
// Launches that overlap.  The result warps wait for the launch before this one to complete before they touch the state, and the
// bounded waits of the other roles (work_empty, o_free, ml_empty) go on meanwhile: what is left of that launch when the first CTA of
// this one starts, at most the blocks that its CTAs have under way, has to take less than their second.  A block takes 13 us per 1000
// keys.
#include "flash_common.cuh"

#include <mutex>

namespace dtb {

namespace {

using namespace flash;

constexpr int kThreads = 512;
constexpr int kRegsLaunch = 128;    // what __launch_bounds__(512, 1) allots; checked before the first launch
constexpr int kRegsSoftmax = 176;
constexpr int kRegsOutput = 104;
constexpr int kRegsOther = 56;
static_assert(2 * kRegsSoftmax + kRegsOutput + kRegsOther == 4 * kRegsLaunch, "register split");
constexpr int kOutWarp = 8;         // first of four
constexpr int kTmaWarp = 12;
constexpr int kMmaWarp = 13;
constexpr int kTailWarp = 14;
constexpr int kSplit = 64;          // keys of a tile whose probabilities are handed over first
constexpr int kPolyPairs = 1;       // pairs of every 8 pairs of scores, exponentiated on the FMA units
constexpr int kWork = 4;            // work items under way in a CTA
constexpr int kWorkReaders = 8 + 4 + 1 + 1;
constexpr int kClaimAhead = 8;      // key tiles before an item's last at which the next item is asked for

constexpr int D = 64;                         // head dimension
constexpr int NB = (512 - kQT * D) / kBN;     // S / P buffers in tensor memory
struct C {
  static constexpr int kTileBytes = kBM * D * 2;          // one Q, K or V tile: one slab
  static constexpr int kQBufs = 2;                        // items whose queries are in shared memory
  static constexpr int kStages = 8;
  static constexpr int kStageOut = 4 * 4096;              // 4 KB per result warp
  // barriers: q_full[QB][2], q_empty[QB], kv_full[S], kv_empty[S], s_full[NB], p_lo[NB], p_hi[NB], pv_done[2], o_final[2],
  // o_free[2], ml_full[2], ml_empty[2], work_full[W], work_empty[W], v_tail[W], tail_go[W], claim
  static constexpr int kBars = 3 * kQBufs + 2 * kStages + 3 * NB + 10 + 4 * kWork + 1;
  static constexpr int kSmemBytes = 1024 + (kQBufs * kQT + kStages) * kTileBytes + kStageOut + kQT * kBM * 8 + kWork * 32 + 16 +
                                    kBars * 8 + 16;
  static constexpr uint32_t kTmemCols = 512;
  static constexpr uint32_t kColS = 0;                    // + buffer * 128
  static constexpr uint32_t kColO = NB * kBN;             // + tile * D
};
static_assert(NB == 3 && C::kColO + kQT * D <= 512, "tensor memory");
static_assert(C::kSmemBytes <= 232448, "shared memory");

struct Item {
  int n_tiles;     // key tiles; 0: a sequence without keys, -1: no more work
  int q0, head, seg;
  int q_begin, q_len, k_len, unused;
};
static_assert(sizeof(Item) == 32, "shared-memory layout");

// Where things are in shared memory.  Every role makes its own from an address that the compiler cannot see through: from one
// that all share it takes the addresses of all roles' barriers out in front of the branch between the roles, and with what is
// left of the registers there reads them back from local memory in each of them.
struct Shared {
  uint8_t* s_q;
  uint8_t* s_kv;
  uint8_t* s_out;
  float2* s_ml;           // [tile][row]: reference and sum of a finished row
  Item* s_work;
  uint8_t* s_claim;
  uint64_t* q_full;       // [item buffer][tile]
  uint64_t* q_empty;      // [item buffer]: the item's last S has read both tiles
  uint64_t* kv_full;
  uint64_t* kv_empty;
  uint64_t* s_full;       // [buffer]: S(u) is in tensor memory
  uint64_t* p_lo;         // [buffer]: first part of P(u) written (one arrival per softmax warp)
  uint64_t* p_hi;         // [buffer]: the rest of P(u) written
  uint64_t* pv_done;      // [tile]: PV(u) has completed
  uint64_t* o_final;      // [tile]: O of the item is complete
  uint64_t* o_free;       // [tile]: ... and has been read (one arrival per result warp)
  uint64_t* ml_full;      // [tile]: references and sums of the item's rows are in s_ml
  uint64_t* ml_empty;     // [tile]: ... and have been read
  uint64_t* work_full;    // [slot]
  uint64_t* work_empty;   // [slot]: no role looks at the slot's item or its two barriers below any more
  uint64_t* tail_go;      // [slot]: every load of the item has been asked for
  uint64_t* v_tail;       // [slot]: the foreign rows of the item's last V tile have been cleared
  uint64_t* claim;
  uint32_t* tmem_slot;

  __device__ __forceinline__ explicit Shared(uint8_t* smem) {
    s_q = smem;
    s_kv = s_q + C::kQBufs * kQT * C::kTileBytes;
    s_out = s_kv + C::kStages * C::kTileBytes;
    s_ml = reinterpret_cast<float2*>(s_out + C::kStageOut);
    s_work = reinterpret_cast<Item*>(s_ml + kQT * kBM);
    s_claim = reinterpret_cast<uint8_t*>(s_work + kWork);
    q_full = reinterpret_cast<uint64_t*>(s_claim + 16);
    q_empty = q_full + 2 * C::kQBufs;
    kv_full = q_empty + C::kQBufs;
    kv_empty = kv_full + C::kStages;
    s_full = kv_empty + C::kStages;
    p_lo = s_full + NB;
    p_hi = p_lo + NB;
    pv_done = p_hi + NB;
    o_final = pv_done + 2;
    o_free = o_final + 2;
    ml_full = o_free + 2;
    ml_empty = ml_full + 2;
    work_full = ml_empty + 2;
    work_empty = work_full + kWork;
    tail_go = work_empty + kWork;
    v_tail = tail_go + kWork;
    claim = v_tail + kWork;
    tmem_slot = reinterpret_cast<uint32_t*>(q_full + C::kBars);
  }
};
// 0, as far as the compiler knows any number.
__device__ __forceinline__ uint32_t opaque_zero() {
  uint32_t z = 0;
  asm volatile("" : "+r"(z));
  return z;
}

// Cluster launch control: ask for a block of this grid that has not started yet ...
__device__ __forceinline__ void claim_request(void* response16, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
               ::"r"(smem_u32(response16)), "r"(smem_u32(bar)) : "memory");
}
// ... and read the answer: false when there was none left (not to be asked again then).
__device__ __forceinline__ bool claim_answer(const void* response16, int& x, int& y, int& z) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .b128 r;\n\t.reg .pred p;\n\t"
      "ld.shared.b128 r, [%4];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "selp.u32 %3, 1, 0, p;\n\t"
      "mov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, %1, %2, _}, r;\n\t}"
      : "=&r"(x), "=&r"(y), "=&r"(z), "=&r"(ok)
      : "r"(smem_u32(response16))
      : "memory");
  return ok != 0;
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 1)
flash_fwd_persistent_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                            const __grid_constant__ CUtensorMap tm_v, const FlashParams p) {
  extern __shared__ uint8_t smem_raw[];
  // (an offset and not a rounded address: the compiler then still knows that it is shared memory, and addresses take one
  // register instead of two)
  uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);
  const Shared sh(smem);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // ------------------------------------------------------------------ set-up
  if (threadIdx.x == kTmaWarp * 32) {
    for (int i = 0; i < C::kQBufs; ++i) {
      mbar_init(&sh.q_full[2 * i], 1);
      mbar_init(&sh.q_full[2 * i + 1], 1);
      mbar_init(&sh.q_empty[i], 1);
    }
    for (int i = 0; i < C::kStages; ++i) {
      mbar_init(&sh.kv_full[i], 1);
      mbar_init(&sh.kv_empty[i], 1);
    }
    for (int i = 0; i < NB; ++i) {
      mbar_init(&sh.s_full[i], 1);
      mbar_init(&sh.p_lo[i], 4);
      mbar_init(&sh.p_hi[i], 4);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh.pv_done[i], 1);
      mbar_init(&sh.o_final[i], 1);
      mbar_init(&sh.o_free[i], 4);
      mbar_init(&sh.ml_full[i], 4);
      mbar_init(&sh.ml_empty[i], 4);
    }
    for (int i = 0; i < kWork; ++i) {
      mbar_init(&sh.work_full[i], 1);
      mbar_init(&sh.work_empty[i], kWorkReaders);
      mbar_init(&sh.tail_go[i], 1);
      mbar_init(&sh.v_tail[i], 1);
    }
    mbar_init(sh.claim, 1);
    fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(sh.tmem_slot, C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  // CTA-uniform view of the status word: a CTA that starts after a failure elsewhere does no work.
  const int aborted = __syncthreads_or(*reinterpret_cast<volatile int*>(p.status) != 0);
  // From here on a launch queued behind this one with the overlap attribute may fill idle SMs (it takes effect once every
  // block of this grid has started or has been claimed); it waits for this grid's completion before it touches results.
  grid_launch_dependents();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(sh.tmem_slot);

  // The next work item as every role but the producer sees it: its slot, or -1 when there is none.  Slots are given back by
  // one arrival per reading warp.
  uint32_t fetched = 0;
  auto take = [&](const Shared& sh, bool there) {
    const uint32_t slot = fetched++ % kWork;
    return there && sh.s_work[slot].n_tiles >= 0 ? static_cast<int>(slot) : -1;
  };
  auto fetch = [&](const Shared& sh) {                       // by one thread
    return take(sh, wait_or_abort(&sh.work_full[fetched % kWork], (fetched / kWork) & 1, p.status, 51));
  };
  auto fetch_warp = [&](const Shared& sh) {                  // by a whole warp
    return take(sh, warp_wait_or_abort(&sh.work_full[fetched % kWork], (fetched / kWork) & 1, p.status, 51));
  };
  auto give_back = [&](const Shared& sh, int slot) {         // by a whole warp
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh.work_empty[slot]);
  };

  if (warp >= kTmaWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
    if (aborted || warp > kTailWarp) {
      // fall through to the tear-down
    } else if (warp == kTmaWarp) {
      // ------------------------------------------------------------ work items and TMA loads
      const Shared sh(smem + opaque_zero());
      if (elect_one()) {
        prefetch_tmap(&tm_q);
        prefetch_tmap(&tm_k);
        prefetch_tmap(&tm_v);
        int it = 0;                // K and V tiles loaded, over all items
        int items = 0;             // items with keys
        int published = 0;
        uint32_t claims = 0;
        bool live = true, asked = false;
        int bx = blockIdx.x, by = blockIdx.y, bz = blockIdx.z;
        auto ask = [&]() {
          fence_proxy_async_smem();            // the answer before this one has been read
          mbar_expect_tx(sh.claim, 16);
          claim_request(sh.s_claim, sh.claim);
          asked = true;
        };
        auto publish = [&](const Item& w) {
          const int slot = published % kWork, round = published / kWork;
          if (round > 0 && !wait_or_abort(&sh.work_empty[slot], (round - 1) & 1, p.status, 13)) return false;
          sh.s_work[slot] = w;
          mbar_arrive(&sh.work_full[slot]);
          ++published;
          return true;
        };
        for (;;) {
          Item w;
          w.head = by;
          w.seg = bz;
          w.q0 = bx * (kQT * kBM);
          w.unused = 0;
          int k_begin;
          if (p.cu_q != nullptr) {
            w.q_begin = p.cu_q[bz];
            w.q_len = p.cu_q[bz + 1] - w.q_begin;
            k_begin = p.cu_k[bz];
            w.k_len = p.cu_k[bz + 1] - k_begin;
          } else {
            w.q_begin = bz * p.seqlen_q;
            w.q_len = p.seqlen_q;
            k_begin = bz * p.seqlen_k;
            w.k_len = p.seqlen_k;
          }
          w.n_tiles = w.k_len > 0 ? (w.k_len + kBN - 1) / kBN : 0;
          asked = false;
          if (w.q0 < w.q_len) {
            if (!publish(w)) break;
            const int n = w.n_tiles;
            if (n > 0) {
              const int qb = items % C::kQBufs, q_round = items / C::kQBufs;
              auto load_kv = [&](const CUtensorMap* tm, int j) {
                const int stage = it % C::kStages;
                const int round = it / C::kStages;
                ++it;
                if (round > 0 && !wait_or_abort(&sh.kv_empty[stage], (round - 1) & 1, p.status, 11)) return false;
                mbar_expect_tx(&sh.kv_full[stage], C::kTileBytes);
                tma_load_2d(sh.s_kv + stage * C::kTileBytes, tm, &sh.kv_full[stage], w.head * D, k_begin + j * kBN);
                return true;
              };
              if (q_round > 0 && !wait_or_abort(&sh.q_empty[qb], (q_round - 1) & 1, p.status, 14)) break;
              // in the order in which the issuer consumes them
              for (int t = 0; live && t < kQT; ++t) {
                uint64_t* full = &sh.q_full[qb * 2 + t];
                mbar_expect_tx(full, C::kTileBytes);
                tma_load_2d(sh.s_q + (qb * kQT + t) * C::kTileBytes, &tm_q, full, w.head * D, w.q_begin + w.q0 + t * kBM);
                if (t == 0) live = load_kv(&tm_k, 0);
              }
              if (live && n > 1) live = load_kv(&tm_k, 1);
              for (int u = 0; live && u < 2 * n; ++u) {
                if (u == 2 * (n > kClaimAhead ? n - kClaimAhead : 0)) ask();
                if ((u & 1) == 0) live = load_kv(&tm_v, u >> 1);
                const int un = u + NB;
                if (live && un < 2 * n && (un & 1) == 0) live = load_kv(&tm_k, un >> 1);
              }
              if (!live) break;
              ++items;
            }
            mbar_arrive(&sh.tail_go[(published - 1) % kWork]);
          }
          if (!asked) ask();
          if (!wait_or_abort(sh.claim, claims & 1, p.status, 15)) break;
          ++claims;
          if (!claim_answer(sh.s_claim, bx, by, bz)) {
            w.n_tiles = -1;
            publish(w);
            break;
          }
        }
      }
      __syncwarp();
    } else if (warp == kTailWarp) {
      // ------------------------------------------------------------ foreign rows of an item's last V tile
      const Shared sh(smem + opaque_zero());
      // (see flash_fwd_sm100.cu: the K step of 16 keys in which a sequence ends holds rows of whatever follows it)
      int it = 0;
      for (int slot; (slot = fetch_warp(sh)) >= 0;) {
        const uint32_t use = ((fetched - 1) / kWork) & 1;
        const int n = sh.s_work[slot].n_tiles;
        const int tail = sh.s_work[slot].k_len - (n - 1) * kBN;
        it += 2 * n;
        if (n > 0 && (tail & 15) != 0) {
          const int stage = (it - 1) % C::kStages;                 // V of the last tile is the last load
          // (the ring slot's barrier is only looked at once this load is the one under way in it)
          if (!warp_wait_or_abort(&sh.tail_go[slot], use, p.status, 16) ||
              !warp_wait_or_abort(&sh.kv_full[stage], ((it - 1) / C::kStages) & 1, p.status, 12))
            break;
          // whole rows of 128 bytes: the swizzle moves 16-byte pieces inside a row only
          uint8_t* first_row = sh.s_kv + stage * C::kTileBytes + tail * 128;
#pragma unroll 1
          for (int i = lane; i < (16 - (tail & 15)) * 8; i += 32)
            *reinterpret_cast<uint4*>(first_row + i * 16) = make_uint4(0u, 0u, 0u, 0u);
          fence_proxy_async_smem();                                // the MMA reads shared memory through the asynchronous proxy
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&sh.v_tail[slot]);
          mbar_arrive(&sh.work_empty[slot]);
        }
      }
    } else {
      // ------------------------------------------------------------ MMA issuer
      const Shared sh(smem + opaque_zero());
      if (elect_one()) {
        constexpr uint32_t idesc_qk = idesc_bf16_f32(kBM, kBN, false, false);
        constexpr uint32_t idesc_pv = idesc_bf16_f32(kBM, D, false, true);
        const uint32_t kv_addr = smem_u32(sh.s_kv);
        const uint64_t q_desc = smem_desc_sw128(smem_u32(sh.s_q), 16, 1024);    // K-major
        const uint64_t k_desc = smem_desc_sw128(kv_addr, 16, 1024);          // K-major
        const uint64_t v_desc = smem_desc_sw128(kv_addr, kSlabBytes, 1024);  // MN-major, slab pitch leading
        // S = Q K^T of the operands that `ready_s` found
        auto issue_s = [&](uint64_t a0, uint64_t b0, uint32_t d) {
#pragma unroll
          for (int k16 = 0; k16 < D / 16; ++k16) {
            const uint32_t off = k16 * 32 >> 4;
            mma_ss(d, a0 + off, b0 + off, idesc_qk, k16 > 0);
          }
        };
        auto issue_pv = [&](int tile, int stage, int buf, bool acc, int k0, int k1, int steps) {
          const uint64_t b0 = v_desc + static_cast<uint32_t>(stage * (C::kTileBytes >> 4));
          const uint32_t d = tmem_base + C::kColO + tile * D;
          const uint32_t a = tmem_base + C::kColS + buf * kBN;
#pragma unroll
          for (int kk = k0; kk < k1; ++kk)
            if (kk < steps) mma_ts(d, a + kk * 8, b0 + (kk * 2048 >> 4), idesc_pv, (acc || kk > 0) ? 1u : 0u);
        };
        int stage = 0;             // next ring slot to consume
        uint32_t round = 0;        // its parity
        auto next_kv = [&](int& held, int code) {
          if (!wait_or_abort(&sh.kv_full[stage], round, p.status, code)) return false;
          tc_fence_after();
          held = stage;
          if (++stage == C::kStages) { stage = 0; round ^= 1; }
          return true;
        };
        int n = 0, tail = 0, slot = 0;      // of the current item: key tiles, keys of the last one, work slot
        auto next_item = [&]() {
          for (;;) {
            slot = fetch(sh);
            if (slot < 0) return false;
            n = sh.s_work[slot].n_tiles;
            tail = sh.s_work[slot].k_len - (n - 1) * kBN;
            if (n > 0) return true;
            mbar_arrive(&sh.work_empty[slot]);
          }
        };
        int k_stage = 0, v_stage = 0;
        int q_tile = 0;            // of the current item: its first tile in s_q, ...
        uint32_t q_use = 0;        // ... the parity of its loads ...
        uint32_t o_use = 1;        // ... and of the reads of the O before it
        bool first = true;
        int buf = 0;               // S / P buffer of the next PV; units are numbered through all items
        uint32_t use = 0;          // parity of its barriers
        // S(un) of the current item into buffer `b`: operands, K fetched for the first Q tile ...
        uint64_t s_a = 0, s_b = 0;
        auto ready_s = [&](int un) {
          const int tile = un & 1;
          if (tile == 0 && !next_kv(k_stage, 22)) return false;
          s_a = q_desc + static_cast<uint32_t>((q_tile + tile) * (C::kTileBytes >> 4));
          s_b = k_desc + static_cast<uint32_t>(k_stage * (C::kTileBytes >> 4));
          return true;
        };
        // ... and what follows its MMAs, K released behind the second Q tile
        auto commit_s = [&](int un, int b) {
          mma_commit(&sh.s_full[b]);
          if (un & 1) {
            mma_commit(&sh.kv_empty[k_stage]);
            if (un == 2 * n - 1) mma_commit(&sh.q_empty[q_tile >> 1]);
          }
        };
        // S(un) itself, un < NB
        auto put_s = [&](int un, int b) {
          if (!ready_s(un)) return false;
          if (un < 2 && !wait_or_abort(&sh.q_full[q_tile + un], q_use, p.status, 21)) return false;
          tc_fence_after();
          issue_s(s_a, s_b, tmem_base + C::kColS + b * kBN);
          commit_s(un, b);
          return true;
        };
        bool ok = next_item();
        for (int u = 0; ok && u < NB && u < 2 * n; ++u) ok = put_s(u, u);
        while (ok) {
          const int n_units = 2 * n;
          for (int u = 0; ok && u < n_units - 2; ++u) {
            const int tile = u & 1;
            // Everything that S(u + NB) needs is waited for in front of P(u): behind P(u) there are the MMAs alone, for the
            // softmax warps of this Q tile then wait for them.
            const bool more_s = u + NB < n_units;
            if (tile == 0 && !next_kv(v_stage, 23)) { ok = false; break; }
            if (more_s && !ready_s(u + NB)) { ok = false; break; }
            if (u < 2 && !first) {
              ok = wait_or_abort(&sh.o_free[tile], o_use, p.status, 30);
              if (!ok) break;
            }
            ok = wait_or_abort(&sh.p_lo[buf], use, p.status, 24 + tile);
            if (!ok) break;
            tc_fence_after();
            issue_pv(tile, v_stage, buf, u > 1, 0, kSplit / 16, kBN / 16);
            ok = wait_or_abort(&sh.p_hi[buf], use, p.status, 26 + tile);
            if (!ok) break;
            tc_fence_after();
            issue_pv(tile, v_stage, buf, true, kSplit / 16, kBN / 16, kBN / 16);
            mma_commit(&sh.pv_done[tile]);
            if (more_s) {
              issue_s(s_a, s_b, tmem_base + C::kColS + buf * kBN);
              commit_s(u + NB, buf);
            }
            if (tile == 1) mma_commit(&sh.kv_empty[v_stage]);
            if (++buf == NB) { buf = 0; use ^= 1; }
          }
          // The last key tile, and in the S buffers that its units leave the first units of the next item, so that the softmax
          // warps find their scores while O is still being read: the third buffer is free now, the others behind their PV.
          const int tail_steps = (tail + 15) >> 4;
          const bool one = n == 1;
          ok = ok && next_kv(v_stage, 23) && ((tail & 15) == 0 || wait_or_abort(&sh.v_tail[slot], ((fetched - 1) / kWork) & 1, p.status, 28));
          mbar_arrive(&sh.work_empty[slot]);
          const bool more = ok && next_item();
          if (more) {
            q_tile += kQT;
            if (q_tile == kQT * C::kQBufs) { q_tile = 0; q_use ^= 1; }
            ok = put_s(0, buf == 0 ? NB - 1 : buf - 1);
          }
#pragma unroll 1
          for (int tile = 0; ok && tile < kQT; ++tile) {
            if (one && !first) {
              ok = wait_or_abort(&sh.o_free[tile], o_use, p.status, 30);
              if (!ok) break;
            }
            ok = wait_or_abort(&sh.p_lo[buf], use, p.status, 24 + tile);
            if (!ok) break;
            tc_fence_after();
            issue_pv(tile, v_stage, buf, !one, 0, kSplit / 16, tail_steps);
            ok = wait_or_abort(&sh.p_hi[buf], use, p.status, 26 + tile);
            if (!ok) break;
            tc_fence_after();
            issue_pv(tile, v_stage, buf, true, kSplit / 16, kBN / 16, tail_steps);
            mma_commit(&sh.o_final[tile]);
            // An arrival that nothing waits for could still be under way when the CTA ends and its shared memory gets a new
            // owner: behind the last PV of all there is only o_final.
            if (more) {
              mma_commit(&sh.pv_done[tile]);
              if (tile == 1) mma_commit(&sh.kv_empty[v_stage]);
              if (tile + 1 < 2 * n) ok = put_s(tile + 1, buf);
            }
            if (++buf == NB) { buf = 0; use ^= 1; }
          }
          if (!more) break;
          first = false;
          o_use ^= 1;
        }
      }
      __syncwarp();
    }
  } else if (warp >= kOutWarp) {
    // -------------------------------------------------------------- results
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOutput));
    if (!aborted) {
      const Shared sh(smem + opaque_zero());
      const int quarter = warp & 3;
      const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      uint8_t* stage = sh.s_out + quarter * 4096;
      const float c = p.scale_log2;
      uint32_t item_use = 0;
      // The launch before this one (which may still be running if this launch overlaps it) must have completed before its
      // state is read for accumulation or its buffers are written.
      grid_dependency_wait();
      for (int slot; (slot = fetch_warp(sh)) >= 0;) {
        const Item w = sh.s_work[slot];
        give_back(sh, slot);
        if (w.n_tiles == 0) {
          if (!p.accumulate)
            for (int r = static_cast<int>(threadIdx.x) - kOutWarp * 32; r < kQT * kBM; r += 128)
              write_empty_row<D>(p, w.seg, w.head, w.q_begin, w.q_len, w.q0 + r);
          continue;
        }
        bool ok = true;
#pragma unroll 1
        for (int tile = 0; ok && tile < kQT; ++tile) {
          const uint32_t o_taddr = lane_base + C::kColO + tile * D;
          const int warp_pos = w.q0 + tile * kBM + quarter * 32;      // position of the warp's first row
          const int rows = w.q_len - warp_pos;
          const int64_t tok0 = static_cast<int64_t>(w.q_begin) + warp_pos;
          const int64_t li = lse_index(p, w.seg, w.head, warp_pos + lane, tok0 + lane);
          const int64_t col = static_cast<int64_t>(w.head) * D;
          float lse_old = -INFINITY;
          OldRows old;
          if (p.accumulate) {                    // under way while the rows are still being computed
            if (lane < rows) lse_old = p.lse[li];
            load_old_rows32(p, tok0, rows, col, old);
          }
          ok = warp_wait_or_abort(&sh.ml_full[tile], item_use, p.status, 42);
          if (!ok) break;
          const float2 ml = sh.s_ml[tile * kBM + quarter * 32 + lane];
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.ml_empty[tile]);
          float w_new, w_old, lse_out;
          merge_weights(p.accumulate != 0, lse_old, (ml.x * c + log2f(ml.y)) * kLn2, ml.y, w_new, w_old, lse_out);
          ok = warp_wait_or_abort(&sh.o_final[tile], item_use, p.status, 41);
          if (!ok) break;
          tc_fence_after();
          if (lane < rows) p.lse[li] = lse_out;
#pragma unroll
          for (int q = 0; q < D / 32; ++q) {
            uint32_t orow[32];
            tmem_ld32(o_taddr + q * 32, orow);
            tmem_wait_ld<32>(orow);
            if (q == D / 32 - 1) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&sh.o_free[tile]);
            }
            if (q > 0 && p.accumulate) load_old_rows32(p, tok0, rows, col + q * 32, old);
            if (rows > 0) store_rows32(p, stage, tok0, rows, col + q * 32, orow, old, w_new, w_old);
          }
        }
        if (!ok) break;
        item_use ^= 1;
      }
    }
  } else {
    // -------------------------------------------------------------- softmax
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
    if (!aborted) {
      const Shared sh(smem + opaque_zero());
      const int tile = warp >> 2;
      const int quarter = warp & 3;
      const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      const uint32_t o_taddr = lane_base + C::kColO + tile * D;
      const float c = p.scale_log2;
      int buf = tile;            // S / P buffer of the next key tile
      uint32_t use = 0;          // parity of its barriers
      uint32_t pv_use = 1;       // parity of PV of the key tile before
      uint32_t items = 0;
      bool ok = true;
      for (int slot; ok && (slot = fetch_warp(sh)) >= 0;) {
        const int n_tiles = sh.s_work[slot].n_tiles;
        const int k_len = sh.s_work[slot].k_len;
        give_back(sh, slot);
        if (n_tiles == 0) continue;
        float m = -INFINITY;     // running max of raw scores (lazily updated)
        float l = 0.f;           // running sum of exp2((s - m) * c)
        for (int j = 0; j < n_tiles; ++j) {
          const uint32_t s_taddr = lane_base + C::kColS + buf * kBN;   // S(u), then P(u) over its first half
          ok = warp_wait_or_abort(&sh.s_full[buf], use, p.status, 31 + tile);
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
              // O is rescaled in place: PV of this Q tile's key tile before must have drained (PV(u) is not issued before this
              // group hands over P(u))
              ok = warp_wait_or_abort(&sh.pv_done[tile], pv_use, p.status, 33 + tile);
              if (!ok) break;
              tc_fence_after();
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
          if (lane == 0) mbar_arrive(&sh.p_lo[buf]);
          exp_part(kSplit, kBN);
          tmem_st32(s_taddr + 32, sr + 32);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.p_hi[buf]);
          float s0, s1, s2, s3;
          unpack2(sum0, s0, s1);
          unpack2(sum1, s2, s3);
          l += (s0 + s1) + (s2 + s3);
          pv_use ^= 1;
          buf += 2;
          if (buf >= NB) { buf -= NB; use ^= 1; }
        }
        if (!ok) break;
        if (items > 0) ok = warp_wait_or_abort(&sh.ml_empty[tile], (items - 1) & 1, p.status, 43);
        if (!ok) break;          // the rows before these have not been read
        sh.s_ml[tile * kBM + quarter * 32 + lane] = make_float2(m, l);
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.ml_full[tile]);
        ++items;
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

cudaError_t launch_flash_persistent(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FlashParams& p,
                                    cudaStream_t stream) {
  static bool configured[64] = {};
  static std::mutex mu;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64) {
    std::lock_guard<std::mutex> lk(mu);
    if (!configured[dev]) {
      // the register hand-over waits for good unless the kernel starts with what it was computed for
      cudaFuncAttributes fa;
      cudaError_t e = cudaFuncGetAttributes(&fa, flash_fwd_persistent_kernel);
      if (e == cudaSuccess && fa.numRegs != kRegsLaunch) e = cudaErrorInvalidKernelImage;
      if (e == cudaSuccess) e = cudaFuncSetAttribute(flash_fwd_persistent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
      if (e != cudaSuccess) return e;
      configured[dev] = true;
    }
  }
  dim3 grid((p.seqlen_q + kQT * kBM - 1) / (kQT * kBM), p.num_heads, p.nseg);
  return launch_attention_kernel(flash_fwd_persistent_kernel, grid, kThreads, C::kSmemBytes, stream, p.overlap_previous != 0, tq, tk, tv, p);
}

}  // namespace dtb
