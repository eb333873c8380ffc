// Prefill attention with the reference's top-8 rule, two heads per CTA (sm_100a).
//
// An item is 128 consecutive positions of TWO query heads of one KV group (two 128-row tiles
// that share every K/V tile).  A CTA works through items, the longest first, as long as there are any
// (see PairItem), and is split into roles:
//   warps 0-3  softmax of tile 0, one thread per row (all 128 columns of a key block);
//   warps 4-7  softmax of tile 1;
//   warp 8     one lane feeds the K and V rings (and Q) with bulk tensor copies;
//   warp 9     one lane issues every tcgen05.mma;
//   warps 10-11 idle: they complete the third warpgroup, which hands most of its
//              registers to the softmax warpgroups (setmaxnreg).
// Tensor memory (512 columns): S0 | S1 | O0 | O1, 128 fp32 columns each.  A softmax
// thread reads its row of S, and writes the bf16 probabilities back over the first 64
// columns of the same S buffer; O' = P V then takes its A operand straight from tensor
// memory, so P never touches shared memory.  The issuing lane alternates between the two
// tiles - S0, S1, then per key block [P0.V, next S0, P1.V, next S1] - so that one tile's
// softmax runs under the other tile's matrix products.  O stays in tensor memory for
// the whole row; a row's running maximum only moves when the new one is more than 2^8
// above it, and the row of O is then rescaled in place by its own thread.
// Every wait is bounded; a wait that runs out sets the status word and the CTA drains.
// Between two items nothing waits for the whole CTA: the next Q is fetched when the last S
// of the item is done, its first S is issued behind the item's last P.V, and the softmax
// threads write the item's output meanwhile.
//
// The top-8 rule is the one of prefill_topk.cu (community-kv.patch,
// hopper/topk_warpselect.h): per row, four classes of columns (class = (j % 8) / 2)
// keep their six best packed candidates, the row reports the eight largest of the 24.

#include "tc_primitives.cuh"

namespace ckv {

namespace {

constexpr int kPairSms = 148;  // one CTA per SM
constexpr int kItemSlots = 4;
constexpr int kPairThreads = 384;  // three warpgroups: two of softmax rows, one of helpers

struct PairSmem {
  static constexpr int kQ = 0;                  // two query tiles
  static constexpr int kK = 2 * kTileBytes;     // two key stages
  static constexpr int kV = 4 * kTileBytes;     // two value stages
  static constexpr int kBars = 6 * kTileBytes;  // barriers, the TMEM slot, the abort flag
  static constexpr int kClaim = kBars + 176;    // what the launch answered to a request for a CTA's item
  static constexpr int kItems = kBars + 192;    // ring of kItemSlots items
  static constexpr int kTotal = kBars + 256;
};

// Operand tiles sit in the 128-byte swizzled layout: [half of the 128 dims][row][128
// bytes], the 16-byte chunks of a row XOR-ed with the row's low three bits (what a bulk
// tensor copy with 128-byte swizzle writes); tiles start on 1024-byte boundaries.

// tcgen05.mma with the descriptors given as 32-bit words (both operands share the high word)
__device__ __forceinline__ void umma_words(uint32_t tmem_d, uint32_t a_low, uint32_t b_low,
                                           uint32_t high, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b64 da, db;\n"
      "setp.ne.b32 p, %5, 0;\n"
      "mov.b64 da, {%1, %3};\n"
      "mov.b64 db, {%2, %3};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, {%6, %6, %6, %6}, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(a_low), "r"(b_low), "r"(high), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void umma_ts_words(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_low,
                                              uint32_t high, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b64 db;\n"
      "setp.ne.b32 p, %5, 0;\n"
      "mov.b64 db, {%2, %3};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, {%6, %6, %6, %6}, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "r"(b_low), "r"(high), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u)
      : "memory");
}

__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two fp32 lanes per instruction (fma.rn.f32x2 / add.f32x2)
__device__ __forceinline__ uint64_t pack_pair(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_pair(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_pair(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Bounded wait that also gives up when another role of the CTA already has.  One thread.
// try_wait parks the thread in hardware for a while instead of spinning.
constexpr uint32_t kPairPolls = 1u << 18;
__device__ __forceinline__ bool pair_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort) {
  for (uint32_t poll = 0; poll < kPairPolls; ++poll) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) {
      return true;
    }
    if ((poll & 15u) == 15u && *abort != 0u) {
      return false;
    }
  }
  *abort = 1u;
  return false;
}

// One look at a barrier.  The answer takes about 200 cycles; what follows may run meanwhile.
__device__ __forceinline__ bool pair_test(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0u;
}

// The same for a whole warp: lane 0 polls, the others take its word.  The barrier's
// completion is made visible to the waiting lanes by one successful test of their own.
__device__ __forceinline__ bool pair_wait_warp(uint32_t bar, uint32_t parity, volatile uint32_t* abort) {
  bool ok = true;
  if ((threadIdx.x & 31) == 0) {
    ok = pair_wait(bar, parity, abort);
  }
  ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
  if (ok) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    (void)done;
  }
  return ok;
}

// The candidate key of the top-8 rule, clamp(rn((raw + 48) * 256)) to 15 bits, without the
// conversion instruction (it shares the special-function unit with the other tile's
// exponentials and would queue behind them): adding 1.5 * 2^23 leaves the integer, rounded
// to nearest even, in the low mantissa bits.
__device__ __forceinline__ uint32_t quantised_key_fma(float raw) {
  const float scaled = fminf(fmaxf(fmaf(raw, 256.0f, 12288.0f), 0.0f), 32767.0f);
  return __float_as_uint(scaled + 12582912.0f) & 0x7fffu;
}

// Insertion into a descending list: slot k becomes the median of its entry, its left
// neighbour's entry and the candidate (two operations per slot, all slots side by side).
template <int kDepth>
__device__ __forceinline__ void sorted_insert(uint32_t (&queue)[kDepth], uint32_t candidate) {
#pragma unroll
  for (int k = kDepth - 1; k > 0; --k) {
    queue[k] = max(queue[k], min(queue[k - 1], candidate));
  }
  queue[0] = max(queue[0], candidate);
}

// Minimum that does not lose a NaN
__device__ __forceinline__ float min_nan(float a, float b) {
  float y;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}

// Candidates of one column class (32 of the 128 columns): the columns that reach the gate
// as a bit mask, then insertion in rounds - every lane with a pending column inserts its
// next one per round, the others zero, without a branch.  The mask is collected from the
// sign of score - gate, one shift each.  The pick of the column's score (a binary tree over
// the index bits) and the insertion are shallow: two warps share a scheduler, so the
// depth of the dependency chain is what a round costs.  A score that is not a number
// passes the sign test and is turned away by the comparison behind the pick.
// `sinks`: that many columns at the front are no candidates.
template <int kClass>
__device__ __forceinline__ void take_candidates(const float (&s)[128], float gate, int key0, int sinks,
                                                uint32_t (&queue)[kLocalK]) {
  const uint64_t minus_gate = pack_pair(-gate, -gate);
  uint32_t below[4] = {0u, 0u, 0u, 0u};  // sign bits of eight columns each
#pragma unroll
  for (int byte = 0; byte < 4; ++byte) {
#pragma unroll
    for (int j = 6; j >= 0; j -= 2) {
      const int c = ((byte * 8 + j) >> 1) * 8 + kClass * 2;
      float lo, hi;
      unpack_pair(add_pair(pack_pair(s[c], s[c + 1]), minus_gate), lo, hi);
      below[byte] = __funnelshift_l(__float_as_uint(hi), below[byte], 1);
      below[byte] = __funnelshift_l(__float_as_uint(lo), below[byte], 1);
    }
  }
  uint32_t takers = ~(below[0] | (below[1] << 8) | (below[2] << 16) | (below[3] << 24));
  if (sinks > 0) {
    // the pairs of whole groups of eight columns, and up to two columns of the next group
    const int pairs = min(sinks >> 3, 15);
    const int more = sinks >= 128 ? 2 : min(max((sinks & 7) - 2 * kClass, 0), 2);
    takers &= ~(((1u << (2 * pairs)) - 1u) | (((1u << more) - 1u) << (2 * pairs)));
  }
  while (__any_sync(0xffffffffu, takers != 0u)) {
    const int i = __ffs(takers) - 1;  // -1: nothing left in this lane
    float pick[16];
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      pick[m] = (i & 1) ? s[m * 8 + kClass * 2 + 1] : s[m * 8 + kClass * 2];
    }
#pragma unroll
    for (int width = 8, bit = 2; width >= 1; width >>= 1, bit <<= 1) {
#pragma unroll
      for (int m = 0; m < width; ++m) {
        pick[m] = (i & bit) ? pick[2 * m + 1] : pick[2 * m];
      }
    }
    const int c = (i >> 1) * 8 + kClass * 2 + (i & 1);
    const uint32_t candidate =
        (quantised_key_fma(pick[0]) << 17) | (static_cast<uint32_t>(key0 + c) & 0x1ffffu);
    sorted_insert<kLocalK>(queue, takers != 0u && pick[0] >= gate ? candidate : 0u);
    takers &= takers - 1;
  }
}

// The items of the launch in descending length: all head pairs' last tiles, then all tiles before
// them; CTA i of the grid begins with item i.  Causal items differ in length: with one head's items
// behind another's, the last head's longest item started when the rest of the chip was nearly done
// (SMs busy for 82 % of a call of 8192 tokens).  A CTA that is done with its item takes the place of
// the next CTA that has not started (clusterlaunchcontrol), and so on until none is left: the next
// item's loads and first product run under the end of the last one, where a CTA per item pays for
// launch, Q and first K, output (about 20000 cycles against 3700 per key block) each time.  Shares dealt
// out before the launch save that too, but a CTA whose SM is held by another kernel then keeps its
// whole share waiting.  32 query on 8 KV heads, us a call, attention alone and with neighbours: a CTA
// per item / shares / so: 4096 tokens 139, 135, 133 and 248, 247, 245; 16384 tokens 1806, 1770, 1748
// and about 2700 each.  Attention alone beside a kernel that holds 16 SMs for 1.7 ms, shares / so:
// 4096 tokens 291 and 189, 16384 tokens 3270 and 1892.
struct PairItem {
  int pos0, head0, kv_head, batch;

  __device__ __forceinline__ void set(const ckv_prefill_args& a, uint32_t item) {
    const uint32_t pairs = static_cast<uint32_t>((a.query_heads / a.kv_heads) >> 1);
    const uint32_t heads = a.kv_heads * pairs;
    const uint32_t lanes = heads * a.batch;  // head pairs of all sequences
    const uint32_t tiles = (a.seq_len + kPfRows - 1) / kPfRows;
    const uint32_t pair = item % lanes;
    batch = static_cast<int>(pair / heads);
    kv_head = static_cast<int>(pair % heads / pairs);
    head0 = static_cast<int>(2u * (pair % heads));
    pos0 = static_cast<int>((tiles - 1u - item / lanes) * kPfRows);
  }
  // key blocks 0 .. its own; the last one holds the diagonal
  __device__ __forceinline__ int blocks() const { return (pos0 >> 7) + 1; }
};

__device__ __forceinline__ void write_item(uint32_t slot, const PairItem& item) {
  asm volatile("st.shared.v4.s32 [%0], {%1, %2, %3, %4};" ::"r"(slot), "r"(item.pos0), "r"(item.head0),
               "r"(item.kv_head), "r"(item.batch)
               : "memory");
}
__device__ __forceinline__ PairItem read_item(uint32_t slot) {
  PairItem item;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(item.pos0), "=r"(item.head0), "=r"(item.kv_head), "=r"(item.batch)
               : "r"(slot)
               : "memory");
  return item;
}

// Asks for the item of a CTA of this grid that has not started (which then never does).  The answer
// arrives at `claim` (16 bytes of shared memory) and on the barrier.
__device__ __forceinline__ void request_item(uint32_t claim, uint32_t bar) {
  mbar_expect_tx(bar, 16u);
  asm volatile(
      "clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(claim),
      "r"(bar)
      : "memory");
}

// The answer: false if every CTA has started.  Nothing may be asked for after that.
__device__ __forceinline__ bool requested_item(uint32_t claim, uint32_t& item) {
  uint32_t taken, first;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b128 answer;\n"
      "ld.shared.b128 answer, [%2];\n"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, answer;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "mov.u32 %1, 0;\n"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, answer;\n"
      "}\n"
      : "=r"(taken), "=r"(first)
      : "r"(claim)
      : "memory");
  async_proxy_fence();  // the next answer is written behind this read
  item = first;
  return taken != 0u;
}

// kMany: more items than SMs, so that a CTA may take several.
template <int kMode, bool kMany>
__global__ void __launch_bounds__(kPairThreads, 1)
    prefill_pair_kernel(const ckv_prefill_args a, const __grid_constant__ CUtensorMap map_q,
                        const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + PairSmem::kBars);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile uint32_t* abort = reinterpret_cast<volatile uint32_t*>(bars + 16);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int length = a.seq_len;

  const uint32_t q_addr = smem_u32(smem + PairSmem::kQ);
  const uint32_t k_addr = smem_u32(smem + PairSmem::kK);
  const uint32_t v_addr = smem_u32(smem + PairSmem::kV);
  const uint32_t bar_q = smem_u32(bars);
  const uint32_t bar_k_full = smem_u32(bars + 1);   // two stages
  const uint32_t bar_v_full = smem_u32(bars + 3);   // two stages
  const uint32_t bar_k_free = smem_u32(bars + 5);   // two stages: both tiles' S of that block done
  const uint32_t bar_s_full = smem_u32(bars + 9);   // per tile: S written
  const uint32_t bar_p_full = smem_u32(bars + 11);  // per tile: P written by its four warps
  const uint32_t bar_o_full = smem_u32(bars + 13);  // per tile: P.V folded into O
  const uint32_t bar_q_free = smem_u32(bars + 7);   // the item's last S of both tiles done
  const uint32_t bar_claim = smem_u32(bars + 8);    // the answer to the producer's request
  const uint32_t bar_item = smem_u32(bars + 17);    // kItemSlots: an item is in its ring slot
  const uint32_t claim = smem_u32(smem + PairSmem::kClaim);
  // Item n of the CTA is in slot n % kItemSlots, pos0 < 0 behind the last.  The producer writes the next
  // one when it has issued the last V of its own, which waited for the S one step before: the softmax
  // warps are at most two items behind, and four slots need no barrier for their reuse.
  const uint32_t ring = smem_u32(smem + PairSmem::kItems);

  PairItem first;  // every role's, worked out while the CTA is set up
  first.set(a, blockIdx.x);
  // a wait already ran out somewhere in this launch: drain the grid quickly
  const bool drained = a.status != nullptr &&
                       (*reinterpret_cast<volatile uint32_t*>(a.status) & CKV_DEV_WAIT_TIMEOUT) != 0u;
  if (__syncthreads_or(drained ? 1 : 0)) {
    return;
  }
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 11; ++i) {
      mbar_init(bar_q + 8 * i, 1);
    }
    mbar_init(bar_p_full, 4);  // one arrival per softmax warp
    mbar_init(bar_p_full + 8, 4);
    mbar_init(bar_o_full, 1);
    mbar_init(bar_o_full + 8, 1);
#pragma unroll
    for (int i = 0; i < kItemSlots; ++i) {
      mbar_init(bar_item + 8 * i, 1);
    }
    *abort = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  bool failed = false;

  auto slot_of = [&](int n) { return ring + 16u * (static_cast<uint32_t>(n) % kItemSlots); };
  auto bar_of = [&](int n) { return bar_item + 8u * (static_cast<uint32_t>(n) % kItemSlots); };
  auto parity_of = [&](int n) { return (static_cast<uint32_t>(n) / kItemSlots) & 1u; };
  auto put_item = [&](int n, const PairItem& item) {
    write_item(slot_of(n), item);
    mbar_arrive(bar_of(n));
  };

  // Register hand-over between the warpgroups.  setmaxnreg.inc blocks until the registers
  // are free, without any bound: the totals must never exceed what the launch allocated
  // (384 threads x 168 registers = 256 x 208 + 128 x 88 = 256 x 216 + 128 x 72).  The helpers' lane
  // that issues the products sets the pace of attention alone, the softmax threads with neighbours:
  // 4096 tokens, 32 query on 8 KV heads, us with 208 / 216: 131 / 138 and 252 / 247.
  constexpr int kSoftmaxRegisters = kMode == 0 ? 208 : 216;
  constexpr int kHelperRegisters = kMode == 0 ? 88 : 72;
  static_assert(256 * kSoftmaxRegisters + 128 * kHelperRegisters <= kPairThreads * 168,
                "register hand-over exceeds the launch allocation");
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kHelperRegisters));
  }
  if (warp >= 10) {
    // nothing to do
  } else if (warp == 8) {
    // ---- producer ----
    if (lane == 0) {
      int step = 0;  // key blocks so far, over all items
      uint32_t index = 0;
      for (int n = 0; !failed; ++n) {
        PairItem item = first;
        if (n > 0) {
          item.set(a, index);
        }
        const int blocks = item.blocks();
        if (n > 0) {
          put_item(n, item);
        }
        for (int block = 0; block < blocks; ++block, ++step) {
          const int stage = step & 1;
          // K goes where K(step - 2) was: free once both tiles' S(step - 2) is done
          if (step >= 2 && !pair_wait(bar_k_free + 8 * stage, ((step >> 1) - 1) & 1, abort)) {
            failed = true;
            break;
          }
          tma_load_tile(k_addr + stage * kTileBytes, &map_k, bar_k_full + 8 * stage, block * kPfKeys,
                        item.kv_head, item.batch);
          if (block == 0) {
            if (n > 0 && !pair_wait(bar_q_free, (n - 1) & 1, abort)) {
              failed = true;
              break;
            }
            mbar_expect_tx(bar_q, 2 * kTileBytes);
            tma_issue_tile(q_addr, &map_q, bar_q, item.pos0, item.head0, item.batch);
            tma_issue_tile(q_addr + kTileBytes, &map_q, bar_q, item.pos0, item.head0 + 1, item.batch);
          }
          // V goes where V(step - 2) was.  S(step - 1) is committed after both
          // P.V(step - 2) were issued, so that barrier covers the products that read the stage.
          if (step >= 2 && !pair_wait(bar_k_free + 8 * (stage ^ 1), ((step - 1) >> 1) & 1, abort)) {
            failed = true;
            break;
          }
          tma_load_tile(v_addr + stage * kTileBytes, &map_v, bar_v_full + 8 * stage, block * kPfKeys,
                        item.kv_head, item.batch);
        }
        if (failed || !kMany) {
          break;
        }
        if (n == 0) {
          put_item(0, item);  // nobody waits for it: every role knows the first item by itself
        }
        // the answer takes about 500 cycles, and a step of products is still to come
        request_item(claim, bar_claim);
        if (!pair_wait(bar_claim, n & 1, abort)) {
          (void)mbar_wait(bar_claim, n & 1);  // it is still written into this CTA's memory
          failed = true;
          break;
        }
        if (!requested_item(claim, index)) {
          item.pos0 = -kPfRows;
          put_item(n + 1, item);
          break;
        }
      }
    }
  } else if (warp == 9) {
    // ---- matrix products ----
    if (lane == 0) {
      const uint32_t idesc_qk = instruction_descriptor(false);
      const uint32_t idesc_pv = instruction_descriptor(true);
      // Descriptors as (low, high) words: the high word (stride between 8-row groups,
      // version, swizzle mode) is the same for every operand, the low word is the
      // address in 16-byte units plus the leading-dimension offset; a step along the
      // reduction only adds a constant to the low word.
      const uint32_t desc_high = (1024u >> 4) | (1u << 14) | (2u << 29);
      const uint32_t q_low = ((q_addr & 0x3ffffu) >> 4) | (1u << 16);
      const uint32_t k_low = ((k_addr & 0x3ffffu) >> 4) | (1u << 16);
      const uint32_t v_low = ((v_addr & 0x3ffffu) >> 4) | (((kTileBytes / 2) >> 4) << 16);
      auto issue_qk = [&](int t, int stage) {
        const uint32_t a_low = q_low + t * (kTileBytes >> 4);
        const uint32_t b_low = k_low + stage * (kTileBytes >> 4);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          // dims 16 ks .. 16 ks + 15: 32 bytes into the row of the half that holds them
          const uint32_t within = ((ks >> 2) * (kTileBytes / 2) + (ks & 3) * 32) >> 4;
          umma_words(tmem + t * 128u, a_low + within, b_low + within, desc_high, idesc_qk, ks > 0);
        }
        umma_commit(bar_s_full + 8 * t);
        if (t == 1) {
          umma_commit(bar_k_free + 8 * stage);
        }
      };
      auto issue_pv = [&](int t, int stage, bool accumulate) {
        const uint32_t b_low = v_low + stage * (kTileBytes >> 4);
        // keys 16 ks .. 16 ks + 15: eight packed columns of P, sixteen 128-byte rows of
        // V in each half (the halves are the leading dimension, 8-key groups the stride)
        umma_ts_words(tmem + 256u + t * 128u, tmem + t * 128u, b_low, desc_high, idesc_pv, accumulate);
#pragma unroll
        for (int ks = 1; ks < 8; ++ks) {
          umma_ts_words(tmem + 256u + t * 128u, tmem + t * 128u + ks * 8u, b_low + ks * (2048 >> 4),
                        desc_high, idesc_pv, true);
        }
      };
      // S(step) behind P.V(step - 1), of the same item or of the one before.  This lane sets the
      // pace of the CTA where there are no neighbours to keep: 32 products of 64 cycles per key
      // block, and the products wait while it waits.  So it asks for the barriers that are usually
      // complete by then (K, V, the second tile's P) one group of products ahead; a barrier asked
      // for when it is needed costs 200 cycles, complete or not.
      int step = 0;
      int blocks = first.blocks(), next_blocks = 0;
      failed = !(pair_wait(bar_q, 0, abort) && pair_wait(bar_k_full, 0, abort));
      if (!failed) {
        tc_fence_after();
        issue_qk(0, 0);
        issue_qk(1, 0);
        if (blocks == 1) {
          umma_commit(bar_q_free);
        }
      }
      bool v_ready = false;
      for (int n = 0; blocks > 0 && !failed; ++n) {
        for (int block = 0; block < blocks; ++block, ++step) {
          const int stage = step & 1;
          const bool last = block + 1 == blocks;
          const uint32_t next_parity = ((step + 1) >> 1) & 1;
          if (!pair_wait(bar_p_full, step & 1, abort) ||
              (!v_ready && !pair_wait(bar_v_full + 8 * stage, (step >> 1) & 1, abort))) {
            failed = true;
            break;
          }
          tc_fence_after();
          const bool k_ready = pair_test(bar_k_full + 8 * (stage ^ 1), next_parity);
          issue_pv(0, stage, block > 0);
          bool p_ready = false;
          if (last) {
            umma_commit(bar_o_full);
          } else {
            if (!k_ready && !pair_wait(bar_k_full + 8 * (stage ^ 1), next_parity, abort)) {
              failed = true;
              break;
            }
            p_ready = pair_test(bar_p_full + 8, step & 1);
            tc_fence_after();
            issue_qk(0, stage ^ 1);
          }
          if (!p_ready && !pair_wait(bar_p_full + 8, step & 1, abort)) {
            failed = true;
            break;
          }
          tc_fence_after();
          v_ready = pair_test(bar_v_full + 8 * (stage ^ 1), next_parity);
          issue_pv(1, stage, block > 0);
          if (!last) {
            issue_qk(1, stage ^ 1);
            if (block + 2 == blocks) {  // the item's last S: Q may be overwritten once it is done
              umma_commit(bar_q_free);
            }
            continue;
          }
          // the next item's first S, if there is one, under the output of this one
          umma_commit(bar_o_full + 8);
          if constexpr (!kMany) {
            break;
          }
          if (!pair_wait(bar_of(n + 1), parity_of(n + 1), abort)) {
            failed = true;
            break;
          }
          next_blocks = read_item(slot_of(n + 1)).blocks();
          if (next_blocks > 0) {
            if (!pair_wait(bar_k_full + 8 * (stage ^ 1), next_parity, abort) || !pair_wait(bar_q, (n + 1) & 1, abort)) {
              failed = true;
              break;
            }
            tc_fence_after();
            issue_qk(0, stage ^ 1);
            issue_qk(1, stage ^ 1);
            if (next_blocks == 1) {
              umma_commit(bar_q_free);
            }
          }
        }
        blocks = next_blocks;
      }
    }
  } else {
    // ---- softmax of tile t, one thread per row ----
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegisters));
    const int t = warp >> 2;
    const int row = tid & (kPfRows - 1);
    const uint32_t lane_base = tmem + (((warp & 3) * 32u) << 16);
    const uint32_t s_addr = lane_base + t * 128u;
    const uint32_t o_addr = lane_base + 256u + t * 128u;
    const float scale_log2 = a.softmax_scale * kLog2e;
    int step = 0;  // key blocks so far, over all items
    int pos0 = first.pos0;
    for (int n = 0; !failed && pos0 >= 0; ++n) {
      const int blocks = (pos0 >> 7) + 1;
      const bool live = pos0 + row < length;
      float run_max = -INFINITY;  // of the raw (unscaled) scores
      float run_sum = 0.f;
      uint32_t q32[4][kLocalK];
      if constexpr (kMode == 1) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
#pragma unroll
          for (int k = 0; k < kLocalK; ++k) {
            q32[c][k] = 0u;
          }
        }
      }

      for (int block = 0; block < blocks; ++block, ++step) {
        const int key0 = block * kPfKeys;
        if (!pair_wait_warp(bar_s_full + 8 * t, step & 1, abort)) {
          failed = true;
          break;
        }
        tc_fence_after();
        uint32_t raw[4][32];
#pragma unroll
        for (int part = 0; part < 4; ++part) {
          tmem_load32_issue(s_addr + part * 32u, raw[part]);
        }
        tmem_wait_load();
        float s[128];
#pragma unroll
        for (int c = 0; c < 128; ++c) {
          s[c] = __uint_as_float(raw[c >> 5][c & 31]);
        }
        // only the last block of a tile meets the diagonal: key pos0 + c, row pos0 + row
        if (block == blocks - 1) {
#pragma unroll
          for (int c = 0; c < 128; ++c) {
            s[c] = c <= row ? s[c] : -INFINITY;
          }
        }
        // eight independent chains (the compiler keeps the order of a single one)
        float part_max[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          part_max[i] = fmaxf(s[i], s[i + 8]);
        }
#pragma unroll
        for (int c = 16; c < 128; c += 16) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            part_max[i] = fmaxf(part_max[i], fmaxf(s[c + i], s[c + i + 8]));
          }
        }
        const float tile_max = fmaxf(fmaxf(fmaxf(part_max[0], part_max[1]), fmaxf(part_max[2], part_max[3])),
                                     fmaxf(fmaxf(part_max[4], part_max[5]), fmaxf(part_max[6], part_max[7])));

        // The running maximum only moves when the new one lies more than 2^8 above it
        // (probabilities up to 256 are harmless in bf16 / fp32); moving it means rescaling
        // the row of O in tensor memory, once the product that still adds to it is done.
        const float new_max = fmaxf(run_max, tile_max);
        const bool move = new_max > run_max && (new_max - run_max) * scale_log2 > 8.0f;
        if (__any_sync(0xffffffffu, move)) {
          float corr = 1.f;
          if (move) {
            corr = run_max == -INFINITY ? 0.f : exp2_fast((run_max - new_max) * scale_log2);
            run_max = new_max;
            run_sum *= corr;
          }
          if (block > 0) {
            // P.V of the last block is done: this block's S was committed after it.  Rare, so
            // rolled and in narrow steps, which take few registers beside the row of scores.
#pragma unroll 1
            for (int part = 0; part < 8; ++part) {
              uint32_t o[16];
              tmem_load16_issue(o_addr + part * 16u, o);
              tmem_wait_load();
#pragma unroll
              for (int c = 0; c < 16; ++c) {
                o[c] = __float_as_uint(__uint_as_float(o[c]) * corr);
              }
              tmem_store16_issue(o_addr + part * 16u, o);
            }
          }
        }
        // ---- probabilities, bf16 pairs, over the first 64 columns of this S buffer ----
        const float offset = (run_max == -INFINITY ? 0.f : run_max) * scale_log2;
        const uint64_t scale_pair = pack_pair(scale_log2, scale_log2);
        const uint64_t offset_pair = pack_pair(-offset, -offset);
        uint64_t sum_pair[2] = {0ull, 0ull};
#pragma unroll
        for (int quarter = 0; quarter < 4; ++quarter) {
          uint32_t packed[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const int c = quarter * 32 + 2 * e;
            float x0, x1;
            unpack_pair(fma_pair(pack_pair(s[c], s[c + 1]), scale_pair, offset_pair), x0, x1);
            const float p0 = exp2_fast(x0);
            const float p1 = exp2_fast(x1);
            sum_pair[e & 1] = add_pair(sum_pair[e & 1], pack_pair(p0, p1));
            packed[e] = pack_bf16(p0, p1);
          }
          tmem_store16_issue(s_addr + quarter * 16u, packed);
        }
        {
          float a0, a1, b0, b1;
          unpack_pair(sum_pair[0], a0, a1);
          unpack_pair(sum_pair[1], b0, b1);
          run_sum += (a0 + a1) + (b0 + b1);
        }
        tmem_wait_store();
        tc_fence_before();
        // one arrival per warp: 128 arrivals on one barrier word queue up behind each other
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar_p_full + 8 * t);
        }

        // The candidate bookkeeping is bound by the ALU and by its rounds of insertion, one at least
        // in most blocks and classes; the gates keep their number down.  32 query on 8 KV heads,
        // against a gate from the lists alone, rounds with a branch, and the rows behind the
        // end taking part: 517 tokens 117 -> 39 us, 6001 tokens 1560 -> 530 us, 16384 tokens
        // 3250 -> 2620 us (attention alone: 20, 326 and 1820 us).
        // It runs from the scores still in registers while the tensor cores work on this
        // tile's P.V and next S: it is off the path between two blocks.
        if constexpr (kMode == 1) {
          const int sinks = a.num_sink - key0;  // columns of this block that are no candidates
          if (sinks > 0) {
            // the groups' maxima without them: the upper 64 columns, if that is far enough
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              part_max[i] = s[64 + i];
#pragma unroll
              for (int c = 72 + i; c < 128; c += 8) {
                part_max[i] = fmaxf(part_max[i], s[c]);
              }
            }
          }
          // A key that is below two keys of every class can never reach the output (the class
          // lists then hold at least eight keys above it), nor one below the top four of two
          // classes.  Two keys of every class: the second-best entries of the lists, or the
          // maxima of this block's two column groups of every class.
          const uint32_t third0 = q32[0][3], third1 = q32[1][3], third2 = q32[2][3], third3 = q32[3][3];
          const uint32_t second_of_fourths =
              max(min(max(third0, third1), max(third2, third3)),
                  max(min(third0, third1), min(third2, third3)));
          const uint32_t row_floor = max(min(min(q32[0][1], q32[1][1]), min(q32[2][1], q32[3][1])),
                                         second_of_fourths);
          float block_floor =
              min_nan(min_nan(min_nan(part_max[0], part_max[1]), min_nan(part_max[2], part_max[3])),
                      min_nan(min_nan(part_max[4], part_max[5]), min_nan(part_max[6], part_max[7])));
          block_floor = sinks > 64 ? -INFINITY : block_floor;
          const uint32_t floor_key = max(row_floor >> 17, quantised_key_fma(block_floor));
          // smallest raw score whose quantised key can reach the floor, a little low
          float gate = floor_key == 0u
                           ? -3.0e38f
                           : (static_cast<float>(floor_key) - 0.75f) * (1.0f / 256.0f) - 48.0f;
          // rows behind the end of a ragged prompt score 0 everywhere: ties that all reach the gate
          gate = live ? gate : INFINITY;
          // (no vote in front of a class: in most blocks some row of the warp has a taker)
          take_candidates<0>(s, gate, key0, sinks, q32[0]);
          take_candidates<1>(s, gate, key0, sinks, q32[1]);
          take_candidates<2>(s, gate, key0, sinks, q32[2]);
          take_candidates<3>(s, gate, key0, sinks, q32[3]);
        }
      }

      // the next item under the last product; the ring's slots up to it are visible then
      if (kMany && !failed && !pair_wait_warp(bar_of(n + 1), parity_of(n + 1), abort)) {
        failed = true;
      }
      if (!failed && !pair_wait_warp(bar_o_full + 8 * t, n & 1, abort)) {
        failed = true;
      }
      if (!failed) {
        tc_fence_after();
        // not held in registers through the loop
        PairItem item;
        if constexpr (kMany) {
          item = read_item(slot_of(n));
        } else {
          uint32_t again = blockIdx.x;
          asm volatile("" : "+r"(again));
          item.set(a, again);
        }
        const int row_pos = item.pos0 + row;
        const int row_head = item.head0 + t;
        const bool row_live = row_pos < length;
        const float inverse = 1.f / run_sum;
        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(a.output) + item.batch * a.o_batch_stride +
                             static_cast<int64_t>(row_live ? row_pos : 0) * a.o_row_stride +
                             row_head * a.o_head_stride;
#pragma unroll
        for (int part = 0; part < 4; ++part) {
          uint32_t o[32];
          tmem_load32_issue(o_addr + part * 32u, o);
          tmem_wait_load();
          if (row_live) {
#pragma unroll
            for (int d = 0; d < 32; d += 8) {
              uint4 v;
              v.x = pack_bf16(__uint_as_float(o[d]) * inverse, __uint_as_float(o[d + 1]) * inverse);
              v.y = pack_bf16(__uint_as_float(o[d + 2]) * inverse, __uint_as_float(o[d + 3]) * inverse);
              v.z = pack_bf16(__uint_as_float(o[d + 4]) * inverse, __uint_as_float(o[d + 5]) * inverse);
              v.w = pack_bf16(__uint_as_float(o[d + 6]) * inverse, __uint_as_float(o[d + 7]) * inverse);
              *reinterpret_cast<uint4*>(dst + part * 32 + d) = v;
            }
          }
        }
        if (row_live) {
          const float lse = run_max * a.softmax_scale + logf(run_sum);
          const int64_t heads_total = a.query_heads;
          a.lse[(item.batch * heads_total + row_head) * length + row_pos] = lse;
          if constexpr (kMode == 1) {
            const int skip = a.num_sink + kKappa - 1;
            if (row_pos >= skip) {
              // merge the four sorted class queues: eight times the largest head, which then
              // leaves its queue (a cursor per queue would put the queues into local memory)
              const int64_t base =
                  ((item.batch * heads_total + row_head) * (length - skip) + (row_pos - skip)) * kKappa;
              const float lse_log2 = lse * kLog2e;
#pragma unroll
              for (int rank = 0; rank < kKappa; ++rank) {
                const uint32_t best = max(max(q32[0][0], q32[1][0]), max(q32[2][0], q32[3][0]));
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                  const bool leaves = q32[c][0] == best;
#pragma unroll
                  for (int k = 0; k < kLocalK; ++k) {
                    q32[c][k] = leaves ? (k + 1 < kLocalK ? q32[c][k + 1] : 0u) : q32[c][k];
                  }
                }
                const float dequant = static_cast<float>(best >> 17) / 256.0f - 48.0f;
                a.topk_val[base + rank] = exp2f(dequant * scale_log2 - lse_log2);
                a.topk_idx[base + rank] = static_cast<int32_t>(best & 0x1ffffu);
              }
            }
          }
        }
      }
      pos0 = kMany ? read_item(slot_of(n + 1)).pos0 : -1;
    }
  }

  if (failed && a.status != nullptr) {
    atomicOr(a.status, CKV_DEV_WAIT_TIMEOUT);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512)
                 : "memory");
  }
}

}  // namespace

cudaError_t launch_prefill_pair(const ckv_prefill_args& a, cudaStream_t stream) {
  const int group = a.query_heads / a.kv_heads;
  if (group < 2 || (group & 1) != 0 || (a.mode != 0 && a.mode != 1)) {
    return cudaErrorInvalidValue;
  }
  CUtensorMap map_q, map_k, map_v;
  if (!tile_map(&map_q, a.query, a, a.query_heads, a.q_row_stride, a.q_head_stride, a.q_batch_stride, true) ||
      !tile_map(&map_k, a.key, a, a.kv_heads, a.k_row_stride, a.k_head_stride, a.k_batch_stride, true) ||
      !tile_map(&map_v, a.value, a, a.kv_heads, a.v_row_stride, a.v_head_stride, a.v_batch_stride, true)) {
    return cudaErrorInvalidValue;
  }
  const int64_t items = static_cast<int64_t>((a.seq_len + kPfRows - 1) / kPfRows) * a.kv_heads * (group / 2) * a.batch;
  if (items > 0x7fffffff) return cudaErrorInvalidConfiguration;
  const unsigned grid = static_cast<unsigned>(items);
  auto run = [&](auto kernel) -> cudaError_t {
    cudaError_t err =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PairSmem::kTotal);
    if (err != cudaSuccess) return err;
    kernel<<<grid, kPairThreads, PairSmem::kTotal, stream>>>(a, map_q, map_k, map_v);
    return cudaGetLastError();
  };
  // No claims where every item has an SM of its own: the loop over items costs a short call about a
  // microsecond (517 tokens of 32 query on 8 KV heads, attention alone, 18.0 -> 16.7 us).
  if (items <= kPairSms) {
    return a.mode == 0 ? run(prefill_pair_kernel<0, false>) : run(prefill_pair_kernel<1, false>);
  }
  return a.mode == 0 ? run(prefill_pair_kernel<0, true>) : run(prefill_pair_kernel<1, true>);
}

}  // namespace ckv
