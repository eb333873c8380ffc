// Edge list -> coalesced adjacency (sm_100a): the consumer of the prefill kernel's
// neighbour edges and the producer of the graph that the host-side partitioner works on.
//
// Reference: build_adjacency, community_kv/graph/partition.py:168-249.  Every row of a
// graph contributes kappa direct edges (row position -> neighbour, weight score * lam / 2)
// and, when lam < 1, kappa (kappa + 1) / 2 co-attention edges between its neighbours
// (weight score_a * score_b * (1 - lam), the diagonal included); an edge is stored as
// (min vertex, max vertex) with vertices numbered graph * seq_len + position, duplicates
// are merged by adding their weights, and the result is sorted by (min, max).
//
// The reference sorts with torch.unique and adds with scatter_add_.  Here: the raw edges
// are enumerated in the reference's order (all direct edges, then all co-attention edges),
// sorted with a stable least-significant-digit radix sort (8 bits per pass), and every run
// of equal keys is summed front to back by one thread - a stable sort keeps equal keys in
// enumeration order, so each weight is the same sequence of fp32 additions a sequential
// scatter-add performs: the result is bit-exact and independent of scheduling.
//
// The sort is a one-sweep radix sort (Adinets and Merrill, "Onesweep", 2022: digit totals of all
// passes up front, one kernel per pass with the decoupled look-back of Merrill and Garland, 2016)
// and carries as few bytes as often as it can:
//   * both ends of an edge lie in one graph, so the key is (graph, min, max) with the
//     positions inside the graph: 31 bits and four passes for 32 graphs of 8192 positions
//     instead of 36 bits and five, and a 4-byte key wherever it fits (else 8 bytes);
//   * the raw edges are never written in enumeration order: the first pass makes them from
//     the rows (64 bytes of neighbours and scores per 44 edges of 8 bytes);
//   * a pass is one kernel: every tile publishes its digit counts and sums its
//     predecessors', and items leave in digit order through shared memory, so that a
//     tile writes runs of consecutive items.
// What bounds a pass now is not the traffic (16 bytes an item, 28 us of 11.5 M items at the copy
// rate; DRAM is busy 15-20 %) but the latency of its chain - shared-memory atomics of the ranking,
// look-back, staging - with 24 warps per SM: long_scoreboard and short_scoreboard lead the stalls.
// Three blocks per SM leave a thread eighty registers.  A tile's items therefore take their places in
// shared memory before the look-back, which then holds only counts, and ranks are kept as halves:
// with the items held across the look-back the 4-byte pass spilled 324 bytes of stores and 392 of
// loads per thread, now 8 (the first pass none, 36 where the neighbours per row are not eight).  The call
// for 32 graphs of 8192 positions, 11.5 M raw edges of random neighbours: 776 -> 697 us, for 8 such graphs
// 343 -> 326, for one of 1024 positions 164 -> 150.
// Five passes over enumerated 12-byte items with separate count and scan kernels took 1.1 ms.

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "../../include/ckv_b200.h"

namespace ckv {
namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kDigits = 256;
constexpr int kMaxPasses = 8;
constexpr int kNarrowItems = 16;  // items per thread with 4-byte keys; half of it with 8-byte keys

template <typename Key>
struct Sort {
  static constexpr int kItems = sizeof(Key) == 4 ? kNarrowItems : kNarrowItems / 2;
  static constexpr int kTile = kSortThreads * kItems;
};

template <typename Key>
struct Runs {
  static constexpr int kItems = sizeof(Key) == 4 ? 8 : 4;
  static constexpr int kTile = kSortThreads * kItems;
};

// The rows that the raw edges are made from.
struct EdgeRows {
  const int32_t* indices;     // [lines, kappa]
  const float* scores;
  const int64_t* positions;   // [lines]
  uint32_t rows;              // lines per graph
  uint32_t direct;            // direct edges in all: lines * kappa
  uint32_t raw;               // raw edges in all
  int kappa;
  int seq_len;
  int position_bits;          // a key is (graph, min, max): graph << 2 bits | min << bits | max
  float direct_scale;
  float co_scale;
};

template <typename Key>
__device__ __forceinline__ Key edge_key(const EdgeRows& e, uint32_t graph, uint32_t a, uint32_t b) {
  const uint32_t low = min(a, b);
  const uint32_t high = max(a, b);
  return (static_cast<Key>(graph) << (2 * e.position_bits)) | (static_cast<Key>(low) << e.position_bits) | high;
}
__device__ __forceinline__ bool in_graph(const EdgeRows& e, int64_t position) {
  return static_cast<uint64_t>(position) < static_cast<uint64_t>(e.seq_len);
}

// ---- digit totals of every pass ----
// One thread per line: it has the line's neighbours at hand and needs no index arithmetic.
// The top digit (graph and the leading bits of min) is the same for most edges of a line, so
// a thread counts runs of it in a register; the other digits go to shared memory one by one.
template <typename Key>
__global__ void __launch_bounds__(kSortThreads) digit_totals_kernel(const EdgeRows e, int passes, uint32_t* totals) {
  __shared__ uint32_t count[kMaxPasses * kDigits];
  for (int i = threadIdx.x; i < passes * kDigits; i += kSortThreads) count[i] = 0u;
  __syncthreads();
  const uint32_t lines = e.direct / e.kappa;
  const uint32_t line = blockIdx.x * kSortThreads + threadIdx.x;
  const int top = passes - 1;
  uint32_t run_digit = 0u, run = 0u;
  auto add = [&](Key key) {
    for (int p = 0; p < top; ++p) {
      atomicAdd(&count[p * kDigits + (static_cast<uint32_t>(key >> (8 * p)) & 255u)], 1u);
    }
    const uint32_t digit = static_cast<uint32_t>(key >> (8 * top)) & 255u;
    if (digit != run_digit) {
      if (run > 0u) atomicAdd(&count[top * kDigits + run_digit], run);
      run_digit = digit;
      run = 0u;
    }
    ++run;
  };
  if (line < lines) {
    const uint32_t graph = line / e.rows;
    const int32_t* own = e.indices + static_cast<int64_t>(line) * e.kappa;
    const int64_t position = e.positions[line];
    const bool co = e.raw > e.direct;
    for (int a = 0; a < e.kappa; ++a) {
      const int32_t u = own[a];
      if (!in_graph(e, u)) continue;
      if (in_graph(e, position)) add(edge_key<Key>(e, graph, u, static_cast<uint32_t>(position)));
      for (int b = a; co && b < e.kappa; ++b) {
        const int32_t v = own[b];
        if (in_graph(e, v)) add(edge_key<Key>(e, graph, u, v));
      }
    }
    if (run > 0u) atomicAdd(&count[top * kDigits + run_digit], run);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * kDigits; i += kSortThreads) {
    if (count[i] > 0u) atomicAdd(&totals[i], count[i]);
  }
}

// Exclusive prefix over the 256 threads of a block; `warp_total` holds one word per warp.
__device__ __forceinline__ uint32_t block_prefix(uint32_t value, uint32_t* warp_total, uint32_t* total) {
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  uint32_t inclusive = value;
#pragma unroll
  for (int delta = 1; delta < 32; delta <<= 1) {
    const uint32_t other = __shfl_up_sync(0xffffffffu, inclusive, delta);
    if (lane >= delta) inclusive += other;
  }
  if (lane == 31) warp_total[warp] = inclusive;
  __syncthreads();
  uint32_t before = 0u, all = 0u;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) {
    before += w < warp ? warp_total[w] : 0u;
    all += warp_total[w];
  }
  *total = all;
  return before + inclusive - value;
}

// One block per pass: digit totals -> where each digit begins, and the number of valid edges.
__global__ void __launch_bounds__(kSortThreads) digit_bases_kernel(uint32_t* totals, uint32_t* valid) {
  __shared__ uint32_t warp_total[kSortWarps];
  uint32_t* row = totals + blockIdx.x * kDigits;
  uint32_t total;
  const uint32_t prefix = block_prefix(row[threadIdx.x], warp_total, &total);
  row[threadIdx.x] = prefix;
  if (blockIdx.x == 0 && threadIdx.x == 0) *valid = total;
}

// ---- decoupled look-back ----
// A tile publishes its count with kPartial, later the sum over all tiles up to it with kComplete;
// flag and value are one 64-bit word.  Tiles take their numbers from a counter when they start, so
// every predecessor is already running and a wait ends; the waits are bounded all the same (`polls`
// looks without progress), and one that runs out is reported and yields a wrong sum (the stores that
// use it check their bounds).
constexpr uint64_t kPartial = 1ull << 62;
constexpr uint64_t kComplete = 2ull << 62;
constexpr uint64_t kValueMask = (1ull << 62) - 1;
constexpr uint32_t kLookPolls = 1u << 22;

__device__ __forceinline__ uint64_t look(const uint64_t* word) {
  uint64_t value;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(value) : "l"(word) : "memory");
  return value;
}
__device__ __forceinline__ void publish(uint64_t* word, uint64_t value) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(word), "l"(value) : "memory");
}

// One thread, one chain: the sum over the tiles in front of `tile`; words of a chain are `stride` apart.
// When a grid starts, a tile finds hundreds of partial words in front of it, so a thread reads
// kLookWords of them at a time.
constexpr int kLookWords = 8;

__device__ __forceinline__ uint32_t look_back(const uint64_t* words, uint32_t tile, uint32_t stride, uint32_t polls,
                                              uint32_t* fault) {
  uint64_t sum = 0;
  uint32_t polled = 0;
  int64_t t = static_cast<int64_t>(tile) - 1;
  bool done = t < 0;
  while (!done) {
    uint64_t word[kLookWords];
#pragma unroll
    for (int i = 0; i < kLookWords; ++i) word[i] = t - i >= 0 ? look(words + (t - i) * stride) : kComplete;
    const int64_t from = t;
#pragma unroll
    for (int i = 0; i < kLookWords; ++i) {
      if (!done && from - i == t && word[i] != 0ull) {
        sum += word[i] & kValueMask;
        done = (word[i] & kComplete) != 0ull;
        --t;
      }
    }
    if (!done && t == from && ++polled > polls) {
      atomicOr(fault, 1u);
      done = true;
    }
  }
  return static_cast<uint32_t>(sum);
}

// ---- one stable radix pass: digit = byte `pass` of the key ----
// Item order inside a tile: warp w holds items [32 kItems w, 32 kItems (w + 1)), round i of the
// warp 32 consecutive ones.  An item's rank among the tile's items of its digit is the count of
// the warps before it, the rounds before it and the lanes before it.  The lanes of a warp that
// share a digit find one another by OR-ing their lane bits into a word of shared memory (a match
// by atomics: about 15 instructions whatever the digit's width; eight ballots take 40), and a
// full tile runs without bounds checks.
template <typename Key>
__device__ __forceinline__ uint32_t digit_of(Key key, int pass) {
  if constexpr (sizeof(Key) == 4) {
    return __byte_perm(static_cast<uint32_t>(key), 0u, 0x4440u | static_cast<uint32_t>(pass));
  } else {
    return static_cast<uint32_t>(key >> (8 * pass)) & 255u;
  }
}

template <typename Key, int kKappa, bool kFirst>
__global__ void __launch_bounds__(kSortThreads, 3)
    radix_pass_kernel(const EdgeRows e, const Key* keys, const float* weights, Key* keys_out, float* weights_out,
                      const uint32_t* digit_base, const uint32_t* valid, int pass, uint64_t* words, uint32_t* ticket,
                      uint32_t polls, uint32_t* fault) {
  constexpr int kItems = Sort<Key>::kItems;
  constexpr int kTile = Sort<Key>::kTile;
  // counts per warp and digit, and the lane masks; the items in digit order reuse the masks' room
  __shared__ uint32_t warp_count[kSortWarps][kDigits];
  union Stage {
    uint32_t lanes[kSortWarps][kDigits];
    struct {
      Key key[kTile];
      float weight[kTile];
    } out;
  };
  __shared__ Stage stage;
  __shared__ uint32_t target_base[kDigits];
  __shared__ uint32_t warp_total[kSortWarps];
  __shared__ uint32_t tile_s;
  __shared__ uint16_t pair_slots[kFirst ? 2080 : 1];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) tile_s = atomicAdd(ticket, 1u);
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) {
    warp_count[w][threadIdx.x] = 0u;
    stage.lanes[w][threadIdx.x] = 0u;
  }
  const uint32_t kappa = kKappa > 0 ? kKappa : static_cast<uint32_t>(e.kappa);
  const uint32_t pairs = kappa * (kappa + 1) / 2;
  if constexpr (kFirst) {
    // pair number -> its two slots, row-major over the upper triangle
    for (uint32_t p = threadIdx.x; p < pairs; p += kSortThreads) {
      uint32_t first = 0, rest = p;
      while (rest >= kappa - first) {
        rest -= kappa - first;
        ++first;
      }
      pair_slots[p] = static_cast<uint16_t>(first | ((first + rest) << 8));
    }
  }
  __syncthreads();
  const uint32_t tile = tile_s;
  const uint32_t n = kFirst ? e.raw : *valid;
  const uint64_t base = static_cast<uint64_t>(tile) * kTile;
  if (base >= n) return;
  const uint32_t item0 = static_cast<uint32_t>(base) + warp * (32 * kItems) + lane;
  uint32_t* const my_count = warp_count[warp];
  uint32_t* const my_lanes = stage.lanes[warp];

  auto work = [&](auto full) {
    constexpr bool kFull = decltype(full)::value;  // every item of the tile takes part
    Key key[kItems];
    float weight[kItems];
    uint32_t live = 0u;  // bit i: item i takes part
    if constexpr (!kFirst) {
#pragma unroll
      for (int i = 0; i < kItems; ++i) {
        const bool here = kFull || item0 + i * 32 < n;
        key[i] = here ? keys[item0 + i * 32] : 0;  // the weights follow: nothing before the look-back needs them
        live |= (here ? 1u : 0u) << i;
      }
    } else {
      uint32_t graph = 0u, next_graph = 0u;  // `next_graph`: first line of the graph after it
      bool placed = false;
      auto graph_of = [&](uint32_t line) {
        if (!placed) {
          graph = line / e.rows;
          next_graph = (graph + 1u) * e.rows;
          placed = true;
        }
        while (line >= next_graph) {
          ++graph;
          next_graph += e.rows;
        }
        return graph;
      };
#pragma unroll
      for (int i = 0; i < kItems; ++i) {
        const uint32_t index = item0 + i * 32;
        key[i] = 0;
        weight[i] = 0.f;
        if (index >= n || index < item0) continue;
        if (index < e.direct) {
          const uint32_t line = index / kappa;
          const int32_t u = e.indices[index];
          const int64_t position = e.positions[line];
          if (in_graph(e, u) && in_graph(e, position)) {
            key[i] = edge_key<Key>(e, graph_of(line), u, static_cast<uint32_t>(position));
            weight[i] = __fmul_rn(e.scores[index], e.direct_scale);
            live |= 1u << i;
          }
        } else {
          const uint32_t j = index - e.direct;
          const uint32_t line = j / pairs;
          const uint32_t slots = pair_slots[j - line * pairs];
          const uint32_t own = line * kappa;  // below raw, which is below 2^32
          const uint32_t first = own + (slots & 255u), second = own + (slots >> 8);
          const int32_t u = e.indices[first], v = e.indices[second];
          if (in_graph(e, u) && in_graph(e, v)) {
            if (index - 32 * i < e.direct) placed = false;  // the direct edges' last line is behind this one's first
            key[i] = edge_key<Key>(e, graph_of(line), u, v);
            weight[i] = __fmul_rn(__fmul_rn(e.scores[first], e.scores[second]), e.co_scale);
            live |= 1u << i;
          }
        }
      }
    }

    uint32_t rank[kItems / 2];  // of two items, below 32 kItems each
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const bool here = kFull || ((live >> i) & 1u);
      const uint32_t digit = digit_of(key[i], pass);
      if (here) atomicOr(&my_lanes[digit], 1u << lane);
      __syncwarp();
      const uint32_t peers = my_lanes[digit];
      const uint32_t before = my_count[digit];
      const uint32_t below = __popc(peers & ((1u << lane) - 1u));
      __syncwarp();
      if (here && below == 0u) {
        my_count[digit] = before + __popc(peers);
        my_lanes[digit] = 0u;
      }
      __syncwarp();
      rank[i / 2] = (i & 1) ? rank[i / 2] | ((before + below) << 16) : before + below;
    }
    __syncthreads();

    // thread d looks after digit d
    const int d = threadIdx.x;
    uint32_t count = 0u, start, total;
    {
#pragma unroll
      for (int w = 0; w < kSortWarps; ++w) count += warp_count[w][d];
      publish(words + static_cast<uint64_t>(tile) * kDigits + d, (tile == 0 ? kComplete : kPartial) | count);
      if constexpr (!kFirst) {
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
          if (kFull || ((live >> i) & 1u)) weight[i] = weights[item0 + i * 32];
        }
      }
      start = block_prefix(count, warp_total, &total);
      uint32_t running = start;  // counts become places in the tile
#pragma unroll
      for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = warp_count[w][d];
        warp_count[w][d] = running;
        running += c;
      }
    }
    __syncthreads();
    // the items take their places in the tile first: nothing but the counts is then held in
    // registers across the look-back, whose predecessors gain the time
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      if (kFull || ((live >> i) & 1u)) {
        const uint32_t slot = my_count[digit_of(key[i], pass)] + ((i & 1) ? rank[i / 2] >> 16 : rank[i / 2] & 0xffffu);
        stage.out.key[slot] = key[i];
        stage.out.weight[slot] = weight[i];
      }
    }
    {
      const uint32_t ahead = look_back(words + d, tile, kDigits, polls, fault);
      if (tile > 0) {
        publish(words + static_cast<uint64_t>(tile) * kDigits + d, kComplete | (static_cast<uint64_t>(ahead) + count));
      }
      target_base[d] = digit_base[d] + ahead - start;
      if (d == 0) tile_s = total;
    }
    __syncthreads();
    const uint32_t here = kFull ? kTile : tile_s;
    const uint32_t limit = *valid;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const uint32_t slot = threadIdx.x + i * kSortThreads;
      if (kFull || slot < here) {
        const Key k = stage.out.key[slot];
        const uint32_t target = target_base[digit_of(k, pass)] + slot;
        if (target < limit) {
          keys_out[target] = k;
          weights_out[target] = stage.out.weight[slot];
        }
      }
    }
  };
  if (!kFirst && base + kTile <= n) {
    work(std::true_type());
  } else {
    work(std::false_type());
  }
}

// ---- runs of equal keys -> edges ----
// A thread holds kRunItems consecutive items; it sums every run that begins among them, reading on
// where the last one goes beyond.  Items come and edges leave through shared memory.
template <typename Key>
__global__ void __launch_bounds__(kSortThreads)
    run_edges_kernel(const Key* keys, const float* weights, const uint32_t* valid, int position_bits, int seq_len,
                     int64_t capacity, uint64_t* words, uint32_t* ticket, uint32_t polls, const uint32_t* fault,
                     int32_t* edge_src, int32_t* edge_dst, float* edge_weight, unsigned long long* edge_count) {
  constexpr int kItems = Runs<Key>::kItems;
  constexpr int kTile = Runs<Key>::kTile;
  __shared__ alignas(16) Key key_in[kTile];
  __shared__ alignas(16) float weight_in[kTile];
  __shared__ Key key_out[kTile];
  __shared__ float weight_out[kTile];
  __shared__ uint32_t warp_total[kSortWarps];
  __shared__ uint32_t tile_s, ahead_s;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) tile_s = atomicAdd(ticket, 1u);
  __syncthreads();
  const uint32_t tile = tile_s;
  const uint32_t n = *valid;
  const uint64_t base = static_cast<uint64_t>(tile) * kTile;
  if (base >= n) return;
  const uint32_t here = n - base < kTile ? static_cast<uint32_t>(n - base) : kTile;
  // four weights and their keys per thread and step
  for (uint32_t i = 4 * threadIdx.x; i < kTile; i += 4 * kSortThreads) {
    if (i + 4 <= here) {
#pragma unroll
      for (int v = 0; v < static_cast<int>(sizeof(Key) / 4); ++v) {
        reinterpret_cast<uint4*>(key_in + i)[v] = reinterpret_cast<const uint4*>(keys + base + i)[v];
      }
      *reinterpret_cast<float4*>(weight_in + i) = *reinterpret_cast<const float4*>(weights + base + i);
    } else {
      for (uint32_t j = i; j < here; ++j) {
        key_in[j] = keys[base + j];
        weight_in[j] = weights[base + j];
      }
    }
  }
  const Key before_tile = base > 0 ? keys[base - 1] : 0;
  __syncthreads();
  const uint32_t first = threadIdx.x * kItems;
  Key key[kItems];
  uint32_t heads = 0u;
  Key previous = first > 0 ? key_in[first - 1] : before_tile;
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    key[i] = key_in[first + i];
    const bool head = first + i < here && ((first + i == 0 && base == 0) || key[i] != previous);
    heads |= (head ? 1u : 0u) << i;
    previous = key[i];
  }
  uint32_t total;
  uint32_t slot = block_prefix(__popc(heads), warp_total, &total);
  if (threadIdx.x < 32) {
    // a warp looks back together: lane l at the l-th tile in front
    if (lane == 0) publish(words + tile, (tile == 0 ? kComplete : kPartial) | total);
    uint64_t sum = 0;
    uint32_t polled = 0;
    int64_t t = static_cast<int64_t>(tile) - 1;
    while (t >= 0) {
      const uint64_t word = t - lane >= 0 ? look(words + (t - lane)) : kComplete;
      const unsigned ready = __ballot_sync(0xffffffffu, word != 0ull);
      const unsigned done = __ballot_sync(0xffffffffu, (word & kComplete) != 0ull);
      const int reach = done ? __ffs(done) : 32;  // lanes 0 .. reach - 1 are wanted
      const unsigned wanted = reach == 32 ? 0xffffffffu : (1u << reach) - 1u;
      if ((ready & wanted) != wanted) {
        if (++polled > polls) {
          if (lane == 0) atomicExch(edge_count, ~0ull);
          break;
        }
        continue;
      }
      uint64_t part = lane < reach ? (word & kValueMask) : 0ull;
#pragma unroll
      for (int offset = 16; offset > 0; offset >>= 1) part += __shfl_xor_sync(0xffffffffu, part, offset);
      sum += part;
      if (done) break;
      t -= 32;
    }
    if (lane == 0) {
      ahead_s = static_cast<uint32_t>(sum);
      if (tile > 0) publish(words + tile, kComplete | (sum + total));
      // The count starts at 0.  Any tile may be the one whose wait ran out, before or after the last
      // tile has its sum: that tile's -1 replaces a count, and no count replaces a -1.  The earlier
      // kernels' waits are reported by the fault word.
      if (base + kTile >= n) {
        if (*fault != 0u) {
          atomicExch(edge_count, ~0ull);
        } else {
          atomicCAS(edge_count, 0ull, sum + total);
        }
      }
    }
  }
  if (heads != 0u) {
    float sum = 0.f;
    Key open = 0;
    bool started = false;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const float weight = weight_in[first + i];
      if ((heads >> i) & 1u) {
        if (started) {
          key_out[slot] = open;
          weight_out[slot] = sum;
          ++slot;
        }
        started = true;
        open = key[i];
        sum = weight;
      } else if (started && first + i < here) {
        sum = __fadd_rn(sum, weight);
      }
    }
    uint32_t j = first + kItems;
    while (j < here && key_in[j] == open) {
      sum = __fadd_rn(sum, weight_in[j]);
      ++j;
    }
    if (j >= here) {
      // the run may go on in the next tiles: four items in flight
      bool more = true;
      for (uint64_t at = base + here; more && at < n; at += 4) {
        Key k[4];
        float w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint64_t from = at + i < n ? at + i : n - 1;
          k[i] = keys[from];
          w[i] = weights[from];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          more = more && at + i < n && k[i] == open;
          if (more) sum = __fadd_rn(sum, w[i]);
        }
      }
    }
    key_out[slot] = open;
    weight_out[slot] = sum;
  }
  __syncthreads();
  const Key mask = (static_cast<Key>(1) << position_bits) - 1;
  for (uint32_t s = threadIdx.x; s < total; s += kSortThreads) {
    const int64_t out = static_cast<int64_t>(ahead_s) + s;
    if (out < capacity) {
      const Key k = key_out[s];
      const int32_t vertex0 = static_cast<int32_t>(k >> (2 * position_bits)) * seq_len;
      edge_src[out] = vertex0 + static_cast<int32_t>((k >> position_bits) & mask);
      edge_dst[out] = vertex0 + static_cast<int32_t>(k & mask);
      edge_weight[out] = weight_out[s];
    }
  }
}

int64_t align256(int64_t bytes) { return (bytes + 255) / 256 * 256; }

// Scratch for `raw` edges.  The key width is not known when the size is asked for, so the layout
// is the one of 8-byte keys; 4-byte keys use part of it.
struct Scratch {
  void* keys[2];
  float* weights[2];
  uint32_t* control;  // cleared: digit totals [kMaxPasses][256], valid, fault, a ticket per kernel
  uint64_t* words;    // cleared: look-back words, [pass][tile][256], then [tile] of the runs
  int64_t bytes;
};
constexpr int64_t kControlWords = kMaxPasses * kDigits + 2 + kMaxPasses + 1;

template <typename Key>
int64_t look_words(int64_t raw, int passes) {
  return passes * ((raw + Sort<Key>::kTile - 1) / Sort<Key>::kTile) * kDigits +
         (raw + Runs<Key>::kTile - 1) / Runs<Key>::kTile;
}

Scratch carve(void* base, int64_t raw) {
  Scratch s = {};
  int64_t offset = 0;
  auto take = [&](int64_t bytes) {
    uint8_t* p = base ? static_cast<uint8_t*>(base) + offset : nullptr;
    offset += align256(bytes);
    return p;
  };
  s.keys[0] = take(raw * 8);
  s.keys[1] = take(raw * 8);
  s.weights[0] = reinterpret_cast<float*>(take(raw * 4));
  s.weights[1] = reinterpret_cast<float*>(take(raw * 4));
  // `control` and `words` are cleared together
  const int64_t words = look_words<uint64_t>(raw, kMaxPasses);
  uint8_t* cleared = take(align256(kControlWords * 4) + words * 8);
  s.control = reinterpret_cast<uint32_t*>(cleared);
  s.words = reinterpret_cast<uint64_t*>(cleared + align256(kControlWords * 4));
  s.bytes = offset;
  return s;
}

template <typename Key, int kKappa>
cudaError_t sort_and_merge(const EdgeRows& e, const Scratch& s, int bits, uint32_t polls, int64_t capacity,
                           int32_t* edge_src, int32_t* edge_dst, float* edge_weight, int64_t* edge_count,
                           cudaStream_t stream) {
  const int passes = bits > 8 ? (bits + 7) / 8 : 1;
  const unsigned tiles = static_cast<unsigned>((static_cast<int64_t>(e.raw) + Sort<Key>::kTile - 1) / Sort<Key>::kTile);
  const unsigned run_tiles = static_cast<unsigned>((static_cast<int64_t>(e.raw) + Runs<Key>::kTile - 1) / Runs<Key>::kTile);
  uint32_t* totals = s.control;
  uint32_t* valid = totals + kMaxPasses * kDigits;
  uint32_t* fault = valid + 1;
  uint32_t* tickets = fault + 1;
  cudaError_t err = cudaMemsetAsync(
      s.control, 0, align256(kControlWords * 4) + static_cast<size_t>(look_words<Key>(e.raw, passes)) * 8, stream);
  if (err != cudaSuccess) return err;
  const unsigned lines = e.direct / e.kappa;
  digit_totals_kernel<Key><<<(lines + kSortThreads - 1) / kSortThreads, kSortThreads, 0, stream>>>(e, passes, totals);
  digit_bases_kernel<<<passes, kSortThreads, 0, stream>>>(totals, valid);
  for (int p = 0; p < passes; ++p) {
    Key* out = static_cast<Key*>(s.keys[p & 1]);
    const Key* in = static_cast<const Key*>(s.keys[1 - (p & 1)]);
    uint64_t* words = s.words + static_cast<int64_t>(p) * tiles * kDigits;
    if (p == 0) {
      radix_pass_kernel<Key, kKappa, true><<<tiles, kSortThreads, 0, stream>>>(
          e, in, s.weights[1], out, s.weights[0], totals, valid, 0, words, tickets, polls, fault);
    } else {
      radix_pass_kernel<Key, 0, false><<<tiles, kSortThreads, 0, stream>>>(
          e, in, s.weights[1 - (p & 1)], out, s.weights[p & 1], totals + p * kDigits, valid, p, words, tickets + p,
          polls, fault);
    }
  }
  const int last = (passes - 1) & 1;
  run_edges_kernel<Key><<<run_tiles, kSortThreads, 0, stream>>>(
      static_cast<const Key*>(s.keys[last]), s.weights[last], valid, e.position_bits, e.seq_len, capacity,
      s.words + static_cast<int64_t>(passes) * tiles * kDigits, tickets + kMaxPasses, polls, fault, edge_src, edge_dst,
      edge_weight, reinterpret_cast<unsigned long long*>(edge_count));
  return cudaGetLastError();
}

int bits_for(int64_t values) {
  int bits = 0;
  while ((1ll << bits) < values) ++bits;
  return bits;
}

}  // namespace
}  // namespace ckv

extern "C" {

int64_t ckv_adjacency_raw_edges(int64_t graphs, int64_t rows, int32_t kappa, double lam) {
  if (graphs <= 0 || rows <= 0 || kappa <= 0) return 0;
  const int64_t per_row = kappa + (lam < 1.0 ? static_cast<int64_t>(kappa) * (kappa + 1) / 2 : 0);
  return graphs * rows * per_row;
}

int64_t ckv_adjacency_scratch_bytes(int64_t graphs, int64_t rows, int32_t kappa, double lam) {
  const int64_t raw = ckv_adjacency_raw_edges(graphs, rows, kappa, lam);
  return raw > 0 ? ckv::carve(nullptr, raw).bytes : 0;
}

int ckv_build_adjacency_polls(const int32_t* topk_indices, const float* topk_scores, const int64_t* query_positions,
                              int32_t graphs, int64_t rows, int32_t kappa, int32_t seq_len, double lam,
                              int32_t* edge_src, int32_t* edge_dst, float* edge_weight, int64_t edge_capacity,
                              int64_t* edge_count, void* scratch, int64_t scratch_bytes, uint32_t look_polls,
                              void* cuda_stream) {
  if (!topk_indices || !topk_scores || !query_positions || !edge_src || !edge_dst || !edge_weight ||
      !edge_count || !scratch) {
    return CKV_ERR_NULL;
  }
  if (graphs <= 0 || rows <= 0 || kappa <= 0 || kappa > 64 || seq_len <= 0 || edge_capacity <= 0 ||
      !(lam >= 0.0 && lam <= 1.0)) {
    return CKV_ERR_SHAPE;
  }
  const int64_t vertices = static_cast<int64_t>(graphs) * seq_len;
  if (vertices >= (1ll << 31)) return CKV_ERR_CAPACITY;  // vertex ids are int32 in the output
  const int64_t raw = ckv_adjacency_raw_edges(graphs, rows, kappa, lam);
  if (raw >= (1ll << 32)) return CKV_ERR_CAPACITY;  // positions inside the sort are 32-bit
  const ckv::Scratch s = ckv::carve(scratch, raw);
  if (scratch_bytes < s.bytes) return CKV_ERR_CAPACITY;
  if (reinterpret_cast<uintptr_t>(scratch) % 256) return CKV_ERR_ALIGN;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  if (cudaMemsetAsync(edge_count, 0, sizeof(int64_t), stream) != cudaSuccess) return CKV_ERR_LAUNCH;
  ckv::EdgeRows e = {};
  e.indices = topk_indices;
  e.scores = topk_scores;
  e.positions = query_positions;
  e.rows = static_cast<uint32_t>(rows);
  e.direct = static_cast<uint32_t>(static_cast<int64_t>(graphs) * rows * kappa);
  e.raw = static_cast<uint32_t>(raw);
  e.kappa = kappa;
  e.seq_len = seq_len;
  e.position_bits = ckv::bits_for(seq_len);
  e.direct_scale = static_cast<float>(lam / 2.0);
  e.co_scale = static_cast<float>(1.0 - lam);
  const int bits = ckv::bits_for(graphs) + 2 * e.position_bits;  // at most 62: the vertex count is below 2^31
  auto run = [&](auto sorter) {
    return sorter(e, s, bits, look_polls, edge_capacity, edge_src, edge_dst, edge_weight, edge_count, stream) ==
                   cudaSuccess
               ? CKV_OK
               : CKV_ERR_LAUNCH;
  };
  if (bits <= 32 && 2 * e.position_bits < 32) {  // and no shift by the width of the key
    return kappa == 8 ? run(ckv::sort_and_merge<uint32_t, 8>) : run(ckv::sort_and_merge<uint32_t, 0>);
  }
  return kappa == 8 ? run(ckv::sort_and_merge<uint64_t, 8>) : run(ckv::sort_and_merge<uint64_t, 0>);
}

int ckv_build_adjacency(const int32_t* topk_indices, const float* topk_scores, const int64_t* query_positions,
                        int32_t graphs, int64_t rows, int32_t kappa, int32_t seq_len, double lam,
                        int32_t* edge_src, int32_t* edge_dst, float* edge_weight, int64_t edge_capacity,
                        int64_t* edge_count, void* scratch, int64_t scratch_bytes, void* cuda_stream) {
  return ckv_build_adjacency_polls(topk_indices, topk_scores, query_positions, graphs, rows, kappa, seq_len, lam,
                                   edge_src, edge_dst, edge_weight, edge_capacity, edge_count, scratch,
                                   scratch_bytes, ckv::kLookPolls, cuda_stream);
}

}  // extern "C"
