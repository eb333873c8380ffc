// Split merge (log-sum-exp) + online community assignment + centroid maintenance.
//
// One CTA of 160 threads per (sequence, retrieval head).  Each of the first four
// warps merges the split partials of one query head at a time with independent
// 16-byte loads.  The fifth warp of the CTA whose head leads its graph merges the per-split
// neighbour candidates into the global top-8, applies the modularity-gain rule
// and updates the graph state in place; it is the single writer of that graph.  Where several
// heads share the graph the same CTA then updates the other heads' tables.

#include "merge_update.cuh"

namespace ckv {

constexpr int kFollowersInFlight = 4;
constexpr int kUpdateMaxThreads = 512;

// The other heads of a graph shared by several retrieval heads take the leader's assignment over into
// their own tables.  The CTA that has just updated the graph does it: what it needs of the decision is
// still in shared memory, and a launch of its own (2.7 us and the gap in front of it) is saved.  Nothing
// else of the launch reads those tables.  Bound by the latency of the rows and the divisions behind
// them: a warp takes a head and has four in flight (eight were slower: 64 heads 18 instead of 12 us),
// and launch_merge_update adds warps for more than twenty heads.
__device__ __forceinline__ void sync_followers(const ckv_layer_args& a, int flat, const UpdateDecision& decision) {
  constexpr int kInFlight = kFollowersInFlight;
  constexpr int kPieces = kHeadDim / 32;  // dimensions lane, lane + 32, ... of a head
  const Unit u = make_unit(a, flat);
  if (u.head != u.graph || decision.overflow != 0) {
    return;
  }
  const int warps = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  const bool wide = (a.flags & CKV_FLAG_FP32_CENTROIDS) != 0;
  const bool reference_division = (a.flags & CKV_FLAG_REFERENCE_DIVISION) != 0;
  for (int base = threadIdx.x >> 5; base < a.retrieval_heads; base += warps * kInFlight) {
    bool follows[kInFlight];
    int64_t index[kInFlight];  // of the community in the head's tables
    int size[kInFlight];
    float key_value[kInFlight][kPieces], old_value[kInFlight][kPieces];
#pragma unroll
    for (int i = 0; i < kInFlight; ++i) {
      const int head = min(base + i * warps, a.retrieval_heads - 1);
      const int other = u.batch * a.retrieval_heads + head;
      follows[i] = base + i * warps < a.retrieval_heads && head != u.head && a.retrieval_to_graph[head] == u.graph;
      index[i] = static_cast<int64_t>(other) * a.community_capacity + decision.assigned;
      size[i] = a.community_sizes[index[i]];
      const __nv_bfloat16* key_row =
          a.current_key != nullptr
              ? reinterpret_cast<const __nv_bfloat16*>(a.current_key) + static_cast<int64_t>(other) * kHeadDim
              : reinterpret_cast<const __nv_bfloat16*>(a.key) + u.batch * a.key_batch_stride +
                    a.retrieval_to_kv[head] * a.key_head_stride +
                    static_cast<int64_t>(decision.current) * a.key_row_stride;
#pragma unroll
      for (int k = 0; k < kPieces; ++k) {
        key_value[i][k] = __bfloat162float(key_row[lane + 32 * k]);
        if (wide) {
          old_value[i][k] = reinterpret_cast<const float*>(a.centroids)[index[i] * kHeadDim + lane + 32 * k];
        } else {
          const __half_raw raw = __nv_cvt_fp8_to_halfraw(
              reinterpret_cast<const __nv_fp8_storage_t*>(a.centroids)[index[i] * kHeadDim + lane + 32 * k], __NV_E4M3);
          old_value[i][k] = __half2float(*reinterpret_cast<const __half*>(&raw));
        }
      }
    }
    __syncwarp();  // every lane has read the sizes
#pragma unroll
    for (int i = 0; i < kInFlight; ++i) {
      if (!follows[i]) {
        continue;
      }
      if (lane == 0) {
        a.community_sizes[index[i]] = size[i] + 1;
        a.community_counts[u.batch * a.retrieval_heads + base + i * warps] = decision.count;
      }
#pragma unroll
      for (int k = 0; k < kPieces; ++k) {
        const float updated = size[i] > 0 ? centroid_mean(old_value[i][k], size[i], key_value[i][k], reference_division)
                                          : key_value[i][k];
        if (wide) {
          reinterpret_cast<float*>(a.centroids)[index[i] * kHeadDim + lane + 32 * k] = updated;
        } else {
          reinterpret_cast<__nv_fp8_storage_t*>(a.centroids)[index[i] * kHeadDim + lane + 32 * k] =
              __nv_cvt_float_to_fp8(updated, __NV_SATFINITE, __NV_E4M3);
        }
      }
    }
  }
}

// kFollowers: several heads share a graph (a kernel of its own, so that the other keeps its registers).
template <bool kFollowers>
__global__ void __launch_bounds__(kFollowers ? kUpdateMaxThreads : kMergeThreads + 32)
    merge_update_kernel(const ckv_layer_args a) {
  __shared__ UpdateDecision decision;
  __shared__ float lse_s;
  pdl_release_dependents();
  pdl_wait_for_predecessor();  // partials and candidates come from the attention kernel
  merge_update_unit<8>(a, blockIdx.x, kMergeThreads / 32, decision, lse_s);
  if constexpr (kFollowers) {
    sync_followers(a, blockIdx.x, decision);
  }
  if (blockIdx.x == 0) {
    wait_for_peer_rows(a);
  }
}

// One warp per unit and pass: lanes 0-15 copy the 256-byte key row, lanes 16-31 the value row.
// Bound by launches and latency (a few kilobytes move), so it is launched early under the kernel
// before it, and with `cursor` it also moves the shared cursor on, which was a launch of its own: one
// CTA then does all the units, so that every row is placed before the cursor changes.  That holds up to
// kOneCtaUnits units; more take the rows and the cursor in two launches.  Six layers of
// 32 heads, budget 4096, a token through the plug-in: 328 -> 292 us; of 8 heads, budget 2048: 245 ->
// 214 us; the launch early alone, four layers of 3 sequences: 138 -> 128 us.  Dependents are
// released behind the wait: released in front of it, the next layer's clusters settle between those
// of the layer still running (32 heads: 309 us; one layer of a million tokens: 75 instead of 66 us).
__global__ void append_kv_kernel(uint4* key_cache, uint4* value_cache, const uint4* new_key, const uint4* new_value,
                                 int64_t units, int64_t unit_stride_vec, const int32_t* row_index,
                                 int64_t row_index_stride, int64_t row, int64_t rows, int32_t* cursor) {
  pdl_wait_for_predecessor();  // the fresh rows and the cursor come from upstream, earlier reads of the row too
  pdl_release_dependents();
  const int lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  const int piece = lane & 15;
  uint4* cache = lane < 16 ? key_cache : value_cache;
  const uint4* fresh = lane < 16 ? new_key : new_value;
  for (int64_t unit = static_cast<int64_t>(blockIdx.x) * warps + (threadIdx.x >> 5); unit < units;
       unit += static_cast<int64_t>(gridDim.x) * warps) {
    const uint4 held = fresh[unit * (kHeadDim * 2 / 16) + piece];
    const int64_t target =
        cursor != nullptr ? *cursor : (row_index != nullptr ? row_index[unit * row_index_stride] : row);
    if (target >= 0 && target < rows) {
      cache[unit * unit_stride_vec + target * (kHeadDim * 2 / 16) + piece] = held;
    }
  }
  if (cursor != nullptr) {
    __syncthreads();
    if (threadIdx.x == 0) {
      *cursor += 1;
    }
  }
}

// Us a call in a captured graph, one CTA for rows and cursor / two launches: 8 units 1.6, 64 2.4,
// 128 3.1, 256 4.6 / 2.2, 512 7.3 / 2.4, 4096 45 / 3.1.  The second launch costs the host 2 us.
constexpr int64_t kOneCtaUnits = 128;

cudaError_t launch_append_kv(void* key_cache, void* value_cache, const void* new_key, const void* new_value,
                             int64_t units, int64_t unit_stride, const int32_t* row_index,
                             int64_t row_index_stride, int64_t row, int32_t* cursor, cudaStream_t stream) {
  // a row that only the device knows may lie behind the unit's last; the caller has seen any other
  const int64_t rows = cursor != nullptr || row_index != nullptr ? unit_stride / kHeadDim : row + 1;
  auto run = [&](unsigned ctas, unsigned warps, int64_t count, const int32_t* index, int32_t* moved) {
    return launch_dependent(append_kv_kernel, dim3(ctas), dim3(32u * warps), 0, stream, static_cast<uint4*>(key_cache),
                            static_cast<uint4*>(value_cache), static_cast<const uint4*>(new_key),
                            static_cast<const uint4*>(new_value), count, unit_stride / 8, index, row_index_stride, row,
                            rows, moved);
  };
  const unsigned ctas = static_cast<unsigned>((units + 3) / 4);
  if (cursor == nullptr) {
    return run(ctas, 4u, units, row_index, nullptr);
  }
  if (units <= kOneCtaUnits) {
    return run(1u, units < 4 ? 4u : static_cast<unsigned>(units < 32 ? units : 32), units, nullptr, cursor);
  }
  const cudaError_t err = run(ctas, 4u, units, cursor, nullptr);
  return err == cudaSuccess ? run(1u, 1u, 0, nullptr, cursor) : err;
}

// One thread polls this GPU's counter a bounded number of times.
// Launched with programmatic stream serialisation: it may start (and poll) while the
// kernel before it in the stream is still running, and it only ends once that kernel
// has completed, so whatever follows sees both the local and the peers' rows.
__global__ void wait_peers_kernel(uint32_t* flag, uint32_t expected, uint32_t* status) {
  pdl_release_dependents();
  constexpr uint32_t kPolls = 1u << 22;  // about two seconds with the back-off below
  bool arrived = false;
  for (uint32_t poll = 0; poll < kPolls; ++poll) {
    uint32_t seen;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(flag) : "memory");
    if (seen >= expected) {
      atomicSub(flag, expected);
      arrived = true;
      break;
    }
    if (poll > 256) {
      __nanosleep(500);
    }
  }
  if (!arrived && status != nullptr) {
    atomicOr(status, CKV_DEV_WAIT_TIMEOUT);
  }
  pdl_wait_for_predecessor();
}

cudaError_t launch_wait_peers(uint32_t* flag, uint32_t expected, uint32_t* status, cudaStream_t stream) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(1);
  config.blockDim = dim3(1);
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, wait_peers_kernel, flag, expected, status);
}

// Nearest-centroid assignment variant: per leader head, the live community whose centroid
// has the largest inner product with the key of the token being decoded (the fp16 value the
// scoring kernel would give a query group made of that key; first maximum).  Eight lanes
// share a centroid row, every product and sum rounded on its own in the scoring kernels'
// fixed order, so a CPU reproduces the choice bit for bit.
// Bound by the latency of the rows: one CTA per head with one row per thread at a time made a
// round trip to memory per 32 communities.  A cluster of eight CTAs now shares a head, four
// rows in flight per thread (1024 communities per round trip), and rank 0 collects
// the eight bests through distributed shared memory.  Four layers of 8 heads and 1500
// communities: 378 -> 234 us a token.
constexpr int kNearestThreads = 256;
constexpr int kNearestCluster = 8;
constexpr int kNearestInFlight = 4;

__global__ void __launch_bounds__(kNearestThreads) nearest_centroid_kernel(const ckv_layer_args a,
                                                                          int32_t* forced) {
  __shared__ unsigned long long warp_best[kNearestThreads / 32];
  __shared__ unsigned long long cta_best[kNearestCluster];  // rank 0's collects
  const int flat = blockIdx.y;
  const int rank = blockIdx.x;
  const Unit u = make_unit(a, flat);
  pdl_release_dependents();
  pdl_wait_for_predecessor();  // the key row and the last step's state come from upstream
  if (u.head != u.graph) {
    return;  // followers of a shared graph take the leader's choice; the whole cluster leaves
  }
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // waited for before the first remote store
  const int capacity = a.community_capacity;
  const int64_t graph_slot = static_cast<int64_t>(u.batch) * a.graphs + u.graph;
  const int current = min(max(a.current_position[graph_slot], 0), a.sequence_capacity - 1);
  const __nv_bfloat16* key_row =
      a.current_key != nullptr
          ? reinterpret_cast<const __nv_bfloat16*>(a.current_key) + static_cast<int64_t>(flat) * kHeadDim
          : reinterpret_cast<const __nv_bfloat16*>(a.key) + u.batch * a.key_batch_stride +
                u.kv * a.key_head_stride + static_cast<int64_t>(current) * a.key_row_stride;
  const int slice = threadIdx.x & 7;
  float q[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    q[k] = __bfloat162float(key_row[slice * 16 + k]);
  }
  const bool wide = (a.flags & CKV_FLAG_FP32_CENTROIDS) != 0;
  const int count = min(a.community_counts[flat], capacity);
  const int32_t* sizes = a.community_sizes + static_cast<int64_t>(flat) * capacity;
  unsigned long long best = 0ull;  // (ordered fp16 key + 1) << 32 | ~row : the first maximum wins
  constexpr int kRows = kNearestThreads / 8;
  constexpr int kStep = kRows * kNearestCluster;
  for (int base = rank * kRows; base < count; base += kNearestInFlight * kStep) {
    float4 held[kNearestInFlight][4];  // a row's slice: 16 floats, or 16 bytes in the first
    int size[kNearestInFlight];
#pragma unroll
    for (int i = 0; i < kNearestInFlight; ++i) {
      size[i] = 0;
      if (base + i * kStep < count) {
        const int row = base + i * kStep + (threadIdx.x >> 3);
        const int64_t element =
            (static_cast<int64_t>(flat) * capacity + min(row, capacity - 1)) * kHeadDim + slice * 16;
        if (wide) {
          const float4* source = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.centroids) + element);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            held[i][k] = source[k];
          }
        } else {
          held[i][0] = *reinterpret_cast<const float4*>(reinterpret_cast<const uint8_t*>(a.centroids) + element);
        }
        size[i] = row < count ? sizes[row] : 0;
      }
    }
#pragma unroll
    for (int i = 0; i < kNearestInFlight; ++i) {
      if (base + i * kStep >= count) {
        break;  // the same for the whole CTA: every lane takes part in the shuffles
      }
      float x[16];
      if (wide) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          x[4 * k] = held[i][k].x;
          x[4 * k + 1] = held[i][k].y;
          x[4 * k + 2] = held[i][k].z;
          x[4 * k + 3] = held[i][k].w;
        }
      } else {
        const uint32_t words[4] = {__float_as_uint(held[i][0].x), __float_as_uint(held[i][0].y),
                                   __float_as_uint(held[i][0].z), __float_as_uint(held[i][0].w)};
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const __half_raw half = __nv_cvt_fp8_to_halfraw(
              static_cast<__nv_fp8_storage_t>((words[k >> 2] >> (8 * (k & 3))) & 0xffu), __NV_E4M3);
          x[k] = __half2float(*reinterpret_cast<const __half*>(&half));
        }
      }
      float acc = __fmul_rn(x[0], q[0]);
#pragma unroll
      for (int k = 1; k < 16; ++k) {
        acc = __fadd_rn(acc, __fmul_rn(x[k], q[k]));
      }
      acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 4));
      acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 2));
      acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 1));
      if (size[i] > 0) {
        const int row = base + i * kStep + (threadIdx.x >> 3);
        uint16_t bits = __half_as_ushort(__float2half_rn(acc));
        bits = bits == 0x8000u ? 0u : bits;  // -0 and +0 compare equal
        const unsigned long long key = static_cast<unsigned long long>(ordered_key16(bits)) + 1ull;
        const unsigned long long packed = (key << 32) | (0xffffffffull - static_cast<unsigned long long>(row));
        best = packed > best ? packed : best;
      }
    }
  }
  best = warp_max_u64(best);
  if ((threadIdx.x & 31) == 0) {
    warp_best[threadIdx.x >> 5] = best;
  }
  __syncthreads();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (threadIdx.x == 0) {
    for (int w = 1; w < kNearestThreads / 32; ++w) {
      best = warp_best[w] > best ? warp_best[w] : best;
    }
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(cta_best + rank)), "r"(0));
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote), "l"(best) : "memory");
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (rank == 0 && threadIdx.x == 0) {
    best = 0ull;
    for (int r = 0; r < kNearestCluster; ++r) {
      best = cta_best[r] > best ? cta_best[r] : best;
    }
    forced[graph_slot] =
        best == 0ull ? -1 : static_cast<int32_t>(0xffffffffull - (best & 0xffffffffull));
  }
}

cudaError_t launch_nearest_centroid(const ckv_layer_args& a, int32_t* forced, cudaStream_t stream) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(kNearestCluster, a.batch * a.retrieval_heads);
  config.blockDim = dim3(kNearestThreads);
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = kNearestCluster;
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = 2;
  return cudaLaunchKernelEx(&config, nearest_centroid_kernel, a, forced);
}

// Warps beyond the five of the merge only serve the followers of a shared graph.  As many as have all of
// them in flight, but no more than leave every CTA resident at once (16 warps per SM at this kernel's
// registers).  One graph for all heads, the update alone in a captured graph, us, a launch of its own for
// the followers / five warps / so: 16 heads 6.8 / 6.3 / 6.1, 32 heads 7.2 / 8.4 / 6.5, 64 heads
// 7.2 / 12.3 / 7.2.  A whole CTA per head, four heads in flight, took 15.2, 27 and 51.
cudaError_t launch_merge_update(const ckv_layer_args& a, cudaStream_t stream) {
  const int units = a.batch * a.retrieval_heads;
  const int fewest = kMergeThreads / 32 + 1;
  if (a.retrieval_heads == a.graphs || (a.flags & CKV_FLAG_SKIP_UPDATE)) {
    return launch_dependent(merge_update_kernel<false>, dim3(units), dim3(32 * fewest), 0, stream, a);
  }
  const int wanted = (a.retrieval_heads + kFollowersInFlight - 1) / kFollowersInFlight;
  const int most = min(kUpdateMaxThreads / 32, 148 * (kUpdateMaxThreads / 32) / units);
  const int warps = max(fewest, min(wanted, most));
  return launch_dependent(merge_update_kernel<true>, dim3(units), dim3(32 * warps), 0, stream, a);
}

}  // namespace ckv
