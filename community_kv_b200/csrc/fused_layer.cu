// One launch per decode layer: a thread-block cluster per (sequence, retrieval head).
//
// Grid (ctas, batch*R), cluster (ctas, 1, 1), 128 threads, three CTAs per SM.  With up to
// eight attention splits a CTA has one split; with more (the usual number for budgets above
// 4096 on few heads) a cluster of nine to sixteen CTAs may share them, up to two consecutive
// splits to a CTA.  The number of splits, and with it every bit of the result, does not
// depend on the number of CTAs.
//
// The CTAs of a cluster are co-scheduled, so they can hand work to one another
// through the hardware cluster barrier instead of through kernel boundaries:
//
//   1. every CTA scores a 1/ctas share of the unit's centroid rows, writes the
//      fp16 scores to the workspace and keeps its slice's keys, sizes and weighted
//      histogram in shared memory;
//   2. the budgeted selection runs across the cluster (select_cluster: three
//      cluster barriers, histograms and the descriptor list exchanged through
//      distributed shared memory); each CTA then resolves only the logical tokens
//      of its own attention splits to cache rows;
//   3. every CTA gathers and attends to its splits and writes their partial
//      (acc, max, sum) rows and neighbour candidates;         -- cluster barrier --
//   4. rank 0 merges the partials, writes the output and applies the online
//      graph update; the other CTAs have already left.
//
// The result is bit for bit the one of the four stand-alone kernels: the same
// device functions run in the same order on the same data.  The path needs per-CTA
// community slices that fit the selection's shared-memory stash.  A graph shared by several
// retrieval heads is updated by its leader while followers may still be reading it, which only a
// kernel boundary orders: step 4 is then a second launch, the merge kernel of the stand-alone path.

#include <atomic>

#include "merge_update.cuh"
#include "score_select.cuh"
#include "segmented_attention.cuh"

namespace ckv {

constexpr int kFusedThreads = 128;
constexpr int kFusedSmem = AttnSmem::kTotal > static_cast<int>(sizeof(ClusterSelectSmem))
                               ? AttnSmem::kTotal
                               : static_cast<int>(sizeof(ClusterSelectSmem));

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// kWide: more than eight CTAs, one or two consecutive splits each; else one CTA per split.
template <int kBlocks, bool kWide>
__global__ void __launch_bounds__(kFusedThreads, 3) decode_cluster_kernel(const ckv_layer_args a) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ UpdateDecision decision;
  __shared__ float lse_s;
  const int flat = blockIdx.y;
  const int rank = blockIdx.x;  // in the cluster
  const int ranks = kWide ? static_cast<int>(gridDim.x) : a.splits;
  // what a thread keeps in flight in the exchanges: sixteen ranks or rows each cost the usual launch
  // registers that it does not need (64 units of 6 CTAs: launch 44.5 -> 41.3 us with eight, of that
  // the merge 6.6 -> 4.6 and the threshold search 6.3 -> 5.4)
  constexpr int kRanks = kWide ? kMaxCluster : 8;
  pdl_release_dependents();
  // This CTA's share of the centroid table does not come from the kernel before it in
  // the stream (that one produces the query): ask for it in L2 while that kernel is
  // still finishing, before the wait below.
  {
    const int limit = score_limit(a, flat);
    const int groups = (limit + 15) / 16;
    const int first_row = 16 * static_cast<int>(static_cast<int64_t>(rank) * groups / ranks);
    const int last_row = min(limit, 16 * static_cast<int>(static_cast<int64_t>(rank + 1) * groups / ranks));
    const uint8_t* rows = reinterpret_cast<const uint8_t*>(a.centroids) +
                          (static_cast<int64_t>(flat) * a.community_capacity + first_row) * kHeadDim;
    for (int row = threadIdx.x; row < last_row - first_row; row += kFusedThreads) {
      asm volatile("prefetch.global.L2 [%0];" ::"l"(rows + static_cast<int64_t>(row) * kHeadDim));
    }
  }
  pdl_wait_for_predecessor();  // the query and last step's state come from upstream
  // ---- 1. centroid scores: this CTA's share of the unit's 16-row groups; the keys
  // stay in shared memory and are counted into the slice's histogram on the way ----
  ClusterSelectSmem& sm = *reinterpret_cast<ClusterSelectSmem*>(smem);
  const int groups = (score_limit(a, flat) + 15) / 16;
  const int first_group = static_cast<int>(static_cast<int64_t>(rank) * groups / ranks);
  const int last_group = static_cast<int>(static_cast<int64_t>(rank + 1) * groups / ranks);
  phase_stamp(a, flat, rank, 0);
  cluster_select_begin<kFusedThreads>(sm);
  // last step's threshold of this unit (-1 before the first step): its high byte is the guess
  int guess_bin = -1;
  if (a.threshold_state != nullptr) {
    const int previous = a.threshold_state[static_cast<int64_t>(flat) * 4];
    guess_bin = previous >= 0 ? (previous >> 8) & 0xff : -1;
  }
  {
    const ScoreSlice slice = {sm.key,       sm.size,      sm.hist_mass, sm.hist_count, first_group * 16,
                              sm.low_mass,  sm.low_count, guess_bin};
    score_groups<kFusedThreads, kClusterStageBytes>(a, flat, first_group, last_group, sm.query, &slice);
  }
  __syncthreads();
  phase_stamp(a, flat, rank, 1);

  // ---- 2. selection across the cluster, then the cache rows of this CTA's splits ----
  const int first_split = kWide ? rank * a.splits / ranks : rank;
  const int last_split = kWide ? (rank + 1) * a.splits / ranks : rank + 1;
  {
    const int steps_total = a.token_budget / kStepTokens;
    const int step_begin = static_cast<int>(static_cast<int64_t>(first_split) * steps_total / a.splits);
    const int step_end = static_cast<int>(static_cast<int64_t>(last_split) * steps_total / a.splits);
    const int row0 = first_group * 16;
    const int rows = min(score_limit(a, flat), last_group * 16) - row0;
    select_cluster<kFusedThreads, kRanks>(a, flat, sm, rank, ranks, row0, rows,
                                          step_begin * kStepTokens, step_end * kStepTokens, guess_bin);
  }
  __syncthreads();  // positions written above are read by other threads of this CTA
  phase_stamp(a, flat, rank, 6);

  // ---- 3. gather + attention over the splits ----
  if constexpr (kWide) {
#pragma unroll 1
    for (int split = first_split; split < last_split; ++split) {
      if (split > first_split) {
        __syncthreads();  // the last split's rows and candidates in shared memory have been read
      }
      attention_split<kBlocks>(a, flat, split, smem);
    }
  } else {
    attention_split<kBlocks>(a, flat, rank, smem);
  }
  phase_stamp(a, flat, rank, 7);
  if (a.flags & CKV_FLAG_ATTENTION_ONLY) {
    return;  // the launch behind this one merges; nothing reads another CTA's shared memory any more
  }
  cluster_arrive();  // release at cluster scope: the partials above are visible to rank 0
  if (rank != 0) {
    return;
  }
  cluster_wait();
  phase_stamp(a, flat, rank, 8);

  // ---- 4. merge, output, online update ----
  merge_update_unit<kRanks>(a, flat, kFusedThreads / 32 - 1, decision, lse_s);
  __syncthreads();
  phase_stamp(a, flat, rank, 9);
  if (flat == 0) {
    wait_for_peer_rows(a);
  }
}

namespace {

cudaError_t configure(int device) {
  static bool configured[64] = {};
  if (configured[device]) {
    return cudaSuccess;
  }
  cudaError_t err = cudaSuccess;
  auto prepare = [&](auto kernel, bool wide) {
    if (err == cudaSuccess) {
      err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFusedSmem);
    }
    if (err == cudaSuccess && wide) {
      err = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
  };
  prepare(decode_cluster_kernel<1, false>, false);
  prepare(decode_cluster_kernel<2, false>, false);
  prepare(decode_cluster_kernel<1, true>, true);
  configured[device] = err == cudaSuccess;
  return err;
}

struct FusedLaunch {
  cudaLaunchAttribute attributes[2];
  cudaLaunchConfig_t config = {};

  FusedLaunch(int ctas, int units, cudaStream_t stream) {
    config.gridDim = dim3(ctas, units);
    config.blockDim = dim3(kFusedThreads);
    config.dynamicSmemBytes = kFusedSmem;
    config.stream = stream;
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = ctas;
    attributes[0].val.clusterDim.y = 1;
    attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attributes;
    config.numAttrs = 2;
  }
};

// Clusters of `ctas` CTAs that are resident at once (0: such a cluster cannot run).  A property of
// the device and the kernel, asked for once; threads that ask at the same time store the same number.
int resident_clusters(int device, int ctas) {
  static std::atomic<int> known[64][kMaxCluster + 1];  // number + 1
  if (device < 0 || device >= 64) {
    return 0;
  }
  std::atomic<int>& slot = known[device][ctas];
  const int seen = slot.load(std::memory_order_relaxed);
  if (seen > 0) {
    return seen - 1;
  }
  int clusters = 0;
  int current = -1;
  if (cudaGetDevice(&current) == cudaSuccess && (current == device || cudaSetDevice(device) == cudaSuccess)) {
    if (configure(device) == cudaSuccess) {
      FusedLaunch launch(ctas, 1, nullptr);
      launch.config.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&clusters, decode_cluster_kernel<1, true>, &launch.config) != cudaSuccess) {
        clusters = 0;
      }
    }
    if (current != device) {
      cudaSetDevice(current);
    }
  }
  (void)cudaGetLastError();
  slot.store(clusters + 1, std::memory_order_relaxed);
  return clusters;
}

// CTAs per unit for more than eight splits; 0: the four kernels are the better route.  Measured
// with back-to-back layers of 4 query heads per unit, budget 8192, us a layer, four kernels / one
// launch, the results the same bits:
//  * one split per CTA, up to sixteen, wins at every number of communities (8 units, 16 splits:
//    512 communities 48.2 / 46.1, 2048 51.9 / 47.7, 16384 80.1 / 63.8) as long as the next layer's
//    clusters find room beside this one's: 30 units of 11 CTAs 73.2 / 70.0, but 27 units of 13
//    69.6 / 73.7, 30 of 12 71.0 / 99.2, 39 of 10 77.0 / 98.4, 45 of 9 80.8 / 120.8.  Hence at most
//    three quarters of the CTA slots.
//  * two splits per CTA cost a second pass of the gather's latency, which only the selection of very
//    many communities by a single CTA outweighs: 8 units, 32 splits: 2048 communities 48.4 / 56.5,
//    8192 56.9 / 62.1, 14336 67.0 / 71.2, 16384 77.2 / 72.1, 32768 184.1 / 91.9.
//  * with more than eight query heads per unit the launch has to score two blocks of heads on few
//    CTAs: 8 units of 16 heads, 16 splits: 8192 communities 86.8 / 97.3, 16384 120.8 / 131.1.
constexpr int kCtaSlots = 3 * 148;
constexpr int kManyCommunities = 16384;

int wide_ctas(const ckv_layer_args& a) {
  if (a.group_size > 8 || (a.splits > kMaxCluster && a.community_capacity < kManyCommunities)) {
    return 0;
  }
  const int ctas = a.splits > kMaxCluster ? (a.splits + 1) / 2 : a.splits;
  const int units = a.batch * a.retrieval_heads;
  return 4 * units * ctas <= 3 * kCtaSlots && resident_clusters(a.device, ctas) >= units ? ctas : 0;
}

}  // namespace

// Graphs shared by several heads take two launches, merge and update in the second.  Beside four they
// save the host two launches and win with more than eight splits; up to eight the scores of few
// communities are faster over the whole chip, and from about one cluster CTA per SM on the merge's CTAs
// find their place late.  One graph for all heads, a row appended and a layer decoded, us in a captured
// graph (eager), four kernels / two launches:
//    4 heads, budget 512, 4 splits, 100 communities   26.0 (27.4) / 28.4 (28.9)
//    4 heads, budget 1024, 8 splits, 1000 communities 32.1 (34.3) / 31.8 (32.3)
//    8 heads, budget 2048, 8 splits, 2000 communities 35.8 (38.0) / 35.8 (36.7)
//   12 heads, budget 1024, 8 splits, 500 communities  30.1 (31.7) / 30.8 (31.4)
//   16 heads, the same                                30.6 (33.0) / 33.3 (33.9)
//   64 heads, the same in 6 splits                    41.0 (42.7) / 46.7 (49.8)
//    6 heads, budget 8192, 16 splits, 2000 communities 44.2 (46.9) / 37.8 (39.0)
constexpr int kSharedCtas = 96;

// CTAs per unit of the one launch; 0: the stand-alone kernels run.
int fused_layer_ctas(const ckv_layer_args& a) {
  if (a.splits < 1 || a.splits > 2 * kMaxCluster ||
      (a.flags & (CKV_FLAG_ATTENTION_ONLY | CKV_FLAG_UPDATE_ONLY | CKV_FLAG_UNFUSED | CKV_FLAG_FP32_CENTROIDS))) {
    return 0;
  }
  const int ctas = a.splits <= 8 ? a.splits : wide_ctas(a);
  if (ctas == 0) {
    return 0;
  }
  if (a.splits <= 8 && a.graphs != a.retrieval_heads && !(a.flags & CKV_FLAG_SKIP_UPDATE) &&
      a.batch * a.retrieval_heads * ctas > kSharedCtas) {
    return 0;
  }
  // every CTA stages the rows it scores: a 1/ctas share of the 16-row groups
  const int groups = (a.community_capacity + 15) / 16;
  return 16 * ((groups + ctas - 1) / ctas) <= kStash ? ctas : 0;
}

cudaError_t launch_fused_layer(const ckv_layer_args& a, int ctas, cudaStream_t stream) {
  const cudaError_t err = configure(a.device >= 0 && a.device < 64 ? a.device : 0);
  if (err != cudaSuccess) return err;
  FusedLaunch launch(ctas, a.batch * a.retrieval_heads, stream);
  auto run = [&](auto kernel) { return cudaLaunchKernelEx(&launch.config, kernel, a); };
  if (a.splits > 8) {
    return run(decode_cluster_kernel<1, true>);
  }
  return a.group_size > 8 ? run(decode_cluster_kernel<2, false>) : run(decode_cluster_kernel<1, false>);
}

}  // namespace ckv
