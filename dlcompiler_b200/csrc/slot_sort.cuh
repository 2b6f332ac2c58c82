// Stable counting sort of routed (token, k) slots by expert, by one thread-block cluster.
//
// The slots are cut into one contiguous segment per warp, in order over the cluster's CTAs.  Every warp
// counts its segment into its own row of a shared-memory table, the table's columns become exclusive
// prefix sums, the CTAs of the cluster exchange their column totals through distributed shared memory,
// and every warp then walks its segment again with its own running counters.  A slot's position follows
// from prefix sums and warp match masks alone, so the order is stable and the result reproducible.
//
// Why a cluster and why a segment per warp: with one CTA that placed 1024 slots per round behind three block
// barriers and an E x 32 scan, 32768 slots took 274 us and 16000 slots over 256 experts 100 us on B200 (the
// serial loops over experts and blocks included); with the walk below, which has no barrier inside and is shared
// by the SMs of a cluster, 16000 slots take 9.7 us and the whole capacity-limited gate behind 32768 slots 22 us.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"

namespace dlb {

constexpr int SORT_THREADS = 1024;
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int SORT_MAX_CLUSTER = 8;     // the portable cluster size

// CTAs for `numel` slots: a warp's segment is at most two rounds of 32 slots up to 16384 slots, with eight CTAs; it grows
// with the slots after that.
inline int sort_cluster_size(int64_t numel) {
  int c = 1;
  while (c < SORT_MAX_CLUSTER && numel > (int64_t)c * 2048) c <<= 1;
  return c;
}
// Row pitch of the table: odd, so that a column walk touches 32 different banks.
__host__ __device__ constexpr int sort_pitch(int experts) { return experts | 1; }
constexpr int SORT_MAX_EXPERTS = 1024;
constexpr size_t sort_smem_ints(int experts) {
  return (size_t)SORT_WARPS * sort_pitch(experts) + 4 * (size_t)experts + 1 + 2 * SORT_WARPS;
}

struct SlotSort {
  int experts, pitch;
  int* table;       // [SORT_WARPS][pitch] counts, then the running position of each warp inside the CTA
  int* total;       // [E] slots of the expert in this CTA's segments (read by the cluster's other CTAs)
  int* count;       // [E] slots of the expert in all segments
  int* before;      // [E] slots of the expert in the segments of earlier CTAs
  int* start;       // [E + 1] exclusive prefix of a per-expert size (block_scan)
  int* scratch;     // [2 * SORT_WARPS]
  int lo, hi;       // this warp's segment
  int rank, ctas;

  __device__ __forceinline__ SlotSort(int* smem, int num_experts, int numel) {
    experts = num_experts;
    pitch = sort_pitch(num_experts);
    table = smem;
    total = table + SORT_WARPS * pitch;
    count = total + experts;
    before = count + experts;
    start = before + experts;
    scratch = start + experts + 1;
    auto cl = cooperative_groups::this_cluster();
    rank = (int)cl.block_rank();
    ctas = (int)cl.num_blocks();
    const int warps = ctas * SORT_WARPS, w = rank * SORT_WARPS + (threadIdx.x >> 5);
    const int seg = ((numel + warps - 1) / warps + 31) & ~31;
    lo = min(numel, w * seg);        // numel < 2^30 and seg is its share rounded up: no overflow
    hi = min(numel, lo + seg);
    for (int i = threadIdx.x; i < SORT_WARPS * pitch; i += SORT_THREADS) table[i] = 0;
    __syncthreads();
  }

  // Calls f(slot, expert or -1, live) for the warp's slots, 32 at a time, the ids fetched four rounds ahead.
  template <typename IdAt, typename F> __device__ __forceinline__ void walk(IdAt id_at, F f) const {
    const int lane = threadIdx.x & 31;
    for (int base = lo; base < hi; base += 128) {
      int e[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int slot = base + j * 32 + lane;
        e[j] = slot < hi ? id_at(slot) : -1;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (base + j * 32 < hi) f(base + j * 32 + lane, e[j]);
    }
  }

  // Fills count / before (all CTAs of the cluster take part).  The caller must keep the CTA alive until every
  // other CTA has passed its own call: finish().
  template <typename IdAt> __device__ __forceinline__ void count_slots(IdAt id_at) {
    int* mine = table + (threadIdx.x >> 5) * pitch;
    walk(id_at, [&](int, int e) {
      if (e >= 0) atomicAdd(&mine[e], 1);      // integer adds commute: still reproducible
    });
    __syncthreads();
    // exclusive prefix over the warps of every column: one warp per column, lane = warp
    const int lane = threadIdx.x & 31;
    for (int e = threadIdx.x >> 5; e < experts; e += SORT_WARPS) {
      const int c = table[lane * pitch + e];
      int inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      table[lane * pitch + e] = inc - c;
      if (lane == 31) total[e] = inc;
    }
    auto cl = cooperative_groups::this_cluster();
    __syncthreads();
    if (ctas > 1) cl.sync();
    for (int e = threadIdx.x; e < experts; e += SORT_THREADS) {
      int all = 0, pre = 0;
      for (int r = 0; r < ctas; ++r) {
        const int v = *cl.map_shared_rank(&total[e], r);
        all += v;
        pre += r < rank ? v : 0;
      }
      count[e] = all;
      before[e] = pre;
    }
    __syncthreads();
    if (ctas > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }

  // After this no CTA reads another's totals any more; global writes of the cluster's CTAs before their
  // count_slots() are visible.
  __device__ __forceinline__ void finish() const {
    __syncthreads();      // the wait is a warp-aligned instruction: loops before it may have left lanes apart
    if (ctas > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }

  // start[e] = sum of size(e') over e' < e, start[E] = the sum of all.
  template <typename Size> __device__ __forceinline__ void block_scan(Size size) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, e = threadIdx.x;   // experts <= SORT_THREADS
    const int c = e < experts ? size(e) : 0;
    int inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) scratch[warp] = inc;
    __syncthreads();
    int add = 0;
    {
      int t = scratch[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += v;
      }
      add = __shfl_sync(0xffffffffu, t, (warp + 31) & 31);
      if (warp == 0) add = 0;
      if (threadIdx.x == SORT_THREADS - 1) start[experts] = t;
    }
    if (e < experts) start[e] = add + inc - c;
    __syncthreads();
  }

  // Calls f(slot, expert, position among the expert's slots) for every slot of a valid expert.
  template <typename IdAt, typename F> __device__ __forceinline__ void place(IdAt id_at, F f) {
    const int lane = threadIdx.x & 31;
    int* mine = table + (threadIdx.x >> 5) * pitch;
    walk(id_at, [&](int slot, int e) {
      const unsigned peers = __match_any_sync(0xffffffffu, e);
      const int rank_in_warp = __popc(peers & ((1u << lane) - 1u));
      int at = 0;
      if (e >= 0) at = mine[e];
      __syncwarp();
      if (e >= 0 && rank_in_warp == 0) mine[e] = at + __popc(peers);
      __syncwarp();
      if (e >= 0) f(slot, e, before[e] + at + rank_in_warp);
    });
  }
};

// Launches `kern` as one cluster of `ctas` CTAs with `smem` bytes of dynamic shared memory.  The kernel's limit is set to
// `max_smem`, the most that any call of it takes: the limit belongs to the process, and a call that set it to its own
// need could lower it between another thread's setting and launch.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_one_cluster(void (*kern)(KArgs...), int ctas, size_t smem, size_t max_smem,
                                      cudaStream_t stream, Args... args) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(SORT_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace dlb
