// The small per-batch passes around a decode: the queue order of the relay legs and
// the result arrays made from the decode's counts and exact weights.
//
// The reference's host code makes them with a handful of torch operations
// (src/pelagos/decoder.py:3839-3873); so did this library's.  Each is a launch of 2-3 us
// on the device and 4-5 us on the host, a dozen of them and a radix sort per call: more
// than the decode of a small batch.  Here each is one launch.  What bounds them is the
// latency of the ordered compaction, a block's rounds of up to 16,384 counts (a warp takes up to
// 512, loads and stores contiguous, ranks from ballots); the rest of a launch's blocks make the
// elementwise results beside it.  From CLUSTER_FROM shots on a cluster of blocks shares the
// walk: each takes a contiguous part, counts it, reads the others' counts from their shared
// memory and compacts its own.  us per call, torch operations / one block for all in rounds of 4,096 /
// now: order of 65,536 shots 87 / 45 / 22, of 1,048,576 97 / 498 / 63, of 4,194,304 157 / 1,947 / 205;
// results 113 / 55 / 43, 111 / 223 / 64, 148 / 778 / 139.

#include "relaybp.h"
#include "relaybp_host.h"

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>

namespace {

namespace cg = cooperative_groups;
using rbph::fail;

constexpr int FT = 1024;  // threads
constexpr int CLUSTER = 8;
// Shots per thread in a compacting block's round (PER): few where one round takes the batch, since a round's
// instructions are the time then.  Order / results on the device: one shot 2.1 / 1.7 us (with 16 per thread, and
// the parts' sizes in 64 bits, 4.7 / 3.3), 16,384 shots 8.0 / 3.9, 32,768 and 65,536 in a cluster 9.9 / 6.8 (32,768
// in one block 14.4 / 6.5).
constexpr int PER_SMALL = 4, PER_LARGE = 16;
constexpr int64_t LARGE_FROM = 2 * PER_SMALL * FT;
constexpr int64_t CLUSTER_FROM = 2 * PER_LARGE * FT;

// The compacting blocks' parts of the B shots: whole rounds, so that loads stay aligned.
struct Part {
  long long i0, i1;
};
template <int PER>
__device__ __forceinline__ Part part_of(long long B, unsigned rank, unsigned n) {
  if (n == 1) return {0, B};
  const unsigned rounds = (unsigned)((B + PER * FT - 1) / (PER * FT));
  const long long each = (long long)((rounds + n - 1) / n) * (PER * FT), i0 = min(B, each * rank);
  return {i0, min(B, i0 + each)};
}

// A warp's PER x 32 counts of a round: bit l of below[k] tells whether found[i + 32 k + l] < limit (past the
// part's end: not), i the warp's first shot.  The loads are contiguous and all in flight; returns the bits' number.
template <int PER>
__device__ __forceinline__ int load_round(const int* found, long long i, long long end, int limit, uint32_t (&below)[PER]) {
  if (i >= end) return 0;  // the whole warp
  int v[PER], n = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const long long at = i + 32 * k + (threadIdx.x & 31);
    v[k] = at < end ? found[at] : limit;
  }
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    below[k] = __ballot_sync(0xffffffffu, v[k] < limit);
    n += __popc(below[k]);
  }
  return n;
}

// Number of found[i] < limit in the part (valid in every thread).
template <int PER>
__device__ __forceinline__ int count_below(const int* found, Part p, int limit, int* counter) {
  if (threadIdx.x == 0) *counter = 0;
  __syncthreads();
  int mine = 0;
  uint32_t below[PER];
  for (long long i = p.i0 + (threadIdx.x >> 5) * (32 * PER); i < p.i1; i += PER * FT)
    mine += load_round<PER>(found, i, p.i1, limit, below);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(counter, mine);
  __syncthreads();
  return *counter;
}

// Exclusive prefix sum of the warps' n, and the block's total in *total.
__device__ __forceinline__ int warps_scan(int n, int* warp_sum, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();  // the last round's sums have been read
  if (lane == 0) warp_sum[warp] = n;
  __syncthreads();
  const int w = warp_sum[lane];  // FT / 32 = 32 warps
  int ws = w;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, ws, o);
    if (lane >= o) ws += t;
  }
  *total = __shfl_sync(0xffffffffu, ws, 31);
  return __shfl_sync(0xffffffffu, ws - w, warp);
}

// The cluster's counts of the parts before this block's, and of all parts in *all.  A cluster of one
// block needs neither.
__device__ __forceinline__ int cluster_base(const cg::cluster_group& cluster, int* counter, int* all) {
  cluster.sync();  // every block's counter is final
  int before = 0, sum = 0;
  const unsigned rank = cluster.block_rank();
  for (unsigned r = 0; r < cluster.num_blocks(); ++r) {
    const int c = *cluster.map_shared_rank(counter, r);
    before += r < rank ? c : 0;
    sum += c;
  }
  cluster.sync();  // no block leaves while another reads its counter
  *all = sum;
  return before;
}

// The first cluster: the indices of shots with found < stop_nconv in ascending order, and their number.
// Other blocks: weights from the exact fixed-point weight (2^-32 units; +inf where there is
// none) and the mask found >= stop_nconv.
template <int PER>
__global__ void __launch_bounds__(FT) results_kernel(const int* found, const long long* wfix, long long B, int S,
                                                     float* w32, double* w64, uint8_t* valid, int* idx, int* count) {
  const cg::cluster_group cluster = cg::this_cluster();
  const unsigned n = cluster.num_blocks();
  if (blockIdx.x >= n) {
    const long long i = (blockIdx.x - n) * (long long)FT + threadIdx.x;
    if (i >= B) return;
    const long long w = wfix[i];
    const double x = w == LLONG_MAX ? __longlong_as_double(0x7ff0000000000000ll)
                                    : __ll2double_rn(w) * 2.3283064365386963e-10;  // 2^-32
    if (w64) w64[i] = x;
    else w32[i] = __double2float_rn(x);
    valid[i] = found[i] >= S ? 1 : 0;
    return;
  }
  __shared__ int warp_sum[32];
  __shared__ int counter;
  const Part p = part_of<PER>(B, blockIdx.x, n);
  int base = 0, all = 0;  // such shots before this block's part, then before the round
  if (n > 1) {
    count_below<PER>(found, p, S, &counter);
    base = cluster_base(cluster, &counter, &all);
  }
  const int lane = threadIdx.x & 31;
  for (long long i0 = p.i0; i0 < p.i1; i0 += PER * FT) {
    const long long i = i0 + (threadIdx.x >> 5) * (32 * PER);
    uint32_t below[PER];
    int total, at = base + warps_scan(load_round<PER>(found, i, p.i1, S, below), warp_sum, &total);
    base += total;
    if (i >= p.i1) continue;  // a warp without shots in the last round: its bits are not set
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      if (below[k] >> lane & 1u) idx[at + __popc(below[k] & ((1u << lane) - 1u))] = (int)i + 32 * k + lane;
      at += __popc(below[k]);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *count = n > 1 ? all : base;
}

// Shots without a solution first, each part in ascending order, and the number of the former.
template <int PER>
__global__ void __launch_bounds__(FT) order_kernel(const int* found, long long B, int* order, int* count) {
  const cg::cluster_group cluster = cg::this_cluster();
  __shared__ int warp_sum[32];
  __shared__ int counter;
  const Part p = part_of<PER>(B, blockIdx.x, cluster.num_blocks());
  int first = count_below<PER>(found, p, 1, &counter);  // unsolved shots of the batch
  int base = 0;                                    // unsolved shots before the round
  if (cluster.num_blocks() > 1) base = cluster_base(cluster, &counter, &first);
  const int lane = threadIdx.x & 31;
  for (long long i0 = p.i0; i0 < p.i1; i0 += PER * FT) {
    const long long i = i0 + (threadIdx.x >> 5) * (32 * PER);
    uint32_t below[PER];
    int total;
    int u = base + warps_scan(load_round<PER>(found, i, p.i1, 1, below), warp_sum, &total);  // unsolved before shot i
    base += total;
    if (i >= p.i1) continue;  // as above
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int shot = (int)i + 32 * k + lane, before = u + __popc(below[k] & ((1u << lane) - 1u));
      if (below[k] >> lane & 1u) order[before] = shot;
      else if (i + 32 * k + lane < p.i1) order[first + shot - before] = shot;
      u += __popc(below[k]);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && count) *count = first;
}

// `blocks` blocks in clusters of `cluster`.
template <typename... P, typename... A>
cudaError_t launch(void (*kernel)(P...), int blocks, int cluster, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = cluster;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(FT);
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = cluster > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace

extern "C" {

int rbp_results(const int32_t* found_count, const int64_t* weight_fixed, int64_t B, int32_t stop_nconv, void* weights,
                int32_t weights_f64, uint8_t* valid, int32_t* unconverged, int32_t* n_unconverged, void* stream) {
  if (B < 0 || B > INT_MAX) return fail(RBP_ERR_ARGUMENT, "rbp_results: batch out of range");
  if (!n_unconverged || (B > 0 && (!found_count || !weight_fixed || !weights || !valid || !unconverged)))
    return fail(RBP_ERR_ARGUMENT, "rbp_results: null buffer");
  const int cluster = B < CLUSTER_FROM ? 1 : CLUSTER;
  const int blocks = cluster + (int)(((B + FT - 1) / FT + cluster - 1) / cluster * cluster);
  RBP_CUDA(launch(B < LARGE_FROM ? results_kernel<PER_SMALL> : results_kernel<PER_LARGE>, blocks, cluster,
                  static_cast<cudaStream_t>(stream), found_count, reinterpret_cast<const long long*>(weight_fixed),
                  (long long)B, (int)stop_nconv, weights_f64 ? nullptr : static_cast<float*>(weights),
                  weights_f64 ? static_cast<double*>(weights) : nullptr, valid, unconverged, n_unconverged));
  return RBP_OK;
}

int rbp_queue_order(const int32_t* found_count, int64_t B, int32_t* order, int32_t* n_unsolved, void* stream) {
  if (B < 0 || B > INT_MAX) return fail(RBP_ERR_ARGUMENT, "rbp_queue_order: batch out of range");
  if (B > 0 && (!found_count || !order)) return fail(RBP_ERR_ARGUMENT, "rbp_queue_order: null buffer");
  const int cluster = B < CLUSTER_FROM ? 1 : CLUSTER;
  RBP_CUDA(launch(B < LARGE_FROM ? order_kernel<PER_SMALL> : order_kernel<PER_LARGE>, cluster, cluster,
                  static_cast<cudaStream_t>(stream), found_count, (long long)B, order, n_unsolved));
  return RBP_OK;
}

}  // extern "C"
