// The small per-batch passes around a decode: the queue order of the relay legs and
// the result arrays made from the decode's counts and exact weights.
//
// The reference's host code makes them with a handful of torch operations
// (src/pelagos/decoder.py:3839-3873); so did this library's.  Each is a launch of 2-3 us
// on the device and 4-5 us on the host, a dozen of them and a radix sort per call: more
// than the decode of a small batch.  Here each is one launch.  What bounds them is the
// latency of one block's walk over the counts (ordered compaction), about 1,000 cycles
// per 4,096 shots; the rest of a launch's blocks make the elementwise results beside it.

#include "relaybp.h"
#include "relaybp_host.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>

namespace {

using rbph::fail;

constexpr int FT = 1024;  // threads; the compacting block takes 4 FT shots per round

// Counts i .. i+3 (past B: `pad`).
__device__ __forceinline__ int4 load4(const int* found, long long i, long long B, int pad) {
  if (i + 3 < B && (reinterpret_cast<uintptr_t>(found) & 15) == 0) return *reinterpret_cast<const int4*>(found + i);
  int4 v = make_int4(pad, pad, pad, pad);
  if (i < B) v.x = found[i];
  if (i + 1 < B) v.y = found[i + 1];
  if (i + 2 < B) v.z = found[i + 2];
  if (i + 3 < B) v.w = found[i + 3];
  return v;
}

// Exclusive prefix sum of n over the block, and the block's total in *total.
__device__ __forceinline__ int block_scan(int n, int* warp_sum, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int s = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += t;
  }
  __syncthreads();  // the last round's sums have been read
  if (lane == 31) warp_sum[warp] = s;
  __syncthreads();
  const int w = warp_sum[lane];  // FT / 32 = 32 warps
  int ws = w;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, ws, o);
    if (lane >= o) ws += t;
  }
  *total = __shfl_sync(0xffffffffu, ws, 31);
  return s - n + __shfl_sync(0xffffffffu, ws - w, warp);
}

// Block 0: the indices of shots with found < stop_nconv in ascending order, and their number.
// Other blocks: weights from the exact fixed-point weight (2^-32 units; +inf where there is
// none) and the mask found >= stop_nconv.
__global__ void __launch_bounds__(FT) results_kernel(const int* found, const long long* wfix, long long B, int S,
                                                     float* w32, double* w64, uint8_t* valid, int* idx, int* count) {
  if (blockIdx.x > 0) {
    const long long i = (blockIdx.x - 1) * (long long)FT + threadIdx.x;
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
  int base = 0;
  for (long long i0 = 0; i0 < B; i0 += 4 * FT) {
    const long long i = i0 + 4 * threadIdx.x;
    const int4 f = load4(found, i, B, S);
    const int n = (f.x < S) + (f.y < S) + (f.z < S) + (f.w < S);
    int total;
    int at = base + block_scan(n, warp_sum, &total);
    if (f.x < S) idx[at++] = (int)i;
    if (f.y < S) idx[at++] = (int)i + 1;
    if (f.z < S) idx[at++] = (int)i + 2;
    if (f.w < S) idx[at++] = (int)i + 3;
    base += total;
  }
  if (threadIdx.x == 0) *count = base;
}

// Shots without a solution first, each part in ascending order, and the number of the former.
__global__ void __launch_bounds__(FT) order_kernel(const int* found, long long B, int* order, int* count) {
  __shared__ int warp_sum[32];
  __shared__ int unsolved;
  if (threadIdx.x == 0) unsolved = 0;
  __syncthreads();
  int mine = 0;
#pragma unroll 4
  for (long long i = 4 * threadIdx.x; i < B; i += 4 * FT) {
    const int4 f = load4(found, i, B, 1);
    mine += (f.x <= 0) + (f.y <= 0) + (f.z <= 0) + (f.w <= 0);
  }
  mine = __reduce_add_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&unsolved, mine);
  __syncthreads();
  const int first = unsolved;
  int base = 0;  // unsolved shots before this round
  for (long long i0 = 0; i0 < B; i0 += 4 * FT) {
    const long long i = i0 + 4 * threadIdx.x;
    const int4 f = load4(found, i, B, 1);
    const int n = (f.x <= 0) + (f.y <= 0) + (f.z <= 0) + (f.w <= 0);
    int total;
    int u = base + block_scan(n, warp_sum, &total);  // unsolved before shot i
    const int v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i + k >= B) break;
      if (v[k] <= 0) order[u++] = (int)i + k;
      else order[first + (int)i + k - u] = (int)i + k;
    }
    base += total;
  }
  if (threadIdx.x == 0 && count) *count = first;
}

}  // namespace

extern "C" {

int rbp_results(const int32_t* found_count, const int64_t* weight_fixed, int64_t B, int32_t stop_nconv, void* weights,
                int32_t weights_f64, uint8_t* valid, int32_t* unconverged, int32_t* n_unconverged, void* stream) {
  if (B < 0 || B > INT_MAX) return fail(RBP_ERR_ARGUMENT, "rbp_results: batch out of range");
  if (!n_unconverged || (B > 0 && (!found_count || !weight_fixed || !weights || !valid || !unconverged)))
    return fail(RBP_ERR_ARGUMENT, "rbp_results: null buffer");
  const int blocks = 1 + (int)((B + FT - 1) / FT);
  results_kernel<<<blocks, FT, 0, static_cast<cudaStream_t>(stream)>>>(
      found_count, reinterpret_cast<const long long*>(weight_fixed), B, stop_nconv,
      weights_f64 ? nullptr : static_cast<float*>(weights), weights_f64 ? static_cast<double*>(weights) : nullptr, valid,
      unconverged, n_unconverged);
  RBP_CUDA(cudaGetLastError());
  return RBP_OK;
}

int rbp_queue_order(const int32_t* found_count, int64_t B, int32_t* order, int32_t* n_unsolved, void* stream) {
  if (B < 0 || B > INT_MAX) return fail(RBP_ERR_ARGUMENT, "rbp_queue_order: batch out of range");
  if (B > 0 && (!found_count || !order)) return fail(RBP_ERR_ARGUMENT, "rbp_queue_order: null buffer");
  order_kernel<<<1, FT, 0, static_cast<cudaStream_t>(stream)>>>(found_count, B, order, n_unsolved);
  RBP_CUDA(cudaGetLastError());
  return RBP_OK;
}

}  // extern "C"
