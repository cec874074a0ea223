// GF(2) products on the device: out[b, r] = XOR over the columns j of row r of
// a sparse 0/1 matrix of x[b, j].  With the check matrix H it turns error rows
// into syndromes (s = H e); with the observables matrix it gives the logical
// observables of true and decoded errors (O e, O e_hat).  The reference does
// both on the host with scipy (src/pelagos/adapter.py:545-560, 601-613, 679).
//
// Shots are bit-sliced: a block takes up to 32 shots, turns their columns into
// words (bit b of word j: column j of shot b) in shared memory, and a row is the
// XOR of its columns' words, so one shared-memory read serves 32 shots.
// Measured with 65,536 shots: the 936 x 2,592 check matrix (231 MB in and out)
// 611 -> 69 us, the 12 observables of long rows 450 -> 42 us, against a
// shot's bytes staged and gathered one by one; reading x once at the copy
// bandwidth takes 26 us.

#include "relaybp.h"
#include "relaybp_host.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

namespace {

using rbph::fail;

constexpr int GF2_THREADS = 256;
constexpr int GF2_SHOTS = 32;  // shots per tile: the bits of a word
constexpr int STAGED = 64;     // in place of the bytes per load: the tile goes through stage_tile

// Bit r of lane c's word becomes bit c of lane r's (5 exchanges of half blocks).
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? (x & ~m) | ((y >> j) & m) : (x & m) | ((y & m) << j);
    m ^= m << (j >> 1);
  }
  return x;
}

// Low bits of a word's four bytes as a nibble, and back.
__device__ __forceinline__ uint32_t pack4(uint32_t v) { return ((v & 0x01010101u) * 0x01020408u) >> 24 & 0xfu; }
__device__ __forceinline__ uint32_t spread4(uint32_t n) { return ((n & 0xfu) * 0x00204081u) & 0x01010101u; }

// Columns j0 .. j0+31 of one shot as a word (columns past N: 0).  VEC: bytes per load
// (16 or 4 where every row's start is aligned to that, else 1).
template <int VEC>
__device__ __forceinline__ uint32_t load_columns(const uint8_t* row, int j0, int N) {
  uint32_t w = 0u;
  if (VEC == 16 && j0 + 32 <= N) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(row + j0 + 16 * h));
      w |= (pack4(u.x) | pack4(u.y) << 4 | pack4(u.z) << 8 | pack4(u.w) << 12) << (16 * h);
    }
  } else if (VEC >= 4 && j0 + 32 <= N) {
#pragma unroll
    for (int h = 0; h < 8; ++h) w |= pack4(__ldg(reinterpret_cast<const uint32_t*>(row + j0 + 4 * h))) << (4 * h);
  } else {
    for (int h = 0; h < 32 && j0 + h < N; ++h) w |= (uint32_t)(row[j0 + h] & 1u) << h;
  }
  return w;
}

// The tile's shots (nb rows of N bytes, one contiguous piece of memory) as packed columns in
// shared memory, [shot][stride] words: 16 bytes per thread and load, four loads in flight, a warp's
// 512 bytes contiguous.  With a lane per shot (load_columns) every load touched 32 lines: the
// 936-row product of 65,536 shots 82 -> 69 us, the failure counts 79 -> 73 us.
// y: XORed in, or null.  magic: ceil(2^32 / (N / 16)), exact for the at most 32 (N / 16) pieces.
__device__ __forceinline__ void stage_tile(const uint8_t* x, const uint8_t* y, int nb, int N, uint32_t magic,
                                           uint32_t* packed, int stride) {
  const uint32_t row = (uint32_t)N / 16, n = row * (uint32_t)nb;
  uint16_t* p16 = reinterpret_cast<uint16_t*>(packed);
  for (uint32_t i0 = threadIdx.x; i0 < n; i0 += 4 * GF2_THREADS) {
    uint4 u[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t i = i0 + k * GF2_THREADS;
      u[k] = i < n ? __ldg(reinterpret_cast<const uint4*>(x) + i) : make_uint4(0u, 0u, 0u, 0u);
      if (y && i < n) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(y) + i);
        u[k] = make_uint4(u[k].x ^ v.x, u[k].y ^ v.y, u[k].z ^ v.z, u[k].w ^ v.w);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t i = i0 + k * GF2_THREADS;
      if (i < n) {
        const uint32_t shot = __umulhi(i, magic);
        p16[shot * (2 * stride) + (i - shot * row)] =
            (uint16_t)(pack4(u[k].x) | pack4(u[k].y) << 4 | pack4(u[k].z) << 8 | pack4(u[k].w) << 12);
      }
    }
  }
}

// The tile's column words (bit b of word j: column j of shot b) from the global rows.
template <int IN>
__device__ __forceinline__ void tile_words(const uint8_t* x, const uint8_t* y, int nb, int N, uint32_t magic,
                                           uint32_t* word) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = GF2_THREADS / 32;
  if constexpr (IN == STAGED) {
    const int stride = ((N + 31) / 32) | 1;  // odd: a column of packed words is read without bank conflicts
    uint32_t* packed = word + (N + 31) / 32 * 32;
    stage_tile(x, y, nb, N, magic, packed, stride);
    __syncthreads();
    for (int j0 = warp * 32; j0 < N; j0 += nwarps * 32)  // a last half word's upper columns are never read
      word[j0 + lane] = transpose32(lane < nb ? packed[lane * stride + j0 / 32] : 0u, lane);
  } else {
    const size_t at = (size_t)min(lane, nb - 1) * N;
    for (int j0 = warp * 32; j0 < N; j0 += nwarps * 32) {
      uint32_t w = 0u;
      if (lane < nb) {
        w = load_columns<IN>(x + at, j0, N);
        if (y) w ^= load_columns<IN>(y + at, j0, N);
      }
      word[j0 + lane] = transpose32(w, lane);
    }
  }
}

// Whether rows of N bytes are staged: whole 16-byte pieces (the caller checked the alignment),
// more than one per row, and two blocks' words within an SM's shared memory.
bool staged(int N) { return N >= 32 && N % 16 == 0 && N <= 12 * 1024; }
size_t words_smem(int N, bool stage) {
  const size_t w = (size_t)(N + 31) / 32;
  return (w * 32 + (stage ? 32 * (w | 1) : 0)) * sizeof(uint32_t);
}
uint32_t piece_magic(int N) { return N >= 32 ? 0xffffffffu / (uint32_t)(N / 16) + 1u : 0u; }

// Bits of w to n (<= 32) bytes.  VEC: 8, 4 or 1, as for load_columns.
template <int VEC>
__device__ __forceinline__ void store_bytes(uint8_t* p, uint32_t w, int n) {
  if (VEC == 8 && n == 32) {
#pragma unroll
    for (int h = 0; h < 4; ++h)
      *reinterpret_cast<uint2*>(p + 8 * h) = make_uint2(spread4(w >> (8 * h)), spread4(w >> (8 * h + 4)));
  } else if (VEC >= 4 && n == 32) {
#pragma unroll
    for (int h = 0; h < 8; ++h) *reinterpret_cast<uint32_t*>(p + 4 * h) = spread4(w >> (4 * h));
  } else {
    for (int h = 0; h < n; ++h) p[h] = (uint8_t)((w >> h) & 1u);
  }
}

// Tiles of `tile` (1..32) shots, grid-stride.  A warp turns 32 columns of the tile's shots
// (lane b: shot b) into 32 column words at a time; then a thread evaluates a row, or with
// few rows (WARP_ROWS; they tend to be long: logical operators) a warp does.
template <int IN, int OUT, bool WARP_ROWS>
__global__ void __launch_bounds__(GF2_THREADS, IN == STAGED ? 6 : 1) gf2_rows_kernel(const uint8_t* x, long long B, int tile, int N,
                                                             uint32_t magic, const int* row_ptr, const int* cols,
                                                             int R, uint8_t* out) {
  extern __shared__ uint32_t word[];  // [N rounded up to 32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = GF2_THREADS / 32;
  for (long long b0 = blockIdx.x * (long long)tile; b0 < B; b0 += gridDim.x * (long long)tile) {
    const int nb = (int)min((long long)tile, B - b0);
    tile_words<IN>(x + b0 * N, nullptr, nb, N, magic, word);
    __syncthreads();
    if constexpr (WARP_ROWS) {
      for (int r = warp; r < R; r += nwarps) {
        uint32_t p = 0u;
        for (int k = row_ptr[r] + lane; k < row_ptr[r + 1]; k += 32) p ^= word[cols[k]];
        p = __reduce_xor_sync(0xffffffffu, p);
        if (lane < nb) out[(b0 + lane) * R + r] = (uint8_t)((p >> lane) & 1u);
      }
    } else {
      for (int r0 = warp * 32; r0 < R; r0 += nwarps * 32) {
        uint32_t p = 0u;
        if (r0 + lane < R)
          for (int k = row_ptr[r0 + lane]; k < row_ptr[r0 + lane + 1]; ++k) p ^= word[cols[k]];
        p = transpose32(p, lane);
        if (lane < nb) store_bytes<OUT>(out + (b0 + lane) * R + r0, p, min(32, R - r0));
      }
    }
    __syncthreads();  // the next tile overwrites the words
  }
}

template <int IN, int OUT>
int launch_rows(const uint8_t* x, long long B, int N, const int* row_ptr, const int* cols, int R, uint8_t* out,
                cudaStream_t st) {
  const size_t smem = words_smem(N, IN == STAGED);
  // fewer than 64 rows do not fill the block's threads
  auto kernel = R < 64 ? gf2_rows_kernel<IN, OUT, true> : gf2_rows_kernel<IN, OUT, false>;
  if (smem > 48 * 1024)
    RBP_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
  // whole words of shots once every SM has work for its resident blocks; small batches are
  // spread over the SMs instead
  const long long spread = 148LL * 4;
  const int tile = (int)std::min<long long>(GF2_SHOTS, std::max<long long>(1, (B + spread - 1) / spread));
  const int blocks = (int)std::min<long long>((B + tile - 1) / tile, 148LL * 8);
  kernel<<<blocks, GF2_THREADS, smem, st>>>(x, B, tile, N, piece_magic(N), row_ptr, cols, R, out);
  RBP_CUDA(cudaGetLastError());
  return RBP_OK;
}

// Failure counts of decoded shots: a shot flips when some row of the observables has odd parity over
// e XOR est, so both arrays are read once, XORed as column words, and nothing but four sums leaves
// the kernel.  counts += (flipped or unsolved, unsolved, flipped but solved, iterations); integer
// adds, so the order of the blocks does not matter.  Bound by reading the two arrays: 65,536
// shots of 2,592 columns, 12 observables 73 us (340 MB at 4.7 TB/s), against 190 us for two
// products of 42 us and a dozen elementwise launches and sums over their results.
template <int IN, bool WARP_ROWS>
__global__ void __launch_bounds__(GF2_THREADS, IN == STAGED ? 6 : 1) gf2_failures_kernel(const uint8_t* e, const uint8_t* est, long long B,
                                                                 int tile, int N, uint32_t magic, const int* row_ptr,
                                                                 const int* cols, int R, const int* found, const int* iters,
                                                                 unsigned long long* counts) {
  extern __shared__ uint32_t word[];  // [N rounded up to 32]
  __shared__ uint32_t s_flip;         // bit b: some observable of the tile's shot b flips
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = GF2_THREADS / 32;
  long long n_fail = 0, n_unsolved = 0, n_flip = 0, n_iter = 0;  // warp 0: its lane's shots
  for (long long b0 = blockIdx.x * (long long)tile; b0 < B; b0 += gridDim.x * (long long)tile) {
    const int nb = (int)min((long long)tile, B - b0);
    tile_words<IN>(e + b0 * N, est + b0 * N, nb, N, magic, word);
    if (threadIdx.x == 0) s_flip = 0u;
    __syncthreads();
    uint32_t any = 0u;
    if constexpr (WARP_ROWS) {
      for (int r = warp; r < R; r += nwarps) {
        uint32_t p = 0u;
        for (int k = row_ptr[r] + lane; k < row_ptr[r + 1]; k += 32) p ^= word[cols[k]];
        any |= __reduce_xor_sync(0xffffffffu, p);
      }
    } else {
      for (int r = threadIdx.x; r < R; r += GF2_THREADS) {
        uint32_t p = 0u;
        for (int k = row_ptr[r]; k < row_ptr[r + 1]; ++k) p ^= word[cols[k]];
        any |= p;
      }
      any = __reduce_or_sync(0xffffffffu, any);
    }
    if (lane == 0 && any) atomicOr(&s_flip, any);
    __syncthreads();  // also: the next tile overwrites the words
    if (warp == 0) {
      if (lane < nb) {
        const bool flip = (s_flip >> lane) & 1u, unsolved = __ldg(found + b0 + lane) <= 0;
        n_fail += flip || unsolved;
        n_unsolved += unsolved;
        n_flip += flip && !unsolved;
        n_iter += __ldg(iters + b0 + lane);
      }
      __syncwarp();  // s_flip is read before the next tile clears it
    }
  }
  if (warp == 0) {
    long long n[4] = {n_fail, n_unsolved, n_flip, n_iter};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) n[i] += __shfl_xor_sync(0xffffffffu, n[i], o);
      if (lane == 0 && n[i]) atomicAdd(counts + i, (unsigned long long)n[i]);
    }
  }
}

template <int IN>
int launch_failures(const uint8_t* e, const uint8_t* est, long long B, int N, const int* row_ptr, const int* cols, int R,
                    const int* found, const int* iters, unsigned long long* counts, cudaStream_t st) {
  const size_t smem = words_smem(N, IN == STAGED);
  auto kernel = R < 64 ? gf2_failures_kernel<IN, true> : gf2_failures_kernel<IN, false>;  // as launch_rows
  if (smem > 48 * 1024 - 64)
    RBP_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
  const long long spread = 148LL * 4;
  const int tile = (int)std::min<long long>(GF2_SHOTS, std::max<long long>(1, (B + spread - 1) / spread));
  const int blocks = (int)std::min<long long>((B + tile - 1) / tile, 148LL * 8);
  RBP_CUDA(cudaMemsetAsync(counts, 0, 4 * sizeof(unsigned long long), st));
  kernel<<<blocks, GF2_THREADS, smem, st>>>(e, est, B, tile, N, piece_magic(N), row_ptr, cols, R, found, iters, counts);
  RBP_CUDA(cudaGetLastError());
  return RBP_OK;
}

}  // namespace

extern "C" int rbp_gf2_failures(const uint8_t* errors, const uint8_t* estimates, int64_t B, int32_t N,
                                const int32_t* row_ptr, const int32_t* cols, int32_t R, const int32_t* found_count,
                                const int32_t* iterations, int64_t* counts, void* stream) {
  if (B <= 0 || N <= 0 || R <= 0) return fail(RBP_ERR_ARGUMENT, "rbp_gf2_failures: sizes must be positive");
  if (!errors || !estimates || !row_ptr || !cols || !found_count || !iterations || !counts)
    return fail(RBP_ERR_ARGUMENT, "rbp_gf2_failures: null buffer");
  if (N > 48 * 1024) return fail(RBP_ERR_UNSUPPORTED, "rbp_gf2_failures: rows longer than 49,152 columns");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const uintptr_t in = reinterpret_cast<uintptr_t>(errors) | reinterpret_cast<uintptr_t>(estimates) | (uintptr_t)N;
  unsigned long long* n = reinterpret_cast<unsigned long long*>(counts);
  if (in % 16 == 0 && staged(N))
    return launch_failures<STAGED>(errors, estimates, B, N, row_ptr, cols, R, found_count, iterations, n, st);
  if (in % 16 == 0) return launch_failures<16>(errors, estimates, B, N, row_ptr, cols, R, found_count, iterations, n, st);
  if (in % 4 == 0) return launch_failures<4>(errors, estimates, B, N, row_ptr, cols, R, found_count, iterations, n, st);
  return launch_failures<1>(errors, estimates, B, N, row_ptr, cols, R, found_count, iterations, n, st);
}

extern "C" int rbp_gf2_matvec(const uint8_t* x, int64_t B, int32_t N, const int32_t* row_ptr, const int32_t* cols,
                              int32_t R, uint8_t* out, void* stream) {
  if (B < 0 || N < 0 || R < 0) return fail(RBP_ERR_ARGUMENT, "rbp_gf2_matvec: negative size");
  if (B == 0 || R == 0) return RBP_OK;
  if (!x || !row_ptr || !out || (!cols && N > 0)) return fail(RBP_ERR_ARGUMENT, "rbp_gf2_matvec: null buffer");
  if (N > 48 * 1024) return fail(RBP_ERR_UNSUPPORTED, "rbp_gf2_matvec: rows longer than 49,152 columns");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const uintptr_t in = reinterpret_cast<uintptr_t>(x) | (uintptr_t)N, o = reinterpret_cast<uintptr_t>(out) | (uintptr_t)R;
  const int iv = in % 16 == 0 ? 16 : (in % 4 == 0 ? 4 : 1), ov = o % 8 == 0 ? 8 : (o % 4 == 0 ? 4 : 1);
  if (iv == 16 && staged(N)) {
    if (ov == 8) return launch_rows<STAGED, 8>(x, B, N, row_ptr, cols, R, out, st);
    if (ov == 4) return launch_rows<STAGED, 4>(x, B, N, row_ptr, cols, R, out, st);
    return launch_rows<STAGED, 1>(x, B, N, row_ptr, cols, R, out, st);
  }
  if (iv == 16 && ov == 8) return launch_rows<16, 8>(x, B, N, row_ptr, cols, R, out, st);
  if (iv == 16 && ov == 4) return launch_rows<16, 4>(x, B, N, row_ptr, cols, R, out, st);
  if (iv == 16) return launch_rows<16, 1>(x, B, N, row_ptr, cols, R, out, st);
  if (iv == 4 && ov >= 4) return launch_rows<4, 4>(x, B, N, row_ptr, cols, R, out, st);
  if (iv == 4) return launch_rows<4, 1>(x, B, N, row_ptr, cols, R, out, st);
  return ov >= 4 ? launch_rows<1, 4>(x, B, N, row_ptr, cols, R, out, st)
                 : launch_rows<1, 1>(x, B, N, row_ptr, cols, R, out, st);
}
