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
#include <type_traits>

namespace {

using rbph::fail;
using rbph::kSMs;

constexpr int GF2_THREADS = 256;
constexpr int GF2_SHOTS = 32;  // shots per tile: the bits of a word
constexpr int STAGED = 64;     // in place of the bytes per load: the tile goes through stage_tile
// Blocks of rows that are not staged have twice the threads from this shared memory on, where few are resident:
// 3,000 shots of 20,001 columns and 12 short rows 88 -> 59 us.
constexpr int WIDE_SMEM = 32 * 1024;
// Below this many rows a warp evaluates one, from it on a thread.  65,536 shots of 2,592 columns, a warp / a thread
// per row, us: 12 rows of 260 entries 53 / 70, of 1,000 58 / 114; 63 rows of 3 entries 62 / 54, of 260 82 / 91, of
// 1,000 121 / 231.  (The host does not see the rows' lengths.)
constexpr int WARP_ROWS_BELOW = 64;

// Threads of the block: known to the compiler for staged rows.
template <int IN>
__device__ __forceinline__ int block_threads() {
  return IN == STAGED ? GF2_THREADS : (int)blockDim.x;
}

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

// The tile's shots (nb rows of N bytes, one contiguous piece of memory) as packed columns in
// shared memory, [shot][stride] words: 16 bytes per thread and load, four loads in flight, a warp's
// 512 bytes contiguous.  With a lane per shot every load touched 32 lines: the
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

// Four bytes from p on, which need not be aligned; bytes outside [lo, hi) are not read (0 instead).
__device__ __forceinline__ uint32_t load4(const uint8_t* p, const uint8_t* lo, const uint8_t* hi) {
  const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3u);
  const uint8_t* a = p - off;
  if (a >= lo && a + 8 <= hi) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(a);
    return __funnelshift_r(__ldg(w), __ldg(w + 1), 8 * off);
  }
  uint32_t v = 0u;
  for (int q = 0; q < 4; ++q)
    if (p + q >= lo && p + q < hi) v |= (uint32_t)p[q] << (8 * q);
  return v;
}

// The tile's column words from rows that are not staged: a thread takes four columns of eight shots,
// whose low bits are one byte of each column's word, so a warp's loads are contiguous whatever the rows'
// alignment (ALIGNED: every row starts at a multiple of four bytes) and eight or more are in flight.  With a
// lane per shot, 32 bytes of a row each, rows of odd length took longer than the shots' bytes staged one by one.
// us, that / a lane per shot / now: 65,536 shots of 1,082 columns and 63 rows 106 / 161 / 61, of 2,594 columns and
// 1,297 rows 762 / 1,000 / 194; 3,000 shots of 20,001 columns and 64 rows 59 / 269 / 60.
// Shots past nb repeat the last one, and a last piece's columns past N are the next row's: bits that are not used.
template <bool ALIGNED>
__device__ __forceinline__ void column_words(const uint8_t* x, const uint8_t* y, size_t at0, size_t size, int nb, int N,
                                             uint32_t* word) {
  uint8_t* bytes = reinterpret_cast<uint8_t*>(word);
  const uint32_t units = ((uint32_t)N + 3) / 4, n = units * (uint32_t)((nb + 7) / 8);
  auto load = [&](size_t at) {
    at += at0;
    uint32_t v = ALIGNED ? __ldg(reinterpret_cast<const uint32_t*>(x + at)) : load4(x + at, x, x + size);
    if (y) v ^= ALIGNED ? __ldg(reinterpret_cast<const uint32_t*>(y + at)) : load4(y + at, y, y + size);
    return v;
  };
  if (nb == 1) {  // batches below one shot per resident block: four pieces of its row in flight instead
#pragma unroll 4
    for (uint32_t u = threadIdx.x; u < units; u += blockDim.x) {
      const uint32_t v = load(4 * u);
#pragma unroll
      for (int q = 0; q < 4; ++q) word[4 * u + q] = v >> (8 * q) & 1u;
    }
    return;
  }
#pragma unroll 1
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const uint32_t oct = i / units, u = i - oct * units;
    uint32_t v[8], bits = 0u;
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = load((size_t)min((int)(8 * oct) + k, nb - 1) * N + 4 * u);
#pragma unroll
    for (int k = 0; k < 8; ++k) bits |= (v[k] & 0x01010101u) << k;
    const uint32_t turn = (threadIdx.x & 31) >> 3;  // the lanes of one bank store different columns
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t c = (q + turn) & 3u;
      bytes[4 * (4 * u + c) + oct] = (uint8_t)(bits >> (8 * c));
    }
  }
}

// The same of rows of at most LANE_COLUMNS columns, a lane per shot: neighbouring rows share the sectors that a
// load touches, and nothing is computed twice (65,536 shots of 25 columns and one row 18 us, by column 23).
constexpr int LANE_COLUMNS = 128;
template <bool ALIGNED>
__device__ __forceinline__ void lane_words(const uint8_t* x, const uint8_t* y, int nb, int N, uint32_t* word) {
  const int lane = threadIdx.x & 31, j0 = (threadIdx.x >> 5) * 32;
  if (j0 >= N) return;
  auto columns = [&](const uint8_t* row) {
    uint32_t w = 0u;
    if (ALIGNED && j0 + 32 <= N) {
#pragma unroll
      for (int h = 0; h < 8; ++h) w |= pack4(__ldg(reinterpret_cast<const uint32_t*>(row + j0 + 4 * h))) << (4 * h);
    } else {
      for (int h = 0; h < 32 && j0 + h < N; ++h) w |= (uint32_t)(row[j0 + h] & 1u) << h;
    }
    return w;
  };
  uint32_t w = 0u;
  if (lane < nb) {
    w = columns(x + (size_t)lane * N);
    if (y) w ^= columns(y + (size_t)lane * N);
  }
  word[j0 + lane] = transpose32(w, lane);
}

// The column words (bit b of word j: column j of shot b) of a tile of staged rows.
__device__ __forceinline__ void staged_words(const uint8_t* x, const uint8_t* y, int nb, int N, uint32_t magic,
                                             uint32_t* word) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = GF2_THREADS / 32;
  const int stride = ((N + 31) / 32) | 1;  // odd: a column of packed words is read without bank conflicts
  uint32_t* packed = word + (N + 31) / 32 * 32;
  stage_tile(x, y, nb, N, magic, packed, stride);
  __syncthreads();
  for (int j0 = warp * 32; j0 < N; j0 += nwarps * 32)  // a last half word's upper columns are never read
    word[j0 + lane] = transpose32(lane < nb ? packed[lane * stride + j0 / 32] : 0u, lane);
}

// The same of other rows, the tile's nb shots from b0 on of the B rows of x (and of y, XORed in, or null).
template <bool ALIGNED>
__device__ __forceinline__ void unstaged_words(const uint8_t* x, const uint8_t* y, long long b0, long long B, int nb, int N,
                                               uint32_t* word) {
  if (N <= LANE_COLUMNS) lane_words<ALIGNED>(x + b0 * N, y ? y + b0 * N : nullptr, nb, N, word);
  else column_words<ALIGNED>(x, y, (size_t)b0 * N, (size_t)B * N, nb, N, word);
}

// Whether rows of N bytes are staged: whole 16-byte pieces (the caller checked the alignment),
// more than one per row, and two blocks' words within an SM's shared memory.
bool staged(int N) { return N >= 32 && N % 16 == 0 && N <= 12 * 1024; }
size_t words_smem(int N, bool stage) {
  const size_t w = (size_t)(N + 31) / 32;
  return (w * 32 + (stage ? 32 * (w | 1) : 0)) * sizeof(uint32_t);
}
uint32_t piece_magic(int N) { return N >= 32 ? 0xffffffffu / (uint32_t)(N / 16) + 1u : 0u; }

// Bits of w to n (<= 32) bytes.  VEC: 8 or 4 bytes per store, where every row's start is aligned to that.
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

// Tiles of `tile` (1..32) shots, grid-stride: the column words, then a thread evaluates a row, or with
// few rows (WARP_ROWS; they tend to be long: logical operators) a warp does.  OUT: bytes per store (8 or 4
// where every output row's start is aligned to that), or 1: a warp's 32 rows of one shot per store.
template <int IN, int OUT, bool WARP_ROWS>
__global__ void __launch_bounds__(IN == STAGED ? GF2_THREADS : 2 * GF2_THREADS, IN == STAGED ? 6 : 3)
gf2_rows_kernel(const uint8_t* x, long long B, int tile, int N, uint32_t magic, const int* row_ptr, const int* cols, int R,
                uint8_t* out) {
  extern __shared__ uint32_t word[];  // [N rounded up to 32]
  __shared__ uint32_t s_row[WARP_ROWS && IN != STAGED ? WARP_ROWS_BELOW : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = block_threads<IN>() / 32;
  for (long long b0 = blockIdx.x * (long long)tile; b0 < B; b0 += gridDim.x * (long long)tile) {
    const int nb = (int)min((long long)tile, B - b0);
    if constexpr (IN == STAGED) staged_words(x + b0 * N, nullptr, nb, N, magic, word);
    else unstaged_words<IN == 4>(x, nullptr, b0, B, nb, N, word);
    __syncthreads();
    if constexpr (WARP_ROWS) {
      for (int r = warp; r < R; r += nwarps) {
        uint32_t p = 0u;
        for (int k = row_ptr[r] + lane; k < row_ptr[r + 1]; k += 32) p ^= word[cols[k]];
        p = __reduce_xor_sync(0xffffffffu, p);
        if (IN == STAGED && lane < nb) out[(b0 + lane) * R + r] = (uint8_t)((p >> lane) & 1u);
        if (IN != STAGED && lane == 0) s_row[r] = p;
      }
      if (IN != STAGED) {  // the tile's outputs are one contiguous piece
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < (uint32_t)(nb * R); i += block_threads<IN>()) {
          const uint32_t b = i / (uint32_t)R;
          out[b0 * R + i] = (uint8_t)((s_row[i - b * (uint32_t)R] >> b) & 1u);
        }
      }
    } else {
      for (int r0 = warp * 32; r0 < R; r0 += nwarps * 32) {
        uint32_t p = 0u;
        if (r0 + lane < R)
          for (int k = row_ptr[r0 + lane]; k < row_ptr[r0 + lane + 1]; ++k) p ^= word[cols[k]];
        if constexpr (OUT == 1) {
          uint8_t* o = out + b0 * R + r0 + lane;
          if (r0 + lane < R)
            for (int b = 0; b < nb; ++b) o[(size_t)b * R] = (uint8_t)((p >> b) & 1u);
        } else {
          p = transpose32(p, lane);
          if (lane < nb) store_bytes<OUT>(out + (b0 + lane) * R + r0, p, min(32, R - r0));
        }
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
  auto kernel = R < WARP_ROWS_BELOW ? gf2_rows_kernel<IN, OUT, true> : gf2_rows_kernel<IN, OUT, false>;
  if (smem > 47 * 1024)  // with the static part
    RBP_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
  // whole words of shots once every SM has work for its resident blocks; small batches are
  // spread over the SMs instead
  const long long spread = 4LL * kSMs;
  const int tile = (int)std::min<long long>(GF2_SHOTS, std::max<long long>(1, (B + spread - 1) / spread));
  const int blocks = (int)std::min<long long>((B + tile - 1) / tile, 8LL * kSMs);
  const int block = IN != STAGED && smem > WIDE_SMEM ? 2 * GF2_THREADS : GF2_THREADS;
  kernel<<<blocks, block, smem, st>>>(x, B, tile, N, piece_magic(N), row_ptr, cols, R, out);
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
__global__ void __launch_bounds__(IN == STAGED ? GF2_THREADS : 2 * GF2_THREADS, IN == STAGED ? 6 : 2)
gf2_failures_kernel(const uint8_t* e, const uint8_t* est, long long B, int tile, int N, uint32_t magic, const int* row_ptr,
                    const int* cols, int R, const int* found, const int* iters, unsigned long long* counts) {
  extern __shared__ uint32_t word[];  // [N rounded up to 32]
  __shared__ uint32_t s_flip;         // bit b: some observable of the tile's shot b flips
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = block_threads<IN>() / 32;
  long long n_fail = 0, n_unsolved = 0, n_flip = 0, n_iter = 0;  // warp 0: its lane's shots
  for (long long b0 = blockIdx.x * (long long)tile; b0 < B; b0 += gridDim.x * (long long)tile) {
    const int nb = (int)min((long long)tile, B - b0);
    if constexpr (IN == STAGED) staged_words(e + b0 * N, est + b0 * N, nb, N, magic, word);
    else unstaged_words<IN == 4>(e, est, b0, B, nb, N, word);
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
      for (int r = threadIdx.x; r < R; r += block_threads<IN>()) {
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
  auto kernel = R < WARP_ROWS_BELOW ? gf2_failures_kernel<IN, true> : gf2_failures_kernel<IN, false>;  // as launch_rows
  if (smem > 47 * 1024)
    RBP_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
  const long long spread = 4LL * kSMs;
  const int tile = (int)std::min<long long>(GF2_SHOTS, std::max<long long>(1, (B + spread - 1) / spread));
  const int blocks = (int)std::min<long long>((B + tile - 1) / tile, 8LL * kSMs);
  const int block = IN != STAGED && smem > WIDE_SMEM ? 2 * GF2_THREADS : GF2_THREADS;
  RBP_CUDA(cudaMemsetAsync(counts, 0, 4 * sizeof(unsigned long long), st));
  kernel<<<blocks, block, smem, st>>>(e, est, B, tile, N, piece_magic(N), row_ptr, cols, R, found, iters, counts);
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
  if (in % 16 == 0 && staged(N)) {
    if (o % 8 == 0) return launch_rows<STAGED, 8>(x, B, N, row_ptr, cols, R, out, st);
    if (o % 4 == 0) return launch_rows<STAGED, 4>(x, B, N, row_ptr, cols, R, out, st);
    return launch_rows<STAGED, 1>(x, B, N, row_ptr, cols, R, out, st);
  }
  if (in % 4 == 0)
    return o % 4 == 0 ? launch_rows<4, 4>(x, B, N, row_ptr, cols, R, out, st)
                      : launch_rows<4, 1>(x, B, N, row_ptr, cols, R, out, st);
  return o % 4 == 0 ? launch_rows<1, 4>(x, B, N, row_ptr, cols, R, out, st)
                    : launch_rows<1, 1>(x, B, N, row_ptr, cols, R, out, st);
}
