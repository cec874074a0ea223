// Device-side pieces of the Relay-BP-S decode kernels (sm_100a): message types,
// group barriers, kernel arguments, the message layout and the block tables.
// The passes are in relaybp_rows.cuh, the decode loop in relaybp_decode.cuh.

#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "relaybp.h"

namespace rbpk {

// ------------------------------------------------------------------ message types

template <typename M>
struct MsgT;
template <>
struct MsgT<float> {
  using A = float;
  static __device__ __forceinline__ float ld(float v) { return v; }
  static __device__ __forceinline__ float st(float v) { return v; }
};
template <>
struct MsgT<double> {
  using A = double;
  static __device__ __forceinline__ double ld(double v) { return v; }
  static __device__ __forceinline__ double st(double v) { return v; }
};
// float16 messages saturate at the largest finite value (+-65504) before
// rounding: posteriors with memory grow past float16's range on hard shots,
// and an infinite message would turn the variable pass's inf - inf into NaN.
__device__ __forceinline__ __half f16_saturate(float v) {
  return __float2half_rn(fminf(fmaxf(v, -65504.0f), 65504.0f));
}
template <>
struct MsgT<__half> {
  using A = float;
  static __device__ __forceinline__ float ld(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half st(float v) { return f16_saturate(v); }
};
template <>
struct MsgT<__nv_bfloat16> {
  using A = float;
  static __device__ __forceinline__ float ld(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 st(float v) { return __float2bfloat16_rn(v); }
};

__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// lambda_mixed = (1 - g) * llr + g * posterior   (kernels.py:1309)
template <typename A>
__device__ __forceinline__ A memory_mix(int mode, A g, A l0, A post) {
  const A one_m = sub_rn(A(1), g);
  if (mode == RBP_MIX_FMA_GP) return fma_rn(g, post, mul_rn(one_m, l0));
  if (mode == RBP_MIX_FMA_LP) return fma_rn(one_m, l0, mul_rn(g, post));
  return add_rn(mul_rn(one_m, l0), mul_rn(g, post));
}

// Weight of one set bit in units of 2^-32; non-finite priors weigh 0
// (decoder.py:741-753).  w * 2^32 is exact in float; rounding to nearest-even.
__device__ __forceinline__ long long weight_units(float w) {
  if (!isfinite(w)) return 0;
  return __float2ll_rn(w * 4294967296.0f);
}

// ------------------------------------------------------------------ group sync

// Barrier over one group: a warp-level sync for 32-thread groups, otherwise a
// named barrier (id 1 + group index) over the group's threads.
__device__ __forceinline__ void group_sync(int id, int n) {
  if (n == 32) {
    __syncwarp();
  } else {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
  }
}

// Barrier + OR-reduction of a predicate over the group.
__device__ __forceinline__ bool group_any(int id, int n, bool p) {
  if (n == 32) return __any_sync(0xffffffffu, p);
  unsigned r;
  asm volatile(
      "{\n\t.reg .pred pi, po;\n\t"
      "setp.ne.u32 pi, %1, 0;\n\t"
      "bar.red.or.pred po, %2, %3, pi;\n\t"
      "selp.u32 %0, 1, 0, po;\n\t}"
      : "=r"(r)
      : "r"((unsigned)p), "r"(id), "r"(n)
      : "memory");
  return r != 0;
}

// ------------------------------------------------------------------ parameters

struct DevGraph {
  int C, V, E;
  int slots;                 // max check degree
  int rows;                  // slot rows of the layout (padded to MAXDC and to whole 16-byte chunks)
  int vslots;                // max variable degree (<= MAXDV of the instantiation)
  const uint8_t* chk_deg;    // [C] (degrees > 255 use the generic check path, which reads chk_ptr)
  const int* chk_ptr;        // [C+1]
  const uint16_t* var_pos;   // [vslots, V] slot position of variable v's k-th edge (summation order),
                             // kNoSlot where v has fewer edges
  const uint16_t* var_chk;   // [V, chk_stride] check of variable v's k-th edge, kNoSlot beyond its degree
  int chk_stride;            // 4 (vslots <= 4) or 8
};

struct DevArgs {
  // parameters
  int pre_iter, num_sets, set_max_iter, stop_nconv;
  int last_leg, use_alpha, use_beta, mix_mode, skip_legs;
  float beta, gamma0;
  // tables
  const float* llr;              // [V]
  const float* gamma_legs;       // [num_sets, V]
  const float* alpha;            // [n_alpha]
  // batch inputs
  long long B;
  const uint8_t* syn;            // [B, C]
  const float* llr_shot;         // [B, V] or null
  const float* gamma_pre;        // [B, V] or null
  const float* gamma_legs_shot;  // [B, shot_leg_rows, V] or null
  int n_shot_legs;
  int shot_leg_rows;             // >= 1; leg l uses row min(l, shot_leg_rows - 1)
  const float* init_post;        // [B, V] or null
  // outputs
  uint8_t* errors;
  uint32_t* errors_packed;
  float* weights;
  long long* wfixed;
  int* found;
  int* iters;
  void* last_post;
  // resumable decoding: shot state after/before a phase (see ShotStateLayout)
  int legs_begin;                // first relay leg when resuming
  int legs_end;                  // relay legs < legs_end run (<= 0: all)
  const unsigned char* resume;   // [B, state_stride] or null: start from the pre-iterations
  unsigned char* suspend;        // [B, state_stride] or null
  int state_stride;
  // scheduling
  int* queue;
  const int* order;              // [B] queue position -> shot index, or null (identity)
  const int* queue_len;          // device count of queue positions to take, or null: B
  // split decode: after the pre-iterations a solved shot runs relay legs < solved_legs at the
  // constant strength solved_gamma; with suspend_unsolved an unsolved shot saves its state and stops
  float solved_gamma;
  int solved_legs;
  int suspend_unsolved;
  int strict;                    // alpha or beta may give a check's output no finite value: masked rows
  int group_threads, groups;
  // shared-memory layout (byte offsets)
  int off_chk_deg, off_llr, off_first, off_group0, group_bytes;
  int g_msg, g_par, g_best, g_first, g_red;
  int keep_sums;                 // 1: the group region has the s1 and lmk arrays
  int g_s1;                      // the shot's first-pass sums, then the memory mixes
};

enum HardSrc { HARD_ZERO = 0, HARD_POST = 1, HARD_BEST = 2 };

// Per-shot decode state between launches (bytes):
//   [0,4) found  [4,8) iterations  [8,12) hard source  [12,16) has-best
//   [16,24) best weight (2^-32 units)  [24,32) unused
//   [32, 32+4W) best-solution bits, [32+4W, 32+8W) first-leg bits,
//   then the posterior [V] (accumulation type) at post_offset.
__host__ __device__ constexpr int state_post_offset(int V) { return (32 + 8 * ((V + 31) / 32) + 15) / 16 * 16; }
__host__ __device__ constexpr int state_stride(int V, int acc_bytes) {
  return (state_post_offset(V) + acc_bytes * V + 15) / 16 * 16;
}
constexpr uint16_t kNoSlot = 0xFFFFu;

// Shared-memory index of slot j of check c.  The slots of a check sit in
// 16-byte chunks of VEC = 16 / sizeof(M) messages, so a check pass moves a row
// with 128-bit loads/stores and consecutive checks occupy consecutive chunks:
//   index = (j / VEC) * (VEC * C) + c * VEC + ((j % VEC) ^ chunk_swizzle(c))
// The XOR swizzle permutes the slots inside a chunk by bits 3-4 of c, so the
// variable pass, whose warps touch the same slot of ~32 consecutive checks,
// spreads those accesses over all 32 banks instead of 8.  The check pass's
// work is symmetric in the slots of a row; it only needs the swizzle to know
// which positions are padding. 
template <typename M>
__host__ __device__ __forceinline__ int chunk_swizzle(int c) {
  constexpr int VEC = 16 / (int)sizeof(M);
  if constexpr (VEC == 8) return ((c >> 3) & 3) << 1;  // 16-bit messages: permute 4-byte words
  else if constexpr (VEC == 4) return (c >> 3) & 3;
  else return (c >> 3) & 1;
}

template <typename M>
__host__ __device__ __forceinline__ int slot_index(int j, int c, int C) {
  constexpr int VEC = 16 / (int)sizeof(M);
  return (j / VEC) * (VEC * C) + c * VEC + ((j % VEC) ^ chunk_swizzle<M>(c));
}

// Index of the first element of chunk q of check c: the 16-byte aligned
// address vector loads and stores use (physical element p of the chunk holds
// slot q * VEC + (p ^ chunk_swizzle(c))).
template <typename M>
__host__ __device__ __forceinline__ int chunk_base(int q, int c, int C) {
  constexpr int VEC = 16 / (int)sizeof(M);
  return q * (VEC * C) + c * VEC;
}

// 16-byte vector access to VEC consecutive slots, converted to/from the
// accumulation type.
template <typename M>
struct VecIO;
template <>
struct VecIO<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void load(const float* p, float* o) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
  static __device__ __forceinline__ void store(float* p, const float* o) {
    *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
  }
};
template <>
struct VecIO<double> {
  static constexpr int N = 2;
  static __device__ __forceinline__ void load(const double* p, double* o) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    o[0] = v.x; o[1] = v.y;
  }
  static __device__ __forceinline__ void store(double* p, const double* o) {
    *reinterpret_cast<double2*>(p) = make_double2(o[0], o[1]);
  }
};
template <typename H, float (*ToF)(H), H (*FromF)(float), unsigned short (*Bits)(H), H (*FromBits)(unsigned short)>
struct VecIO16 {
  static constexpr int N = 8;
  static __device__ __forceinline__ void load(const H* p, float* o) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[2 * i] = ToF(FromBits((unsigned short)(w[i] & 0xFFFFu)));
      o[2 * i + 1] = ToF(FromBits((unsigned short)(w[i] >> 16)));
    }
  }
  static __device__ __forceinline__ void store(H* p, const float* o) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      w[i] = (uint32_t)Bits(FromF(o[2 * i])) | ((uint32_t)Bits(FromF(o[2 * i + 1])) << 16);
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  }
};
__device__ __forceinline__ float h2f(__half h) { return __half2float(h); }
__device__ __forceinline__ __half f2h(float f) { return f16_saturate(f); }
__device__ __forceinline__ unsigned short hbits(__half h) { return __half_as_ushort(h); }
__device__ __forceinline__ __half hfrom(unsigned short b) { return __ushort_as_half(b); }
__device__ __forceinline__ float b2f(__nv_bfloat16 h) { return __bfloat162float(h); }
__device__ __forceinline__ __nv_bfloat16 f2b(float f) { return __float2bfloat16_rn(f); }
__device__ __forceinline__ unsigned short bbits(__nv_bfloat16 h) { return __bfloat16_as_ushort(h); }
__device__ __forceinline__ __nv_bfloat16 bfrom(unsigned short b) { return __ushort_as_bfloat16(b); }
template <>
struct VecIO<__half> : VecIO16<__half, h2f, f2h, hbits, hfrom> {};
template <>
struct VecIO<__nv_bfloat16> : VecIO16<__nv_bfloat16, b2f, f2b, bbits, bfrom> {};

// Bit set of the hard decisions post <= 0 of the group's variables into dst
// (one ballot per warp and owned-variable slot).
template <typename A, int VPT>
__device__ __forceinline__ void ballot_post(const A (&post)[VPT], uint32_t* dst, int warp, int lane, int G, int V) {
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int v0 = warp * 32 + k * G;
    const unsigned m = __ballot_sync(0xffffffffu, v0 + lane < V && post[k] <= A(0));
    if (lane == 0 && v0 < V) dst[v0 >> 5] = m;
  }
}

// ------------------------------------------------------------------ block tables
//
// Template parameters here and in the kernels:
// M     message storage type (float, __half, __nv_bfloat16, double)
// MAXDC check degree bound held in registers by the check pass (0: generic loop)
// VPT   variables owned per thread
// MAXDV variable degree bound (slot positions held in registers)

// Negate every message of a 16-byte chunk (IEEE sign flip, exact in every
// storage type: float16 / bfloat16 saturate and round symmetrically).
template <typename M>
__device__ __forceinline__ uint4 flip_signs(uint4 v) {
  if constexpr (sizeof(M) == 2) {
    v.x ^= 0x80008000u; v.y ^= 0x80008000u; v.z ^= 0x80008000u; v.w ^= 0x80008000u;
  } else if constexpr (sizeof(M) == 4) {
    v.x ^= 0x80000000u; v.y ^= 0x80000000u; v.z ^= 0x80000000u; v.w ^= 0x80000000u;
  } else {
    v.y ^= 0x80000000u; v.w ^= 0x80000000u;
  }
  return v;
}

// The first check pass of every phase reads mu_e = llr[var(e)]: it is the same
// for every shot except for the syndrome bit, which only negates the check's
// outputs (par flips, the magnitudes do not change).  This computes that pass
// once per block for s = 0, with the same operations the check pass uses
// (alpha of iteration 0, beta, the degree-1 rule, storage rounding), into the
// table at off_first; the kernel then copies a row, negated when s = 1.
template <typename M, int MAXDC>
__device__ void build_first_pass_table(const DevGraph& g, const DevArgs& a, unsigned char* smem) {
  if constexpr (MAXDC > 0) {
    using IO = MsgT<M>;
    using A = typename IO::A;
    constexpr int VEC = VecIO<M>::N;
    constexpr int NQ = MAXDC / VEC;
    M* tab = reinterpret_cast<M*>(smem + a.off_first);
    const float* s_llr = reinterpret_cast<const float*>(smem + a.off_llr);
    const uint8_t* s_chk_deg = smem + a.off_chk_deg;
    for (int v = threadIdx.x; v < g.V; v += blockDim.x)
      for (int j = 0; j < g.vslots; ++j) {
        const uint16_t p = g.var_pos[j * g.V + v];
        if (p != kNoSlot) tab[p] = IO::st(A(s_llr[v]));
      }
    __syncthreads();
    const A alpha = a.use_alpha ? A(__ldg(a.alpha)) : A(1);
    const A beta = A(a.beta);
    const A kInf = A(__int_as_float(0x7f800000));
    for (int c = threadIdx.x; c < g.C; c += blockDim.x) {
      const int deg = s_chk_deg[c];
      const int swz = chunk_swizzle<M>(c);
      A mv[MAXDC];
#pragma unroll
      for (int q = 0; q < NQ; ++q) VecIO<M>::load(tab + chunk_base<M>(q, c, g.C), mv + q * VEC);
      int neg = 0;
      A min1 = A(1e30), min2 = A(1e30);
#pragma unroll
      for (int j = 0; j < MAXDC; ++j) {
        const bool in = ((j % VEC) ^ swz) < deg - (j / VEC) * VEC;
        neg ^= (in && mv[j] < A(0)) ? 1 : 0;
        const A x = in ? fmin(fabs(mv[j]), kInf) : kInf;
        min2 = fmin(min2, fmax(min1, x));
        min1 = fmin(min1, x);
      }
      const bool par = (neg & 1) != 0;  // syndrome bit 0
      A lo = deg == 1 ? A(0) : min1;
      A hi = deg == 1 ? A(0) : min2;
      if (a.use_alpha) {
        lo = mul_rn(alpha, lo);
        hi = mul_rn(alpha, hi);
      }
      if (a.use_beta) {
        lo = fmax(sub_rn(lo, beta), A(0));
        hi = fmax(sub_rn(hi, beta), A(0));
      }
      A out[MAXDC];
#pragma unroll
      for (int j = 0; j < MAXDC; ++j) {
        const A m = mv[j];
        const A mag = (fabs(m) == min1) ? hi : lo;
        out[j] = (par != !(m >= A(0))) ? -mag : mag;
      }
#pragma unroll
      for (int q = 0; q < NQ; ++q) VecIO<M>::store(tab + chunk_base<M>(q, c, g.C), out + q * VEC);
    }
    __syncthreads();
  }
}

// Copy the code's block-wide tables (check degrees, prior LLRs) to shared memory.
__device__ __forceinline__ void load_block_tables(const DevGraph& g, const DevArgs& a, unsigned char* smem) {
  uint8_t* s_chk_deg = smem + a.off_chk_deg;
  float* s_llr = reinterpret_cast<float*>(smem + a.off_llr);
  for (int i = threadIdx.x; i < g.C; i += blockDim.x) s_chk_deg[i] = g.chk_deg[i];
  for (int i = threadIdx.x; i < g.V; i += blockDim.x) s_llr[i] = a.llr[i];
}

}  // namespace rbpk
