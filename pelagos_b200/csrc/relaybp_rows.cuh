// Check rows and variable updates of one decode iteration (sm_100a), on a
// group's message slots in shared memory.  Included by relaybp_decode.cuh.
//
// What bounds them: instruction issue.  An iteration of the [[144,12,12]]
// phenomenological code (936 rows of up to 8 messages, 2,592 variables) is 30
// warp-rows and 81 warp-variables; the messages cross the shared-memory pipe
// in about 1,400 wavefronts.  So both passes are written for few instructions:
//
// * Padding slots (rows shorter than MAXDC) always hold +inf: the minimum
//   scan and the sign product run over all MAXDC slots without masks, and only
//   rows that have padding put it back after their vector stores.
// * The sign product is an XOR of the messages' raw bits (three operands per
//   instruction); an output is its edge's minimum times +-alpha (+-1 without
//   normalization), whose sign bit is the row's XOR the message's.
// * Each edge's minimum over the other edges (min2 for a unique smallest, min1
//   for the rest) comes from minima of pairs, quadruples and halves of the row,
//   as three-input minima.
// * 16-bit rows stay packed: two messages per instruction.
// * The dummy slot of absent variable edges always holds 0, so sums need no
//   mask; only the store to it is skipped.
//
// Equality with the reference's operations (kernels.py:1128-1202), which the
// masked form below (check_row_masked) restates literally:
//   sign: a message is never -0.0 where signs are read as bits.  float32: a
//     message is add(lm, sub(sum, nv)); sum starts at +0 and adding never
//     turns it into -0, so sub(sum, nv) is -0 for no nv, and the result is not
//     either.  Initial messages are made by init_msg, which maps -0 to +0.
//     16 bits: rounding a tiny negative gives -0; packed rows add +0 first.
//   NaN: the reference ignores a NaN magnitude, counts it as not negative, and
//     its output to that edge only ever meets the variable's NaN again.  The
//     checks' outputs are finite (magnitudes are capped at 1e30), so a message
//     is NaN only when its memory mix is; float32 / bfloat16 variables then
//     send +inf (edge_mix), which every other edge sees as the same thing.
//     float16 messages saturate and cannot be NaN or inf.
//   min1/min2: min(1e30, .) of the two smallest magnitudes.  Here the cap is
//     one more operand of the minima; a minimum does not depend on the order of
//     its operands, so each edge receives min(1e30, the others) all the same.
// An alpha table or beta that could make a check's output non-finite
// (DevArgs::strict) runs the masked form; so do float64 rows.

#pragma once

#include "relaybp_kernel.cuh"

namespace rbpk {

template <typename M>
__device__ __forceinline__ M pad_value() {
  if constexpr (sizeof(M) == 8) return __longlong_as_double(0x7ff0000000000000ll);
  else if constexpr (sizeof(M) == 4) return __int_as_float(0x7f800000);
  else if constexpr (std::is_same<M, __half>::value) return __ushort_as_half((unsigned short)0x7c00u);
  else return __ushort_as_bfloat16((unsigned short)0x7f80u);
}

// +inf into the padding slots deg..MAXDC-1 of check c.
template <typename M, int MAXDC>
__device__ __forceinline__ void fill_padding(M* msg, int c, int C, int deg) {
#pragma unroll 1
  for (int j = deg; j < MAXDC; ++j) msg[slot_index<M>(j, c, C)] = pad_value<M>();
}

// Packed pairs of 16-bit messages.
template <typename M>
struct Pair16;
template <>
struct Pair16<__half> {
  using T = __half2;
  static constexpr uint32_t kInf = 0x7c007c00u;
  static constexpr uint32_t kCap = 0x7bff7bffu;  // 65504: where float16 messages saturate
};
template <>
struct Pair16<__nv_bfloat16> {
  using T = __nv_bfloat162;
  static constexpr uint32_t kInf = 0x7f807f80u;
  static constexpr uint32_t kCap = 0x714a714au;  // 1e30 rounded to bfloat16
};
template <typename T>
__device__ __forceinline__ uint32_t word_of(T x) {
  return *reinterpret_cast<const uint32_t*>(&x);
}
template <typename T>
__device__ __forceinline__ T pair_of(uint32_t w) {
  return *reinterpret_cast<const T*>(&w);
}

__device__ __forceinline__ float vmin(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ __half2 vmin(__half2 a, __half2 b) { return __hmin2(a, b); }
__device__ __forceinline__ __nv_bfloat162 vmin(__nv_bfloat162 a, __nv_bfloat162 b) { return __hmin2(a, b); }

// Nested minima of two become one three-input instruction: half the ALU work of a scan.
template <typename T>
__device__ __forceinline__ T vmin(T a, T b, T c) {
  return vmin(vmin(a, b), c);
}

// e[j] = min(cap, every m[i] with i != j) for N = 4, 8 or 16 values, as three-input minima.
template <int N, typename T>
__device__ __forceinline__ void exclusive_min(const T (&m)[N], T cap, T (&e)[N]) {
  T p[N / 2];
#pragma unroll
  for (int i = 0; i < N / 2; ++i) p[i] = vmin(m[2 * i], m[2 * i + 1]);
  if constexpr (N == 4) {
#pragma unroll
    for (int j = 0; j < 4; ++j) e[j] = vmin(m[j ^ 1], p[(j >> 1) ^ 1], cap);
  } else if constexpr (N == 8) {
    const T h[2] = {vmin(p[0], p[1], cap), vmin(p[2], p[3], cap)};
#pragma unroll
    for (int j = 0; j < 8; ++j) e[j] = vmin(m[j ^ 1], p[(j >> 1) ^ 1], h[(j >> 2) ^ 1]);
  } else {
    T q[4], o[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = vmin(p[2 * i], p[2 * i + 1]);
    const T h[2] = {vmin(q[0], q[1], cap), vmin(q[2], q[3], cap)};
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = vmin(p[i ^ 1], q[(i >> 1) ^ 1], h[(i >> 2) ^ 1]);
#pragma unroll
    for (int j = 0; j < 16; ++j) e[j] = vmin(m[j ^ 1], o[j >> 1]);
  }
}

// One check row (c2v min-sum, kernels.py:1052-1215) whose padding holds +inf: each
// edge receives the smallest magnitude among the others, which is min2 for a unique
// minimum and min1 for the rest.  sign: the syndrome bit in bit 31 (other bits 0).
// BETA: the offset may be on.  The padding receives values too: restore_row.
template <typename M, int MAXDC, bool BETA>
__device__ __forceinline__ void check_row_packed(M* msg, int c, int C, uint32_t sign, float alpha, bool use_alpha,
                                                 bool use_beta, float beta) {
  constexpr int NW = MAXDC * (int)sizeof(M) / 4;  // 32-bit words of the row
  if constexpr (sizeof(M) == 4) {
    float w[NW], m[NW], e[NW];
    uint32_t x = sign;
#pragma unroll
    for (int q = 0; q < NW / 4; ++q) VecIO<M>::load(msg + chunk_base<M>(q, c, C), w + 4 * q);
#pragma unroll
    for (int j = 0; j < NW; ++j) {
      x ^= __float_as_uint(w[j]);
      m[j] = fabsf(w[j]);
    }
    exclusive_min<NW, float>(m, 1e30f, e);
    float factor = alpha;  // 1 without normalization: the products below only set signs
    if (BETA && use_beta) {
#pragma unroll
      for (int j = 0; j < NW; ++j) e[j] = fmaxf(sub_rn(mul_rn(alpha, e[j]), beta), 0.f);
      factor = 1.f;
    }
    const uint32_t f = (x & 0x80000000u) ^ __float_as_uint(factor);
#pragma unroll
    for (int j = 0; j < NW; ++j)
      e[j] = mul_rn(e[j], __uint_as_float((__float_as_uint(w[j]) & 0x80000000u) ^ f));
#pragma unroll
    for (int q = 0; q < NW / 4; ++q) VecIO<M>::store(msg + chunk_base<M>(q, c, C), e + 4 * q);
  } else {
    uint32_t w[NW];
#pragma unroll
    for (int q = 0; q < NW / 4; ++q) {
      const uint4 u = *reinterpret_cast<const uint4*>(msg + chunk_base<M>(q, c, C));
      w[4 * q] = u.x;
      w[4 * q + 1] = u.y;
      w[4 * q + 2] = u.z;
      w[4 * q + 3] = u.w;
    }
    using T = typename Pair16<M>::T;
    T m[NW], e[NW];
    uint32_t x = 0u;
#pragma unroll
    for (int j = 0; j < NW; ++j) {
      w[j] = word_of(__hadd2_rn(pair_of<T>(w[j]), pair_of<T>(0u)));  // -0 -> +0
      x ^= w[j];
      m[j] = pair_of<T>(w[j] & 0x7fff7fffu);
    }
    x = ((x ^ (x << 16) ^ sign) & 0x80000000u) ? 0x80008000u : 0u;
    // the two halves of the words: each half's minimum bounds the other half's edges
    const bool scaled = use_alpha || (BETA && use_beta);
    const T cap = pair_of<T>(scaled ? Pair16<M>::kInf : Pair16<M>::kCap);  // scaled rows cap in float32 below
    T all = cap;
#pragma unroll
    for (int j = 0; j < NW; ++j) all = vmin(all, m[j]);
    const uint32_t a = word_of(all);
    exclusive_min<NW, T>(m, pair_of<T>(__byte_perm(a, a, 0x1032)), e);
    if (scaled) {
#pragma unroll
      for (int j = 0; j < NW; ++j) {
        float lo = fminf(MsgT<M>::ld(e[j].x), 1e30f), hi = fminf(MsgT<M>::ld(e[j].y), 1e30f);
        if (use_alpha) {
          lo = mul_rn(alpha, lo);
          hi = mul_rn(alpha, hi);
        }
        if (BETA && use_beta) {
          lo = fmaxf(sub_rn(lo, beta), 0.f);
          hi = fmaxf(sub_rn(hi, beta), 0.f);
        }
        e[j].x = MsgT<M>::st(lo);
        e[j].y = MsgT<M>::st(hi);
      }
    }
#pragma unroll
    for (int j = 0; j < NW; ++j) w[j] = word_of(e[j]) ^ ((w[j] & 0x80008000u) ^ x);
#pragma unroll
    for (int q = 0; q < NW / 4; ++q)
      *reinterpret_cast<uint4*>(msg + chunk_base<M>(q, c, C)) =
          make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
  }
}

// After check_row_packed of a row with fewer than MAXDC edges: its padding back to +inf, and
// the only edge of a check receives 0 (kernels.py:1176; the sign of a zero is lost in the sums).
template <typename M, int MAXDC>
__device__ __forceinline__ void restore_row(M* msg, int c, int C, int deg) {
  if (deg == 1) msg[slot_index<M>(0, c, C)] = MsgT<M>::st(0.f);
  fill_padding<M, MAXDC>(msg, c, C, deg);
}

// The same row with its padding masked: any alpha and beta, any message type.
template <typename M, int MAXDC>
__device__ __forceinline__ void check_row_masked(M* msg, int c, int C, int deg, int s, typename MsgT<M>::A alpha,
                                                 bool use_alpha, bool use_beta, typename MsgT<M>::A beta) {
  using A = typename MsgT<M>::A;
  constexpr int VEC = VecIO<M>::N;
  constexpr int NQ = MAXDC / VEC;
  const int swz = chunk_swizzle<M>(c);
  A mv[MAXDC];
#pragma unroll
  for (int q = 0; q < NQ; ++q) VecIO<M>::load(msg + chunk_base<M>(q, c, C), mv + q * VEC);
  const A kInf = A(__int_as_float(0x7f800000));
  int neg = 0;
  A min1 = A(1e30), min2 = A(1e30);
#pragma unroll
  for (int j = 0; j < MAXDC; ++j) {
    // physical position j holds slot (j / VEC) * VEC + ((j % VEC) ^ swz)
    const bool in = ((j % VEC) ^ swz) < deg - (j / VEC) * VEC;
    neg ^= (in && mv[j] < A(0)) ? 1 : 0;
    const A x = in ? fmin(fabs(mv[j]), kInf) : kInf;
    min2 = fmin(min2, fmax(min1, x));
    min1 = fmin(min1, x);
  }
  const bool par = ((neg ^ s) & 1) != 0;
  A lo = deg == 1 ? A(0) : min1;
  A hi = deg == 1 ? A(0) : min2;
  if (use_alpha) {
    lo = mul_rn(alpha, lo);
    hi = mul_rn(alpha, hi);
  }
  if (use_beta) {
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
  for (int q = 0; q < NQ; ++q) VecIO<M>::store(msg + chunk_base<M>(q, c, C), out + q * VEC);
}

// The same row with any number of slots, read one by one (MAXDC 0 kernels).
template <typename M>
__device__ __forceinline__ void check_row_generic(M* msg, int c, int C, int deg, int s, typename MsgT<M>::A alpha,
                                                  bool use_alpha, bool use_beta, typename MsgT<M>::A beta) {
  using IO = MsgT<M>;
  using A = typename IO::A;
  int neg = 0, cnt1 = 0;
  A min1 = A(1e30), min2 = A(1e30);
  for (int j = 0; j < deg; ++j) {
    const A m = IO::ld(msg[slot_index<M>(j, c, C)]);
    neg ^= (m < A(0)) ? 1 : 0;
    const A x = fabs(m);
    if (x < min1) { min2 = min1; min1 = x; cnt1 = 1; }
    else if (x == min1) { cnt1 += 1; }
    else if (x < min2) { min2 = x; }
  }
  const bool par = ((neg ^ s) & 1) != 0;
  for (int j = 0; j < deg; ++j) {
    const int ix = slot_index<M>(j, c, C);
    const A m = IO::ld(msg[ix]);
    A mag = (cnt1 == 1 && fabs(m) == min1) ? min2 : min1;
    if (deg == 1) mag = A(0);
    if (use_alpha) mag = mul_rn(alpha, mag);
    if (use_beta) mag = fmax(sub_rn(mag, beta), A(0));
    msg[ix] = IO::st((par != !(m >= A(0))) ? -mag : mag);
  }
}

// Message of an edge at a phase's start (kernels.py:904-1000): the prior LLR.
template <typename M>
__device__ __forceinline__ M init_msg(typename MsgT<M>::A llr) {
  if constexpr (sizeof(M) == 4) return fminf(add_rn(llr, 0.0f), __int_as_float(0x7f800000));
  else if constexpr (std::is_same<M, __nv_bfloat16>::value) return MsgT<M>::st(fminf(llr, __int_as_float(0x7f800000)));
  else return MsgT<M>::st(llr);
}

// The memory mix as the outgoing messages take it: +inf for NaN (see above).
template <typename M>
__device__ __forceinline__ typename MsgT<M>::A edge_mix(typename MsgT<M>::A lm) {
  if constexpr (sizeof(M) == 4 || std::is_same<M, __nv_bfloat16>::value) return fminf(lm, __int_as_float(0x7f800000));
  else return lm;
}

// Outgoing messages of a variable: lm + (sum - nv[j]) to every present edge.
// off: byte offsets from smem of the variable's edge slots.
template <typename M, int MAXDV>
__device__ __forceinline__ void store_edges(unsigned char* smem, const uint32_t (&off)[MAXDV], uint32_t dummy,
                                            typename MsgT<M>::A lm, typename MsgT<M>::A sum,
                                            const typename MsgT<M>::A (&nv)[MAXDV]) {
  const typename MsgT<M>::A le = edge_mix<M>(lm);
#pragma unroll
  for (int j = 0; j < MAXDV; ++j)
    if (off[j] != dummy) *reinterpret_cast<M*>(smem + off[j]) = MsgT<M>::st(add_rn(le, sub_rn(sum, nv[j])));
}

// Incoming messages and their sum in the graph's edge order (the dummy slot holds 0).
template <typename M, int MAXDV>
__device__ __forceinline__ typename MsgT<M>::A load_edges(const unsigned char* smem, const uint32_t (&off)[MAXDV],
                                                          typename MsgT<M>::A (&nv)[MAXDV]) {
  using A = typename MsgT<M>::A;
  A sum = A(0);
#pragma unroll
  for (int j = 0; j < MAXDV; ++j) {
    nv[j] = MsgT<M>::ld(*reinterpret_cast<const M*>(smem + off[j]));
    sum = add_rn(sum, nv[j]);
  }
  return sum;
}

}  // namespace rbpk
