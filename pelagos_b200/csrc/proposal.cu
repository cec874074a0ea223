// Learned relay-leg proposal: a 2-layer edge-conditioned message-passing
// network on the Tanner graph that maps a shot's syndrome and pre-iteration
// posterior to per-variable memory strengths for the first relay legs.
//
// The reference has no learned proposal.  Its interface is the one these
// strengths go through: per-shot leg gammas, used like explicit_gammas rows
// (src/pelagos/decoder.py:338-340, 481-491, 3685-3688) and bounded by
// gamma_dist_interval (src/pelagos/utils.py:128-160).
//
// Network (widths: node state H=64, message D=16; per shot):
//   z_v = (tanh(P_v/16), [P_v<=0], unsat_v, tanh(llr_v/16)), P clipped to +-1e4
//   t_v = 2[P_v<=0] + [|P_v|<8]                     edge type of v's edges
//   x_c = (s_c, mean_{v in c} z_v, 1)
//   g0  = relu(E x^)
//   layer l = 1, 2:
//     m_c = (W_l g^_c)^,  n_v = (sum_{c in M(v)} m_c)^
//     a_c = sum_{v in N(c)} G_l[t_v] * (n_v - m_c)
//     g_c = relu(g_c + U_l a^_c + b_l)
//   o_c = O . g2^_c,  r_v = sum_{c in M(v)} o_c / deg_v + Oz . z_v + ob
//   gamma_v = lo + (hi - lo) sigmoid(r_v)
// ^ = rounded to bf16.  Weights are bf16 (an fp32 master copy is what AdamW
// updates); every sum accumulates in fp32.
//
// Three implementations of the forward pass:
//   * training kernels: a thread owns one or two rows (checks of a shot), fp32 arithmetic, rounded layer
//     inputs (bf16) and relu bits kept in device memory for the backward kernels; then loss, gradients, AdamW;
//   * net_propose_kernel: the inference pass, one 512-thread block per SM
//     looping over shots, with the graph, a shot's features, messages and
//     per-variable sums in shared memory and the dense layers on the tensor
//     cores (mma.sync m16n8k16 bf16 -> fp32).  A warp owns 16 checks at a
//     time; the 64-wide node states g0/g1/g2 never leave its registers (they
//     are recomputed from the saved 16-wide inputs x, a1, a2 instead of stored);
//   * net_propose_fast_kernel: the same pass, bit for bit, for graphs of low degrees.
// All round at the same points, so training and inference agree to fp32 summation order.

#include "relaybp.h"
#include "relaybp_host.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <type_traits>
#include <vector>

namespace {

using rbph::DevBuf;
using rbph::DeviceGuard;
using rbph::fail;
using rbph::kSMs;
using bf16 = __nv_bfloat16;

constexpr int NH = 64;   // node state width
constexpr int ND = 16;   // message width
constexpr int NF = 4;    // variable features
constexpr int NTY = 4;   // edge types
constexpr int NX = 6;    // check inputs

// flat parameter layout (offsets into theta)
constexpr int P_E = 0;
constexpr int P_W1 = P_E + NH * NX;
constexpr int P_G1 = P_W1 + ND * NH;
constexpr int P_U1 = P_G1 + NTY * ND;
constexpr int P_B1 = P_U1 + NH * ND;
constexpr int P_W2 = P_B1 + NH;
constexpr int P_G2 = P_W2 + ND * NH;
constexpr int P_U2 = P_G2 + NTY * ND;
constexpr int P_B2 = P_U2 + NH * ND;
constexpr int P_O = P_B2 + NH;
constexpr int P_OZ = P_O + NH;
constexpr int P_OB = P_OZ + NF;
constexpr int N_PARAMS = P_OB + 1;
static_assert(N_PARAMS == 4805, "parameter layout");
static_assert(P_W1 % 2 == 0 && P_U1 % 2 == 0 && P_W2 % 2 == 0 && P_U2 % 2 == 0 && P_O % 2 == 0 && P_B1 % 2 == 0 &&
                  P_B2 % 2 == 0,
              "paired bf16 weight loads need even offsets");
static_assert(P_G1 % 8 == 0 && P_G2 % 8 == 0, "gate rows are read as 16-byte vectors");

struct NetGraph {
  int C, V, E;
  const int* chk_ptr;     // [C+1]
  const int* chk_var;     // [E] variable of each edge, check-major
  const int* var_ptr;     // [V+1]
  const int* var_chk;     // [E] check of each edge, variable-major
  const float* llr_feat;  // [V] tanh(llr/16)
};

__device__ __forceinline__ float rbf(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float ldw(const bf16* p, int i) { return __bfloat162float(p[i]); }

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&p);
}

__device__ __forceinline__ void unpack8(const uint4& q, float (&f)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 q;
  q.x = pack_bf16(f[0], f[1]);
  q.y = pack_bf16(f[2], f[3]);
  q.z = pack_bf16(f[4], f[5]);
  q.w = pack_bf16(f[6], f[7]);
  return q;
}

// Sum over the block (valid in thread 0); every thread of the block must call it.
__device__ __forceinline__ float block_sum(float v, float* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float s = 0.f;
  if (threadIdx.x == 0)
    for (int i = 0; i < nw; ++i) s += red[i];
  return s;
}

// ------------------------------------------------------------------ features (training path)

__global__ void feat_var_kernel(NetGraph g, long long B, const uint8_t* syn, const float* post, float* z,
                                uint8_t* ty) {
  const long long n = B * g.V;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long b = i / g.V;
    const int v = (int)(i - b * g.V);
    const float pc = fminf(fmaxf(post[i], -1e4f), 1e4f);
    const bool hard = pc <= 0.f;
    const int k0 = g.var_ptr[v], k1 = g.var_ptr[v + 1];
    int cnt = 0;
    for (int k = k0; k < k1; ++k) cnt += syn[b * g.C + g.var_chk[k]] & 1;
    const float deg = (float)max(k1 - k0, 1);
    float4 f;
    f.x = tanhf(pc * 0.0625f);
    f.y = hard ? 1.f : 0.f;
    f.z = (float)cnt / deg;
    f.w = g.llr_feat[v];
    reinterpret_cast<float4*>(z)[i] = f;
    ty[i] = (uint8_t)((hard ? 2 : 0) + (fabsf(pc) < 8.f ? 1 : 0));
  }
}

// ------------------------------------------------------------------ rows (training path)
//
// A "row" is a check of a shot (row = b C + c), a "node" a variable of a shot.  A thread
// owns a row: its 16- and 64-wide vectors stay in registers or pass through them one
// channel at a time, weights come from shared memory as broadcasts (four per load), and
// every sum runs in the order of a plain loop, in fp32.  What is kept for the backward
// pass is what it needs: the rounded layer inputs (bf16 values, stored as such) and one
// bit per channel for the relu; the 64-wide fp32 node states are recomputed, not stored.
// Arrays are stored in 16-byte columns ([chunk][row]), so a warp's accesses are
// contiguous.  With one thread per output element, each layer re-reading and re-writing
// the node states (245 MB each for 1,024 shots of the 936 x 2,592 graph), a step of
// 1,024 shots took 9.71 ms; now 1.78.

// Gradients are summed in three steps: fp32 within a block (over its rows), one partial sum
// per block in memory, and the blocks' sums in double.  With an atomic add per block the
// additions to the running fp32 sum were the larger part of the error.
constexpr int GRAD_BLOCKS = kSMs * 4;               // at most so many blocks add to a parameter
constexpr int GRAD_STRIDE = (N_PARAMS + 1 + 3) / 4 * 4;  // the loss comes after the parameters
constexpr int RT = 128;       // threads (rows) of a row kernel's tile
// Rows per thread of the row kernels: each weight read from shared memory serves that many rows.
// us per launch at 958,464 rows, one row / two rows: forward stages 1-3 108, 204, 217 / 86, 178,
// 191 (four rows: 108, 253, 266); backward stages 0-2 305, 250, 190 / 274, 240, 234.  So two,
// one in the last of these, and one where two would leave SMs without a block: a step of 16
// shots (14,976 rows) takes 141 us with one row and 156 with two, of 64 shots 246 and 237.
constexpr unsigned TWO_ROWS_FROM = kSMs * 2 * RT;
__host__ __device__ constexpr int forward_blocks(int rows) { return rows == 1 ? 6 : 4; }  // resident per SM
__host__ __device__ constexpr int backward_blocks(int rows) { return rows == 1 ? 4 : 2; }
constexpr int SY = NH + 4;    // padded shared-memory rows of the gradient tiles
constexpr int SX = ND + 4;

struct NetWork {
  float* z;                      // [nv][4] variable features
  uint8_t* ty;                   // [nv] edge type
  uint4* x;                      // [nc] check inputs x^ (8 bf16, 6 used)
  uint4 *m1, *m2, *a1, *a2;      // [2][nc] messages, rounded aggregates
  uint4 *n1, *n2;                // [2][nv] variable sums
  uint4 *g1, *g2;                // [8][nc] round(relu(q)) of layers 1 and 2
  unsigned long long *k1, *k2;   // [nc] bit j: q_j > 0
  float *o, *dout;               // [nc]
  float4 *da, *dm1, *dm2;        // [4][nc]
  float4* dn;                    // [4][nv]
};

__device__ __forceinline__ void load16(const uint4* p, size_t n, size_t i, float (&f)[16]) {
  float h[8];
  unpack8(__ldg(p + i), h);
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = h[j];
  unpack8(__ldg(p + n + i), h);
#pragma unroll
  for (int j = 0; j < 8; ++j) f[8 + j] = h[j];
}

__device__ __forceinline__ void load16(const float4* p, size_t n, size_t i, float (&f)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 v = __ldg(p + q * n + i);
    f[4 * q] = v.x;
    f[4 * q + 1] = v.y;
    f[4 * q + 2] = v.z;
    f[4 * q + 3] = v.w;
  }
}

__device__ __forceinline__ void store16(uint4* p, size_t n, size_t i, const float (&f)[16]) {
  float h[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) h[j] = f[j];
  p[i] = pack8(h);
#pragma unroll
  for (int j = 0; j < 8; ++j) h[j] = f[8 + j];
  p[n + i] = pack8(h);
}

__device__ __forceinline__ void store16(float4* p, size_t n, size_t i, const float (&f)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) p[q * n + i] = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
}

// acc[r] + sum_k f[r][k] w[k], k ascending, w 16 floats in shared memory
template <int R>
__device__ __forceinline__ void dot16(const float (&f)[R][16], const float* w, float (&acc)[R]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 v = *reinterpret_cast<const float4*>(w + 4 * q);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      acc[r] = fmaf(f[r][4 * q], v.x, acc[r]);
      acc[r] = fmaf(f[r][4 * q + 1], v.y, acc[r]);
      acc[r] = fmaf(f[r][4 * q + 2], v.z, acc[r]);
      acc[r] = fmaf(f[r][4 * q + 3], v.w, acc[r]);
    }
  }
}

// acc[r][k] += y[r] w[k]
template <int R>
__device__ __forceinline__ void axpy16(const float (&y)[R], const float* w, float (&acc)[R][16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 v = *reinterpret_cast<const float4*>(w + 4 * q);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      acc[r][4 * q] = fmaf(y[r], v.x, acc[r][4 * q]);
      acc[r][4 * q + 1] = fmaf(y[r], v.y, acc[r][4 * q + 1]);
      acc[r][4 * q + 2] = fmaf(y[r], v.z, acc[r][4 * q + 2]);
      acc[r][4 * q + 3] = fmaf(y[r], v.w, acc[r][4 * q + 3]);
    }
  }
}

// q0_j = E_j . x^
template <int R>
__device__ __forceinline__ void embed(const float (&x)[R][8], const float* e, float (&acc)[R]) {
  const float4 u = *reinterpret_cast<const float4*>(e);
  const float2 v = *reinterpret_cast<const float2*>(e + 4);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    acc[r] = fmaf(x[r][0], u.x, 0.f);
    acc[r] = fmaf(x[r][1], u.y, acc[r]);
    acc[r] = fmaf(x[r][2], u.z, acc[r]);
    acc[r] = fmaf(x[r][3], u.w, acc[r]);
    acc[r] = fmaf(x[r][4], v.x, acc[r]);
    acc[r] = fmaf(x[r][5], v.y, acc[r]);
  }
}

// Weights as fp32 in shared memory: E as [64][8], W (given [16][64]) transposed to [64][16].
__device__ __forceinline__ void stage_e(const bf16* theta, float* s) {
  for (int i = threadIdx.x; i < NH * 8; i += blockDim.x) s[i] = i % 8 < NX ? ldw(theta, P_E + i / 8 * NX + i % 8) : 0.f;
}
__device__ __forceinline__ void stage_t(const bf16* w, float* s) {
  for (int i = threadIdx.x; i < NH * ND; i += blockDim.x) s[i] = ldw(w, i % ND * NH + i / ND);
}
__device__ __forceinline__ void stage(const bf16* w, int n, float* s) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) s[i] = ldw(w, i);
}

// Forward of a row up to its next message (STAGE 1: x^ -> m1; 2: a1 -> m2) or readout (3: a2 -> o).
template <int STAGE, int FR>
__global__ void __launch_bounds__(RT, forward_blocks(FR)) rows_forward_kernel(NetGraph g, unsigned nc, unsigned nv,
                                                                              NetWork w, const bf16* theta,
                                                                              const uint8_t* syn, const float* lmean) {
  __shared__ __align__(16) float sE[NH * 8], sW[NH * ND], sU1[NH * ND], sU2[STAGE == 3 ? NH * ND : 4];
  __shared__ float sb1[NH], sb2[NH], sO[NH];
  __shared__ __align__(16) float sG[NTY * SX];
  stage_e(theta, sE);
  if (STAGE == 1) stage_t(theta + P_W1, sW);
  if (STAGE == 2) stage_t(theta + P_W2, sW);
  if (STAGE >= 2) {
    stage(theta + P_U1, NH * ND, sU1);
    stage(theta + P_B1, NH, sb1);
    const bf16* G = theta + (STAGE == 2 ? P_G1 : P_G2);
    for (int i = threadIdx.x; i < NTY * ND; i += RT) sG[i / ND * SX + i % ND] = ldw(G, i);
  }
  if (STAGE == 3) {
    stage(theta + P_U2, NH * ND, sU2);
    stage(theta + P_B2, NH, sb2);
    stage(theta + P_O, NH, sO);
  }
  __syncthreads();
  for (unsigned r0 = blockIdx.x * (RT * FR) + threadIdx.x; r0 < nc; r0 += gridDim.x * (RT * FR)) {
    float x[FR][8], a[FR][16], al[FR][16];  // al: layer 1's aggregates in stage 3
#pragma unroll
    for (int i = 0; i < FR; ++i) {
      const unsigned row = min(r0 + i * RT, nc - 1);  // past the end: the last row once more, not stored
      const bool in = r0 + i * RT < nc;
      const unsigned b = row / (unsigned)g.C, c = row - b * (unsigned)g.C;
      const int e0 = g.chk_ptr[c], e1 = g.chk_ptr[c + 1];
      const size_t v0 = (size_t)b * g.V;
      if constexpr (STAGE == 1) {
        float s0 = 0.f, s1 = 0.f, s2 = 0.f;
        for (int e = e0; e < e1; ++e) {
          const float4 f = __ldg(reinterpret_cast<const float4*>(w.z) + v0 + g.chk_var[e]);
          s0 += f.x;
          s1 += f.y;
          s2 += f.z;
        }
        const float deg = (float)max(e1 - e0, 1);
        const float xi[8] = {(float)(syn[row] & 1), s0 / deg, s1 / deg, s2 / deg, lmean[c], 1.f, 0.f, 0.f};
        const uint4 q = pack8(xi);
        if (in) w.x[row] = q;
        unpack8(q, x[i]);
      } else {
        unpack8(__ldg(w.x + row), x[i]);
      }
      if constexpr (STAGE >= 2) {
        // a_c = sum_{v in N(c)} G[t_v] (n_v - m_c)
        const uint4* n = STAGE == 2 ? w.n1 : w.n2;
        float mc[16];
        load16(STAGE == 2 ? w.m1 : w.m2, nc, row, mc);
#pragma unroll
        for (int k = 0; k < 16; ++k) a[i][k] = 0.f;
        for (int e = e0; e < e1; ++e) {
          const size_t v = v0 + g.chk_var[e];
          float nf[16];
          load16(n, nv, v, nf);
          const float* gt = sG + __ldg(w.ty + v) * SX;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 t = *reinterpret_cast<const float4*>(gt + 4 * q);
            a[i][4 * q] = fmaf(t.x, nf[4 * q] - mc[4 * q], a[i][4 * q]);
            a[i][4 * q + 1] = fmaf(t.y, nf[4 * q + 1] - mc[4 * q + 1], a[i][4 * q + 1]);
            a[i][4 * q + 2] = fmaf(t.z, nf[4 * q + 2] - mc[4 * q + 2], a[i][4 * q + 2]);
            a[i][4 * q + 3] = fmaf(t.w, nf[4 * q + 3] - mc[4 * q + 3], a[i][4 * q + 3]);
          }
        }
        if (in) store16(STAGE == 2 ? w.a1 : w.a2, nc, row, a[i]);
#pragma unroll
        for (int k = 0; k < 16; ++k) a[i][k] = rbf(a[i][k]);  // the layer's input
        if constexpr (STAGE == 3) load16(w.a1, nc, row, al[i]);
      }
    }
    float m[FR][16] = {}, o[FR] = {};
    unsigned long long mask[FR] = {};
#pragma unroll 1
    for (int ch = 0; ch < NH / 8; ++ch) {
      float gv[FR][8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int j = ch * 8 + k;
        float q[FR], y[FR];
        embed(x, sE + j * 8, q);
        if constexpr (STAGE >= 2) {
          float u[FR] = {};
          if constexpr (STAGE == 2) dot16(a, sU1 + j * ND, u);
          else dot16(al, sU1 + j * ND, u);
#pragma unroll
          for (int i = 0; i < FR; ++i) q[i] = u[i] + sb1[j] + fmaxf(q[i], 0.f);
        }
        if constexpr (STAGE == 3) {
          float u[FR] = {};
          dot16(a, sU2 + j * ND, u);
#pragma unroll
          for (int i = 0; i < FR; ++i) q[i] = u[i] + sb2[j] + fmaxf(q[i], 0.f);
        }
#pragma unroll
        for (int i = 0; i < FR; ++i) {
          if (q[i] > 0.f) mask[i] |= 1ull << j;
          gv[i][k] = y[i] = rbf(fmaxf(q[i], 0.f));
          if constexpr (STAGE == 3) o[i] = fmaf(y[i], sO[j], o[i]);
        }
        if constexpr (STAGE < 3) axpy16(y, sW + j * ND, m);
      }
      if constexpr (STAGE >= 2) {
#pragma unroll
        for (int i = 0; i < FR; ++i)
          if (r0 + i * RT < nc) (STAGE == 2 ? w.g1 : w.g2)[(size_t)ch * nc + r0 + i * RT] = pack8(gv[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < FR; ++i) {
      const unsigned row = r0 + i * RT;
      if (row >= nc) break;
      if constexpr (STAGE == 1) store16(w.m1, nc, row, m[i]);
      if constexpr (STAGE == 2) {
        store16(w.m2, nc, row, m[i]);
        w.k1[row] = mask[i];
      }
      if constexpr (STAGE == 3) {
        w.o[row] = o[i];
        w.k2[row] = mask[i];
      }
    }
  }
}

// n_v = round(sum_{c in M(v)} m_c): a thread per node and half of the channels.
__global__ void varsum_kernel(NetGraph g, unsigned nc, unsigned nv, const uint4* m, uint4* n) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const unsigned b = i / (unsigned)g.V, v = i - b * (unsigned)g.V;
  const uint4* mh = m + (size_t)blockIdx.y * nc + (size_t)b * g.C;
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int k = g.var_ptr[v]; k < g.var_ptr[v + 1]; ++k) {
    float f[8];
    unpack8(__ldg(mh + g.var_chk[k]), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] += f[j];
  }
  n[(size_t)blockIdx.y * nv + i] = pack8(s);
}

// dn_v = G[t_v] sum_{c in M(v)} da_c: a thread per node and quarter of the channels.
__global__ void dn_kernel(NetGraph g, unsigned nc, unsigned nv, const bf16* G, const uint8_t* ty, const float4* da,
                          float4* dn) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const int q = blockIdx.y;
  const unsigned b = i / (unsigned)g.V, v = i - b * (unsigned)g.V;
  const float4* dc = da + (size_t)q * nc + (size_t)b * g.C;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k = g.var_ptr[v]; k < g.var_ptr[v + 1]; ++k) {
    const float4 d = __ldg(dc + g.var_chk[k]);
    s.x += d.x;
    s.y += d.y;
    s.z += d.z;
    s.w += d.w;
  }
  const bf16* gt = G + ty[i] * ND + 4 * q;
  dn[(size_t)q * nv + i] = make_float4(ldw(gt, 0) * s.x, ldw(gt, 1) * s.y, ldw(gt, 2) * s.z, ldw(gt, 3) * s.w);
}

// Backward of the aggregation and of the variable sums: dm_c = -(sum_v G[t_v]) da_c + sum_v dn_v and
// dG[t] += da_c (n_v - m_c), a thread per row and quarter of the channels; the gate gradients stay
// in the thread's registers over all its rows.
__global__ void __launch_bounds__(512) dm_kernel(NetGraph g, unsigned nc, unsigned nv, const bf16* G, const uint8_t* ty,
                                                 const uint4* m, const uint4* n, const float4* da, const float4* dn,
                                                 float4* dm, float* dG) {
  __shared__ __align__(16) float gs[NTY * ND];
  __shared__ float acc[16][NTY * ND];
  for (int i = threadIdx.x; i < NTY * ND; i += blockDim.x) gs[i] = ldw(G, i);
  __syncthreads();
  const int q = threadIdx.x & 3;
  float part[NTY][4] = {};
  for (unsigned row = blockIdx.x * 128 + (threadIdx.x >> 2); row < nc; row += gridDim.x * 128) {
    const unsigned b = row / (unsigned)g.C, c = row - b * (unsigned)g.C;
    const size_t v0 = (size_t)b * g.V;
    auto quad = [&](const uint4* p, size_t i) {  // channels 4q .. 4q+3 of a bf16 half row
      const uint2 u = __ldg(reinterpret_cast<const uint2*>(p + i) + (q & 1));
      const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
      const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
      return make_float4(lo.x, lo.y, hi.x, hi.y);
    };
    const float4 mc = quad(m + (size_t)(q >> 1) * nc, row);
    const float4 d = __ldg(da + (size_t)q * nc + row);
    float4 gsum = make_float4(0.f, 0.f, 0.f, 0.f), s = gsum;
    for (int e = g.chk_ptr[c]; e < g.chk_ptr[c + 1]; ++e) {
      const size_t v = v0 + g.chk_var[e];
      const int t = __ldg(ty + v);
      const float4 nf = quad(n + (size_t)(q >> 1) * nv, v);
      const float4 gt = *reinterpret_cast<const float4*>(gs + t * ND + 4 * q);
      const float4 dv = __ldg(dn + (size_t)q * nv + v);
      gsum.x += gt.x;
      gsum.y += gt.y;
      gsum.z += gt.z;
      gsum.w += gt.w;
      s.x += dv.x;
      s.y += dv.y;
      s.z += dv.z;
      s.w += dv.w;
#pragma unroll
      for (int tt = 0; tt < NTY; ++tt)
        if (t == tt) {
          part[tt][0] = fmaf(d.x, nf.x - mc.x, part[tt][0]);
          part[tt][1] = fmaf(d.y, nf.y - mc.y, part[tt][1]);
          part[tt][2] = fmaf(d.z, nf.z - mc.z, part[tt][2]);
          part[tt][3] = fmaf(d.w, nf.w - mc.w, part[tt][3]);
        }
    }
    dm[(size_t)q * nc + row] =
        make_float4(-gsum.x * d.x + s.x, -gsum.y * d.y + s.y, -gsum.z * d.z + s.z, -gsum.w * d.w + s.w);
  }
#pragma unroll
  for (int tt = 0; tt < NTY; ++tt)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float p = part[tt][i];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
      if ((threadIdx.x & 31) < 4) acc[threadIdx.x >> 5][tt * ND + 4 * q + i] = p;
    }
  __syncthreads();
  if (threadIdx.x < NTY * ND) {
    float s = 0.f;
    for (int k = 0; k < 16; ++k) s += acc[k][threadIdx.x];
    dG[(size_t)blockIdx.x * GRAD_STRIDE + threadIdx.x] = s;
  }
}

// acc[i][k] += sum over a warp's tile of y[j(i)] x[4 kq + k], j(i) = 4 jq + i, then 32 + 4 jq + i - 4: a lane's
// 8 x 4 block of the 64 x 16 outer products, 32 fmas per three 16-byte shared-memory loads.
template <int WR>
__device__ __forceinline__ void outer_sum(const float* sy, const float* sx, int jq, int kq, float (&acc)[8][4]) {
#pragma unroll 4
  for (int r = 0; r < WR; ++r) {
    const float4 y0 = *reinterpret_cast<const float4*>(sy + r * SY + 4 * jq);
    const float4 y1 = *reinterpret_cast<const float4*>(sy + r * SY + 32 + 4 * jq);
    const float4 x = *reinterpret_cast<const float4*>(sx + r * SX + 4 * kq);
    const float y[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      acc[i][0] = fmaf(y[i], x.x, acc[i][0]);
      acc[i][1] = fmaf(y[i], x.y, acc[i][1]);
      acc[i][2] = fmaf(y[i], x.z, acc[i][2]);
      acc[i][3] = fmaf(y[i], x.w, acc[i][3]);
    }
  }
}

// Backward of a row from the readout (STAGE 2) or from dm2 (1) to the aggregates' gradients da,
// or from dm1 to the inputs (0), and the weight gradients of that stretch: per warp and
// tile of rows each 64-wide vector (dq, then the layer's input g) is laid in shared memory next
// to the 16-wide one it multiplies, and a lane adds up its 8 x 4 block of the outer products
// over the warp's own rows, without a block barrier until the warps' sums are added up at the
// end.  Shared-memory loads bound these kernels more than the fmas: with a tile per block and
// 2 x 4 blocks (two loads per 8 fmas) the stages took 339, 307 and 255 us, now 274, 241 and 190.
//   dq2_j = dout O_j [q2_j > 0],  dq1 = (dq2 + W2^T dm2) [q1 > 0],  dq0 = (dq1 + W1^T dm1) [q0 > 0]
//   2: dO += dout g2, dU2 += dq2 a2^T, db2 += dq2, da = U2^T dq2
//   1: dW2 += dm2 g1^T, dU1 += dq1 a1^T, db1 += dq1, da = U1^T dq1
//   0: dW1 += dm1 g0^T, dE += dq0 x^T
template <int STAGE, int BR>
__global__ void __launch_bounds__(RT, backward_blocks(BR)) rows_backward_kernel(NetGraph g, unsigned nc, NetWork w,
                                                                                const bf16* theta, const float* dr,
                                                                                float* grad) {
  constexpr int WR = 32 * BR;  // rows of a warp's tile
  extern __shared__ __align__(16) float sm[];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, jq = lane >> 2, kq = lane & 3;
  float* sy = sm + warp * (WR * (SY + SX));      // this warp's [WR][SY]
  float* sx = sy + WR * SY;                      // [WR][SX]
  float* sO = sm + RT / 32 * (WR * (SY + SX));   // [64]
  float* sW2 = sO + NH;                          // [64][16] transposed (stages 1, 0)
  float* sU = sW2 + (STAGE == 2 ? 0 : NH * ND);  // [64][16]: U2 or U1 (stages 2, 1)
  float* sW1 = sU;                               // [64][16] transposed (stage 0)
  float* sE = sW1 + NH * ND;                     // [64][8] (stage 0)
  stage(theta + P_O, NH, sO);
  if (STAGE == 2) stage(theta + P_U2, NH * ND, sU);
  if (STAGE == 1) stage(theta + P_U1, NH * ND, sU);
  if (STAGE <= 1) stage_t(theta + P_W2, sW2);
  if (STAGE == 0) {
    stage_t(theta + P_W1, sW1);
    stage_e(theta, sE);
  }
  __syncthreads();
  float acc_y[8][4] = {}, acc_g[8][4] = {}, acc_b[2] = {}, acc_o[2] = {};
  const unsigned nt = (nc + WR - 1) / WR;  // tiles of a warp's rows
  for (unsigned tile = blockIdx.x * (RT / 32) + warp; tile < nt; tile += gridDim.x * (RT / 32)) {
    float da[BR][16] = {}, dm2[BR][16] = {}, dm1[BR][16] = {}, x[BR][8] = {}, dout[BR] = {};
    unsigned long long k2[BR] = {}, k1[BR] = {};
    __syncwarp();  // the last tile's sums are done
#pragma unroll
    for (int i = 0; i < BR; ++i) {
      const unsigned row = tile * WR + i * 32 + lane;
      const bool in = row < nc;
      float* myx = sx + (i * 32 + lane) * SX;
      if (in) {
        k2[i] = w.k2[row];
        if constexpr (STAGE == 2) {
          const unsigned b = row / (unsigned)g.C, c = row - b * (unsigned)g.C;
          for (int e = g.chk_ptr[c]; e < g.chk_ptr[c + 1]; ++e) {
            const int v = g.chk_var[e];
            dout[i] += __ldg(dr + (size_t)b * g.V + v) / (float)max(g.var_ptr[v + 1] - g.var_ptr[v], 1);
          }
          w.dout[row] = dout[i];
        } else {
          dout[i] = w.dout[row];
          k1[i] = w.k1[row];
          load16(w.dm2, nc, row, dm2[i]);
        }
        if constexpr (STAGE == 0) {
          load16(w.dm1, nc, row, dm1[i]);
          unpack8(__ldg(w.x + row), x[i]);
        }
      }
      // the 16-wide factor of dq: a2, a1 or x^
      float a[16] = {};
      if constexpr (STAGE == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = x[i][k];
      } else if (in) {
        load16(STAGE == 2 ? w.a2 : w.a1, nc, row, a);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<float4*>(myx + 4 * q) = make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
    }
#pragma unroll 1
    for (int j0 = 0; j0 < NH; j0 += 4) {
      float dq[BR][4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int j = j0 + k;
        float d[BR], u[BR] = {};
#pragma unroll
        for (int i = 0; i < BR; ++i) d[i] = (k2[i] >> j) & 1ull ? dout[i] * sO[j] : 0.f;
        if constexpr (STAGE <= 1) {
          dot16(dm2, sW2 + j * ND, u);
#pragma unroll
          for (int i = 0; i < BR; ++i) d[i] = (k1[i] >> j) & 1ull ? d[i] + u[i] : 0.f;
        }
        if constexpr (STAGE == 0) {
          float u1[BR] = {}, q0[BR];
          dot16(dm1, sW1 + j * ND, u1);
          embed(x, sE + j * 8, q0);
#pragma unroll
          for (int i = 0; i < BR; ++i) d[i] = q0[i] > 0.f ? d[i] + u1[i] : 0.f;
        } else {
          axpy16(d, sU + j * ND, da);
        }
#pragma unroll
        for (int i = 0; i < BR; ++i) dq[i][k] = d[i];
      }
#pragma unroll
      for (int i = 0; i < BR; ++i)
        *reinterpret_cast<float4*>(sy + (i * 32 + lane) * SY + j0) =
            make_float4(dq[i][0], dq[i][1], dq[i][2], dq[i][3]);
    }
    if constexpr (STAGE >= 1) {
#pragma unroll
      for (int i = 0; i < BR; ++i) {
        const unsigned row = tile * WR + i * 32 + lane;
        if (row < nc) store16(w.da, nc, row, da[i]);
      }
    }
    __syncwarp();
    outer_sum<WR>(sy, sx, jq, kq, acc_y);
    if constexpr (STAGE >= 1) {  // biases: lane and lane + 32
#pragma unroll 8
      for (int r = 0; r < WR; ++r) {
        acc_b[0] += sy[r * SY + lane];
        acc_b[1] += sy[r * SY + 32 + lane];
      }
    }
    __syncwarp();
    // the layer's input g and its factor: dout, dm2 or dm1
#pragma unroll
    for (int i = 0; i < BR; ++i) {
      const unsigned row = tile * WR + i * 32 + lane;
      const bool in = row < nc;
      float* y = sy + (i * 32 + lane) * SY;
      float* myx = sx + (i * 32 + lane) * SX;
      if constexpr (STAGE != 0) {
#pragma unroll
        for (int ch = 0; ch < NH / 8; ++ch) {
          float gv[8] = {};
          if (in) unpack8(__ldg((STAGE == 2 ? w.g2 : w.g1) + (size_t)ch * nc + row), gv);
          *reinterpret_cast<float4*>(y + ch * 8) = make_float4(gv[0], gv[1], gv[2], gv[3]);
          *reinterpret_cast<float4*>(y + ch * 8 + 4) = make_float4(gv[4], gv[5], gv[6], gv[7]);
        }
      }
      if constexpr (STAGE == 2) {
        myx[0] = dout[i];
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float* f = (STAGE == 1 ? dm2[i] : dm1[i]) + 4 * q;
          *reinterpret_cast<float4*>(myx + 4 * q) = make_float4(f[0], f[1], f[2], f[3]);
        }
      }
    }
    if constexpr (STAGE == 0) {
#pragma unroll 1
      for (int j0 = 0; j0 < NH; j0 += 4) {
        float gv[BR][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float q0[BR];
          embed(x, sE + (j0 + k) * 8, q0);
#pragma unroll
          for (int i = 0; i < BR; ++i) gv[i][k] = rbf(fmaxf(q0[i], 0.f));
        }
#pragma unroll
        for (int i = 0; i < BR; ++i)
          *reinterpret_cast<float4*>(sy + (i * 32 + lane) * SY + j0) =
              make_float4(gv[i][0], gv[i][1], gv[i][2], gv[i][3]);
      }
    }
    __syncwarp();
    if constexpr (STAGE == 2) {
#pragma unroll 8
      for (int r = 0; r < WR; ++r) {
        const float d = sx[r * SX];
        acc_o[0] = fmaf(d, sy[r * SY + lane], acc_o[0]);
        acc_o[1] = fmaf(d, sy[r * SY + 32 + lane], acc_o[1]);
      }
    } else {
      outer_sum<WR>(sy, sx, jq, kq, acc_g);
    }
  }
  // the warps' sums, one after another in shared memory
  __syncthreads();
  float* red = sm;  // [4][1024] a warp's outer products as [j][k]
  float* out = grad + (size_t)blockIdx.x * GRAD_STRIDE;
  static_assert(RT / 32 * NH * ND <= RT / 32 * WR * (SY + SX), "the warps' sums fit their tiles");
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    if (STAGE == 2 && pass == 1) break;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float* f = pass ? acc_g[i] : acc_y[i];
      const int j = 4 * jq + (i < 4 ? i : 28 + i);
      *reinterpret_cast<float4*>(red + (warp * NH + j) * ND + 4 * kq) = make_float4(f[0], f[1], f[2], f[3]);
    }
    __syncthreads();
    for (int i = t; i < NH * ND; i += RT) {
      float q = 0.f;
      for (int k = 0; k < RT / 32; ++k) q += red[k * NH * ND + i];
      const int j = i / ND, k = i % ND;
      if (pass) out[(STAGE == 1 ? P_W2 : P_W1) + k * NH + j] = q;
      else if (STAGE >= 1) out[(STAGE == 2 ? P_U2 : P_U1) + i] = q;
      else if (k < NX) out[P_E + j * NX + k] = q;
    }
    __syncthreads();
  }
  if constexpr (STAGE >= 1) {
    red[(warp * 2) * NH + lane] = acc_b[0];
    red[(warp * 2) * NH + 32 + lane] = acc_b[1];
    red[(warp * 2 + 1) * NH + lane] = acc_o[0];
    red[(warp * 2 + 1) * NH + 32 + lane] = acc_o[1];
    __syncthreads();
    if (t < (STAGE == 2 ? 2 : 1) * NH) {
      float q = 0.f;
      for (int k = 0; k < RT / 32; ++k) q += red[k * 2 * NH + t];
      out[t < NH ? (STAGE == 2 ? P_B2 : P_B1) + t : P_O + t - NH] = q;
    }
  }
}
constexpr int rows_backward_smem(int stage, int rows) {
  return (RT * rows * (SY + SX) + NH + (stage == 2 ? 1 : 2) * NH * ND + (stage == 0 ? NH * 8 : 0)) * 4;
}

// ------------------------------------------------------------------ readout and loss (training path)

// r = sum_{c in M(v)} o_c / deg_v + Oz.z_v + ob.  With targets: the weighted
// logistic loss (divided by B V), dr, and the Oz / ob gradients, as the block's partial sums.
__global__ void __launch_bounds__(256) readout_kernel(NetGraph g, long long B, const bf16* theta, const float* o,
                                                      const float* z, const uint8_t* y, float w_neg, float* r,
                                                      float* dr, float* grad) {
  __shared__ float red[32];
  const float oz0 = ldw(theta, P_OZ), oz1 = ldw(theta, P_OZ + 1), oz2 = ldw(theta, P_OZ + 2),
              oz3 = ldw(theta, P_OZ + 3), ob = ldw(theta, P_OB);
  const long long tot = B * g.V;
  const float inv_n = 1.f / (float)tot;
  float l_acc = 0.f, g0 = 0.f, g1 = 0.f, g2 = 0.f, g3 = 0.f, gb = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot; i += (long long)gridDim.x * blockDim.x) {
    const long long b = i / g.V;
    const int v = (int)(i - b * g.V);
    const int k0 = g.var_ptr[v], k1 = g.var_ptr[v + 1];
    float s = 0.f;
    for (int k = k0; k < k1; ++k) s += o[b * g.C + g.var_chk[k]];
    const float4 f = reinterpret_cast<const float4*>(z)[i];
    const float rv = s / (float)max(k1 - k0, 1) + (oz0 * f.x + oz1 * f.y + oz2 * f.z + oz3 * f.w) + ob;
    r[i] = rv;
    if (y) {
      const float yv = (float)(y[i] & 1);
      const float w = yv > 0.f ? 1.f : w_neg;
      const float sp = fmaxf(rv, 0.f) + log1pf(expf(-fabsf(rv)));
      l_acc += w * (sp - yv * rv);
      const float d = w * (1.f / (1.f + expf(-rv)) - yv) * inv_n;
      dr[i] = d;
      g0 += d * f.x;
      g1 += d * f.y;
      g2 += d * f.z;
      g3 += d * f.w;
      gb += d;
    }
  }
  if (!y) return;  // uniform over the block
  const float vals[6] = {l_acc * inv_n, g0, g1, g2, g3, gb};
  float* out = grad + (size_t)blockIdx.x * GRAD_STRIDE;
  const int dst[6] = {N_PARAMS, P_OZ, P_OZ + 1, P_OZ + 2, P_OZ + 3, P_OB};
  for (int q = 0; q < 6; ++q) {
    const float t = block_sum(vals[q], red);
    if (threadIdx.x == 0) out[dst[q]] = t;
  }
}

// The blocks' partial sums of each parameter (and of the loss), added in double: 32 warps share
// 32 parameters, so that the latency of a few loads bounds the kernel (8 warps: 36 us for 592
// rows of partial sums, now 11).  rows / last / gates / vars: blocks of the kernels behind a parameter (last: the
// second layer's update and readout).
__global__ void __launch_bounds__(1024) grad_sum_kernel(const float* partial, int rows, int last, int gates, int vars,
                                                       float* grad, float* loss) {
  __shared__ double part[32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, p = blockIdx.x * 32 + lane;
  const bool gate = (p >= P_G1 && p < P_U1) || (p >= P_G2 && p < P_U2);
  const int n = p > N_PARAMS ? 0 : (gate ? gates : (p >= P_OZ ? vars : (p >= P_U2 ? last : rows)));
  double s = 0.0;
#pragma unroll 4
  for (int k = warp; k < n; k += 32) s += (double)partial[(size_t)k * GRAD_STRIDE + p];
  part[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && p <= N_PARAMS) {
    for (int k = 1; k < 32; ++k) s += part[k][lane];
    if (p < N_PARAMS) grad[p] = (float)s;
    else *loss = (float)s;
  }
}

// AdamW with decoupled weight decay and bias-corrected moments; refreshes the bf16 copy.
__global__ void adamw_kernel(int n, float* theta, float* m, float* v, const float* grad, bf16* theta_bf, float lr,
                             float beta1, float beta2, float eps, float wd, float bc1, float bc2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = grad[i];
    float p = theta[i] * (1.f - lr * wd);
    const float mi = beta1 * m[i] + (1.f - beta1) * gi;
    const float vi = beta2 * v[i] + (1.f - beta2) * gi * gi;
    p -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    m[i] = mi;
    v[i] = vi;
    theta[i] = p;
    theta_bf[i] = __float2bfloat16_rn(p);
  }
}

__global__ void to_bf16_kernel(int n, const float* x, bf16* y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = __float2bfloat16_rn(x[i]);
}

// ------------------------------------------------------------------ fused inference (tensor cores)
//
// One 512-thread block per SM takes shots from a grid-stride loop.  Shared
// memory (bf16 rows unless noted):
//   s_w  all weights, staged once per block     s_g  the graph's index arrays (u16), once per block
//   s_x  [C][8]  check inputs x^ (6 used)       s_th [V] f32 tanh feature
//   s_m  [C][16] messages of the current layer  s_tu [V] u8  type | unsat-count << 2
//   s_n  [V][8]  their per-variable sums, for   s_syn [C] u8
//                one half of the channels at a time
//   s_a1, s_a2 [C][16] aggregated layer inputs a^ (kept: the tile passes
//                recompute g0 and g1 from x^ and a1^ instead of storing them)
// Phases per shot, separated by block barriers: variable features; check
// inputs; per layer: tile pass (messages), then per half of the channels the
// variable sums and the check aggregation; tile pass 3 (layer-2 update and
// o); variable readout.  A warp's tile is 16 checks: x^ / a^ rows are loaded
// as mma A fragments, weights as B fragments from s_w, and each layer's fp32
// accumulators become the next layer's A fragments in registers.

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float sw_f(const bf16* w, int i) { return __bfloat162float(w[i]); }

// B operands of the tensor-core layers, stored per fragment so that a warp
// reads each fragment as 32 consecutive words (lane l at word l): no bank
// conflicts, unlike reading the [n][k] weight rows directly (a 128-byte row
// stride puts the 8 rows of a fragment in one bank).
constexpr int FR_E = 0;                   // [nt 8] (k 0..7; k >= 6 is zero)
constexpr int FR_W1 = FR_E + 8 * 32;      // [nt 2][kk 4][half 2]
constexpr int FR_W2 = FR_W1 + 16 * 32;
constexpr int FR_U1 = FR_W2 + 16 * 32;    // [nt 8][half 2]
constexpr int FR_U2 = FR_U1 + 16 * 32;
constexpr int FR_O = FR_U2 + 16 * 32;     // [kk 4][half 2], column 0 only
constexpr int FR_WORDS = FR_O + 8 * 32;

__device__ __forceinline__ uint32_t theta_pair(const bf16* th, int i) {
  return (uint32_t)__bfloat16_as_ushort(th[i]) | ((uint32_t)__bfloat16_as_ushort(th[i + 1]) << 16);
}

// Word w of the fragment table (lane = w % 32: row n = nt*8 + lane/4, columns k, k+1 with k = ... + 2 (lane%4)).
__device__ uint32_t fragment_word(const bf16* th, int w) {
  const int lane = w & 31, f = w >> 5, gq = lane >> 2, k2 = 2 * (lane & 3);
  if (w < FR_W1) {
    const int n = f * 8 + gq;
    return k2 < NX ? theta_pair(th, P_E + n * NX + k2) : 0u;
  }
  if (w < FR_U1) {
    const int base = w < FR_W2 ? P_W1 : P_W2;
    const int ff = f - (w < FR_W2 ? FR_W1 : FR_W2) / 32;
    const int nt = ff >> 3, kk = (ff >> 1) & 3, half = ff & 1;
    return theta_pair(th, base + (nt * 8 + gq) * NH + kk * 16 + half * 8 + k2);
  }
  if (w < FR_O) {
    const int base = w < FR_U2 ? P_U1 : P_U2;
    const int ff = f - (w < FR_U2 ? FR_U1 : FR_U2) / 32;
    const int nt = ff >> 1, half = ff & 1;
    return theta_pair(th, base + (nt * 8 + gq) * ND + half * 8 + k2);
  }
  const int ff = f - FR_O / 32;
  const int kk = ff >> 1, half = ff & 1;
  return gq == 0 ? theta_pair(th, P_O + kk * 16 + half * 8 + k2) : 0u;
}

struct ProposeArgs {
  long long B;
  const uint8_t* syn;       // [B, C]
  const float* post;        // row b at post + b * post_stride
  long long post_stride;    // elements between rows (>= V)
  float lo, hi;
  float* gammas;            // [B, V] or null
  float* logits;            // [B, V] or null
  const int32_t* shot_list;   // [B] shots to evaluate, or null: all
  const int32_t* list_count;  // device count of shot_list entries, or null: B
  const bf16* theta;        // [N_PARAMS]
  const float* chk_lmean;   // [C] mean of the check's variables' tanh(llr/16)
  const uint16_t* graph16;  // chk_ptr [C+1], chk_var [E], var_ptr [V+1], var_chk [E]
  int graph16_len;          // entries, a multiple of 8
  int off_w, off_fr, off_g, off_x, off_m, off_n, off_a1, off_a2, off_th, off_tu, off_syn;  // shared-memory byte offsets
};

// Rows r0, r0+8 of a bf16 [rows][16] array as an A fragment (zero past C).
__device__ __forceinline__ void load_a16(const bf16* s, int r0, int tq, int C, uint32_t (&a)[4]) {
  const int r1 = r0 + 8;
  a[0] = r0 < C ? *reinterpret_cast<const uint32_t*>(s + r0 * ND + 2 * tq) : 0u;
  a[1] = r1 < C ? *reinterpret_cast<const uint32_t*>(s + r1 * ND + 2 * tq) : 0u;
  a[2] = r0 < C ? *reinterpret_cast<const uint32_t*>(s + r0 * ND + 8 + 2 * tq) : 0u;
  a[3] = r1 < C ? *reinterpret_cast<const uint32_t*>(s + r1 * ND + 8 + 2 * tq) : 0u;
}

// q0 = x^ E^T for the warp's 16 checks (8 n-tiles of 8 columns); x rows are 8 wide.
__device__ __forceinline__ void tile_embed(const uint32_t* fr, const bf16* s_x, int r0, int lane, int tq, int C,
                                           float (&acc)[8][4]) {
  uint32_t a[4];
  a[0] = (r0 < C && tq < 3) ? *reinterpret_cast<const uint32_t*>(s_x + r0 * 8 + 2 * tq) : 0u;
  a[1] = (r0 + 8 < C && tq < 3) ? *reinterpret_cast<const uint32_t*>(s_x + (r0 + 8) * 8 + 2 * tq) : 0u;
  a[2] = 0u;
  a[3] = 0u;
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    mma_bf16(acc[nt], a, fr[FR_E + nt * 32 + lane], 0u);
  }
}

// A fragments (4 k-tiles of 16) of round(relu(acc)).
__device__ __forceinline__ void relu_to_a(const float (&acc)[8][4], uint32_t (&ga)[4][4]) {
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    ga[kk][0] = pack_bf16(fmaxf(acc[2 * kk][0], 0.f), fmaxf(acc[2 * kk][1], 0.f));
    ga[kk][1] = pack_bf16(fmaxf(acc[2 * kk][2], 0.f), fmaxf(acc[2 * kk][3], 0.f));
    ga[kk][2] = pack_bf16(fmaxf(acc[2 * kk + 1][0], 0.f), fmaxf(acc[2 * kk + 1][1], 0.f));
    ga[kk][3] = pack_bf16(fmaxf(acc[2 * kk + 1][2], 0.f), fmaxf(acc[2 * kk + 1][3], 0.f));
  }
}

// m = round(g^ W^T) for the tile, stored as bf16 rows of 16.
__device__ __forceinline__ void tile_message(const uint32_t* fr, int fw, const uint32_t (&ga)[4][4], int r0,
                                             int lane, int tq, int C, bf16* s_m) {
  float mc[2][4];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    mc[nt][0] = mc[nt][1] = mc[nt][2] = mc[nt][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const uint32_t* f = fr + fw + (nt * 8 + kk * 2) * 32 + lane;
      mma_bf16(mc[nt], ga[kk], f[0], f[32]);
    }
  }
  const int r1 = r0 + 8;
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    if (r0 < C) *reinterpret_cast<uint32_t*>(s_m + r0 * ND + nt * 8 + 2 * tq) = pack_bf16(mc[nt][0], mc[nt][1]);
    if (r1 < C) *reinterpret_cast<uint32_t*>(s_m + r1 * ND + nt * 8 + 2 * tq) = pack_bf16(mc[nt][2], mc[nt][3]);
  }
}

// acc <- relu(acc) + b + a^ U^T  (the residual update of one layer)
__device__ __forceinline__ void tile_update(const bf16* sw, const uint32_t* fr, int fu, int pb, const bf16* s_a,
                                            int r0, int lane, int tq, int C, float (&acc)[8][4]) {
  uint32_t a[4];
  load_a16(s_a, r0, tq, C, a);
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    const int col = nt * 8 + 2 * tq;
    const float2 bb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sw + pb + col));
    acc[nt][0] = fmaxf(acc[nt][0], 0.f) + bb.x;
    acc[nt][1] = fmaxf(acc[nt][1], 0.f) + bb.y;
    acc[nt][2] = fmaxf(acc[nt][2], 0.f) + bb.x;
    acc[nt][3] = fmaxf(acc[nt][3], 0.f) + bb.y;
    const uint32_t* f = fr + fu + nt * 64 + lane;
    mma_bf16(acc[nt], a, f[0], f[32]);
  }
}

constexpr int PROPOSE_THREADS = 512;

__global__ void __launch_bounds__(PROPOSE_THREADS, 1) net_propose_kernel(NetGraph g, ProposeArgs pa) {
  extern __shared__ __align__(16) unsigned char smem[];
  bf16* sw = reinterpret_cast<bf16*>(smem + pa.off_w);
  uint32_t* fr = reinterpret_cast<uint32_t*>(smem + pa.off_fr);
  bf16* s_x = reinterpret_cast<bf16*>(smem + pa.off_x);
  bf16* s_m = reinterpret_cast<bf16*>(smem + pa.off_m);
  float* s_o = reinterpret_cast<float*>(smem + pa.off_m);  // reuses the message rows after layer 2
  bf16* s_n = reinterpret_cast<bf16*>(smem + pa.off_n);
  bf16* s_a1 = reinterpret_cast<bf16*>(smem + pa.off_a1);
  bf16* s_a2 = reinterpret_cast<bf16*>(smem + pa.off_a2);
  float* s_th = reinterpret_cast<float*>(smem + pa.off_th);
  uint8_t* s_tu = smem + pa.off_tu;
  uint8_t* s_syn = smem + pa.off_syn;
  const int C = g.C, V = g.V, E = g.E;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const int ntiles = (C + 15) >> 4;
  uint16_t* sg = reinterpret_cast<uint16_t*>(smem + pa.off_g);
  const uint16_t* chk_ptr = sg;
  const uint16_t* chk_var = chk_ptr + C + 1;
  const uint16_t* var_ptr = chk_var + E;
  const uint16_t* var_chk = var_ptr + V + 1;

  for (int i = tid; i < N_PARAMS; i += blockDim.x) sw[i] = pa.theta[i];
  for (int i = tid; i < FR_WORDS; i += blockDim.x) fr[i] = fragment_word(pa.theta, i);
  for (int i = tid; i < pa.graph16_len / 8; i += blockDim.x)
    reinterpret_cast<uint4*>(sg)[i] = __ldg(reinterpret_cast<const uint4*>(pa.graph16) + i);
  __syncthreads();

  const long long n_items = pa.shot_list && pa.list_count ? (long long)min(max(*pa.list_count, 0), (int)pa.B) : pa.B;
  for (long long item = blockIdx.x; item < n_items; item += gridDim.x) {
    const long long b = pa.shot_list ? (long long)pa.shot_list[item] : item;
    if (b < 0 || b >= pa.B) continue;  // block-uniform: no barrier is skipped by part of the block
    // variable features
    for (int c = tid; c < C; c += blockDim.x) s_syn[c] = pa.syn[b * C + c] & 1;
    __syncthreads();
    for (int v = tid; v < V; v += blockDim.x) {
      const float pc = fminf(fmaxf(pa.post[b * pa.post_stride + v], -1e4f), 1e4f);
      int cnt = 0;
      for (int k = var_ptr[v]; k < var_ptr[v + 1]; ++k) cnt += s_syn[var_chk[k]];
      s_th[v] = tanhf(pc * 0.0625f);
      s_tu[v] = (uint8_t)((pc <= 0.f ? 2 : 0) + (fabsf(pc) < 8.f ? 1 : 0) + (cnt << 2));
    }
    __syncthreads();
    // check inputs x^ = (s, mean tanh, mean hard, mean unsat, mean tanh(llr/16), 1, 0, 0)
    for (int c = tid; c < C; c += blockDim.x) {
      const int e0 = chk_ptr[c], e1 = chk_ptr[c + 1];
      float s0 = 0.f, s1 = 0.f, s2 = 0.f;
      for (int e = e0; e < e1; ++e) {
        const int v = chk_var[e];
        const int tu = s_tu[v];
        s0 += s_th[v];
        s1 += (float)((tu >> 1) & 1);
        s2 += (float)(tu >> 2) / (float)max(var_ptr[v + 1] - var_ptr[v], 1);
      }
      const float deg = (float)max(e1 - e0, 1);
      uint4 q;
      q.x = pack_bf16((float)s_syn[c], s0 / deg);
      q.y = pack_bf16(s1 / deg, s2 / deg);
      q.z = pack_bf16(__ldg(pa.chk_lmean + c), 1.f);
      q.w = 0u;
      *reinterpret_cast<uint4*>(s_x + c * 8) = q;
    }
    __syncthreads();
#pragma unroll 1
    for (int layer = 1; layer <= 2; ++layer) {
      const int pg = layer == 1 ? P_G1 : P_G2;
      bf16* s_a = layer == 1 ? s_a1 : s_a2;
      // tile pass: this layer's messages
      for (int tile = warp; tile < ntiles; tile += nwarps) {
        float acc[8][4];
        uint32_t ga[4][4];
        const int r0 = tile * 16 + gq;
        tile_embed(fr, s_x, r0, lane, tq, C, acc);
        if (layer == 2) tile_update(sw, fr, FR_U1, P_B1, s_a1, r0, lane, tq, C, acc);
        relu_to_a(acc, ga);
        tile_message(fr, layer == 1 ? FR_W1 : FR_W2, ga, r0, lane, tq, C, s_m);
      }
      __syncthreads();
      // per half h of the 16 channels: n_v = round(sum_{c in M(v)} m_c), then
      // a_c = sum_{v in N(c)} G[t_v] (n_v - m_c)
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        for (int v = tid; v < V; v += blockDim.x) {
          float n[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
          for (int k = var_ptr[v]; k < var_ptr[v + 1]; ++k) {
            float f[8];
            unpack8(*reinterpret_cast<const uint4*>(s_m + var_chk[k] * ND + h * 8), f);
#pragma unroll
            for (int j = 0; j < 8; ++j) n[j] += f[j];
          }
          *reinterpret_cast<uint4*>(s_n + v * 8) = pack8(n);
        }
        __syncthreads();
        for (int c = tid; c < C; c += blockDim.x) {
          float mc[8], a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
          unpack8(*reinterpret_cast<const uint4*>(s_m + c * ND + h * 8), mc);
          for (int e = chk_ptr[c]; e < chk_ptr[c + 1]; ++e) {
            const int v = chk_var[e];
            float n[8], gt[8];
            unpack8(*reinterpret_cast<const uint4*>(s_n + v * 8), n);
            unpack8(*reinterpret_cast<const uint4*>(sw + pg + (s_tu[v] & 3) * ND + h * 8), gt);
#pragma unroll
            for (int j = 0; j < 8; ++j) a[j] = fmaf(gt[j], n[j] - mc[j], a[j]);
          }
          *reinterpret_cast<uint4*>(s_a + c * ND + h * 8) = pack8(a);
        }
        __syncthreads();
      }
    }
    // layer-2 update and the check readout o_c = O . g2^
    for (int tile = warp; tile < ntiles; tile += nwarps) {
      float acc[8][4];
      uint32_t ga[4][4];
      const int r0 = tile * 16 + gq;
      tile_embed(fr, s_x, r0, lane, tq, C, acc);
      tile_update(sw, fr, FR_U1, P_B1, s_a1, r0, lane, tq, C, acc);
      tile_update(sw, fr, FR_U2, P_B2, s_a2, r0, lane, tq, C, acc);
      relu_to_a(acc, ga);
      float oc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) mma_bf16(oc, ga[kk], fr[FR_O + kk * 64 + lane], fr[FR_O + kk * 64 + 32 + lane]);
      if (tq == 0) {
        if (r0 < C) s_o[r0] = oc[0];
        if (r0 + 8 < C) s_o[r0 + 8] = oc[2];
      }
    }
    __syncthreads();
    // variable readout
    const float oz0 = sw_f(sw, P_OZ), oz1 = sw_f(sw, P_OZ + 1), oz2 = sw_f(sw, P_OZ + 2), oz3 = sw_f(sw, P_OZ + 3),
                ob = sw_f(sw, P_OB);
    for (int v = tid; v < V; v += blockDim.x) {
      const int k0 = var_ptr[v], k1 = var_ptr[v + 1];
      float s = 0.f;
      for (int k = k0; k < k1; ++k) s += s_o[var_chk[k]];
      const float deg = (float)max(k1 - k0, 1);
      const int tu = s_tu[v];
      const float r = s / deg +
                      (oz0 * s_th[v] + oz1 * (float)((tu >> 1) & 1) + oz2 * ((float)(tu >> 2) / deg) +
                       oz3 * __ldg(g.llr_feat + v)) +
                      ob;
      if (pa.logits) pa.logits[b * V + v] = r;
      if (pa.gammas) pa.gammas[b * V + v] = pa.lo + (pa.hi - pa.lo) / (1.f + expf(-r));
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ fused inference, low degrees
//
// The same network for graphs with at most 8 edges per check and 4 per variable (and
// V <= 3072, C <= 1024): every value is computed by the same operations in the same order,
// so outputs equal net_propose_kernel's bit for bit.  A shot there took 110 K cycles, 63 K
// of them in the two message sums: one thread walked a row's edges through dependent
// loads of bounds, indices and 16-byte rows, half of each 32-byte row's banks unused, and
// every pass ran once per half of the channels.  Here
//   * index rows are padded (8 checks' or 4 variables' indices in one load), absent edges
//     pointing at a zero row (sums) or a zero gate (aggregation), so a row's loads are
//     independent;
//   * messages and sums lie as two arrays of 16-byte half rows: consecutive rows cover
//     every bank;
//   * a layer's aggregate overwrites the layer's messages in place (a check reads only its
//     own message row), which makes room for the sums of all 16 channels at once;
//   * the tanh feature stays in its owner's registers after the check inputs are formed;
//   * unsat / deg comes from a table of the quotients;
//   * the next shot's posterior and syndrome are loaded while this one is evaluated;
//   * a check's edge types are packed into one word per shot.
// Measured on the 936 x 2,592 graph: 16,384 shots 6.53 -> 3.55 ms.  Of a shot's 58 K cycles
// the aggregations take 21 K (issue, ALU and shared-memory work within 25 % of each other),
// the tile passes (mma.sync chains of 16 checks) 18 K, the sums 9 K, the rest 10 K.

constexpr int FP_DC = 8, FP_DV = 4, FP_KV = 6, FP_KC = 2;  // index rows; variables and checks per thread
constexpr int FP_LUT = (FP_DV + 1) * (FP_DV + 1);

struct FastArgs {
  const uint16_t* chk_idx;  // [C][8] variable of each edge, V beyond the degree
  const uint16_t* var_idx;  // [V][4] check of each edge, C beyond the degree
  int off_fr, off_gate, off_bias, off_lut, off_ci, off_vi, off_x, off_a1, off_a2, off_n, off_tu, off_ct, off_syn;
};

// Rows r0, r0+8 of an array of half rows ([2][C + 1][8] bf16) as an A fragment (zero past C).
__device__ __forceinline__ void load_a_halves(const bf16* s, int r0, int tq, int C, uint32_t (&a)[4]) {
  const int r1 = r0 + 8;
  const bf16* h1 = s + (C + 1) * 8;
  a[0] = r0 < C ? *reinterpret_cast<const uint32_t*>(s + r0 * 8 + 2 * tq) : 0u;
  a[1] = r1 < C ? *reinterpret_cast<const uint32_t*>(s + r1 * 8 + 2 * tq) : 0u;
  a[2] = r0 < C ? *reinterpret_cast<const uint32_t*>(h1 + r0 * 8 + 2 * tq) : 0u;
  a[3] = r1 < C ? *reinterpret_cast<const uint32_t*>(h1 + r1 * 8 + 2 * tq) : 0u;
}

__device__ __forceinline__ void tile_message_halves(const uint32_t* fr, int fw, const uint32_t (&ga)[4][4], int r0,
                                                    int lane, int tq, int C, bf16* s_m) {
  float mc[2][4];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    mc[nt][0] = mc[nt][1] = mc[nt][2] = mc[nt][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const uint32_t* f = fr + fw + (nt * 8 + kk * 2) * 32 + lane;
      mma_bf16(mc[nt], ga[kk], f[0], f[32]);
    }
  }
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    bf16* h = s_m + nt * (C + 1) * 8;
    if (r0 < C) *reinterpret_cast<uint32_t*>(h + r0 * 8 + 2 * tq) = pack_bf16(mc[nt][0], mc[nt][1]);
    if (r0 + 8 < C) *reinterpret_cast<uint32_t*>(h + (r0 + 8) * 8 + 2 * tq) = pack_bf16(mc[nt][2], mc[nt][3]);
  }
}

// acc <- relu(acc) + b + a^ U^T, a^ from half rows, b the layer's 64 biases
__device__ __forceinline__ void tile_update_halves(const uint32_t* fr, int fu, const bf16* bias, const bf16* s_a, int r0,
                                                   int lane, int tq, int C, float (&acc)[8][4]) {
  uint32_t a[4];
  load_a_halves(s_a, r0, tq, C, a);
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    const float2 bb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(bias + nt * 8 + 2 * tq));
    acc[nt][0] = fmaxf(acc[nt][0], 0.f) + bb.x;
    acc[nt][1] = fmaxf(acc[nt][1], 0.f) + bb.y;
    acc[nt][2] = fmaxf(acc[nt][2], 0.f) + bb.x;
    acc[nt][3] = fmaxf(acc[nt][3], 0.f) + bb.y;
    const uint32_t* f = fr + fu + nt * 64 + lane;
    mma_bf16(acc[nt], a, f[0], f[32]);
  }
}

// DV: variable degree bound (3 or 4).
template <int DV>
__global__ void __launch_bounds__(PROPOSE_THREADS, 1) net_propose_fast_kernel(NetGraph g, ProposeArgs pa, FastArgs fa) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t* fr = reinterpret_cast<uint32_t*>(smem + fa.off_fr);
  bf16* s_gate = reinterpret_cast<bf16*>(smem + fa.off_gate);  // [2][5][16], row 4 zero
  bf16* s_bias = reinterpret_cast<bf16*>(smem + fa.off_bias);  // [2][64]
  float* s_lut = reinterpret_cast<float*>(smem + fa.off_lut);  // [deg][unsat] quotients
  const uint16_t* s_ci = reinterpret_cast<const uint16_t*>(smem + fa.off_ci);
  const uint16_t* s_vi = reinterpret_cast<const uint16_t*>(smem + fa.off_vi);
  bf16* s_x = reinterpret_cast<bf16*>(smem + fa.off_x);    // [C][8]
  bf16* s_a1 = reinterpret_cast<bf16*>(smem + fa.off_a1);  // layer 1: messages, then aggregates
  bf16* s_a2 = reinterpret_cast<bf16*>(smem + fa.off_a2);  // layer 2
  bf16* s_n = reinterpret_cast<bf16*>(smem + fa.off_n);    // [2][V + 1][8]
  float* s_th = reinterpret_cast<float*>(smem + fa.off_n);  // [V + 1] until the check inputs are formed
  float* s_o = reinterpret_cast<float*>(smem + fa.off_n);   // [C + 1] after the last aggregation
  uint8_t* s_tu = smem + fa.off_tu;                         // [V + 1] type | (deg * 5 + unsat) << 3
  uint32_t* s_ct = reinterpret_cast<uint32_t*>(smem + fa.off_ct);  // [C] types of a check's edges, 3 bits each
  uint8_t* s_syn = smem + fa.off_syn;                       // [C + 1]
  const int C = g.C, V = g.V;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = PROPOSE_THREADS >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const int ntiles = (C + 15) >> 4;

  for (int i = tid; i < FR_WORDS; i += PROPOSE_THREADS) fr[i] = fragment_word(pa.theta, i);
  for (int i = tid; i < 2 * 5 * ND; i += PROPOSE_THREADS) {
    const int layer = i / (5 * ND), t = i / ND % 5;
    s_gate[i] = t < NTY ? pa.theta[(layer ? P_G2 : P_G1) + t * ND + i % ND] : __float2bfloat16_rn(0.f);
  }
  for (int i = tid; i < 2 * NH; i += PROPOSE_THREADS) s_bias[i] = pa.theta[(i < NH ? P_B1 : P_B2) + i % NH];
  for (int i = tid; i < FP_LUT; i += PROPOSE_THREADS)
    s_lut[i] = (float)(i % (FP_DV + 1)) / (float)max(i / (FP_DV + 1), 1);
  for (int i = tid; i < C; i += PROPOSE_THREADS)
    reinterpret_cast<uint4*>(smem + fa.off_ci)[i] = __ldg(reinterpret_cast<const uint4*>(fa.chk_idx) + i);
  for (int i = tid; i < V; i += PROPOSE_THREADS)
    reinterpret_cast<uint2*>(smem + fa.off_vi)[i] = __ldg(reinterpret_cast<const uint2*>(fa.var_idx) + i);
  if (tid < 4) {  // the zero rows absent edges point at
    bf16* z = (tid & 1 ? s_a2 : s_a1) + (tid >> 1) * (C + 1) * 8 + C * 8;
    *reinterpret_cast<uint4*>(z) = make_uint4(0u, 0u, 0u, 0u);
  }
  if (tid == 0) {
    s_syn[C] = 0;
    s_tu[V] = 4;  // the zero gate
  }
  const float oz0 = ldw(pa.theta, P_OZ), oz1 = ldw(pa.theta, P_OZ + 1), oz2 = ldw(pa.theta, P_OZ + 2),
              oz3 = ldw(pa.theta, P_OZ + 3), ob = ldw(pa.theta, P_OB);

  const long long n_items = pa.shot_list && pa.list_count ? (long long)min(max(*pa.list_count, 0), (int)pa.B) : pa.B;
  auto shot_of = [&](long long item) -> long long {
    if (item >= n_items) return -1;
    const long long b = pa.shot_list ? (long long)pa.shot_list[item] : item;
    return b < pa.B ? b : -1;
  };
  float nx[FP_KV] = {};      // the next shot's posterior and syndrome (this thread's variables and checks)
  uint32_t ny[FP_KC] = {};
  auto fetch = [&](long long b) {
#pragma unroll
    for (int k = 0; k < FP_KV; ++k) {
      const int v = tid + k * PROPOSE_THREADS;
      if (v < V) nx[k] = __ldg(pa.post + b * pa.post_stride + v);
    }
#pragma unroll
    for (int k = 0; k < FP_KC; ++k) {
      const int c = tid + k * PROPOSE_THREADS;
      if (c < C) ny[k] = __ldg(pa.syn + b * C + c) & 1u;
    }
  };
  long long item = blockIdx.x, b = shot_of(item);
  if (b >= 0) fetch(b);
  for (; item < n_items; item += gridDim.x) {
    const long long next = shot_of(item + gridDim.x);
    if (b < 0) {  // block-uniform: no barrier is skipped by part of the block
      b = next;
      if (b >= 0) fetch(b);
      continue;
    }
    float th[FP_KV];
#pragma unroll
    for (int k = 0; k < FP_KC; ++k) {
      const int c = tid + k * PROPOSE_THREADS;
      if (c < C) s_syn[c] = (uint8_t)ny[k];
    }
    __syncthreads();
    // variable features
#pragma unroll
    for (int k = 0; k < FP_KV; ++k) {
      const int v = tid + k * PROPOSE_THREADS;
      if (v < V) {
        const float pc = fminf(fmaxf(nx[k], -1e4f), 1e4f);
        const uint2 u = reinterpret_cast<const uint2*>(s_vi)[v];
        const int c[4] = {(int)(u.x & 0xffffu), (int)(u.x >> 16), (int)(u.y & 0xffffu), (int)(u.y >> 16)};
        int cnt = 0, deg = 0;
#pragma unroll
        for (int j = 0; j < DV; ++j) {
          cnt += s_syn[c[j]];
          deg += c[j] < C;
        }
        th[k] = tanhf(pc * 0.0625f);
        s_th[v] = th[k];
        s_tu[v] = (uint8_t)((pc <= 0.f ? 2 : 0) + (fabsf(pc) < 8.f ? 1 : 0) + ((deg * (FP_DV + 1) + cnt) << 3));
      }
    }
    if (tid == 0) s_th[V] = 0.f;
    __syncthreads();
    if (next >= 0) fetch(next);
    // check inputs x^ = (s, mean tanh, mean hard, mean unsat, mean tanh(llr/16), 1, 0, 0)
#pragma unroll
    for (int k = 0; k < FP_KC; ++k) {
      const int c = tid + k * PROPOSE_THREADS;
      if (c < C) {
        const uint4 u = reinterpret_cast<const uint4*>(s_ci)[c];
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
        float s0 = 0.f, s1 = 0.f, s2 = 0.f;
        int d = 0;
        uint32_t types = 0u;
#pragma unroll
        for (int e = 0; e < FP_DC; ++e) {
          const int v = (int)(e & 1 ? w[e >> 1] >> 16 : w[e >> 1] & 0xffffu);
          const int tu = s_tu[v];
          s0 += s_th[v];
          s1 += (float)((tu >> 1) & 1);
          s2 += s_lut[tu >> 3];
          d += v < V;
          types |= (uint32_t)(tu & 7) << (3 * e);
        }
        s_ct[c] = types;
        const float deg = (float)max(d, 1);
        uint4 q;
        q.x = pack_bf16((float)s_syn[c], s0 / deg);
        q.y = pack_bf16(s1 / deg, s2 / deg);
        q.z = pack_bf16(__ldg(pa.chk_lmean + c), 1.f);
        q.w = 0u;
        *reinterpret_cast<uint4*>(s_x + c * 8) = q;
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int layer = 1; layer <= 2; ++layer) {
      bf16* s_m = layer == 1 ? s_a1 : s_a2;
      // tile pass: this layer's messages
      for (int tile = warp; tile < ntiles; tile += nwarps) {
        float acc[8][4];
        uint32_t ga[4][4];
        const int r0 = tile * 16 + gq;
        tile_embed(fr, s_x, r0, lane, tq, C, acc);
        if (layer == 2) tile_update_halves(fr, FR_U1, s_bias, s_a1, r0, lane, tq, C, acc);
        relu_to_a(acc, ga);
        tile_message_halves(fr, layer == 1 ? FR_W1 : FR_W2, ga, r0, lane, tq, C, s_m);
      }
      __syncthreads();
      // n_v = round(sum_{c in M(v)} m_c), a thread per variable and half of the channels
      for (int i = tid; i < 2 * V; i += PROPOSE_THREADS) {
        const int h = i >= V ? 1 : 0, v = i - h * V;
        const uint2 u = reinterpret_cast<const uint2*>(s_vi)[v];
        const int c[4] = {(int)(u.x & 0xffffu), (int)(u.x >> 16), (int)(u.y & 0xffffu), (int)(u.y >> 16)};
        const uint4* m = reinterpret_cast<const uint4*>(s_m + h * (C + 1) * 8);
        uint4 r[DV];
#pragma unroll
        for (int j = 0; j < DV; ++j) r[j] = m[c[j]];
        float n[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < DV; ++j) {
          float f[8];
          unpack8(r[j], f);
#pragma unroll
          for (int q = 0; q < 8; ++q) n[q] += f[q];
        }
        reinterpret_cast<uint4*>(s_n + h * (V + 1) * 8)[v] = pack8(n);
      }
      if (tid < 2) reinterpret_cast<uint4*>(s_n + tid * (V + 1) * 8)[V] = make_uint4(0u, 0u, 0u, 0u);
      __syncthreads();
      // a_c = sum_{v in N(c)} G[t_v] (n_v - m_c), a thread per check and half of the channels
      for (int i = tid; i < 2 * C; i += PROPOSE_THREADS) {
        const int h = i >= C ? 1 : 0, c = i - h * C;
        const uint4 u = reinterpret_cast<const uint4*>(s_ci)[c];
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
        const uint4* nh = reinterpret_cast<const uint4*>(s_n + h * (V + 1) * 8);
        const unsigned char* gate = reinterpret_cast<const unsigned char*>(s_gate + (layer - 1) * 5 * ND + h * 8);
        const uint32_t types = s_ct[c];
        uint4* own = reinterpret_cast<uint4*>(s_m + h * (C + 1) * 8) + c;
        float mc[8], a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        unpack8(*own, mc);
#pragma unroll
        for (int e = 0; e < FP_DC; ++e) {
          const int v = (int)(e & 1 ? w[e >> 1] >> 16 : w[e >> 1] & 0xffffu);
          float n[8], gt[8];
          unpack8(nh[v], n);
          const uint32_t off = (3 * e >= 5 ? types >> (3 * e - 5) : types << (5 - 3 * e)) & 0xe0u;  // type * 32 bytes
          unpack8(*reinterpret_cast<const uint4*>(gate + off), gt);
#pragma unroll
          for (int j = 0; j < 8; ++j) a[j] = fmaf(gt[j], n[j] - mc[j], a[j]);
        }
        *own = pack8(a);
      }
      __syncthreads();
    }
    // layer-2 update and the check readout o_c = O . g2^
    for (int tile = warp; tile < ntiles; tile += nwarps) {
      float acc[8][4];
      uint32_t ga[4][4];
      const int r0 = tile * 16 + gq;
      tile_embed(fr, s_x, r0, lane, tq, C, acc);
      tile_update_halves(fr, FR_U1, s_bias, s_a1, r0, lane, tq, C, acc);
      tile_update_halves(fr, FR_U2, s_bias + NH, s_a2, r0, lane, tq, C, acc);
      relu_to_a(acc, ga);
      float oc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) mma_bf16(oc, ga[kk], fr[FR_O + kk * 64 + lane], fr[FR_O + kk * 64 + 32 + lane]);
      if (tq == 0) {
        if (r0 < C) s_o[r0] = oc[0];
        if (r0 + 8 < C) s_o[r0 + 8] = oc[2];
      }
    }
    if (tid == 0) s_o[C] = 0.f;
    __syncthreads();
    // variable readout
#pragma unroll
    for (int k = 0; k < FP_KV; ++k) {
      const int v = tid + k * PROPOSE_THREADS;
      if (v < V) {
        const uint2 u = reinterpret_cast<const uint2*>(s_vi)[v];
        const int c[4] = {(int)(u.x & 0xffffu), (int)(u.x >> 16), (int)(u.y & 0xffffu), (int)(u.y >> 16)};
        float s = 0.f;
        int d = 0;
#pragma unroll
        for (int j = 0; j < DV; ++j) {
          s += s_o[c[j]];
          d += c[j] < C;
        }
        const float deg = (float)max(d, 1);
        const int tu = s_tu[v];
        const float r = s / deg + (oz0 * th[k] + oz1 * (float)((tu >> 1) & 1) + oz2 * s_lut[tu >> 3] +
                                   oz3 * __ldg(g.llr_feat + v)) + ob;
        if (pa.logits) pa.logits[b * V + v] = r;
        if (pa.gammas) pa.gammas[b * V + v] = pa.lo + (pa.hi - pa.lo) / (1.f + expf(-r));
      }
    }
    b = next;
    __syncthreads();
  }
}

int grid_for(long long n, int threads = 256) {
  const long long b = (n + threads - 1) / threads;
  return (int)std::max(1LL, std::min(b, 16LL * kSMs));
}

}  // namespace

// ------------------------------------------------------------------ host object

struct rbp_net {
  int device = 0;
  int C = 0, V = 0, E = 0;
  DevBuf<int> chk_ptr, chk_var, var_ptr, var_chk;
  DevBuf<float> llr_feat, chk_lmean;
  DevBuf<uint16_t> graph16;
  DevBuf<float> theta, adam_m, adam_v, grad, loss;
  DevBuf<bf16> theta_bf;
  long long step = 0;
  long long ws_B = 0;
  DevBuf<uint4> slab;           // the training workspace, one allocation
  NetWork ws{};
  float *r = nullptr, *dr = nullptr;
  float* partial = nullptr;     // [GRAD_BLOCKS][GRAD_STRIDE]
  int propose_smem = 0, propose_blocks = 0;
  ProposeArgs layout{};
  DevBuf<uint16_t> chk_idx, var_idx;  // padded index rows of net_propose_fast_kernel
  int fast_smem = 0;                  // 0: the graph does not fit that kernel
  void (*fast_kernel)(NetGraph, ProposeArgs, FastArgs) = nullptr;
  FastArgs fast{};

  NetGraph graph() const { return NetGraph{C, V, E, chk_ptr.p, chk_var.p, var_ptr.p, var_chk.p, llr_feat.p}; }

  int workspace(long long B) {
    if (B <= ws_B) return RBP_OK;
    const size_t nc = (size_t)B * C, nv = (size_t)B * V;
    ws_B = 0;
    unsigned char* base = nullptr;
    size_t off = 0;
    auto take = [&](auto*& p, size_t count) {
      p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + off);
      off += (count * sizeof(*p) + 255) / 256 * 256;
    };
    for (int pass = 0; pass < 2; ++pass) {  // sizes, then places
      if (pass == 1) {
        const int rc = slab.upload(nullptr, off / sizeof(uint4));
        if (rc != RBP_OK) return rc;
        base = reinterpret_cast<unsigned char*>(slab.p);
        off = 0;
      }
      take(ws.z, nv * NF);
      take(ws.ty, nv);
      take(ws.x, nc);
      for (uint4** p : {&ws.m1, &ws.m2, &ws.a1, &ws.a2}) take(*p, nc * 2);
      for (uint4** p : {&ws.n1, &ws.n2}) take(*p, nv * 2);
      for (uint4** p : {&ws.g1, &ws.g2}) take(*p, nc * 8);
      for (unsigned long long** p : {&ws.k1, &ws.k2}) take(*p, nc);
      for (float** p : {&ws.o, &ws.dout}) take(*p, nc);
      for (float4** p : {&ws.da, &ws.dm1, &ws.dm2}) take(*p, nc * 4);
      take(ws.dn, nv * 4);
      for (float** p : {&r, &dr}) take(*p, nv);
      take(partial, (size_t)GRAD_BLOCKS * GRAD_STRIDE);
    }
    ws_B = B;
    return RBP_OK;
  }

  static int rows_per_thread(unsigned nc) { return nc >= TWO_ROWS_FROM ? 2 : 1; }

  // Training-path forward; leaves what the backward pass needs in the workspace.
  void forward(long long B, const uint8_t* syn, const float* post, cudaStream_t st) {
    const NetGraph g = graph();
    const NetWork& w = ws;
    const unsigned nc = (unsigned)(B * C), nv = (unsigned)(B * V);
    // weights are staged once per block: the resident blocks loop over their rows
    const int R = rows_per_thread(nc);
    const unsigned rows = std::min<unsigned>((nc + RT * R - 1) / (RT * R), kSMs * forward_blocks(R));
    const dim3 halves((nv + 255) / 256, 2);
    const bf16* t = theta_bf.p;
    feat_var_kernel<<<grid_for(nv), 256, 0, st>>>(g, B, syn, post, w.z, w.ty);
    (R == 2 ? rows_forward_kernel<1, 2> : rows_forward_kernel<1, 1>)<<<rows, RT, 0, st>>>(g, nc, nv, w, t, syn, chk_lmean.p);
    varsum_kernel<<<halves, 256, 0, st>>>(g, nc, nv, w.m1, w.n1);
    (R == 2 ? rows_forward_kernel<2, 2> : rows_forward_kernel<2, 1>)<<<rows, RT, 0, st>>>(g, nc, nv, w, t, syn, chk_lmean.p);
    varsum_kernel<<<halves, 256, 0, st>>>(g, nc, nv, w.m2, w.n2);
    (R == 2 ? rows_forward_kernel<3, 2> : rows_forward_kernel<3, 1>)<<<rows, RT, 0, st>>>(g, nc, nv, w, t, syn, chk_lmean.p);
  }

  // Gradients of everything behind the readout (dr), summed with the readout's own into grad and loss.
  void backward(long long B, int vars, cudaStream_t st) {
    const NetGraph g = graph();
    const NetWork& w = ws;
    const unsigned nc = (unsigned)(B * C), nv = (unsigned)(B * V);
    const dim3 quarters((nv + 255) / 256, 4);
    const auto blocks = [&](int rows) { return (int)std::min<unsigned>((nc + RT * rows - 1) / (RT * rows), kSMs * backward_blocks(rows)); };
    const int R = rows_per_thread(nc), tiles = blocks(R), last = blocks(1);
    const int gather = (int)std::min<unsigned>((nc + 127) / 128, GRAD_BLOCKS);
    float* pg = partial;
    const bf16* t = theta_bf.p;
    rows_backward_kernel<2, 1><<<last, RT, rows_backward_smem(2, 1), st>>>(g, nc, w, t, dr, pg);
    dn_kernel<<<quarters, 256, 0, st>>>(g, nc, nv, t + P_G2, w.ty, w.da, w.dn);
    dm_kernel<<<gather, 512, 0, st>>>(g, nc, nv, t + P_G2, w.ty, w.m2, w.n2, w.da, w.dn, w.dm2, pg + P_G2);
    (R == 2 ? rows_backward_kernel<1, 2> : rows_backward_kernel<1, 1>)<<<tiles, RT, rows_backward_smem(1, R), st>>>(
        g, nc, w, t, dr, pg);
    dn_kernel<<<quarters, 256, 0, st>>>(g, nc, nv, t + P_G1, w.ty, w.da, w.dn);
    dm_kernel<<<gather, 512, 0, st>>>(g, nc, nv, t + P_G1, w.ty, w.m1, w.n1, w.da, w.dn, w.dm1, pg + P_G1);
    (R == 2 ? rows_backward_kernel<0, 2> : rows_backward_kernel<0, 1>)<<<tiles, RT, rows_backward_smem(0, R), st>>>(
        g, nc, w, t, dr, pg);
    grad_sum_kernel<<<(N_PARAMS + 32) / 32, 1024, 0, st>>>(pg, tiles, last, gather, vars, grad.p, loss.p);
  }
};

extern "C" {

int rbp_net_param_count(int64_t* n) {
  if (!n) return fail(RBP_ERR_ARGUMENT, "rbp_net_param_count: null argument");
  *n = N_PARAMS;
  return RBP_OK;
}

int rbp_net_create(const rbp_graph* g, const float* llr, rbp_net** out) {
  if (!out) return fail(RBP_ERR_ARGUMENT, "rbp_net_create: out is null");
  *out = nullptr;
  if (!g || !llr) return fail(RBP_ERR_ARGUMENT, "rbp_net_create: null graph or llr");
  const int C = g->C, V = g->V, E = g->E;
  std::vector<int> chk_ptr(C + 1, 0), edge_var(E), var_chk(E);
  for (int e = 0; e < E; ++e) chk_ptr[g->edge_chk[e] + 1]++;
  for (int c = 0; c < C; ++c) chk_ptr[c + 1] += chk_ptr[c];
  int max_dv = 0;
  for (int v = 0; v < V; ++v) {
    const int k0 = g->var_ptr[v], k1 = g->var_ptr[v + 1];
    max_dv = std::max(max_dv, k1 - k0);
    for (int k = k0; k < k1; ++k) {
      edge_var[g->var_edges[k]] = v;
      var_chk[k] = g->edge_chk[g->var_edges[k]];
    }
    std::sort(var_chk.begin() + k0, var_chk.begin() + k1);
  }
  if (max_dv > 63) return fail(RBP_ERR_UNSUPPORTED, "rbp_net_create: variable degree above 63");
  std::vector<float> lf(V), lmean(C);
  for (int v = 0; v < V; ++v) lf[v] = std::tanh(llr[v] / 16.0f);
  for (int c = 0; c < C; ++c) {
    float s = 0.f;  // edge order, float sums
    for (int e = chk_ptr[c]; e < chk_ptr[c + 1]; ++e) s += lf[edge_var[e]];
    lmean[c] = s / (float)std::max(chk_ptr[c + 1] - chk_ptr[c], 1);
  }
  DeviceGuard dg(g->device);
  if (!dg.ok) return fail(RBP_ERR_CUDA, "rbp_net_create: cannot select the CUDA device");
  rbp_net* n = new rbp_net();
  n->device = g->device;
  n->C = C;
  n->V = V;
  n->E = E;
  int rc;
  std::vector<float> zeros(N_PARAMS, 0.f);
  if ((rc = n->chk_ptr.upload(chk_ptr.data(), C + 1)) || (rc = n->chk_var.upload(edge_var.data(), E)) ||
      (rc = n->var_ptr.upload(g->var_ptr.data(), V + 1)) || (rc = n->var_chk.upload(var_chk.data(), E)) ||
      (rc = n->llr_feat.upload(lf.data(), V)) || (rc = n->chk_lmean.upload(lmean.data(), C)) ||
      (rc = n->theta.upload(zeros.data(), N_PARAMS)) || (rc = n->adam_m.upload(zeros.data(), N_PARAMS)) ||
      (rc = n->adam_v.upload(zeros.data(), N_PARAMS)) || (rc = n->grad.upload(zeros.data(), N_PARAMS)) ||
      (rc = n->loss.upload(zeros.data(), 1)) || (rc = n->theta_bf.upload(nullptr, N_PARAMS))) {
    delete n;
    return rc;
  }
  to_bf16_kernel<<<4, 256>>>(N_PARAMS, n->theta.p, n->theta_bf.p);
  for (const void* k : {reinterpret_cast<const void*>(rows_backward_kernel<0, 1>),
                        reinterpret_cast<const void*>(rows_backward_kernel<0, 2>),
                        reinterpret_cast<const void*>(rows_backward_kernel<1, 1>),
                        reinterpret_cast<const void*>(rows_backward_kernel<1, 2>),
                        reinterpret_cast<const void*>(rows_backward_kernel<2, 1>)})
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_backward_smem(0, 2)) != cudaSuccess) {
      delete n;
      return fail(RBP_ERR_CUDA, "rbp_net_create: cannot reserve shared memory for the training kernels");
    }
  // inference kernel shared memory (see net_propose_kernel)
  int off = 0;
  auto take = [&](int bytes) {
    const int o = off;
    off = rbph::align16(off + bytes);
    return o;
  };
  const int g16 = (2 * C + 2 * V + 2 + 2 * E + 7) / 8 * 8;
  n->layout.graph16_len = g16;
  n->layout.off_w = take(N_PARAMS * 2);
  n->layout.off_fr = take(FR_WORDS * 4);
  n->layout.off_g = take(g16 * 2);
  n->layout.off_x = take(C * 8 * 2);
  n->layout.off_m = take(std::max(C * ND * 2, C * 4));
  n->layout.off_n = take(V * 8 * 2);
  n->layout.off_a1 = take(C * ND * 2);
  n->layout.off_a2 = take(C * ND * 2);
  n->layout.off_th = take(V * 4);
  n->layout.off_tu = take(V);
  n->layout.off_syn = take(C);
  n->propose_smem = off;
  const bool small_graph = C < 65536 && V < 65536 && E < 65536;
  if (small_graph) {
    std::vector<uint16_t> h16(g16, 0);
    size_t o = 0;
    for (int c = 0; c <= C; ++c) h16[o++] = (uint16_t)chk_ptr[c];
    for (int e = 0; e < E; ++e) h16[o++] = (uint16_t)edge_var[e];
    for (int v = 0; v <= V; ++v) h16[o++] = (uint16_t)g->var_ptr[v];
    for (int k = 0; k < E; ++k) h16[o++] = (uint16_t)var_chk[k];
    if ((rc = n->graph16.upload(h16.data(), g16))) {
      delete n;
      return rc;
    }
  }
  int optin = 0, sms = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, n->device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, n->device);
  int max_dc = 0;
  for (int c = 0; c < C; ++c) max_dc = std::max(max_dc, chk_ptr[c + 1] - chk_ptr[c]);
  if (max_dc <= FP_DC && max_dv <= FP_DV && V <= FP_KV * PROPOSE_THREADS && C <= FP_KC * PROPOSE_THREADS) {
    off = 0;
    FastArgs& f = n->fast;
    f.off_fr = take(FR_WORDS * 4);
    f.off_gate = take(2 * 5 * ND * 2);
    f.off_bias = take(2 * NH * 2);
    f.off_lut = take(FP_LUT * 4);
    f.off_ci = take(C * FP_DC * 2);
    f.off_vi = take(V * FP_DV * 2);
    f.off_x = take(C * 8 * 2);
    f.off_a1 = take(2 * (C + 1) * 8 * 2);
    f.off_a2 = take(2 * (C + 1) * 8 * 2);
    f.off_n = take(std::max(2 * (V + 1) * 8 * 2, std::max(V, C) * 4 + 4));
    f.off_tu = take(V + 1);
    f.off_ct = take(C * 4);
    f.off_syn = take(C + 1);
    if (off <= optin) {
      std::vector<uint16_t> ci((size_t)C * FP_DC, (uint16_t)V), vi((size_t)V * FP_DV, (uint16_t)C);
      for (int c = 0; c < C; ++c)
        for (int e = chk_ptr[c]; e < chk_ptr[c + 1]; ++e) ci[(size_t)c * FP_DC + e - chk_ptr[c]] = (uint16_t)edge_var[e];
      for (int v = 0; v < V; ++v)
        for (int k = g->var_ptr[v]; k < g->var_ptr[v + 1]; ++k)
          vi[(size_t)v * FP_DV + k - g->var_ptr[v]] = (uint16_t)var_chk[k];
      if ((rc = n->chk_idx.upload(ci.data(), ci.size())) || (rc = n->var_idx.upload(vi.data(), vi.size()))) {
        delete n;
        return rc;
      }
      n->fast_kernel = max_dv <= 3 ? net_propose_fast_kernel<3> : net_propose_fast_kernel<4>;
      if (cudaFuncSetAttribute(reinterpret_cast<const void*>(n->fast_kernel),
                               cudaFuncAttributeMaxDynamicSharedMemorySize, off) != cudaSuccess) {
        delete n;
        return fail(RBP_ERR_CUDA, "rbp_net_create: cannot reserve shared memory for the inference kernel");
      }
      f.chk_idx = n->chk_idx.p;
      f.var_idx = n->var_idx.p;
      n->fast_smem = off;
    }
    off = n->propose_smem;
  }
  if (small_graph && off <= optin) {
    if (cudaFuncSetAttribute(net_propose_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, off) != cudaSuccess) {
      delete n;
      return fail(RBP_ERR_CUDA, "rbp_net_create: cannot reserve shared memory for the inference kernel");
    }
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, net_propose_kernel, PROPOSE_THREADS, off);
    n->propose_blocks = std::max(1, per_sm) * sms;
  }
  if (cudaDeviceSynchronize() != cudaSuccess) {
    delete n;
    return fail(RBP_ERR_CUDA, "rbp_net_create: device error");
  }
  *out = n;
  return RBP_OK;
}

int rbp_net_destroy(rbp_net* n) {
  if (!n) return RBP_OK;
  DeviceGuard dg(n->device);
  delete n;
  return RBP_OK;
}

int rbp_net_set_params(rbp_net* n, const float* theta, void* stream) {
  if (!n || !theta) return fail(RBP_ERR_ARGUMENT, "rbp_net_set_params: null argument");
  DeviceGuard dg(n->device);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  RBP_CUDA(cudaMemcpyAsync(n->theta.p, theta, N_PARAMS * sizeof(float), cudaMemcpyDeviceToDevice, st));
  RBP_CUDA(cudaMemsetAsync(n->adam_m.p, 0, N_PARAMS * sizeof(float), st));
  RBP_CUDA(cudaMemsetAsync(n->adam_v.p, 0, N_PARAMS * sizeof(float), st));
  to_bf16_kernel<<<4, 256, 0, st>>>(N_PARAMS, n->theta.p, n->theta_bf.p);
  RBP_CUDA(cudaGetLastError());
  n->step = 0;
  return RBP_OK;
}

int rbp_net_get_params(const rbp_net* n, float* theta, void* stream) {
  if (!n || !theta) return fail(RBP_ERR_ARGUMENT, "rbp_net_get_params: null argument");
  DeviceGuard dg(n->device);
  RBP_CUDA(cudaMemcpyAsync(theta, n->theta.p, N_PARAMS * sizeof(float), cudaMemcpyDeviceToDevice,
                           static_cast<cudaStream_t>(stream)));
  return RBP_OK;
}

int rbp_net_forward(rbp_net* n, int64_t B, const uint8_t* syn, const float* post, float* logits, void* stream) {
  if (!n) return fail(RBP_ERR_ARGUMENT, "rbp_net_forward: null network");
  if (B < 0) return fail(RBP_ERR_ARGUMENT, "rbp_net_forward: negative batch");
  if (B == 0) return RBP_OK;
  if (!syn || !post || !logits) return fail(RBP_ERR_ARGUMENT, "rbp_net_forward: null buffer");
  DeviceGuard dg(n->device);
  int rc;
  if ((rc = n->workspace(B))) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  n->forward(B, syn, post, st);
  readout_kernel<<<grid_for(B * n->V), 256, 0, st>>>(n->graph(), B, n->theta_bf.p, n->ws.o, n->ws.z, nullptr, 0.f,
                                                      logits, nullptr, nullptr);
  RBP_CUDA(cudaGetLastError());
  return RBP_OK;
}

int rbp_net_train_step(rbp_net* n, int64_t B, const uint8_t* syn, const float* post, const uint8_t* target,
                       const rbp_net_hparams* hp, float* loss, float* grads, void* stream) {
  if (!n || !hp) return fail(RBP_ERR_ARGUMENT, "rbp_net_train_step: null argument");
  if (B <= 0) return fail(RBP_ERR_ARGUMENT, "rbp_net_train_step: batch must be positive");
  if (!syn || !post || !target) return fail(RBP_ERR_ARGUMENT, "rbp_net_train_step: null buffer");
  if (!(hp->w_neg > 0.f) || hp->lr < 0.f) return fail(RBP_ERR_ARGUMENT, "rbp_net_train_step: bad hyper-parameters");
  DeviceGuard dg(n->device);
  int rc;
  if ((rc = n->workspace(B))) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  n->forward(B, syn, post, st);
  const int vars = std::min(grid_for(B * n->V), GRAD_BLOCKS);
  readout_kernel<<<vars, 256, 0, st>>>(n->graph(), B, n->theta_bf.p, n->ws.o, n->ws.z, target, hp->w_neg, n->r,
                                       n->dr, n->partial);
  n->backward(B, vars, st);
  if (loss) RBP_CUDA(cudaMemcpyAsync(loss, n->loss.p, sizeof(float), cudaMemcpyDeviceToDevice, st));
  if (grads) RBP_CUDA(cudaMemcpyAsync(grads, n->grad.p, N_PARAMS * sizeof(float), cudaMemcpyDeviceToDevice, st));
  if (hp->lr > 0.f) {
    n->step += 1;
    const float bc1 = 1.f - std::pow(hp->beta1, (float)n->step), bc2 = 1.f - std::pow(hp->beta2, (float)n->step);
    adamw_kernel<<<(N_PARAMS + 255) / 256, 256, 0, st>>>(N_PARAMS, n->theta.p, n->adam_m.p, n->adam_v.p, n->grad.p,
                                                         n->theta_bf.p, hp->lr, hp->beta1, hp->beta2, hp->eps,
                                                         hp->weight_decay, bc1, bc2);
  }
  RBP_CUDA(cudaGetLastError());
  return RBP_OK;
}

int rbp_net_propose(rbp_net* n, int64_t B, const uint8_t* syn, const float* post, int64_t post_stride, float lo,
                    float hi, const int32_t* shot_list, const int32_t* list_count, float* gammas, float* logits,
                    void* stream) {
  if (!n) return fail(RBP_ERR_ARGUMENT, "rbp_net_propose: null network");
  if (B < 0) return fail(RBP_ERR_ARGUMENT, "rbp_net_propose: negative batch");
  if (B == 0) return RBP_OK;
  if (!syn || !post || (!gammas && !logits)) return fail(RBP_ERR_ARGUMENT, "rbp_net_propose: null buffer");
  if (!(lo <= hi)) return fail(RBP_ERR_ARGUMENT, "rbp_net_propose: lo must not exceed hi");
  if (post_stride != 0 && post_stride < n->V) return fail(RBP_ERR_ARGUMENT, "rbp_net_propose: post_stride below V");
  if (n->propose_blocks == 0)
    return fail(RBP_ERR_UNSUPPORTED, "rbp_net_propose: the graph and a shot's state (" +
                                         std::to_string(n->propose_smem) +
                                         " B) exceed shared memory, or the graph exceeds 65535 edges");
  DeviceGuard dg(n->device);
  ProposeArgs pa = n->layout;
  pa.B = B;
  pa.syn = syn;
  pa.post = post;
  pa.post_stride = post_stride ? post_stride : n->V;
  pa.lo = lo;
  pa.hi = hi;
  pa.gammas = gammas;
  pa.logits = logits;
  pa.shot_list = shot_list;
  pa.list_count = list_count;
  pa.theta = n->theta_bf.p;
  pa.chk_lmean = n->chk_lmean.p;
  pa.graph16 = n->graph16.p;
  const int blocks = (int)std::min<long long>(B, n->propose_blocks);
  if (n->fast_smem) {
    n->fast_kernel<<<blocks, PROPOSE_THREADS, n->fast_smem, static_cast<cudaStream_t>(stream)>>>(n->graph(), pa, n->fast);
    RBP_CUDA(cudaGetLastError());
    return RBP_OK;
  }
  net_propose_kernel<<<blocks, PROPOSE_THREADS, n->propose_smem, static_cast<cudaStream_t>(stream)>>>(n->graph(), pa);
  RBP_CUDA(cudaGetLastError());
  return RBP_OK;
}

}  // extern "C"
