// The decode loop and its kernels (sm_100a).
//
// A group of G threads decodes one shot at a time, start to finish (first phase,
// relay legs, selection, outputs), then takes the next position of a global work
// queue: shots that converge early free their group instead of waiting for the
// slowest shot of a batch, and there is no host round trip per iteration.
// run_group below is the loop; three kernels run it:
//   relaybp_decode_kernel   several groups per block (or one), one block per SM's
//                           worth of registers; groups meet at named barriers;
//   relaybp_decode2_kernel  one group per block, compiled for two resident blocks
//                           per SM: one block's barrier and dependency waits are
//                           the other's issue slots;
//   relaybp_mixed_kernel    several codes' queues in one launch.
// Results do not depend on the kernel, the shape or the queue order.
//
// Ownership.  Thread t of a group owns variables v = t + k G (k < VPT) and checks
// c = t + k G.  Everything per variable stays in that thread's registers: the
// byte offsets of its edges' message slots (loaded once per kernel), its
// posterior (carried across legs: the memory) and the leg's memory strength.
// Shared memory per group holds
//   msg[rows * C + 1]  edge messages; the slots of a check sit in 16-byte chunks
//                      (slot_index).  A slot holds mu after a variable pass and nu
//                      after a check pass; padding and dummy slots: relaybp_rows.cuh.
//   mis[ceil(C/32)]    bit c%32 of word c/32: (parity of check c's current hard
//                      decisions) XOR (its syndrome bit).  Decisions start at 0, so it
//                      starts as the syndrome; a decision that flips XORs its
//                      checks' bits (shared atomics, no return value).
//   best[W], first[W]  bit sets (W = ceil(V/32)): best solution, first-leg decision.
//                      Word w + k (G/32) holds the bits of warp w's variables, so only
//                      that warp touches it and __syncwarp orders the accesses.
//   red[]              weight sum of a selection (entries 0 and 4 used in turn),
//                      the claimed shot index (entries 1 and 2 used in turn, so a claim
//                      never overwrites one a thread has not read yet).
//   s1[], lmk[]        per owned-variable slot: the shot's first-pass sums, and the
//                      memory mixes of a leg's first iteration (see below); left out
//                      where they would not fit (DevArgs::keep_sums 0).
//
// An iteration (decoder.py:2610-2875) is check pass (c2v min-sum,
// kernels.py:1052-1215) -> barrier -> variable pass (memory mix, posterior, hard
// decision, v2c, kernels.py:1220-1350) -> barrier -> test.  It has converged when
// every mis word is 0 (the parity + all-checks test of kernels.py:510-741): each
// warp reads the words for itself, so the test needs no barrier of its own.  The
// steady iterations of a phase are one small loop (phase starts, selections and the
// variants below stay outside it): with the loop's control spread over the shot
// state machine, an iteration of a lone shot spent 950 of its 5,950 cycles there.
//
// A relay leg's first iteration usually converges (most legs of solved shots repeat
// their solution), and then its outgoing messages are never read: the next leg
// restarts them.  That variable pass keeps its memory mixes in lmk and stores the
// messages only once the iteration is known not to have converged.  And a leg
// restarts the messages, so its first check pass is the same at every leg (with
// shared priors the block's table with the shot's syndrome signs): the shot's first leg in a launch
// keeps each variable's sum of those messages (s1), and later legs add the kept
// sum to the memory mix instead of running the check pass and the message loads.
// Both give the same values bit for bit.  For per-shot priors, which have no table
// and set up and check a leg's first messages in full, the kept sums took 2,047 shots
// of 1,080 variables from 262 to 245 us, 8,000 shots of 2,592 from 1,375 to 1,227.
//
// Numerics follow the reference kernels operation by operation with one rounding
// per operation (explicit _rn intrinsics; built with --fmad=false); the memory-mix
// rounding is selectable.  Incoming messages are summed in the graph's var_edges
// order.  Solution weights are exact 64-bit fixed point.

#pragma once

#include <type_traits>

#include "relaybp_kernel.cuh"
#include "relaybp_rows.cuh"

namespace rbpk {

// Largest block an instantiation of the kernels for one and for two resident blocks per
// SM is compiled for; bounds the registers the owned-variable state may take (at two
// blocks: 64 registers up to 4 owned variables, 72 at 6, 80 at 8, else 128).
__host__ __device__ constexpr int max_block_threads(int vpt) {
  return vpt <= 2 ? 1024 : (vpt == 3 ? 896 : (vpt == 4 ? 768 : (vpt <= 8 ? 512 : 256)));
}
__host__ __device__ constexpr int max_block_threads2(int vpt) {
  return vpt <= 4 ? 512 : (vpt == 6 ? 448 : (vpt == 8 ? 384 : 256));
}

// The checks of the variables in `flips` (bit k: variable t + k G) change their mis bit.
// A thread takes its flips one by one, so a warp runs as many rounds as its busiest lane
// has flips (one or two on hard shots), whichever variables they are; the check indices
// come from the graph's table in one load (registers cannot be indexed).
template <int MAXDV>
__device__ __forceinline__ void flip_checks(uint32_t* mis, const DevGraph& g, uint32_t flips, int t, int G) {
  while (flips) {
    const int v = t + (__ffs(flips) - 1) * G;
    flips &= flips - 1;
    const uint2* row = reinterpret_cast<const uint2*>(g.var_chk + (size_t)v * g.chk_stride);
#pragma unroll
    for (int h = 0; h < (MAXDV + 3) / 4; ++h) {
      if (h > 0 && g.chk_stride <= 4) break;
      const uint2 u = __ldg(row + h);
      const uint32_t c[4] = {u.x & 0xffffu, u.x >> 16, u.y & 0xffffu, u.y >> 16};
#pragma unroll
      for (int j = 0; j < (MAXDV < 4 ? MAXDV : 4); ++j)
        if (c[j] != kNoSlot) atomicXor(mis + (c[j] >> 5), 1u << (c[j] & 31u));
    }
  }
}

// Group gid of this block decodes shots of one code until the work queue is empty.
// The block-wide tables must be in shared memory.  BLOCK or solo: the group is the block
// (the block barrier costs half a named one with register operands).
template <typename M, int MAXDC, int VPT, int MAXDV, bool BLOCK>
__device__ __forceinline__ void run_group(const DevGraph& g, const DevArgs& a, unsigned char* smem, bool solo) {
  using IO = MsgT<M>;
  using A = typename IO::A;
  constexpr bool PACKED = MAXDC > 0 && sizeof(M) < 8;  // rows with a packed form (relaybp_rows.cuh)

  const int C = g.C, V = g.V;
  const int G = BLOCK ? (int)blockDim.x : a.group_threads;
  const int gid = BLOCK ? 0 : (int)threadIdx.x / G;
  if (!BLOCK && gid >= a.groups) return;
  const int t = (int)threadIdx.x - gid * G;
  const int lane = t & 31;
  const int warp = t >> 5;
  const int nwarps = G >> 5;
  const int W = (V + 31) >> 5;
  const int Wc = (C + 31) >> 5;
  const A beta = A(a.beta);
  const uint8_t* s_chk_deg = smem + a.off_chk_deg;
  const float* s_llr = reinterpret_cast<const float*>(smem + a.off_llr);
  const M* first_tab = reinterpret_cast<const M*>(smem + a.off_first);
  unsigned char* region = smem + a.off_group0 + gid * a.group_bytes;
  M* msg = reinterpret_cast<M*>(region + a.g_msg);
  uint32_t* mis = reinterpret_cast<uint32_t*>(region + a.g_par);
  uint32_t* best = reinterpret_cast<uint32_t*>(region + a.g_best);
  uint32_t* first = reinterpret_cast<uint32_t*>(region + a.g_first);
  long long* red = reinterpret_cast<long long*>(region + a.g_red);
  A* s1 = reinterpret_cast<A*>(region + a.g_s1);
  A* lmk = s1 + VPT * G;

  const bool first_from_table = MAXDC > 0 && a.llr_shot == nullptr;
  // the default rounding of the memory mix, shared priors, no offset and finite check outputs:
  // the steady loop without per-launch choices
  const bool usual = a.mix_mode == RBP_MIX_SEPARATE && a.llr_shot == nullptr && !a.use_beta && !a.strict;

  auto sync = [&]() {
    if (BLOCK || solo) __syncthreads();
    else group_sync(1 + gid, G);
  };
  auto sync_or = [&](bool p) -> bool {
    if (BLOCK || solo) return __syncthreads_or(p) != 0;
    return group_any(1 + gid, G, p);
  };

  // byte offsets from smem of the owned variables' edge slots in summation order;
  // absent edges (degree < MAXDV) point at the dummy slot after the last row
  const uint32_t msg0 = (uint32_t)(reinterpret_cast<unsigned char*>(msg) - smem);
  const uint32_t dummy = msg0 + (uint32_t)(g.rows * C) * (uint32_t)sizeof(M);
  uint32_t vpos[VPT][MAXDV];
  uint32_t owned = 0u;  // bit k: variable t + k G exists
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int v = t + k * G;
    owned |= (v < V ? 1u : 0u) << k;
#pragma unroll
    for (int j = 0; j < MAXDV; ++j) {
      uint32_t p = kNoSlot;
      if (v < V && j < g.vslots) p = g.var_pos[j * V + v];
      vpos[k][j] = p == kNoSlot ? dummy : msg0 + p * (uint32_t)sizeof(M);
    }
  }
  uint32_t padm = 0u;  // bit k: the row of check t + k G has padding
  if constexpr (MAXDC > 0) {
    for (int k = 0; t + k * G < C; ++k) {
      const int c = t + k * G;
      padm |= (s_chk_deg[c] < MAXDC ? 1u : 0u) << k;
      fill_padding<M, MAXDC>(msg, c, C, s_chk_deg[c]);
    }
  }
  if (t == 0) {
    msg[g.rows * C] = IO::st(A(0));
    red[0] = 0;
    red[4] = 0;
  }

  A post[VPT];  // posteriors of the owned variables (the memory)
  A gam[VPT];   // memory strengths of the running phase
  uint32_t hmask = 0u;      // bit k: hard decision of variable t + k G
  uint32_t hmask_sel = 0u;  // the decisions at the shot's last computed selection
  uint32_t synm = 0u;       // bit k: syndrome of check t + k G
  // Everything below runs under group-uniform control: each thread holds the same
  // control values, so barriers are reached by every thread of the group.
  int claim = 0;  // which red[1 + claim] entry the next claim writes
  int wsel = 0;   // the next selection sums into red[0] (0) or red[4] (1)

  // ---------------------------------------------------------------- passes
  // A phase's first check pass from the block's table, rows negated where the syndrome is 1.
  auto table_pass = [&]() {
    if constexpr (MAXDC > 0) {
#pragma unroll 1
      for (int k = 0; t + k * G < C; ++k) {
        const int c = t + k * G;
#pragma unroll
        for (int q = 0; q < MAXDC / VecIO<M>::N; ++q) {
          uint4 w = *reinterpret_cast<const uint4*>(first_tab + chunk_base<M>(q, c, C));
          if ((synm >> k) & 1u) w = flip_signs<M>(w);
          *reinterpret_cast<uint4*>(msg + chunk_base<M>(q, c, C)) = w;
        }
        if ((padm >> k) & 1u) fill_padding<M, MAXDC>(msg, c, C, s_chk_deg[c]);
      }
    }
  };

  // Check pass of iteration `it`, one owned row per step (two interleaved rows per step took
  // longer: 936 rows by 704 threads 934 cycles against 1,153).  USUAL: packed rows only.
  auto check_pass = [&](int it, auto kind) {
    constexpr bool USUAL = decltype(kind)::value;
    const A alpha = a.use_alpha ? A(__ldg(a.alpha + it)) : A(1);
    if constexpr (PACKED) {
      if (USUAL || !a.strict) {
        uint32_t s = synm;
#pragma unroll 1
        for (int c = t; c < C; c += G, s >>= 1)
          check_row_packed<M, MAXDC, !USUAL>(msg, c, C, s << 31, alpha, a.use_alpha, a.use_beta, beta);
        for (uint32_t pm = padm; pm; pm &= pm - 1) {
          const int c = t + (__ffs(pm) - 1) * G;
          restore_row<M, MAXDC>(msg, c, C, s_chk_deg[c]);
        }
        return;
      }
    }
    if constexpr (!PACKED || !USUAL) {
#pragma unroll 1
      for (int k = 0; t + k * G < C; ++k) {
        const int c = t + k * G, s = (int)((synm >> k) & 1u);
        if constexpr (MAXDC > 0)
          check_row_masked<M, MAXDC>(msg, c, C, s_chk_deg[c], s, alpha, a.use_alpha, a.use_beta, beta);
        else
          check_row_generic<M>(msg, c, C, g.chk_ptr[c + 1] - g.chk_ptr[c], s, alpha, a.use_alpha, a.use_beta, beta);
      }
    }
  };

  // The decisions after a variable pass (those beyond V masked out); the few that
  // changed flip their checks' mis bits.
  auto decide = [&](uint32_t hnew) {
    hnew &= owned;
    const uint32_t flips = hnew ^ hmask;
    hmask = hnew;
    if (flips) flip_checks<MAXDV>(mis, g, flips, t, G);
  };

  // Prior LLR of owned variable slot v; beyond V some word of the block's memory, whose
  // results are masked out.
  auto prior = [&](int v, const float* llr_row) -> A {
    if (llr_row != nullptr) return v < V ? A(__ldg(llr_row + v)) : A(1);
    return A(s_llr[v]);
  };

  // Variable pass, straight-line over the owned variables: no branch splits the loop body.
  // With DEFER the outgoing messages are not stored: the mixes go to lmk and the sums to s1.
  auto var_pass = [&](const float* llr_row, auto defer, auto kind) {
    constexpr bool DEFER = decltype(defer)::value, USUAL = decltype(kind)::value;
    uint32_t hnew = 0u;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int v = t + k * G;
      const A l0 = USUAL ? A(s_llr[v]) : prior(v, llr_row);
      const A lm = memory_mix<A>(USUAL ? (int)RBP_MIX_SEPARATE : a.mix_mode, gam[k], l0, post[k]);
      A nv[MAXDV];
      const A sum = load_edges<M, MAXDV>(smem, vpos[k], nv);
      const A pv = add_rn(lm, sum);
      post[k] = pv;
      if constexpr (DEFER) {
        lmk[v] = lm;  // lmk and s1 entries are read back only by the thread that wrote them
        s1[v] = sum;
      } else {
        store_edges<M, MAXDV>(smem, vpos[k], dummy, lm, sum, nv);
      }
      hnew |= (pv <= A(0) ? 1u : 0u) << k;
    }
    decide(hnew);
  };

  // A relay leg's first iteration from the kept sums.
  auto var_pass_quick = [&](const float* llr_row) {
    uint32_t hnew = 0u;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int v = t + k * G;
      const A lm = memory_mix<A>(a.mix_mode, gam[k], prior(v, llr_row), post[k]);
      lmk[v] = lm;
      const A pv = add_rn(lm, s1[v]);
      post[k] = pv;
      hnew |= (pv <= A(0) ? 1u : 0u) << k;
    }
    decide(hnew);
  };

  // The messages a deferred pass did not store: the incoming ones are reloaded (still in
  // their slots) and summed in the same order, so the values are those it would have stored.
  auto store_deferred = [&]() {
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      A nv[MAXDV];
      const A sum = load_edges<M, MAXDV>(smem, vpos[k], nv);
      store_edges<M, MAXDV>(smem, vpos[k], dummy, lmk[t + k * G], sum, nv);
    }
  };

  // After a variable pass and its barrier: whether every check holds.
  auto all_satisfied = [&]() -> bool {
    const volatile uint32_t* words = mis;
    uint32_t bad = words[min(lane, Wc - 1)];
    if (Wc > 32) {
#pragma unroll 1
      for (int w = lane + 32; w < Wc; w += 32) bad |= words[w];
    }
    return !__any_sync(0xffffffffu, bad != 0u);
  };

  // ---------------------------------------------------------------- shots
  bool fresh = true;  // no shot decoded yet
  long long b = 0, best_w = LLONG_MAX;
  int found = 0, iters = 0, hard_src = HARD_ZERO;
  bool has_best = false, stopped = false;

  while (true) {
    // Claim the next queue position (its atomic's latency overlaps the last shot's outputs).
    int q = 0;
    if (t == 0) q = atomicAdd(a.queue, 1);

    if (!fresh) {
      // Outputs of shot b (decoder.py:3839-3873) and the optional saved state.
      __syncwarp();
      if (a.suspend && (!a.suspend_unsolved || stopped)) {
        unsigned char* sst = a.suspend + b * (long long)a.state_stride;
        if (t == 0) {
          int* hdr = reinterpret_cast<int*>(sst);
          hdr[0] = found;
          hdr[1] = iters;
          hdr[2] = hard_src;
          hdr[3] = has_best ? 1 : 0;
          *reinterpret_cast<long long*>(sst + 16) = best_w;
        }
        uint32_t* bits = reinterpret_cast<uint32_t*>(sst + 32);
        if (lane < VPT) {
          const int w = warp + lane * nwarps;
          if (w < W) {
            bits[w] = best[w];
            bits[W + w] = first[w];
          }
        }
        A* sp = reinterpret_cast<A*>(sst + state_post_offset(V));
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
          const int v = t + k * G;
          if (v < V) sp[v] = post[k];
        }
      }
      const uint32_t* src_bits = has_best ? best : first;
      const bool from_post = !has_best && a.last_leg && hard_src == HARD_POST;
      const bool zero_bits = !has_best && a.last_leg && hard_src != HARD_POST;
      if (a.errors) {
        uint8_t* erow = a.errors + b * (long long)V;
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
          const int v = t + k * G;
          if (v < V) {
            uint8_t e;
            if (from_post) e = post[k] <= A(0) ? 1 : 0;
            else if (zero_bits) e = 0;
            else e = (src_bits[v >> 5] >> (v & 31)) & 1u;
            erow[v] = e;
          }
        }
      }
      if (a.errors_packed) {
        uint32_t* prow = a.errors_packed + b * (long long)W;
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
          const int v0 = warp * 32 + k * G;
          unsigned m;
          if (from_post) m = __ballot_sync(0xffffffffu, v0 + lane < V && post[k] <= A(0));
          else if (zero_bits) m = 0u;
          else m = v0 < V ? src_bits[v0 >> 5] : 0u;
          if (lane == 0 && v0 < V) prow[v0 >> 5] = m;
        }
      }
      if (a.last_post) {
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
          const int v = t + k * G;
          if (v < V) {
            if constexpr (sizeof(A) == 8) reinterpret_cast<double*>(a.last_post)[b * (long long)V + v] = post[k];
            else reinterpret_cast<float*>(a.last_post)[b * (long long)V + v] = post[k];
          }
        }
      }
      if (t == 0) {
        if (a.weights)
          a.weights[b] = has_best ? __ll2float_rn(best_w) * 2.3283064365386963e-10f  // 2^-32
                                  : __int_as_float(0x7f800000);
        if (a.wfixed) a.wfixed[b] = has_best ? best_w : LLONG_MAX;
        a.found[b] = found;
        a.iters[b] = iters;
      }
    }

    // Shot index of the claimed position: B when the queue is exhausted, -1 for an order
    // entry that is not a shot index (skipped).
    if (t == 0) {
      const long long qq = (long long)q;
      const long long qn = a.queue_len ? (long long)max(0, min(*a.queue_len, (int)a.B)) : a.B;
      long long sb = qq < qn ? qq : a.B;
      if (qq < qn && a.order) {
        sb = (long long)a.order[qq];
        if (sb < 0 || sb >= a.B) sb = -1;
      }
      reinterpret_cast<volatile long long*>(red)[1 + claim] = sb;
    }
    sync();
    b = reinterpret_cast<volatile long long*>(red)[1 + claim];
    claim ^= 1;
    if (b >= a.B) return;
    fresh = b < 0;
    if (fresh) continue;

    // Set-up (decoder.py:3429-3478): inputs, bit sets, mis bits.  Every load of the shot's
    // inputs is issued before any of them is used, so their latencies overlap.
    const uint8_t* syn_row = a.syn + b * (long long)C;
    const float* llr_row = a.llr_shot ? a.llr_shot + b * (long long)V : nullptr;
    best_w = LLONG_MAX;
    found = iters = 0;
    hard_src = HARD_ZERO;
    int has_best_raw = 0;
    const unsigned char* sst = a.resume ? a.resume + b * (long long)a.state_stride : nullptr;
    if (sst) {
      // continue a shot suspended after an earlier phase
      const int* hdr = reinterpret_cast<const int*>(sst);
      found = hdr[0];
      iters = hdr[1];
      hard_src = hdr[2];
      has_best_raw = hdr[3];
      best_w = *reinterpret_cast<const long long*>(sst + 16);
      const uint32_t* bits = reinterpret_cast<const uint32_t*>(sst + 32);
      if (lane < VPT) {
        const int w = warp + lane * nwarps;
        if (w < W) {
          best[w] = bits[w];
          first[w] = bits[W + w];
        }
      }
      const A* sp = reinterpret_cast<const A*>(sst + state_post_offset(V));
#pragma unroll
      for (int k = 0; k < VPT; ++k) {
        const int v = t + k * G;
        post[k] = v < V ? sp[v] : A(1);
      }
    } else {
      if (lane < VPT) {
        const int w = warp + lane * nwarps;
        if (w < W) {
          best[w] = 0u;
          first[w] = 0u;
        }
      }
#pragma unroll
      for (int k = 0; k < VPT; ++k) {
        const int v = t + k * G;
        post[k] = a.init_post && v < V ? A(__ldg(a.init_post + b * (long long)V + v)) : prior(v, llr_row);
      }
    }
    // syndrome bits of the owned checks, four loads in flight per round
    synm = 0u;
    for (int k = 0, c = t; c < C; k += 4, c += 4 * G) {
      const uint32_t s0 = syn_row[c];
      const uint32_t s1b = c + G < C ? (uint32_t)syn_row[c + G] : 0u;
      const uint32_t s2 = c + 2 * G < C ? (uint32_t)syn_row[c + 2 * G] : 0u;
      const uint32_t s3 = c + 3 * G < C ? (uint32_t)syn_row[c + 3 * G] : 0u;
      synm |= ((s0 & 1u) | ((s1b & 1u) << 1) | ((s2 & 1u) << 2) | ((s3 & 1u) << 3)) << k;
    }
    // Decisions restart at 0, so each check's mis bit is its syndrome bit (every thread read
    // the last shot's mis words before the claim's barrier).
    for (int k = 0; k * G < C; ++k) {
      const int c = t + k * G;
      const unsigned m = __ballot_sync(0xffffffffu, c < C && ((synm >> k) & 1u));
      const int w = warp + k * nwarps;
      if (lane == 0 && w < Wc) mis[w] = m;
    }
    hmask = hmask_sel = 0u;
    bool sel_seen = false;  // a selection has been computed for this shot
    bool s1_ok = false;     // the kept first-pass sums belong to this shot
    bool synced = false;    // a barrier followed the last test of the mis words
    has_best = has_best_raw != 0;
    stopped = false;
    // a shot resumed at leg 0 was solved by the pre-iterations if it found a solution there
    bool solved_pre = (a.resume && a.legs_begin == 0) ? found > 0 : false;
    const int legs_stop = (a.legs_end > 0 && a.legs_end < a.num_sets) ? a.legs_end : a.num_sets;

    // Phase -1: the pre-iterations (decoder.py:3480-3616); phase l >= 0: relay leg l
    // (decoder.py:3672-3837).
    for (int phase = a.resume ? a.legs_begin : -1;; ++phase) {
      if (phase >= legs_stop || (phase >= 0 && found >= a.stop_nconv)) break;
      int max_iter;
      const float* grow;
      float gs = 0.f;
      if (phase < 0) {
        max_iter = a.pre_iter;
        grow = a.gamma_pre ? a.gamma_pre + b * (long long)V : nullptr;
        gs = a.gamma0;
      } else {
        max_iter = a.set_max_iter;
        grow = (a.gamma_legs_shot && phase < a.n_shot_legs)
                   ? a.gamma_legs_shot + (b * (long long)a.shot_leg_rows + min(phase, a.shot_leg_rows - 1)) * V
                   : a.gamma_legs + (long long)phase * V;
        if (solved_pre && phase < a.solved_legs) {
          grow = nullptr;
          gs = a.solved_gamma;
        }
      }

      if (max_iter <= 0) {
        // freeze_finished_lanes_kernel(count_iteration=False) after an empty phase
        if (found >= min(phase < 0 ? 1 : found + 1, a.stop_nconv)) hard_src = HARD_BEST;
      } else {
        // memory strengths of this phase: loaded here, first used by the variable pass
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
          const int v = t + k * G;
          gam[k] = A(gs);
          if (grow && v < V) gam[k] = A(__ldg(grow + v));
        }
        int it = 0;
        bool conv = false;
        // a leg's first iteration: its messages are stored only if it does not converge, and from
        // the shot's second leg on it needs no messages at all
        const bool defer = phase >= 0 && a.keep_sums, quick = defer && s1_ok;
        if (quick) {
          // the variable pass flips mis bits: every thread's read of them in the last
          // iteration's test must come first (a convergence's selection ordered them)
          if (!synced) sync();
          var_pass_quick(llr_row);
          sync();
          it = 1;
          conv = all_satisfied();
        }
        if (!quick || (!conv && it < max_iter)) {  // quick: the incoming messages the deferred stores re-sum
          if (!first_from_table) {
            // message init mu_e = llr[var(e)] (kernels.py:904-1000), read by the first check pass
#pragma unroll
            for (int k = 0; k < VPT; ++k) {
              const M m0 = init_msg<M>(prior(t + k * G, llr_row));
#pragma unroll
              for (int j = 0; j < MAXDV; ++j)
                if (vpos[k][j] != dummy) *reinterpret_cast<M*>(smem + vpos[k][j]) = m0;
            }
            sync();
          }
          if (defer || first_from_table) {
            if (first_from_table) table_pass();
            else check_pass(0, std::false_type{});
            sync();
            if (!quick) {
              if (defer) var_pass(llr_row, std::true_type{}, std::false_type{});
              else var_pass(llr_row, std::false_type{}, std::false_type{});
              s1_ok = defer;
              sync();
              it = 1;
              conv = all_satisfied();
            }
            if (defer && !conv && it < max_iter) {
              store_deferred();
              sync();  // the next check pass reads them
            }
          }
        }
        if (usual) {
          while (!conv && it < max_iter) {
            check_pass(it, std::true_type{});
            sync();
            var_pass(llr_row, std::false_type{}, std::true_type{});
            sync();
            ++it;
            conv = all_satisfied();
          }
        } else {
          while (!conv && it < max_iter) {
            check_pass(it, std::false_type{});
            sync();
            var_pass(llr_row, std::false_type{}, std::false_type{});
            sync();
            ++it;
            conv = all_satisfied();
          }
        }
        iters += it;
        synced = conv;
        if (!conv) {
          hard_src = HARD_POST;
        } else {
          // check_and_select_kernel (kernels.py:609-741).  Decisions equal to the shot's last
          // selection's have its weight, so the best cannot change: after the shot's first selection
          // the "decisions differ" test comes first (one OR-barrier) and the weight sum, with a second
          // barrier, only when they do.  The sum goes to red[0] or red[4], alternating: once a
          // selection's sum barrier has passed, the other entry's last readers (the previous
          // selection's) are done and thread 0 clears it.
          bool select = true;
          if (sel_seen) select = sync_or(hmask != hmask_sel);
          if (select) {
            long long* wsum = red + (wsel ? 4 : 0);
            long long w = 0;  // weight of the owned variables decided 1, in 2^-32 units (decoder.py:741-753)
#pragma unroll
            for (int k = 0; k < VPT; ++k) {
              const int v = t + k * G;
              if ((hmask >> k) & 1u) w += weight_units(llr_row ? __ldg(llr_row + v) : s_llr[v]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
            if (lane == 0 && w != 0) atomicAdd(reinterpret_cast<unsigned long long*>(wsum), (unsigned long long)w);
            sync();
            if (t == 0) red[wsel ? 0 : 4] = 0;
            hmask_sel = hmask;
            sel_seen = true;
            const long long tot = *reinterpret_cast<volatile long long*>(wsum);
            if (!has_best || tot < best_w) {
              best_w = tot;
              has_best = true;
              ballot_post<A, VPT>(post, best, warp, lane, G, V);
            }
            wsel ^= 1;
          }
          // freeze_finished_lanes_kernel (kernels.py:746-847): a convergence always freezes
          found += 1;
          hard_src = HARD_BEST;
        }
      }

      // first-leg hard decision: after the pre-iterations, or after relay leg 0 when there
      // were none (decoder.py:3595-3598, 3807-3810)
      if (!a.last_leg && (phase < 0 || (phase == 0 && a.pre_iter == 0))) {
        if (hard_src == HARD_POST) {
          ballot_post<A, VPT>(post, first, warp, lane, G, V);
        } else {
          __syncwarp();
          if (lane < VPT) {
            const int w = warp + lane * nwarps;
            if (w < W) first[w] = hard_src == HARD_BEST ? best[w] : 0u;
          }
        }
      }
      if (phase < 0) {
        if (found >= a.stop_nconv || a.skip_legs) break;
        solved_pre = found > 0;
        if (!solved_pre && a.suspend_unsolved) {
          stopped = true;
          break;
        }
      }
    }
  }
}

// Tables of one code for the block's groups.
template <typename M, int MAXDC>
__device__ __forceinline__ void block_tables(const DevGraph& g, const DevArgs& a, unsigned char* smem) {
  load_block_tables(g, a, smem);
  __syncthreads();
  build_first_pass_table<M, MAXDC>(g, a, smem);
}

// One code, one launch (rbp_decode, rbp_decode_static): a.groups groups per block.
template <typename M, int MAXDC, int VPT, int MAXDV>
__global__ void __launch_bounds__(max_block_threads(VPT))
relaybp_decode_kernel(DevGraph g, DevArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  block_tables<M, MAXDC>(g, a, smem);
  run_group<M, MAXDC, VPT, MAXDV, false>(g, a, smem, a.groups == 1);
}

// The same with one group per block and two resident blocks per SM.
template <typename M, int MAXDC, int VPT, int MAXDV>
__global__ void __launch_bounds__(max_block_threads2(VPT), 2)
relaybp_decode2_kernel(DevGraph g, DevArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  block_tables<M, MAXDC>(g, a, smem);
  run_group<M, MAXDC, VPT, MAXDV, true>(g, a, smem, true);
}

// Several codes in one launch (rbp_mixed_*).  Block b starts on the code whose
// block range holds b (first_block[], from the host's work estimate).  When
// that code's queue is empty the whole block moves to the next code that still
// has shots, re-partitioning its threads into that code's group shape, until
// every queue is empty.  Queue counters only grow, so the loop ends.
constexpr int kMaxMixedCodes = 8;

struct MixedCode {
  DevGraph g;
  DevArgs a;
};

struct MixedArgs {
  MixedCode code[kMaxMixedCodes];
  int ncodes;
  int first_block[kMaxMixedCodes + 1];
};

template <typename M, int MAXDC, int VPT, int MAXDV>
__global__ void __launch_bounds__(max_block_threads(VPT))
relaybp_mixed_kernel(const __grid_constant__ MixedArgs m) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_next;
  int code = 0;
  while (code + 1 < m.ncodes && (int)blockIdx.x >= m.first_block[code + 1]) ++code;
  while (code >= 0) {
    const DevGraph g = m.code[code].g;
    const DevArgs a = m.code[code].a;
    block_tables<M, MAXDC>(g, a, smem);
    run_group<M, MAXDC, VPT, MAXDV, false>(g, a, smem, false);
    __syncthreads();
    if (threadIdx.x == 0) {
      int next = -1;
      for (int i = 1; i <= m.ncodes && next < 0; ++i) {
        const int c = (code + i) % m.ncodes;
        if (*reinterpret_cast<volatile const int*>(m.code[c].a.queue) < m.code[c].a.B) next = c;
      }
      s_next = next;
    }
    __syncthreads();
    code = s_next;
    __syncthreads();
  }
}

using KernelFn = void (*)(DevGraph, DevArgs);

// Kernel for (check degree bound, variable degree, owned variables per thread),
// or null when this build has no such instantiation.  One per message type.
KernelFn pick_f32(int dc, int dv, int vpt);
KernelFn pick_f16(int dc, int dv, int vpt);
KernelFn pick_bf16(int dc, int dv, int vpt);
KernelFn pick_f64(int dc, int dv, int vpt);
// The same for two resident blocks per SM (check degrees up to 16).
KernelFn pick2_f32(int dc, int dv, int vpt);
KernelFn pick2_f16(int dc, int dv, int vpt);
KernelFn pick2_bf16(int dc, int dv, int vpt);
KernelFn pick2_f64(int dc, int dv, int vpt);

using MixedKernelFn = void (*)(MixedArgs);
MixedKernelFn pick_mixed_f32(int dc, int dv, int vpt);

// Supported owned-variable counts, ascending.
constexpr int kVptChoices[] = {1, 2, 3, 4, 6, 8, 12, 16};

}  // namespace rbpk

// Instantiation tables (used by relaybp_inst*.cu).
#define RBPK_DV(KERNEL, M, DC, VPT)                          \
  if (dv <= 3) return &rbpk::KERNEL<M, DC, VPT, 3>;          \
  if (dv <= 8) return &rbpk::KERNEL<M, DC, VPT, 8>;          \
  return nullptr;
#define RBPK_DC(KERNEL, M, VPT)                              \
  if (dc <= 8) { RBPK_DV(KERNEL, M, 8, VPT) }                \
  if (dc <= 16) { RBPK_DV(KERNEL, M, 16, VPT) }
#define RBPK_DC_ANY(KERNEL, M, VPT)                          \
  RBPK_DC(KERNEL, M, VPT)                                    \
  { RBPK_DV(KERNEL, M, 0, VPT) }
#define RBPK_DEFINE_PICK(NAME, M)                            \
  rbpk::KernelFn rbpk::NAME(int dc, int dv, int vpt) {       \
    switch (vpt) {                                           \
      case 1: { RBPK_DC_ANY(relaybp_decode_kernel, M, 1) }   \
      case 2: { RBPK_DC_ANY(relaybp_decode_kernel, M, 2) }   \
      case 3: { RBPK_DC_ANY(relaybp_decode_kernel, M, 3) }   \
      case 4: { RBPK_DC_ANY(relaybp_decode_kernel, M, 4) }   \
      case 6: { RBPK_DC_ANY(relaybp_decode_kernel, M, 6) }   \
      case 8: { RBPK_DC_ANY(relaybp_decode_kernel, M, 8) }   \
      case 12: { RBPK_DC_ANY(relaybp_decode_kernel, M, 12) } \
      case 16: { RBPK_DC_ANY(relaybp_decode_kernel, M, 16) } \
      default: return nullptr;                               \
    }                                                        \
  }
#define RBPK_DEFINE_PICK2(NAME, M)                           \
  rbpk::KernelFn rbpk::NAME(int dc, int dv, int vpt) {       \
    switch (vpt) {                                           \
      case 1: { RBPK_DC(relaybp_decode2_kernel, M, 1) break; }   \
      case 2: { RBPK_DC(relaybp_decode2_kernel, M, 2) break; }   \
      case 3: { RBPK_DC(relaybp_decode2_kernel, M, 3) break; }   \
      case 4: { RBPK_DC(relaybp_decode2_kernel, M, 4) break; }   \
      case 6: { RBPK_DC(relaybp_decode2_kernel, M, 6) break; }   \
      case 8: { RBPK_DC(relaybp_decode2_kernel, M, 8) break; }   \
      case 12: { RBPK_DC(relaybp_decode2_kernel, M, 12) break; } \
      case 16: { RBPK_DC(relaybp_decode2_kernel, M, 16) break; } \
    }                                                        \
    return nullptr;                                          \
  }
#define RBPK_DEFINE_PICK_MIXED(NAME, M)                      \
  rbpk::MixedKernelFn rbpk::NAME(int dc, int dv, int vpt) {  \
    switch (vpt) {                                           \
      case 4: { RBPK_DC_ANY(relaybp_mixed_kernel, M, 4) }    \
      case 8: { RBPK_DC_ANY(relaybp_mixed_kernel, M, 8) }    \
      case 16: { RBPK_DC_ANY(relaybp_mixed_kernel, M, 16) }  \
      default: return nullptr;                               \
    }                                                        \
  }
