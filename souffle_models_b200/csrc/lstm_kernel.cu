// Stacked-LSTM wavefront megakernel for sm_100a (batch 1).
//
// Replaces cpp/lstm/lstm_reuse_shared_memory.cu:179-337 (lstm_reuse_shared_memory_v10_vec: 320
// blocks, 109 grid.sync(), fp32 weights partly in registers).  Cell semantics are the
// reference's (python/models/lstm/tf_lstm.py:59-70; cpp/lstm/lstm_reuse_shared_memory.cu:309-318):
// gates i, j, f, o;  c' = c*sigmoid(f+1) + sigmoid(i)*tanh(j);  h' = tanh(c')*sigmoid(o).
//
// Design: every layer is owned by one thread-block cluster of kLstmParts CTAs; a CTA keeps its 4*U gate rows of both
// weight matrices (fp16) in the registers of its cell warps for the whole sequence, and its units' cell state.  Every
// path through the (layer, step) grid has steps-1 hops along time and layers-1 hops across layers, so the hop along time
// is the one that has to be short:
// * The products run on the tensor cores (mma.sync m16n8k16; tcgen05 has no shape for a one-column product).  A warp owns
//   one 16-row tile -- the four gates of four units -- over the whole of K, so nothing is reduced across warps.  The fp32
//   vector enters as three fp16 columns (value, remainder, remainder of the remainder, each scaled by 2^11 against the one
//   before: 33 bits) of the eight the shape has, so the products are those of the fp32 vector; four accumulators per
//   half of K keep the chains of additions short.
// * A step's input half W_in x(t) does not depend on the hidden state: it is multiplied while h(t-1) travels.
// * Hidden states go straight into the shared memory of the eight CTAs of the cluster (distributed shared memory,
//   st.async: the store itself counts as a transfer on the receiver's mbarrier, no fence on either side), and every cell
//   warp waits for them itself: there is no CTA barrier in the step.
// A step of hidden 256 takes 2.3 k cycles (hidden 64: 1.5 k); with the products on the CUDA cores (128 conversions and FMAs
// per thread, partial sums by shuffle, one waiting thread and a CTA barrier) it took 3.5 k (2.4 k): 10 layers x 100 steps
// 228 -> 155 us, 12 x 64 x 200 266 -> 175 us.
// Only the hop to the next layer goes through global memory: one slot per (layer, step) and unit, a 64-bit word of the hidden
// state and the launch's tag.  A word is written as a whole, so the reader, which polls the vector itself, needs neither a
// fence in front of the store nor a counter behind it, and a unit that lags cannot be covered by its peers.  With counters (a release
// behind the stored states, a poll of eight counters, then the vector) a hop took a fence and a round trip through L2 more:
// 10 layers x 100 steps of hidden 256 155 -> 141 us, 3 x 37 of hidden 128 38.7 -> 34.8 a call.
// A fetch warp keeps that hop off the cell arithmetic's path: it brings the layer's input vectors into shared memory up to four steps
// ahead.
// There is no grid-wide barrier.  All waits in the step loop are bounded; on expiry the CTA records a
// status word, leaves the loop and waits for its cluster at the final cluster barrier (shared
// memory must outlive the peers' remote stores).  That barrier does not cover the stores themselves: st.async completes on
// the receiver's mbarrier only.  So every hidden vector is waited for, the last one too, which nobody reads, and a CTA that
// gave up on a wait stays a while longer for whatever is still on its way to it.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "sm100_ptx.cuh"
#include "stage_program.h"

namespace souffle {

constexpr int kLstmParts = 8;                      // CTAs per layer = cluster size
constexpr int kLstmXBufs = 4;                      // input vectors the fetch warp may run ahead
constexpr int kLstmMaxLayers = 18;
static_assert(kLstmMaxLayers * kLstmParts <= (int)kLaunchSteps, "more CTAs than a launch number has steps for");
// threads of a CTA: a cell warp per 32 hidden units of the layer (it owns four of the CTA's), and the fetch warp
__host__ __device__ constexpr int lstm_block(int H) { return (H / 32 + 1) * 32; }

struct LstmParams {
  const __half* w_in;     // [4*L][H][H], row = output unit, col = input
  const __half* w_state;  // [4*L][H][H]
  const float* bias;      // [L][H] or null; added to all four gates of a unit (reference layout)
  const float* x;         // [T][H]
  float* y;               // [T][H]: top layer's h per step
  uint64_t* h_all;        // [L][T][H] scratch: every published hidden state (low half) beside the launch's tag
  unsigned long long* epoch;      // counter of the launches on this scratch (see launch_step): the tag is one more than this one's
                                  // number, which no word of the scratch holds yet
  int* status;
  int* expired;           // host memory or null: set by a CTA that gave up on a wait
  int layers, hidden, steps, ref_input_delay;
  unsigned long long timeout_ns;
};

// sigmoid(v) = 1 / (1 + e^-v), or tanh(v) = 1 - 2 / (1 + e^2v) where is_tanh: ex2-based, absolute error of a few 1e-7 on values
// in [-1, 1].  No branch: a step is one dependent chain, and its lanes differ.
__device__ __forceinline__ float gate_f(float v, bool is_tanh) {
  const float r = __fdividef(is_tanh ? 2.0f : 1.0f, 1.0f + __expf(is_tanh ? 2.0f * v : -v));
  return is_tanh ? 1.0f - r : r;
}

// What the bounded waits look at.  Hidden 64 and 128: a WaitCtl on the stack.  In shared memory every step was slower (3 x 128 x 37
// 38.1 -> 38.9 us, 8 x 128 x 150 161.7 -> 163.8), and so were the places below (163.0 with a call at the limit, 167 without).  Hidden 256,
// whose step loop has no register left: places known at compile time and no call, where the WaitCtl spilled a word
// (12 x 256 x 200 284.5 -> 281.5 us).
struct LstmWait {
  int* abort;                                   // of the CTA, in shared memory
  const unsigned long long* deadline_ns;        // in shared memory
  int* status;
};
template <int H>
using LstmWaitOf = std::conditional_t<(H < 256), WaitCtl, LstmWait>;
// One thread, now and then: true if it has to give up.
__device__ __forceinline__ bool lstm_expired(const WaitCtl& w, int code, int where) {
  if (*w.abort_smem) return true;
  if (globaltimer_ns() <= w.deadline_ns) return false;
  record_timeout(w, code, where);
  return true;
}
__device__ __forceinline__ bool lstm_expired(const LstmWait& w, int code, int where) {
  if (*const_cast<volatile int*>(w.abort)) return true;
  if (globaltimer_ns() <= *const_cast<const volatile unsigned long long*>(w.deadline_ns)) return false;
  *const_cast<volatile int*>(w.abort) = 1;
  if (atomicCAS(w.status, 0, code) == 0) {
    w.status[1] = where;
    w.status[2] = (int)blockIdx.x;
  }
  return true;
}

// Bounded wait of a whole warp on an mbarrier; every lane sees the phase itself.  kCluster: its transfers come from other
// CTAs of the cluster.  `stop` (0: none) is the address of a shared word: once it is set, a wait whose phase is not
// complete by then ends as well.
template <bool kCluster>
__device__ __forceinline__ bool lstm_try(uint32_t bar, uint32_t parity) {
  if constexpr (kCluster) return mbar_try_wait_cluster(bar, parity);
  else return mbar_try_wait(bar, parity);
}
template <bool kCluster, class W>
__device__ __forceinline__ bool lstm_wait_loop(uint32_t bar, uint32_t parity, const W& w, int where, uint32_t stop) {
  uint32_t spins = 0;
  while (!lstm_try<kCluster>(bar, parity)) {
    ++spins;
    if (stop && (spins & 0xF) == 0 && ld_acquire_cta_shared_u32(stop)) return lstm_try<kCluster>(bar, parity);
    if ((spins & 0xFF) == 0 && lstm_expired(w, DEV_TIMEOUT_MBAR, where)) return false;
  }
  return true;
}
template <bool kCluster, class W>
__device__ __forceinline__ bool lstm_wait_warp(uint32_t bar, uint32_t parity, const W& w, int where, int lane, uint32_t stop = 0) {
  if (__all_sync(0xffffffffu, lstm_try<kCluster>(bar, parity))) return true;
  if (__all_sync(0xffffffffu, lstm_try<kCluster>(bar, parity))) return true;
  int ok = 1;
  if (lane == 0) ok = lstm_wait_loop<kCluster>(bar, parity, w, where, stop) ? 1 : 0;
  if (__shfl_sync(0xffffffffu, ok, 0) == 0) return false;
  return __all_sync(0xffffffffu, lstm_try<kCluster>(bar, parity));       // complete: lane 0 has seen it
}

// D (16 x 8, fp32) += A (16 x 16, fp16) B (16 x 8, fp16).  Lane 4 g + q holds rows g and g + 8 of A and columns 2 q, 2 q + 1 of
// D, and column g of B.
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A vector in shared memory: its three fp16 parts, one row each; the pad puts the rows 16 banks apart.
constexpr float kLstmPart = 2048.0f;                 // scale of a part against the one before
constexpr float kLstmHScale = 32768.0f;              // hidden states (at most 1 in magnitude) are scaled by this
__host__ __device__ constexpr int lstm_row(int H) { return H + 32; }

// v (scaled into the range of fp16) = hi + mid / 2^11 + lo / 2^22.  An infinity has no remainder.
__device__ __forceinline__ void lstm_split(float v, __half& hi, __half& mid, __half& lo) {
  hi = __float2half_rn(v);
  const float r = __hisinf(hi) ? 0.0f : (v - __half2float(hi)) * kLstmPart;
  mid = __float2half_rn(r);
  lo = __float2half_rn((r - __half2float(mid)) * kLstmPart);
}

// One half of the gate rows' products (W_in x or W_state h): K = H in blocks of 32.  The order of K inside a block is
// chosen so that a lane's weights and vector elements are 16 contiguous bytes: lane q of a row takes elements
// 8 q .. 8 q + 7, four for each of the block's two MMAs.
// The first kReg blocks' weights are in registers, the others' come from shared memory (`rest`: this thread's pieces, two
// per block, `rest_step` apart).
template <int H, int kReg>
__device__ __forceinline__ void lstm_product(const uint4 (&w)[2][kReg], const uint4* rest, int rest_step, const __half* vec, int lane, float (&out)[4]) {
  float acc[4][4];
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[s][i] = 0.0f;
  const int n = lane >> 2, q = lane & 3;
#pragma unroll
  for (int b = 0; b < H / 32; ++b) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (n < 3) v = *reinterpret_cast<const uint4*>(vec + n * lstm_row(H) + b * 32 + q * 8);
    const uint4 w0 = b < kReg ? w[0][b < kReg ? b : 0] : rest[2 * (b - kReg) * rest_step],
                w1 = b < kReg ? w[1][b < kReg ? b : 0] : rest[(2 * (b - kReg) + 1) * rest_step];
    mma_16816(acc[(2 * b) & 3], w0.x, w1.x, w0.y, w1.y, v.x, v.y);
    mma_16816(acc[(2 * b + 1) & 3], w0.z, w1.z, w0.w, w1.w, v.z, v.w);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) out[i] = (acc[0][i] + acc[1][i]) + (acc[2][i] + acc[3][i]);
}

// The parts of a vector end 2^-61 below its largest element.  Where that may be large enough for a gate to notice (from
// 2^20 on: the large elements' own weights may be zero), and for infinities and NaN, which have no scale, the caller's vector
// goes to the cell warps in pieces, largest elements first, whose products add up: a piece takes the elements within 2^37
// of its largest, all of whose 24 bits the parts hold.  The first such vector moves the cell warps of its layer to a step loop of
// their own: one more branch in the loop that all others run made a step 150 cycles longer (1 x 256 x 200: 232 -> 248 us).
constexpr uint32_t kLstmWide = 127u + 20u;           // biased exponent of 2^20
constexpr uint32_t kLstmPieceRange = 37u;

// What the warps of a CTA share.
template <int H>
struct LstmShared {
  static constexpr int kWarps = H / 32;         // cell warps: four units each
  static constexpr int kRow = lstm_row(H);
  // Hidden 256: a cell thread's weights are 128 registers of the 168 that nine warps leave it (registers are handed out per
  // four warps); two blocks of the input half stay in shared memory instead.
  static constexpr int kXReg = H == 256 ? 6 : H / 32;
  alignas(16) __half x[kLstmXBufs][3 * kRow];   // input vectors
  alignas(16) __half h[2][3 * kRow];            // hidden vectors, written by the whole cluster
  uint4 wx_rest[H == 256 ? 2 * (H / 32 - kXReg) * kWarps * 32 : 1];
  float x_scale[kLstmXBufs];                    // takes the products back to the vector's scale; negative: another piece follows
  uint64_t x_full[kLstmXBufs], x_empty[kLstmXBufs], h_full[2], pieces_ready;
  unsigned long long deadline_ns;
  int abort;
  uint32_t pieces;                              // 1: from the next input vector on, vectors come in pieces
  int piece[kWarps];                            // then: pieces a cell warp has multiplied so far
  uint32_t tag;                                 // of this launch's words in h_all
};

template <int H>
__device__ __forceinline__ void lstm_wait_set(LstmWaitOf<H>& w, LstmShared<H>& sh, const LstmParams& p) {
  if constexpr (H < 256) {
    w.abort_smem = &sh.abort;
    w.status_g = p.status;
    w.deadline_ns = sh.deadline_ns;
  } else {
    w.abort = &sh.abort;
    w.deadline_ns = &sh.deadline_ns;
    w.status = p.status;
  }
}

// The cell arithmetic of all steps from t on (c_state: the cell state, before step t, of the lane's unit: the same value in its
// eight lanes); both are brought up to date.
// kPieces: input vectors may come in several pieces; without, the loop ends (false) in front of the first step whose vector
// does.  False with the abort flag set: a wait has run out.
template <int H, bool kPieces>
__device__ __forceinline__ bool lstm_steps(const LstmParams& p, LstmShared<H>& sh, const LstmWaitOf<H>& ctl, int layer, int part, int tid,
                                           int& t, float& c_state) {
  constexpr int U = H / kLstmParts, kWarps = LstmShared<H>::kWarps, kRow = LstmShared<H>::kRow, kXReg = LstmShared<H>::kXReg;
  constexpr uint32_t kStepBytes = 6u * H;
  const int L = p.layers, T = p.steps, warp = tid >> 5, lane = tid & 31;
  const uint32_t xfull0 = smem_u32(sh.x_full), xempty0 = smem_u32(sh.x_empty), hfull0 = smem_u32(sh.h_full);
  // Rows of a warp's tile: row r < 8 is gate r / 4 (i, j) of unit r % 4, row 8 + r gate 2 + r / 4 (f, o).  So lane 4 g + q
  // meets the sums of gates g / 4 and 2 + g / 4 of unit g % 4: q = 0 finishes the first, q = 1 the second.
  const int g = lane >> 2, q = lane & 3, unit0 = part * U + warp * 4, unit = unit0 + (g & 3);
  const float bias_u = p.bias ? p.bias[layer * H + unit] : 0.0f;
  const float bias_g = bias_u + (q == 1 && g < 4 ? 1.0f : 0.0f);       // the forget gate's + 1
  const bool is_tanh = q == 0 && g >= 4;                               // gate j
  uint4 wx[2][kXReg], wh[2][H / 32];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const size_t row = ((size_t)(layer * 4 + 2 * r + (g >> 2)) * H + unit) * H + q * 8;
#pragma unroll
    for (int b = 0; b < H / 32; ++b) {
      const uint4 w = __ldg(reinterpret_cast<const uint4*>(p.w_in + row + b * 32));
      if (b < kXReg) wx[r][b < kXReg ? b : 0] = w;
      else sh.wx_rest[(2 * (b - kXReg) + r) * kWarps * 32 + tid] = w;          // read by this thread only
      wh[r][b] = __ldg(reinterpret_cast<const uint4*>(p.w_state + row + b * 32));
    }
  }
  // lane 8 k + d sends part k of the warp's four hidden states to CTA d; lane 24 stores them to global memory
  const int send_part = lane >> 3;
  const uint32_t send_to = map_shared_rank(smem_u32(&sh.h[0][(send_part < 3 ? send_part : 0) * kRow + unit0]), (uint32_t)(lane & 7));
  const uint32_t send_bar = map_shared_rank(hfull0, (uint32_t)(lane & 7));
  float cx[4];                                // W_in x(t), scaled back
  bool ok = true;
  auto input_half = [&](int step) {
    if constexpr (!kPieces) {
      const int xb = step % kLstmXBufs;
      ok = lstm_wait_warp<false>(xfull0 + 8 * xb, (uint32_t)(step / kLstmXBufs) & 1u, ctl, 910, lane, smem_u32(&sh.pieces));
      if (!ok) return;
      lstm_product<H, kXReg>(wx, sh.wx_rest + (H == 256 ? tid : 0), kWarps * 32, sh.x[xb], lane, cx);
      const float down = sh.x_scale[xb];
#pragma unroll
      for (int i = 0; i < 4; ++i) cx[i] *= down;
      __syncwarp();
      if (lane == 0) mbar_arrive(xempty0 + 8 * xb);       // this warp has read x(step)
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) cx[i] = 0.0f;
      bool more = true;
      while (more) {
        const int piece = *const_cast<volatile int*>(sh.piece + warp), xb = piece % kLstmXBufs;
        ok = lstm_wait_warp<false>(xfull0 + 8 * xb, (uint32_t)(piece / kLstmXBufs) & 1u, ctl, 910, lane);
        if (!ok) return;
        float px[4];
        lstm_product<H, kXReg>(wx, sh.wx_rest + (H == 256 ? tid : 0), kWarps * 32, sh.x[xb], lane, px);
        const float down = sh.x_scale[xb];
#pragma unroll
        for (int i = 0; i < 4; ++i) cx[i] = fmaf(px[i], fabsf(down), cx[i]);
        more = __any_sync(0xffffffffu, down < 0.0f);
        if (lane == 0) {
          sh.piece[warp] = piece + 1;
          mbar_arrive(xempty0 + 8 * xb);
        }
        __syncwarp();
      }
    }
  };
  input_half(t);
  for (; ok && t < T; ++t) {
    const int hb = t & 1;                               // h(t) goes to sh.h[hb]; h(t-1) is in sh.h[hb ^ 1]
    if (t > 0) {
      ok = lstm_wait_warp<true>(hfull0 + 8 * (hb ^ 1), (uint32_t)((t - 1) >> 1) & 1u, ctl, 800 + layer, lane);
      if (!ok) break;
      // that barrier's next phase receives h(t+1); nobody sends it before having this warp's h(t)
      if (tid == 0 && t + 1 < T) mbar_expect_tx(hfull0 + 8 * (hb ^ 1), kStepBytes);
    }
    float ch[4];
    lstm_product<H, H / 32>(wh, sh.wx_rest, 0, sh.h[hb ^ 1], lane, ch);
#pragma unroll
    for (int i = 0; i < 4; ++i) ch[i] = fmaf(ch[i], 1.0f / kLstmHScale, cx[i]);
    // columns 0, 1 (lane q = 0) and 2 (q = 1) are the three parts of the vector
    const float first = q == 0 ? fmaf(ch[1], 1.0f / kLstmPart, ch[0]) : ch[0] * (1.0f / (kLstmPart * kLstmPart));
    const float second = q == 0 ? fmaf(ch[3], 1.0f / kLstmPart, ch[2]) : ch[2] * (1.0f / (kLstmPart * kLstmPart));
    const float other = __shfl_xor_sync(0xffffffffu, q == 0 ? second : first, 1);
    const float pre = (q == 0 ? first : second) + other + bias_g;
    const float act = gate_f(pre, is_tanh);
    const int base = 4 * (g & 3);
    const float gi = __shfl_sync(0xffffffffu, act, base), gf = __shfl_sync(0xffffffffu, act, base + 1);
    const float gj = __shfl_sync(0xffffffffu, act, base + 16), go = __shfl_sync(0xffffffffu, act, base + 17);
    c_state = c_state * gf + gi * gj;
    const float h = gate_f(c_state, true) * go;
    // lanes 4 u .. 4 u + 3 offer the three parts of unit u's hidden state and the fp32 value itself; lane 8 k + d collects
    // offer k of all four units
    uint32_t offer;
    {
      const float s0 = h * kLstmHScale;
      const __half hi = __float2half_rn(s0);
      const float s1 = (s0 - __half2float(hi)) * kLstmPart;
      const __half mid = __float2half_rn(s1);
      const __half lo = __float2half_rn((s1 - __half2float(mid)) * kLstmPart);
      offer = q == 0 ? __half_as_ushort(hi) : q == 1 ? __half_as_ushort(mid) : q == 2 ? __half_as_ushort(lo) : __float_as_uint(h);
    }
    uint32_t got[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) got[i] = __shfl_sync(0xffffffffu, offer, 4 * i + send_part);
    if (lane < 24) {
      const uint64_t word = (uint64_t)(got[0] | (got[1] << 16)) | ((uint64_t)(got[2] | (got[3] << 16)) << 32);
      st_async_b64(send_to + (uint32_t)(hb * 3 * kRow * 2), word, send_bar + 8u * (uint32_t)hb);
    }
    if (lane == 24) {
      if (layer == L - 1) {
        *reinterpret_cast<float4*>(p.y + (size_t)t * H + unit0) =
            make_float4(__uint_as_float(got[0]), __uint_as_float(got[1]), __uint_as_float(got[2]), __uint_as_float(got[3]));
      } else {                                  // for the next layer
        const uint32_t tag = *const_cast<volatile uint32_t*>(&sh.tag);
        uint64_t* to = p.h_all + (size_t)(uint32_t)(layer * T) * H;
        to += (size_t)(uint32_t)t * H;
        to += unit0;
        st_relaxed_tagged(to, got[0], got[1], tag);
        st_relaxed_tagged(to + 2, got[2], got[3], tag);
      }
    }
    if (t + 1 < T) input_half(t + 1);
  }
  // h(T - 1) has no reader, but it has to be here before this CTA's shared memory goes (not to send it would take a condition
  // in every step: 10 x 256 x 100 161.4 us against 156.6, 1 x 256 x 200 233.6 against 227.5)
  if (ok) ok = lstm_wait_warp<true>(hfull0 + 8 * ((T - 1) & 1), (uint32_t)((T - 1) >> 1) & 1u, ctl, 930, lane);
  return ok;
}
// Out of line: rare, and inlined its registers would be taken from the loop above.
template <int H>
__device__ __noinline__ void lstm_steps_in_pieces(const LstmParams& p, LstmShared<H>& sh, float c_state) {
  int t = *const_cast<volatile int*>(sh.piece + (threadIdx.x >> 5));       // every vector before this one came whole
  LstmWaitOf<H> ctl;
  lstm_wait_set<H>(ctl, sh, p);
  lstm_steps<H, true>(p, sh, ctl, blockIdx.x / kLstmParts, (int)cluster_cta_rank(), threadIdx.x, t, c_state);
}

// H = 64, 128 or 256 (= p.hidden).
template <int H>
__global__ void __launch_bounds__(lstm_block(H), 1) souffle_lstm_wavefront(const __grid_constant__ LstmParams p) {
  constexpr int kWarps = LstmShared<H>::kWarps, kRow = LstmShared<H>::kRow;
  constexpr uint32_t kStepBytes = 6u * H;       // a hidden vector: three fp16 parts
  __shared__ LstmShared<H> sh;
  const int L = p.layers, T = p.steps;
  const uint32_t xfull0 = smem_u32(sh.x_full), xempty0 = smem_u32(sh.x_empty), hfull0 = smem_u32(sh.h_full);
  const int layer = blockIdx.x / kLstmParts;
  const int part = (int)cluster_cta_rank();     // == blockIdx.x % kLstmParts for clusters along x
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    sh.abort = 0;
    sh.deadline_ns = globaltimer_ns() + p.timeout_ns;
    sh.pieces = 0;
    sh.tag = (uint32_t)(*const_cast<volatile unsigned long long*>(p.epoch) / kLaunchSteps) + 1u;
    for (int i = 0; i < kLstmXBufs; ++i) {
      mbar_init(xfull0 + 8 * i, 32);            // the 32 lanes of the fetch warp
      mbar_init(xempty0 + 8 * i, kWarps);       // one lane of every cell warp
    }
    mbar_init(smem_u32(&sh.pieces_ready), kWarps);            // one lane of every cell warp
    for (int i = 0; i < 2; ++i) {               // h(0) and h(1): one local arrival that announces the bytes of a vector
      mbar_init(hfull0 + 8 * i, 1);
      mbar_expect_tx(hfull0 + 8 * i, kStepBytes);
    }
    fence_mbar_init();
  }
  for (int i = tid; i < 2 * 3 * kRow; i += lstm_block(H)) (&sh.h[0][0])[i] = __ushort_as_half(0);    // h before the first step
  __syncthreads();
  cluster_sync_all();                           // every CTA's barriers exist before anyone arrives on them

  LstmWaitOf<H> ctl;
  lstm_wait_set<H>(ctl, sh, p);

  if (warp == kWarps) {
    // ---------------- fetch warp: the layer's input vector of every step -> shared memory ----------------
    // The vector of the layer below is polled as a whole, and the next one is requested before this one is unpacked: where the layer
    // below is ahead, a step costs no round trip.
    constexpr int E = H / 32;                   // elements of this lane: lane * E ...
    // vector or piece number n of this CTA: the wait for its slot, and its way into it
    auto slot_free = [&](int n) -> int {
      const int xb = n % kLstmXBufs, use = n / kLstmXBufs;
      if (use == 0) return 1;
      int free = 1;
      if (lane == 0) free = lstm_wait_loop<false>(xempty0 + 8 * xb, (uint32_t)(use - 1) & 1u, ctl, 900, 0) ? 1 : 0;
      free = __shfl_sync(0xffffffffu, free, 0);
      __syncwarp();
      return free;
    };
    auto hand_over = [&](int n, const float (&val)[E], float up, float down) {
      const int xb = n % kLstmXBufs;
      __half hi[E], mid[E], lo[E];
#pragma unroll
      for (int i = 0; i < E; ++i) lstm_split(val[i] * up, hi[i], mid[i], lo[i]);
#pragma unroll
      for (int i = 0; i < E; i += 2) {
        __half* dst = sh.x[xb] + lane * E + i;
        *reinterpret_cast<__half2*>(dst) = __halves2half2(hi[i], hi[i + 1]);
        *reinterpret_cast<__half2*>(dst + kRow) = __halves2half2(mid[i], mid[i + 1]);
        *reinterpret_cast<__half2*>(dst + 2 * kRow) = __halves2half2(lo[i], lo[i + 1]);
      }
      if (lane == 0) sh.x_scale[xb] = down;
      mbar_arrive(xfull0 + 8 * xb);             // release: this lane's stores are visible to whoever waits
    };
    if (layer > 0) {
      const uint64_t* src = p.h_all + (size_t)(layer - 1) * T * H + lane * E;
      const uint32_t tag = *const_cast<volatile uint32_t*>(&sh.tag);
      uint64_t word[E];
      auto request = [&](const uint64_t* from, uint64_t (&w)[E]) {
#pragma unroll
        for (int i = 0; i < E; i += 2) ld_relaxed_2x64(from + i, w[i], w[i + 1]);
      };
      request(src, word);
      for (int t = 0; t < T; ++t, src += H) {
        int ok = 1;
        uint32_t spins = 0;
        for (;;) {
          bool there = true;
#pragma unroll
          for (int i = 0; i < E; ++i) there = there && (uint32_t)(word[i] >> 32) == tag;
          if (__all_sync(0xffffffffu, there)) break;
          if (((++spins) & 0x3F) == 0) {
            int give_up = 0;
            if (lane == 0) give_up = lstm_expired(ctl, DEV_TIMEOUT_FLAG, 700 + layer) ? 1 : 0;
            if (__shfl_sync(0xffffffffu, give_up, 0)) {
              ok = 0;
              break;
            }
          }
          request(src, word);
        }
        float v[E];
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = __uint_as_float((uint32_t)word[i]);
        if (ok && t + 1 < T) request(src + H, word);
        if (ok) ok = slot_free(t);
        if (!ok) {
          if (lane == 0) *const_cast<volatile int*>(&sh.abort) = 1;
          break;
        }
        hand_over(t, v, kLstmHScale, 1.0f / kLstmHScale);          // hidden states: a constant scale
      }
    }
    int piece = 0;                              // layer 0: pieces handed over so far (the steps so far, unless one had several)
    bool in_pieces = false;                     // the cell warps expect several
    for (int t = 0; layer == 0 && t < T; ++t) {
      const int tx = p.ref_input_delay ? t - 1 : t;
      const float* src = p.x + (size_t)tx * H + lane * E;
      float v[E];
#pragma unroll
      for (int i = 0; i < E; i += 2) {
        const float2 f = tx >= 0 ? __ldcg(reinterpret_cast<const float2*>(src + i)) : make_float2(0.f, 0.f);
        v[i] = f.x;
        v[i + 1] = f.y;
      }
      int ok = 1;
      for (bool more = true; more && ok;) {
        // power-of-two scale that takes the piece's largest element into the upper range of fp16
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < E; ++i) m = max(m, __float_as_uint(v[i]) & 0x7fffffffu);
        m = __reduce_max_sync(0xffffffffu, m);
        uint32_t e = m >> 23, least = 0;        // biased exponents: of the largest element, of the smallest this piece takes
        more = false;
        if (e >= kLstmWide) {
          least = e == 255u ? 255u : e - kLstmPieceRange;
          bool rest = false;
#pragma unroll
          for (int i = 0; i < E; ++i) rest = rest || (v[i] != 0.0f && ((__float_as_uint(v[i]) >> 23) & 255u) < least);
          more = __any_sync(0xffffffffu, rest);
          if (more && !in_pieces) {             // the cell warps have to expect it: they stop in front of this vector
            if (lane == 0) {
              st_release_cta_shared_u32(smem_u32(&sh.pieces), 1u);
              ok = lstm_wait_loop<false>(smem_u32(&sh.pieces_ready), 0u, ctl, 920, 0) ? 1 : 0;
            }
            ok = __shfl_sync(0xffffffffu, ok, 0);
            in_pieces = true;
          }
        }
        float up = 1.0f, down = 1.0f;           // an infinity or NaN passes through as it is
        if (e != 255u) {
          e = e < 15u ? 15u : e;                // 2^-112 and below need no more than the largest scale
          up = __uint_as_float((268u - e) << 23);        // 2^(14 - (e - 127))
          down = __uint_as_float((e - 14u) << 23);
        }
        float part_v[E];
#pragma unroll
        for (int i = 0; i < E; ++i) {
          const bool take = ((__float_as_uint(v[i]) >> 23) & 255u) >= least;
          part_v[i] = take ? v[i] : 0.0f;
          if (take) v[i] = 0.0f;
        }
        if (ok) ok = slot_free(piece);
        if (ok) hand_over(piece++, part_v, up, more ? -down : down);
      }
      if (!ok) {
        if (lane == 0) *const_cast<volatile int*>(&sh.abort) = 1;
        break;
      }
    }
  } else {
    // ---------------- cell arithmetic ----------------
    int t = 0;
    float c_state = 0.0f;
    const bool ok = lstm_steps<H, false>(p, sh, ctl, layer, part, tid, t, c_state);
    if (!ok && *const_cast<volatile int*>(&sh.abort) == 0) {          // not given up: vector t comes in pieces, all before it came whole
      if (lane == 0) {
        sh.piece[warp] = t;
        mbar_arrive(smem_u32(&sh.pieces_ready));
      }
      __syncwarp();
      lstm_steps_in_pieces<H>(p, sh, c_state);
    }
  }
  // Nobody leaves while a peer may still store into its shared memory.
  __syncthreads();
  cluster_sync_all();
  if (*const_cast<volatile int*>(&sh.abort)) {   // sent by peers before they came here, and not waited for: 200 us are ample
    if (tid == 0 && p.expired) *p.expired = 1;
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  // The steps of the cluster's CTAs, all of which have read the counter.  (At hidden 256 the register allocation hangs on this place:
  // taken with the read, the step leaves a spill in the prologue, behind the barrier or by a thread per CTA the loop is 0.5-0.7 % slower.)
  if (part == 0 && tid < kLstmParts) atomicAdd(p.epoch, (unsigned long long)launch_step(blockIdx.x + tid, gridDim.x));
}

}  // namespace souffle
