// Squeeze-and-excite module as one global-sync launch (fp32, NCHW).
//
// The reference's fused kernel (cpp/efficientnet/kernels/se_module_global_fused.cu:316-444) runs four phases
// separated by three grid.sync(): per-channel average pool (the channel's image kept in shared memory), the
// reduce GEMV with x*sigmoid(x), the expand GEMV with sigmoid, and the broadcast add of the gate onto the image.
// Here a channel's image is cut into slices handed out per warp, so that small channel counts still fill the GPU
// and small images cost no CTA-wide synchronisation; every warp keeps as many of its slices in shared memory across the
// one grid barrier as fit, and both tiny GEMVs are recomputed by every CTA that needs them instead of being exchanged
// through two more barriers: the input is read from HBM once and the output written once.
// The module is bound by memory: 16 warps of an SM have to keep some 40 KB of loads in flight to draw the full HBM rate,
// so a warp issues eight 16-byte loads per lane before it touches the first of them.  One 4-byte load per lane and four in
// flight took 107-114 us of GPU time for 32 x 144 x 56 x 56 (1.1 TB/s of the 116 MB the module cannot do without), this
// form 33 us (3.6 TB/s).
// Small images with many channels are bound by the reduce weights instead (1 x 1152 x 7 x 7: 221 KB, which every CTA needs,
// against 0.2 MB of image): a CTA brings them to shared memory while it waits at the barrier, 16 bytes at a time, eight
// loads in flight (19.7 us under ncu with the rows of the GEMV read from L2 four 4-byte loads at a time, 13.8 so).  Larger
// weights stay in L2 and are read 16 bytes at a time (1 x 4096 x 8 x 8, 1 MB of weights: 62 us by 4-byte loads, 24.5 so).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "sm100_ptx.cuh"

namespace souffle {

constexpr int kSeThreads = 512;
constexpr int kSeWarps = kSeThreads / 32;
constexpr int kSeSmemBytes = 231424;          // 226 KiB of dynamic shared memory at most
constexpr int kSeMaxReduce = 64;              // reduce channels
constexpr int kSeMaxChannels = 4096;          // channels (their means are staged in shared memory)
constexpr int kSeUnroll = 8;                  // 16-byte loads a lane has in flight

// Floats of shared memory a cached slice takes: up to three in front of it, so that the 16-byte pieces of the slice sit on
// 16-byte boundaries there too, wherever it starts in global memory.
__host__ __device__ inline int se_slice_floats(int slice_len) { return (slice_len + 3 + 3) & ~3; }

struct SeParams {
  const float* input;      // [batch][channels][hw]
  const float* w_reduce;   // [reduce][channels]
  const float* w_expand;   // [channels][reduce]
  float* out;              // [batch][channels][hw]
  float* pooled;           // optional [batch][channels] channel means (the reference returns them)
  float* partial;          // [batch*channels][slices] partial sums of the pool
  unsigned* sync;          // arrival counter of the grid barrier (zero at launch, left zero by the last CTA out)
  int* status;             // [0] code, [1] where, [2] cta
  int* expired;            // host memory: set by a CTA that gave up on the barrier
  int batch, channels, hw, reduce;
  int slices, slice_len;   // a channel image = slices pieces of slice_len floats (the last one shorter)
  int items;               // batch * channels * slices
  int per_cta;             // CTA b owns items [b * per_cta, (b + 1) * per_cta): few images per CTA
  int cached;              // of the (up to ceil(per_cta / 16)) slices of a warp, those kept in shared memory
  int stage_weights;       // 1: w_reduce is brought to shared memory while the CTA loads its slices
  unsigned long long timeout_ns;
};

__device__ __forceinline__ float se_sigmoid(float x) { return 1.0f / (1.0f + __expf(-x)); }

// The first element of a slice that sits on a 16-byte boundary.
__device__ __forceinline__ int se_head(const float* p, int len) {
  const int h = (4 - (int)((reinterpret_cast<uintptr_t>(p) >> 2) & 3)) & 3;
  return h < len ? h : len;
}

// Sum of one slice (per lane: the lane's share); the slice is copied to `keep` unless that is null.  `keep` has the slice's
// own offset from a 16-byte boundary.
__device__ __forceinline__ float se_load_slice(const float* __restrict__ src, float* keep, int len, int lane) {
  const int head = se_head(src, len), n4 = (len - head) >> 2, tail = head + 4 * n4;
  float s = 0.0f, edge = 0.0f;
  const bool has_edge = lane < head || tail + lane < len;          // up to three floats at either end
  const int at = lane < head ? lane : tail + lane;
  if (has_edge) edge = __ldg(src + at);
  const bool has_edge2 = lane < head && tail + lane < len;         // a lane with one at each end
  float edge2 = 0.0f;
  if (has_edge2) edge2 = __ldg(src + tail + lane);
  const float4* s4 = reinterpret_cast<const float4*>(src + head);
  float4* k4 = reinterpret_cast<float4*>(keep + head);
  for (int i0 = lane; i0 < n4; i0 += 32 * kSeUnroll) {
    float4 v[kSeUnroll];
#pragma unroll
    for (int u = 0; u < kSeUnroll; ++u) {
      const int i = i0 + 32 * u;
      v[u] = i < n4 ? __ldg(s4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < kSeUnroll; ++u) {
      const int i = i0 + 32 * u;
      if (keep && i < n4) k4[i] = v[u];
      s += (v[u].x + v[u].y) + (v[u].z + v[u].w);
    }
  }
  if (keep && has_edge) keep[at] = edge;
  if (keep && has_edge2) keep[tail + lane] = edge2;
  return s + (edge + edge2);
}

// dst = src + g over one slice; 16 bytes at a time where src and dst have the same offset from a 16-byte boundary.
__device__ __forceinline__ void se_add_slice(const float* src, float* __restrict__ dst, int len, float g, int lane) {
  if (((reinterpret_cast<uintptr_t>(src) ^ reinterpret_cast<uintptr_t>(dst)) & 15) != 0) {
    for (int i = lane; i < len; i += 32) dst[i] = src[i] + g;
    return;
  }
  const int head = se_head(src, len), n4 = (len - head) >> 2, tail = head + 4 * n4;
  const float4* s4 = reinterpret_cast<const float4*>(src + head);
  float4* d4 = reinterpret_cast<float4*>(dst + head);
  for (int i0 = lane; i0 < n4; i0 += 32 * kSeUnroll) {
    float4 v[kSeUnroll];
#pragma unroll
    for (int u = 0; u < kSeUnroll; ++u)
      if (i0 + 32 * u < n4) v[u] = s4[i0 + 32 * u];
#pragma unroll
    for (int u = 0; u < kSeUnroll; ++u)
      if (i0 + 32 * u < n4) d4[i0 + 32 * u] = make_float4(v[u].x + g, v[u].y + g, v[u].z + g, v[u].w + g);
  }
  if (lane < head) dst[lane] = src[lane] + g;
  if (tail + lane < len) dst[tail + lane] = src[tail + lane] + g;
}

// Work is handed out per WARP: an item is one slice of one channel image; warp w of CTA b takes items
// b * per_cta + w, + 16, ...  Everything but the grid barrier and the per-image reduce GEMV is warp-local, so a 7 x 7
// image costs no CTA-wide synchronisation.
__global__ void __launch_bounds__(kSeThreads, 1) souffle_se_module(const SeParams p) {
  extern __shared__ __align__(16) float se_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int keep_floats = se_slice_floats(p.slice_len);
  float* my_cache = se_smem + (size_t)warp * p.cached * keep_floats;                 // this warp's kept slices
  float* w_red = se_smem + (size_t)kSeWarps * p.cached * keep_floats;                // [reduce][channels] when staged
  float* pooled_s = w_red + (p.stage_weights ? p.reduce * p.channels : 0);           // channel means of one image
  float* gate_in = pooled_s + p.channels;                                            // reduce GEMV outputs of one image
  __shared__ int abort_flag;
  const int item0 = blockIdx.x * p.per_cta, item1 = min(item0 + p.per_cta, p.items);
  if (threadIdx.x == 0) abort_flag = 0;

  // ---- phase 1: this warp's slices, their partial sums ----
  int slot = 0;
  for (int item = item0 + warp; item < item1; item += kSeWarps, ++slot) {
    const int ch = item / p.slices, sl = item - ch * p.slices;          // ch = image * channels + channel
    const int begin = sl * p.slice_len;
    const int len = min(p.slice_len, p.hw - begin);
    const float* src = p.input + (size_t)ch * p.hw + begin;
    float* keep = slot < p.cached ? my_cache + slot * keep_floats + ((reinterpret_cast<uintptr_t>(src) >> 2) & 3) : nullptr;
    const float s = warp_sum(se_load_slice(src, keep, len, lane));
    if (lane == 0) p.partial[(size_t)ch * p.slices + sl] = s;
  }

  // ---- the one grid barrier: every partial sum is published; the weights come in while this CTA waits ----
  __syncthreads();
  if (threadIdx.x == 0) {
    red_add_release_u32(p.sync, 1u);
    const unsigned long long t0 = globaltimer_ns();
    uint32_t spins = 0;
    while (ld_acquire_u32(p.sync) < gridDim.x) {
      if (((++spins) & 0x3F) == 0 && globaltimer_ns() - t0 > p.timeout_ns) {
        if (atomicCAS(p.status, (int)DEV_OK, (int)DEV_TIMEOUT_GRID) == (int)DEV_OK) {   // first CTA to give up records where
          p.status[1] = 900;
          p.status[2] = (int)blockIdx.x;
        }
        *p.expired = 1;
        abort_flag = 1;
        break;
      }
    }
  } else if (warp > 0 && p.stage_weights) {
    const int n = p.reduce * p.channels, n4 = (reinterpret_cast<uintptr_t>(p.w_reduce) & 15) == 0 ? n >> 2 : 0;
    constexpr int kStep = kSeThreads - 32;
    for (int i0 = threadIdx.x - 32; i0 < n4; i0 += kStep * kSeUnroll) {
      float4 v[kSeUnroll];
#pragma unroll
      for (int u = 0; u < kSeUnroll; ++u)
        if (i0 + u * kStep < n4) v[u] = __ldg(reinterpret_cast<const float4*>(p.w_reduce) + i0 + u * kStep);
#pragma unroll
      for (int u = 0; u < kSeUnroll; ++u)
        if (i0 + u * kStep < n4) reinterpret_cast<float4*>(w_red)[i0 + u * kStep] = v[u];
    }
    for (int i = 4 * n4 + threadIdx.x - 32; i < n; i += kStep) w_red[i] = __ldg(p.w_reduce + i);
  }
  __syncthreads();
  if (abort_flag) return;

  // ---- phases 2-4: per image the channel means and the reduce GEMV (x * sigmoid x) once per CTA, then per
  //      item this channel's gate (expand GEMV row, sigmoid) and the add ----
  const float inv_hw = 1.0f / (float)p.hw;
  const int items_per_img = p.channels * p.slices;
  int cur_img = -1;
  slot = 0;
  for (int first = item0; first < item1; first += kSeWarps, ++slot) {    // item of warp 0 in this round
    const int last = min(first + kSeWarps, item1) - 1;
    for (int img = first / items_per_img; img <= last / items_per_img; ++img) {
      // a round of one CTA spans at most a few images; (re)build the image's reduce outputs when it changes
      if (img != cur_img) {
        __syncthreads();
        for (int k = threadIdx.x; k < p.channels; k += kSeThreads) {
          const float* pp = p.partial + (size_t)(img * p.channels + k) * p.slices;
          float s = 0.0f;
#pragma unroll 8
          for (int s2 = 0; s2 < p.slices; ++s2) s += __ldcg(pp + s2);       // written by other CTAs: read at L2
          pooled_s[k] = s * inv_hw;
        }
        __syncthreads();
        for (int j = warp; j < p.reduce; j += kSeWarps) {
          float acc = 0.0f;
          if (p.stage_weights) {
#pragma unroll 4
            for (int k = lane; k < p.channels; k += 32) acc = fmaf(pooled_s[k], w_red[j * p.channels + k], acc);
          } else {                                           // too large to stage: rows from L2, eight loads in flight
            const float* row = p.w_reduce + (size_t)j * p.channels;
            if (p.channels % 4 == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
#pragma unroll 8
              for (int k = lane; k < p.channels / 4; k += 32) {
                const float4 w = __ldg(reinterpret_cast<const float4*>(row) + k), m = reinterpret_cast<const float4*>(pooled_s)[k];
                acc = fmaf(m.w, w.w, fmaf(m.z, w.z, fmaf(m.y, w.y, fmaf(m.x, w.x, acc))));
              }
            } else {
#pragma unroll 8
              for (int k = lane; k < p.channels; k += 32) acc = fmaf(pooled_s[k], __ldg(row + k), acc);
            }
          }
          acc = warp_sum(acc);
          if (lane == 0) gate_in[j] = acc * se_sigmoid(acc);
        }
        __syncthreads();
        cur_img = img;
      }
      const int item = first + warp;
      if (item <= last && item / items_per_img == img) {
        const int ch = item / p.slices, sl = item - ch * p.slices;
        const int c = ch - img * p.channels;
        float g = 0.0f;                                      // expand GEMV row of this channel: lanes over the reduce outputs
        for (int j = lane; j < p.reduce; j += 32) g = fmaf(gate_in[j], __ldg(p.w_expand + (size_t)c * p.reduce + j), g);
        g = se_sigmoid(warp_sum(g));
        if (p.pooled && sl == 0 && lane == 0) p.pooled[ch] = pooled_s[c];
        const int begin = sl * p.slice_len;
        const int len = min(p.slice_len, p.hw - begin);
        const float* src = p.input + (size_t)ch * p.hw + begin;
        if (slot < p.cached) src = my_cache + slot * keep_floats + ((reinterpret_cast<uintptr_t>(src) >> 2) & 3);
        se_add_slice(src, p.out + (size_t)ch * p.hw + begin, len, g, lane);
      }
    }
  }

  // ---- leave the barrier word clean for the next launch: the last CTA out resets it ----
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned old = atomicAdd(p.sync + 1, 1u);
    if (old == gridDim.x - 1) {
      p.sync[0] = 0u;
      p.sync[1] = 0u;
    }
  }
}

}  // namespace souffle
