// Squeeze-and-excite module as one global-sync launch (fp32, NCHW).
//
// The reference's fused kernel (cpp/efficientnet/kernels/se_module_global_fused.cu:316-444) runs four phases
// separated by three grid.sync(): per-channel average pool (the channel's image kept in shared memory), the
// reduce GEMV with x*sigmoid(x), the expand GEMV with sigmoid, and the broadcast add of the gate onto the image.
// Here a channel's image is cut into slices handed out per warp, so that small channel counts still fill the GPU
// and small images cost no CTA-wide synchronisation; every warp keeps as many of its slices in shared memory across the
// one grid barrier as fit, and both tiny GEMVs are recomputed by every CTA that needs them instead of being exchanged
// through two more barriers: the input is read from HBM once and the output written once.
// The module is bound by memory.  A warp owns a contiguous run of slices; as many of them as fit shared memory come in as one bulk copy
// that no register waits for, the others are summed from registers meanwhile, sixteen 16-byte loads per lane in flight, and read again in
// the end.  With eight loads per lane in flight, slice by slice, 58 MB (32 x 144 x 56 x 56) took 15 us to come in (12.5 so), 7 MB in
// slices of 196 bytes (32 x 1152 x 7 x 7) 12 us (8 so).
// The gates of a CTA's channels are worked out by all threads at once, a channel each, for all images that the CTA meets: one warp-wide
// GEMV row per slice, each a round trip to L2, had made 32 x 1152 x 7 x 7 spend 23 us in its last phase, and a second image's chain of
// reads cost 6 us of 30 in 32 x 144 x 56 x 56.  A launch of (us, before -> now): 32 x 144 x 56 x 56 33.5 -> 30.9, 32 x 32 x 112 x 112
// 31.3 -> 28.1, 32 x 672 x 14 x 14 31.3 -> 15.0, 32 x 1152 x 7 x 7 44.0 -> 17.3, 13 x 480 x 14 x 14 11.5 -> 8.9.
// The first two move 2.5 times their input: what shared memory does not hold is read again, from L2.
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

// Floats of shared memory that a warp's kept run of `n` slices takes: up to three in front of it, so that its 16-byte pieces sit on 16-byte
// boundaries there too, wherever it starts in global memory, and as many behind it.
__host__ __device__ inline int se_run_floats(int n, int slice_len) { return n ? (n * slice_len + 3 + 3) & ~3 : 0; }

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
  uint32_t mg_hw;          // multiplier of the divisor hw over a CTA's elements, or 0: images of 512 floats and more are added one by one
  int slices, slice_len;   // a channel image = slices pieces of slice_len floats (the last one shorter)
  int items;               // batch * channels * slices
  int per_cta;             // CTA b owns items [b * per_cta, (b + 1) * per_cta): few images per CTA
  int per_warp;            // warp w owns per_warp of them from b * per_cta + w * per_warp on
  int cached;              // of the slices of a warp, those kept in shared memory (the first ones)
  int stage_weights;       // 1: w_reduce is brought to shared memory while the CTA waits at the barrier
  int expand_rows;         // the same for w_expand: room for that many rows, or 0
  int group;               // images of a CTA worked on at a time
  unsigned long long timeout_ns;
};

__device__ __forceinline__ float se_sigmoid(float x) { return 1.0f / (1.0f + __expf(-x)); }

// The first element of a slice that sits on a 16-byte boundary.
__device__ __forceinline__ int se_head(const float* p, int len) {
  const int h = (4 - (int)((reinterpret_cast<uintptr_t>(p) >> 2) & 3)) & 3;
  return h < len ? h : len;
}

// A lane's share of the sum of one slice in global memory.
__device__ __forceinline__ float se_sum_slice(const float* __restrict__ src, int len, int lane) {
  const int head = se_head(src, len), n4 = (len - head) >> 2, tail = head + 4 * n4;
  float s = 0.0f;
  if (lane < head) s += __ldg(src + lane);                         // up to three floats at either end
  if (tail + lane < len) s += __ldg(src + tail + lane);
  const float4* s4 = reinterpret_cast<const float4*>(src + head);
  constexpr int kDeep = 2 * kSeUnroll;
  for (int i0 = lane; i0 < n4; i0 += 32 * kDeep) {
    float4 v[kDeep];
#pragma unroll
    for (int u = 0; u < kDeep; ++u) {
      const int i = i0 + 32 * u;
      v[u] = i < n4 ? __ldg(s4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < kDeep; ++u) s += (v[u].x + v[u].y) + (v[u].z + v[u].w);
  }
  return s;
}
// The same in shared memory, where the slice starts `off` floats behind a 16-byte boundary.
__device__ __forceinline__ float se_sum_kept(const float* src, int off, int len, int lane) {
  int head = (4 - off) & 3;
  if (head > len) head = len;
  const int n4 = (len - head) >> 2, tail = head + 4 * n4;
  float s = 0.0f;
  if (lane < head) s += src[lane];
  if (tail + lane < len) s += src[tail + lane];
  const float4* s4 = reinterpret_cast<const float4*>(src + head);
#pragma unroll 4
  for (int i = lane; i < n4; i += 32) {
    const float4 v = s4[i];
    s += (v.x + v.y) + (v.z + v.w);
  }
  return s;
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

// The one grid barrier: every partial sum is published, and the weights (the reduce weights where they fit, the rows of the CTA's channels
// of the expand weights where they are few) come in while this CTA waits.  False: it was given up.
__device__ __forceinline__ bool se_barrier(const SeParams& p, volatile int* abort_flag, float* w_red, float* w_exp, int expand_pitch, int ch0, int ch1) {
  const int warp = threadIdx.x >> 5;
  __syncthreads();
  if (threadIdx.x == 0 && !*abort_flag) {
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
        *abort_flag = 1;
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
  if (w_exp && warp > 0 && p.expand_rows) {
    const int n = (ch1 - ch0 + 1) * p.reduce, c = ch0 % p.channels;
#pragma unroll 4
    for (int i = threadIdx.x - 32; i < n; i += kSeThreads - 32) {
      const int r = i / p.reduce, j = i - r * p.reduce;
      int row = c + r;
      while (row >= p.channels) row -= p.channels;
      w_exp[r * expand_pitch + j] = __ldg(p.w_expand + row * p.reduce + j);
    }
  }
  __syncthreads();
  return *abort_flag == 0;
}

// Channel means and reduce GEMV (x * sigmoid x) of images img..img + ni - 1; the means whose first slice lies in [lo, hi) of the items go to
// the caller's array.
__device__ __forceinline__ void se_means_and_reduce(const SeParams& p, int img, int ni, int lo, int hi, const float* w_red, float* pooled_s, float* gate_in) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float inv_hw = 1.0f / (float)p.hw;
  const int img0 = img * p.channels * p.slices;
  for (int k = threadIdx.x; k < ni * p.channels; k += kSeThreads) {
    const float* pp = p.partial + (size_t)(img * p.channels + k) * p.slices;
    float s = 0.0f;
#pragma unroll 8
    for (int s2 = 0; s2 < p.slices; ++s2) s += __ldcg(pp + s2);       // written by other CTAs: read at L2
    s *= inv_hw;
    pooled_s[k] = s;
    if (p.pooled && img0 + k * p.slices >= lo && img0 + k * p.slices < hi) p.pooled[img * p.channels + k] = s;
  }
  __syncthreads();
  if (p.stage_weights) {
    for (int t = warp; t < ni * p.reduce; t += kSeWarps) {
      const int im = t / p.reduce, j = t - im * p.reduce;
      const float* mean = pooled_s + im * p.channels;
      float acc = 0.0f;
#pragma unroll 4
      for (int k = lane; k < p.channels; k += 32) acc = fmaf(mean[k], w_red[j * p.channels + k], acc);
      acc = warp_sum(acc);
      if (lane == 0) gate_in[im * kSeMaxReduce + j] = acc * se_sigmoid(acc);
    }
  } else {                                             // too large to stage: rows from L2, a warp's (up to four) at once
    constexpr int kRows = kSeMaxReduce / kSeWarps;
#pragma unroll 1
    for (int im = 0; im < ni; ++im) {
      const float* mean = pooled_s + im * p.channels;
      float acc[kRows];
#pragma unroll
      for (int r = 0; r < kRows; ++r) acc[r] = 0.0f;
      if (p.channels % 4 == 0 && ((reinterpret_cast<uintptr_t>(p.w_reduce) | reinterpret_cast<uintptr_t>(mean)) & 15) == 0) {
#pragma unroll 2
        for (int k = lane; k < p.channels / 4; k += 32) {
          const float4 m = reinterpret_cast<const float4*>(mean)[k];
#pragma unroll
          for (int r = 0; r < kRows; ++r) {
            const int j = warp + r * kSeWarps;
            const float4 w = j < p.reduce ? __ldg(reinterpret_cast<const float4*>(p.w_reduce + (size_t)j * p.channels) + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            acc[r] = fmaf(m.w, w.w, fmaf(m.z, w.z, fmaf(m.y, w.y, fmaf(m.x, w.x, acc[r]))));
          }
        }
      } else {
#pragma unroll 4
        for (int k = lane; k < p.channels; k += 32)
#pragma unroll
          for (int r = 0; r < kRows; ++r) {
            const int j = warp + r * kSeWarps;
            if (j < p.reduce) acc[r] = fmaf(mean[k], __ldg(p.w_reduce + (size_t)j * p.channels + k), acc[r]);
          }
      }
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        const int j = warp + r * kSeWarps;
        const float v = warp_sum(acc[r]);
        if (lane == 0 && j < p.reduce) gate_in[im * kSeMaxReduce + j] = v * se_sigmoid(v);
      }
    }
  }
  __syncthreads();
}

// ---- leave the barrier word clean for the next launch: the last CTA out resets it ----
__device__ __forceinline__ void se_leave(const SeParams& p) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned old = atomicAdd(p.sync + 1, 1u);
    if (old == gridDim.x - 1) {
      p.sync[0] = 0u;
      p.sync[1] = 0u;
    }
  }
}

// Few slices: a warp has one, of 1024 floats at most, and keeps it in registers, as it does its row of the expand weights.  Such a call is
// a chain of latencies (image, barrier, partial sums, two tiny GEMVs), so nothing else stands in it: 1 x 32 x 112 x 112 takes 6.4 us here,
// 7.5 in the kernel below and 6.7 where slices went through shared memory and a gate's weights came in behind the barrier (1 x 96 x 56 x
// 56: 5.7, 7.0 and 6.1).
__global__ void __launch_bounds__(kSeThreads, 1) souffle_se_module_small(const SeParams p) {
  extern __shared__ __align__(16) float se_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* w_red = se_smem;
  float* pooled_s = w_red + (p.stage_weights ? p.reduce * p.channels : 0);
  float* gate_in = pooled_s + p.group * p.channels;
  __shared__ int abort_flag;
  const int item0 = blockIdx.x * p.per_cta, item1 = min(item0 + p.per_cta, p.items), item = item0 + warp;
  if (threadIdx.x == 0) abort_flag = 0;
  const bool mine = item < item1;
  const int ch = item / p.slices, at = ch * p.hw + (item - ch * p.slices) * p.slice_len;
  const int len = mine ? min(p.slice_len, p.hw - (item - ch * p.slices) * p.slice_len) : 0;
  const float* src = p.input + at;
  const int head = mine ? se_head(src, len) : 0, n4 = (len - head) >> 2, tail = head + 4 * n4;
  float4 v[kSeUnroll];
  float e0 = 0.0f, e1 = 0.0f, w0 = 0.0f, w1 = 0.0f;
#pragma unroll
  for (int u = 0; u < kSeUnroll; ++u) {
    const int i = lane + 32 * u;
    v[u] = i < n4 ? __ldg(reinterpret_cast<const float4*>(src + head) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (lane < head) e0 = __ldg(src + lane);
  if (tail + lane < len) e1 = __ldg(src + tail + lane);
  if (mine) {
    const float* row = p.w_expand + (ch % p.channels) * p.reduce;
    if (lane < p.reduce) w0 = __ldg(row + lane);
    if (lane + 32 < p.reduce) w1 = __ldg(row + lane + 32);
    float s = e0 + e1;
#pragma unroll
    for (int u = 0; u < kSeUnroll; ++u) s += (v[u].x + v[u].y) + (v[u].z + v[u].w);
    s = warp_sum(s);
    if (lane == 0) p.partial[item] = s;
  }
  if (!se_barrier(p, &abort_flag, w_red, nullptr, 0, 0, 0)) return;
  const int items_per_img = p.channels * p.slices, img_end = (item1 - 1) / items_per_img + 1;
  for (int img = item0 / items_per_img; img < img_end; img += p.group) {
    const int ni = min(p.group, img_end - img);
    const int img0 = img * items_per_img, lo = max(item0, img0), hi = min(item1, img0 + ni * items_per_img);
    se_means_and_reduce(p, img, ni, lo, hi, w_red, pooled_s, gate_in);
    if (item >= lo && item < hi) {
      const float* in = gate_in + (ch / p.channels - img) * kSeMaxReduce;
      float g = lane < p.reduce ? in[lane] * w0 : 0.0f;
      if (lane + 32 < p.reduce) g = fmaf(in[lane + 32], w1, g);
      g = se_sigmoid(warp_sum(g));
      float* dst = p.out + at;
      if (((reinterpret_cast<uintptr_t>(src) ^ reinterpret_cast<uintptr_t>(dst)) & 15) == 0) {
#pragma unroll
        for (int u = 0; u < kSeUnroll; ++u)
          if (lane + 32 * u < n4)
            reinterpret_cast<float4*>(dst + head)[lane + 32 * u] = make_float4(v[u].x + g, v[u].y + g, v[u].z + g, v[u].w + g);
      } else {
#pragma unroll
        for (int u = 0; u < kSeUnroll; ++u)
          if (lane + 32 * u < n4) {
            float* d = dst + head + 4 * (lane + 32 * u);
            d[0] = v[u].x + g; d[1] = v[u].y + g; d[2] = v[u].z + g; d[3] = v[u].w + g;
          }
      }
      if (lane < head) dst[lane] = e0 + g;
      if (tail + lane < len) dst[tail + lane] = e1 + g;
    }
    if (img + p.group < img_end) __syncthreads();        // the next group's means go over this one's
  }
  se_leave(p);
}

// Work is handed out per WARP: an item is one slice of one channel image, items lie one behind the other in memory, and warp w of CTA b takes
// per_warp of them from b * per_cta + w * per_warp on.  Everything but the grid barrier and the per-image GEMVs is warp-local, so a 7 x 7
// image costs no CTA-wide synchronisation.
__global__ void __launch_bounds__(kSeThreads, 1) souffle_se_module(const SeParams p) {
  extern __shared__ __align__(16) float se_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int run_floats = se_run_floats(p.cached, p.slice_len);
  float* my_run = se_smem + (size_t)warp * run_floats;                               // this warp's kept slices
  float* w_red = se_smem + (size_t)kSeWarps * run_floats;                            // [reduce][channels] when staged
  float* pooled_s = w_red + (p.stage_weights ? p.reduce * p.channels : 0);           // channel means of a group of images, then the gates
  float* gate_in = pooled_s + p.group * p.channels;                                  // reduce GEMV outputs of the group
  float* w_exp = gate_in + p.group * kSeMaxReduce;                                   // rows of the CTA's channels, `expand_pitch` apart
  const int expand_pitch = p.reduce | 1;                                             // (odd: a thread reads a row)
  __shared__ int abort_flag;
  __shared__ uint64_t run_full[kSeWarps];
  const int item0 = blockIdx.x * p.per_cta, item1 = min(item0 + p.per_cta, p.items);
  const int mine0 = min(item0 + warp * p.per_warp, item1), mine1 = min(mine0 + p.per_warp, item1), kept1 = min(mine0 + p.cached, mine1);
  // first element of an item, as an offset in the tensor
  const bool whole = p.slices == 1;                                  // (no division where an item is a channel image)
  auto channel_of = [&](int item) -> int { return whole ? item : item / p.slices; };
  auto item_at = [&](int item) -> int { const int ch = channel_of(item); return ch * p.hw + (item - ch * p.slices) * p.slice_len; };
  auto item_len = [&](int item) -> int { return whole ? p.hw : min(p.slice_len, p.hw - (item % p.slices) * p.slice_len); };
  if (threadIdx.x == 0) abort_flag = 0;
  const uint32_t full = smem_u32(&run_full[warp]);
  const int run_at = item_at(mine0), run_len = item_at(kept1) - run_at;
  const int run_off = (int)((reinterpret_cast<uintptr_t>(p.input + run_at) >> 2) & 3);
  float* run = my_run + run_off;

  // ---- phase 1: this warp's slices, their partial sums ----
  const bool bulk = mine0 < kept1;
  if (bulk) {
    const float* src = p.input + run_at;
    const int head = se_head(src, run_len), n4 = (run_len - head) >> 2, tail = head + 4 * n4;
    if (lane == 0) {
      mbar_init(full, 1);
      fence_mbar_init();
      mbar_expect_tx(full, 16u * (uint32_t)n4);
      if (n4) bulk_load(smem_u32(run + head), src + head, 16u * (uint32_t)n4, full);
    }
    if (lane < head) run[lane] = __ldg(src + lane);
    if (tail + lane < run_len) run[tail + lane] = __ldg(src + tail + lane);
    __syncwarp();
  }
  for (int item = kept1; item < mine1; ++item) {
    const float s = warp_sum(se_sum_slice(p.input + item_at(item), item_len(item), lane));
    if (lane == 0) p.partial[item] = s;
  }
  if (bulk) {
    int ok = 1;
    if (lane == 0) {
      uint32_t spins = 0;
      unsigned long long t0 = 0;
      while (!mbar_try_wait(full, 0u)) {
        if (((++spins) & 0xFF) == 0) {
          const unsigned long long now = globaltimer_ns();
          if (!t0) t0 = now;
          if (now - t0 > p.timeout_ns) {
            ok = 0;
            break;
          }
        }
      }
    }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (ok) ok = mbar_try_wait(full, 0u);        // complete: every lane sees the phase itself
    if (!__all_sync(0xffffffffu, ok) && lane == 0) {
      if (atomicCAS(p.status, (int)DEV_OK, (int)DEV_TIMEOUT_MBAR) == (int)DEV_OK) {
        p.status[1] = 901;
        p.status[2] = (int)blockIdx.x;
      }
      *p.expired = 1;
      abort_flag = 1;
    }
    // four slices' sums at a time: their reductions across the lanes do not depend on one another
    for (int item = mine0; item < kept1; item += 4) {
      float s[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        s[u] = 0.0f;
        if (item + u < kept1) {
          const int at = item_at(item + u) - run_at;
          s[u] = se_sum_kept(run + at, (run_off + at) & 3, item_len(item + u), lane);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < 4; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
      const float mine = lane == 0 ? s[0] : lane == 1 ? s[1] : lane == 2 ? s[2] : s[3];
      if (lane < 4 && item + lane < kept1) p.partial[item + lane] = mine;
    }
  }

  if (!se_barrier(p, &abort_flag, w_red, w_exp, expand_pitch, channel_of(item0), channel_of(item1 - 1))) {
    const unsigned long long t0 = globaltimer_ns();        // copies of a run that was given up may still be on their way: 200 us are ample
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    return;
  }

  // ---- phases 2-4: per group of images the channel means and the reduce GEMV (x * sigmoid x), the gates of this CTA's channels
  //      (expand GEMV, sigmoid), and the add ----
  const int items_per_img = p.channels * p.slices, img_end = (item1 - 1) / items_per_img + 1;
  for (int img = item0 / items_per_img; img < img_end; img += p.group) {
    const int ni = min(p.group, img_end - img);
    const int img0 = img * items_per_img, lo = max(item0, img0), hi = min(item1, img0 + ni * items_per_img);
    se_means_and_reduce(p, img, ni, lo, hi, w_red, pooled_s, gate_in);
    const int c_end = channel_of(hi - 1 - img0) + 1, staged0 = channel_of(item0) - img * p.channels;
    for (int c = channel_of(lo - img0) + (int)threadIdx.x; c < c_end; c += kSeThreads) {
      const int im = c / p.channels;
      const float* in = gate_in + im * kSeMaxReduce;
      const float* row = p.w_expand + (c - im * p.channels) * p.reduce;
      float g = 0.0f, g2 = 0.0f;
      if (p.expand_rows) {
        row = w_exp + (c - staged0) * expand_pitch;
#pragma unroll 8
        for (int j = 0; j < p.reduce; ++j) g = fmaf(in[j], row[j], g);
      } else if (p.reduce % 4 == 0 && (reinterpret_cast<uintptr_t>(p.w_expand) & 15) == 0) {
#pragma unroll 4
        for (int j = 0; j < p.reduce; j += 4) {
          const float4 w = __ldg(reinterpret_cast<const float4*>(row + j));
          g = fmaf(in[j + 1], w.y, fmaf(in[j], w.x, g));
          g2 = fmaf(in[j + 3], w.w, fmaf(in[j + 2], w.z, g2));
        }
      } else {
#pragma unroll 8
        for (int j = 0; j < p.reduce; ++j) g = fmaf(in[j], __ldg(row + j), g);
      }
      pooled_s[c] = se_sigmoid(g + g2);                  // (the group's means have been used)
    }
    __syncthreads();
    int item = max(mine0, lo);
    const int kept_hi = min(kept1, hi);
    if (whole && p.mg_hw && item < kept_hi && ((reinterpret_cast<uintptr_t>(p.input) ^ reinterpret_cast<uintptr_t>(p.out)) & 15) == 0) {
      // small channel images: 16 bytes of the run at a time, whichever channels they belong to (image by image, 49 floats each, a warp
      // took 1.1 k cycles per image)
      const int at = item * p.hw, n = (kept_hi - item) * p.hw;
      const float* src = run + (at - run_at);
      float* dst = p.out + at;
      const float* gate = pooled_s + (item - img0);
      auto gate_at = [&](int i) -> float { return gate[__umulhi((uint32_t)i, p.mg_hw)]; };
      const int head = se_head(dst, n), n4 = (n - head) >> 2, tail = head + 4 * n4;
#pragma unroll 2
      for (int i = lane; i < n4; i += 32) {
        const int e = head + 4 * i;
        const float4 v = *reinterpret_cast<const float4*>(src + e);
        *reinterpret_cast<float4*>(dst + e) = make_float4(v.x + gate_at(e), v.y + gate_at(e + 1), v.z + gate_at(e + 2), v.w + gate_at(e + 3));
      }
      if (lane < head) dst[lane] = src[lane] + gate_at(lane);
      if (tail + lane < n) dst[tail + lane] = src[tail + lane] + gate_at(tail + lane);
      item = kept_hi;
    }
    for (; item < min(mine1, hi); ++item) {
      const int at = item_at(item), len = item_len(item);
      const float g = pooled_s[channel_of(item - img0)];
      se_add_slice(item < kept1 ? run + (at - run_at) : p.input + at, p.out + at, len, g, lane);
    }
    __syncthreads();                                     // the next group's means go over the gates
  }

  se_leave(p);
}

}  // namespace souffle
