// Persistent global-sync megakernel for sm_100a.
//
// One CTA per SM interprets a stage program (stage_program.h).  Dense contractions run on
// tcgen05.mma with fp32 accumulators in tensor memory, operands arrive by TMA into a
// 128B-swizzled shared-memory ring, and the softmax / LayerNorm / GELU epilogues read the
// accumulators straight out of TMEM.  Stages are separated by a bounded grid barrier.
//
// Reference behaviour covered (paths relative to the reference project root):
//   cpp/bert/kernels/fused_sqq_bert.cu:34-2305   whole encoder layer in one cooperative launch
//   cpp/bert/kernels/fused_sqq_bert.cu:2308-3785 attention half (QKV, QK^T, softmax, PV, proj, LN)
//   cpp/bert/kernels/fused_sqq_feedforward.cu:1728-2617 FFN half (FC1+act, FC2+residual, LN)
//   cpp/swin_transformer/kernels/swin_fused_ffn_m256n2048k512_m256n512k2048.cu:9-769 fc1 -> fc2
//   cpp/swin_transformer/kernels/gemm_three_stages.h:8-379 and kernels/gemm_k6.cu:9-339 single GEMMs
//
// Warp roles (384 threads): warp 0 = feeder (a lone lane: grid barrier, activation tiles), warp 1 = MMA issuer and
// TMEM owner, warps 2..9 = epilogue (warp w reads TMEM lanes 32*(w%4) .. +31; two warps share a
// lane quarter and take alternate 32-column chunks) and attention softmax warps, warp 10 = arrivals, L2 prefetch and drops,
// warp 11 = weight tiles and stage records.  All twelve take rows of the LayerNorm stages.
// Every wait (mbarrier, grid barrier) is bounded by a wall-clock deadline; on expiry the CTA
// records a status word, drains and returns, so a fault never leaves the GPU spinning.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "sm100_ptx.cuh"
#include "stage_program.h"

namespace souffle {

constexpr int kThreads = 384;               // registers are handed out per four warps: a block of ten warps is charged for
                                            // twelve, so the last two cost nothing
constexpr int kEpiWarps = 8, kEpiThreads = kEpiWarps * 32;
constexpr int kSpareWarp = 2 + kEpiWarps, kWeightWarp = kSpareWarp + 1;
constexpr int kRingBytes = 196608;          // 192 KiB operand ring (4 x 48 KiB, 3 x 64 KiB or 6 x 32 KiB slots)
constexpr int kCtlBytes = 3072;             // barriers, control words, two stage records, two tiles' bias
constexpr int kVecBytes = 16384;             // per-stage vectors (LayerNorm stages)
constexpr int kStageRow = 64;                // bytes per staged row; the 16-byte pieces of a row are XOR-swizzled (see below)
constexpr int kStageWarp = 32 * kStageRow;   // one epilogue warp's transpose buffer
constexpr int kStageBytes = 8 * kStageWarp;  // 16 KiB
// Layout after the control block: ring | vectors | store staging.  The attention stage with three
// key blocks needs 208 KiB and simply runs over all three regions (it uses neither of the other two); the boxes of a GEMM stage's
// TMA stores take the last two together.
constexpr int kSmemBytes = kCtlBytes + kRingBytes + kVecBytes + kStageBytes;
constexpr int kMaxSlots = 8;
constexpr uint32_t kTmemCols = 512;
constexpr int kATileBytes = 128 * 64 * 2;   // 128 rows x 64 halves
constexpr int kAccStride = 256;             // TMEM columns between the two accumulator buffers
constexpr int kUnitBytes = 64 * 64 * 2;     // the unit matrix that adds residuals (of a pair: each CTA has half)
constexpr int kOCol = 384;                  // TMEM column of the attention output accumulator

struct MegaParams {
  const Stage* stages;        // plan-owned stage list, or null to use the inline stages
  int n_stages;
  const CUtensorMap* maps;    // plan-owned tensor maps (indices >= 0)
  int n_maps;
  const void* x;
  void* y;
  const int* lens;
  unsigned* sync;       // [0] arrival count, [1] generation used by this launch
  unsigned* sync_next;  // the pair the next launch will use; cleared by this launch
  unsigned* epoch;      // plan-owned counter (see launch_step) whose launch numbers tag EPI_LN statistics, or null
  int* status;        // [0] code, [1] where, [2] cta
  int* expired;       // host memory or null: set by a CTA that gave up on a wait
  unsigned long long timeout_ns;
  int max_slots;      // experiment knob: cap on operand ring slots, 0 = as many as fit
  int skip_arrival;   // test hook: CTA (low 16 bits - 1) leaves without arriving after stage (high 16 bits); 0 = off; -1: see kSmemAlign
  long long* prof;    // optional [n_stages][grid][8]: clock64 at stage start, work done, barrier left, then GEMM
                      // role cycles: MMA waiting for operands, MMA waiting for a free accumulator, producer
                      // waiting for a free slot, epilogue waiting for an accumulator, epilogue busy
};

// Everything a launch needs, passed in parameter space: per-call tensor maps (negative map
// indices: -1 -> call_maps[0], -2 -> call_maps[1], ...), up to two inline stages for the
// plan-less entry points, and the pointers above.
constexpr int kCallMaps = 6;
struct CallArgs {
  CUtensorMap call_maps[kCallMaps];
  Stage inline_stages[3];
  MegaParams p;
};
__device__ __forceinline__ const CUtensorMap* map_ptr(const CallArgs& a, int idx) {
  return idx < 0 ? &a.call_maps[-idx - 1] : a.p.maps + idx;
}

constexpr uint32_t kSmemAlign = 1024;        // of swizzled tiles: descriptors and copies take it for granted, so the prologue looks
extern __shared__ __align__(kSmemAlign) uint8_t smem_raw[];

struct __align__(8) SmemCtl {
  uint64_t full[kMaxSlots];
  uint64_t empty[kMaxSlots];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint64_t qk_full, qk_empty, v_full, v_empty, s_full, p_full, o_full;   // attention, pipeline 0
  uint64_t attn1[7];                                                     // attention, pipeline 1 (same order)
  uint64_t o_empty[2];                                                   // pair attention: output accumulator read out
  uint64_t ln_full[4], ln_empty[4];
  uint32_t tmem_base;
  int abort;
  int leave[2];                     // a wait has run out: all warps leave the stage loop together
  uint32_t arrived;                 // stages whose arrival this CTA has sent
  uint32_t go;                      // stages that may start, as published by the feeder (publish_go / wait_go / stage_go)
  uint32_t epoch;                   // this launch's number x kLaunchSteps, see RowStat
  WaitCtl wait;                     // here and not on the stack: see RoleState
  alignas(16) float bias[2][256];   // of this tile's and the next tile's columns
  alignas(16) Stage stage[2];       // records of this stage and the next, by the parity of their ordinals
};
static_assert(sizeof(SmemCtl) <= kCtlBytes, "control block too large");

// Per-thread view of the pipelines; identical arithmetic in every role keeps them in step.  Out-of-line stage functions take and
// return it packed into one register: every grid barrier's acquire empties L1, so a word on the stack costs a round trip to L2.
struct RoleState {
  uint32_t slot = 0;       // next ring slot
  uint32_t slot_bits = 0;  // phase bit per ring slot
  uint32_t acc_bits = 0;   // bits 0, 1: phase bit per accumulator buffer; bit 2: next accumulator buffer
  uint32_t attn_bit = 0;   // phase bit of the attention barriers, pipeline 0
  uint32_t attn_bit1 = 0;  // phase bit of the attention barriers, pipeline 1
  uint32_t ln_bits = 0;    // phase bit per LayerNorm batch buffer
  uint32_t o_bits = 0;     // pair attention: phase bit of the o_empty barrier of each pipeline (MMA lane)
  __device__ __forceinline__ uint32_t pack() const {
    return slot | (slot_bits << 4) | (acc_bits << 12) | (attn_bit << 15) | (attn_bit1 << 16) | (ln_bits << 17) | (o_bits << 21);
  }
  static __device__ __forceinline__ RoleState unpack(uint32_t w) {
    RoleState r;
    r.slot = w & 15u; r.slot_bits = (w >> 4) & 255u; r.acc_bits = (w >> 12) & 7u; r.attn_bit = (w >> 15) & 1u;
    r.attn_bit1 = (w >> 16) & 1u; r.ln_bits = (w >> 17) & 15u; r.o_bits = (w >> 21) & 3u;
    return r;
  }
};
static_assert(kMaxSlots <= 8, "a slot index and a phase bit per slot are packed into four and eight bits");

// SM clock for the stage-level stamps of the in-kernel profile.  The memory clobber keeps the read where it is
// written: a plain clock64() may be scheduled above a preceding barrier, which charges a stage's work to the wait
// that follows it.
__device__ __forceinline__ long long clock_now() {
  long long t;
  asm volatile("mov.u64 %0, %%clock64;" : "=l"(t) :: "memory");
  return t;
}

__device__ __forceinline__ const void* sel_ptr(int sel, const void* plan, const MegaParams& p) {
  return sel == PTR_CALL_X ? p.x : (sel == PTR_CALL_Y ? (const void*)p.y : plan);
}

// ------------------------------------------------------------------------------------
// grid barrier: one monotonic arrival counter per launch, bounded spin
//
// Its two halves lie with different warps, so that a stage's set-up runs while the CTA waits.  At the end of a stage all
// threads of a CTA meet once (the end of the stage loop); a lane of a spare warp then adds the CTA's arrival to the counter,
// whose release covers every thread's writes and takes ~1 k cycles.  Meanwhile every warp has gone on to the next stage: the
// epilogue warps stage the bias, the row warps load gamma and beta, and the weight warp requests the first weight tiles, none of
// which the stage before has written.  Only the feeder (the lone lane of warp 0 that issues the stage's copies) looks at the
// counter (grid_wait), and what it does next is issue the stage's first activation copy.  All other warps of a GEMM or
// attention stage are behind the data the feeder asks for; the warps of a LayerNorm stage, which read what earlier stages wrote
// by themselves, all get the feeder's one verdict (stage_go).
// ------------------------------------------------------------------------------------
// The polls in front stand in straight line (a loop's way out costs some 150 cycles, see mbar_wait_hot); a CTA that waits
// longer than they last goes on out of line.
__device__ __noinline__ bool grid_wait_loop(const unsigned* count, unsigned target, const WaitCtl& ctl, int where) {
  uint32_t spins = 0;
  while (ld_acquire_u32(count) < target) {
    if (((++spins) & 0x3F) == 0) {
      if (*ctl.abort_smem) return false;
      if (globaltimer_ns() > ctl.deadline_ns) {
        record_timeout(ctl, DEV_TIMEOUT_GRID, where);
        return false;
      }
    }
  }
  return true;
}
// One thread: waits until every CTA has finished the stage before `st`.  Its acquire and the proxy fence order the other CTAs'
// writes before this thread's TMA and bulk copies.  False: the wait has run out.
__device__ __forceinline__ bool grid_wait(const MegaParams& p, const WaitCtl& ctl, const Stage& st) {
  bool there = st.ordinal == 0;
  if (!there) {
    // The counter only grows during a launch: the barrier in front of `st` is passed once every CTA has added 1 for each stage
    // that runs before it.  (The launch that runs next clears the other counter, see the prologue.)
    const unsigned* count = p.sync;
    const unsigned target = (unsigned)st.ordinal * gridDim.x;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (!there) there = ld_acquire_u32(count) >= target;
    if (!there) there = grid_wait_loop(count, target, ctl, st.prev);
    fence_proxy_async_global();
  }
  if (p.prof) {
    const long long now = clock_now();
    p.prof[((size_t)st.position * gridDim.x + blockIdx.x) * kProfSlots + 0] = now;
    if (st.ordinal > 0) p.prof[((size_t)st.prev * gridDim.x + blockIdx.x) * kProfSlots + 2] = now;
  }
  return there;
}
// Bounded wait for a word of this CTA's shared memory that only grows.
__device__ __noinline__ bool wait_word_loop(uint32_t word, uint32_t want, const WaitCtl& ctl, int where) {
  uint32_t spins = 0;
  while (ld_acquire_cta_shared_u32(word) < want) {
    if (((++spins) & 0xFF) == 0) {
      if (*ctl.abort_smem) return false;
      if (globaltimer_ns() > ctl.deadline_ns + kWaitGraceNs) {
        record_timeout(ctl, DEV_TIMEOUT_FLAG, where);
        return false;
      }
    }
  }
  return true;
}
__device__ __forceinline__ bool wait_word(uint32_t word, uint32_t want, const WaitCtl& ctl, int where) {
  return ld_acquire_cta_shared_u32(word) >= want || wait_word_loop(word, want, ctl, where);
}
// One thread: this CTA's arrival for the stage before the one of ordinal si is on its way.  Copies issued before that would delay it: its release waits for
// them too.
__device__ __forceinline__ bool wait_arrived(SmemCtl& cs, int si, const WaitCtl& ctl) { return wait_word(smem_u32(&cs.arrived), (uint32_t)si, ctl, 700); }
// The feeder's word that stage si may start.
__device__ __forceinline__ void publish_go(SmemCtl& cs, int si) { st_release_cta_shared_u32(smem_u32(&cs.go), (uint32_t)si + 1u); }
// For a warp whose part the stage's result does not depend on (what it skips when it gives up is a drop from L2).
__device__ __forceinline__ bool wait_go(SmemCtl& cs, int si, const WaitCtl& ctl) {
  return __all_sync(0xffffffffu, wait_word(smem_u32(&cs.go), (uint32_t)si + 1u, ctl, 701));
}
// All threads of the CTA: true if stage si may start.  The feeder alone looks at the clock, and its verdict reaches every warp
// through a barrier: warps that judged the limit one by one could part ways when it passes, and those that went on would miss
// the others' rows or wait for them in a barrier.
constexpr int kGoBarrier = 15;
__device__ __forceinline__ bool stage_go(const MegaParams& p, SmemCtl& cs, const Stage& st, const WaitCtl& ctl, int warp, int lane) {
  if (warp == 0) {
    if (lane == 0 && grid_wait(p, ctl, st)) publish_go(cs, st.ordinal);
    __syncwarp();
  }
  named_barrier_sync(kGoBarrier, kThreads);
  return ld_acquire_cta_shared_u32(smem_u32(&cs.go)) > (uint32_t)st.ordinal;      // not written again before all have met at the stage's end
}

// The warp's index as a value the compiler knows to be the same in all its lanes (see elect_one).
__device__ __forceinline__ int uniform_warp(int warp) { return __shfl_sync(0xffffffffu, warp, 0); }

// ------------------------------------------------------------------------------------
// GEMM stage
// ------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t fast_div(uint32_t n, uint32_t d, uint32_t mg) {
  return d == 1u ? n : __umulhi(n, mg);
}

struct GemmGeom {
  int tiles_n, splitk, items, kchunks, kper, bn, bm, nh, slot_bytes, nslots;
};
__device__ __forceinline__ GemmGeom gemm_geom(const Stage& st) {
  GemmGeom g;
  g.bn = st.bn;
  g.bm = st.bm;
  g.nh = st.bm >> 7;                       // 128-row halves per tile, each with its own accumulator
  g.tiles_n = st.tiles_n;
  g.splitk = st.splitk;
  g.items = st.items;
  g.kchunks = st.kchunks;
  g.kper = st.kper;
  g.slot_bytes = st.slot_bytes;
  g.nslots = st.nslots;
  return g;
}
// work item -> (m tile, n tile, k split)
__device__ __forceinline__ void gemm_item(const Stage& st, int item, int& mt, int& nt, int& ks) {
  const uint32_t q = fast_div((uint32_t)item, (uint32_t)st.splitk, st.mg_splitk);
  ks = item - (int)q * st.splitk;
  const uint32_t m = fast_div(q, (uint32_t)st.tiles_n, st.mg_tiles_n);
  nt = (int)q - (int)m * st.tiles_n;
  mt = (int)m;
}

// Epilogue parameters of a stage, copied into registers once (the stage record itself lives in
// shared memory and would otherwise be re-read around every asm statement).
struct EpiCtx {
  int epi, act, M, N, ldo;
  __half* out;
  float* partial;
  const CUtensorMap* tm_out;   // store map
  bool prof;
};
constexpr uint32_t kNoRow = 0xFFFFFFFFu;      // "this row is outside the matrix"

// A thread that owns one row of a 32-row block holds 64 bytes of that row.  Written straight to global
// memory, one store instruction would touch 32 different lines with 16 bytes each.  Going through the
// warp's staging buffer turns that around: afterwards lanes 4j..4j+3 hold the 64 bytes of row j (+8, +16,
// +24), so every store instruction writes eight rows with 64 contiguous bytes each.
// `rowptr[i]` is the global byte address of row (8*i + lane/4) at this chunk's first column, or null.
__device__ __forceinline__ void staged_store_64B(uint8_t* sbuf, const uint32_t (&w)[16], uint8_t* const (&rowptr)[4], int lane) {
  // Piece i (16 bytes) of row r sits at r * 64 + ((i ^ (r >> 1)) & 3) * 16: the eight lanes of a quarter warp then hit
  // distinct banks both when every lane writes piece i of its own row and when four lanes read one row each of two
  // neighbouring rows (padded rows avoided the conflicts of the writes only: two thirds of the reads were replays).
  const int sw_w = (lane >> 1) & 3;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<uint4*>(sbuf + lane * kStageRow + ((i ^ sw_w) << 4)) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  __syncwarp();
  uint4 v[4];                    // all four loads are issued before the first store waits for its data
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = 8 * i + (lane >> 2);
    v[i] = *reinterpret_cast<const uint4*>(sbuf + r * kStageRow + ((((lane & 3) ^ (r >> 1)) & 3) << 4));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (rowptr[i]) *reinterpret_cast<uint4*>(rowptr[i] + (lane & 3) * 16) = v[i];
  __syncwarp();
}

// Output addressing is split into a row part, computed once per tile, and a column part, computed once
// per chunk; both are element offsets that fit 32 bits (the host rejects larger buffers).
// Row part: offset of matrix row `row` in the stage's output (kNoRow past the end).
__device__ __forceinline__ uint32_t epi_row_offset(const Stage& st, const EpiCtx& e, int row, int ks) {
  if (row >= e.M) return kNoRow;
  if (e.epi == EPI_PARTIAL) return (uint32_t)(ks * e.M + row) * (uint32_t)e.N;
  if (e.epi == EPI_QKV) {
    // [3][B][heads][S][d]: row -> (sequence, token)
    const uint32_t b = fast_div((uint32_t)row, (uint32_t)st.seq, st.mg_seq), sq = (uint32_t)row - b * (uint32_t)st.seq;
    return (b * (uint32_t)(st.heads * st.seq) + sq) * (uint32_t)st.head_dim;
  }
  return (uint32_t)row * (uint32_t)e.ldo;
}
// Column part: offset of column `col` (a multiple of 16; a chunk never straddles a head or a q/k/v plane).
__device__ __forceinline__ uint32_t epi_col_offset(const Stage& st, const EpiCtx& e, int col) {
  if (e.epi == EPI_QKV) {
    const uint32_t g = fast_div((uint32_t)col, (uint32_t)st.head_dim, st.mg_head_dim), dd = (uint32_t)col - g * (uint32_t)st.head_dim;
    const uint32_t which = fast_div(g, (uint32_t)st.heads, st.mg_heads), hh = g - which * (uint32_t)st.heads;
    const uint32_t head_plane = (uint32_t)(st.seq * st.head_dim);
    return (which * (uint32_t)(st.batch * st.heads) + hh) * head_plane + dd;
  }
  return (uint32_t)col;
}

// Bias, activation and conversion of a 32-column chunk: r[i] = column i of this thread's own row, `bias` = the chunk's in shared
// memory.  Written phase by phase over the whole chunk -- every loop is 16 independent operations -- instead of element by
// element: an epilogue warp has at most one other warp on its scheduler, so a dependent chain per element (add, pack, seven GELU
// steps) runs at one instruction per ALU latency.
__device__ __forceinline__ void epilogue_values32(const EpiCtx& e, const uint32_t (&r)[32], const float* bias, uint32_t (&w)[16]) {
  const float4* b4 = reinterpret_cast<const float4*>(bias);     // fp32: no conversions here
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float4 b = b4[i];
    w[2 * i] = pack_h2_sum(r[4 * i], r[4 * i + 1], b.x, b.y);
    w[2 * i + 1] = pack_h2_sum(r[4 * i + 2], r[4 * i + 3], b.z, b.w);
  }
  if (e.act == ACT_RELU) {
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = relu_h2(w[i]);
  } else if (e.act == ACT_GELU) {
    gelu_tanh_h2x16(w);                                          // on fp16 pairs
  }
}

// Stores through the TMA: a lane writes 64 bytes of its row (32 fp16 or 16 fp32 columns) into a box of 32 rows (the layout of a
// 64B-swizzled box), one lane hands the box to the copy engine.  A warp has kRingBoxes boxes inside the operand ring for the CTA's
// last tile, whose operands have all been consumed, and two beside the ring before that, used round robin; a box is
// written again once the copy issued from it has read it, for which the issuing lane waits right behind the next copy.
// With fp16 outputs going through shared memory twice (written by rows, read back and stored by eight rows of 64 bytes), addresses
// per chunk and the stage's whole bias vector read from there, a chunk of 32 columns took ~1.9 k cycles of its warp, now ~1.0 k
// (without GELU 0.9 k): 7 x 112 QKV 13.5 k -> 12.7 k cycles, FC1 17.0 k -> 15.5 k; 64 x 128 FC1 61.9 k -> 59.6 k, on pairs 56.9 k -> 53.2 k.
constexpr int kRingBoxes = 12;
struct StoreBoxes {
  uint8_t* base;
  int box, n;
};
template <class Issue>
__device__ __forceinline__ void store_box(StoreBoxes& sb, const uint32_t* w, int lane, Issue issue) {
  uint8_t* buf = sb.base + sb.box * kStageWarp;
  const int sw = (lane >> 1) & 3;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<uint4*>(buf + lane * kStageRow + ((i ^ sw) << 4)) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  fence_proxy_async_smem();
  __syncwarp();
  if (elect_one()) {
    issue(smem_u32(buf));
    bulk_commit_group();
    if (sb.n == 2) bulk_wait_group_read<1>(); else bulk_wait_group_read<kRingBoxes - 1>();
  }
  __syncwarp();
  sb.box = sb.box + 1 == sb.n ? 0 : sb.box + 1;
}

// 16-column tail chunk (tile widths that are an odd multiple of 16): direct stores.
__device__ __forceinline__ void epilogue_chunk16(const Stage& st, const EpiCtx& e, const uint32_t (&r)[16], const float* bias, uint32_t own, int col) {
  if (own == kNoRow) return;
  if (e.epi == EPI_PARTIAL) {
    float4* dst = reinterpret_cast<float4*>(e.partial + own + col);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      dst[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]),
                           __uint_as_float(r[4 * i + 3]));
    return;
  }
  float v[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]) + bias[i];
  if (e.act == ACT_RELU) {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.0f);
  } else if (e.act == ACT_GELU) {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = gelu_tanh(v[i]);
  }
  uint4* d4 = reinterpret_cast<uint4*>(e.out + (own + epi_col_offset(st, e, col)));
  d4[0] = make_uint4(pack_h2(v[0], v[1]), pack_h2(v[2], v[3]), pack_h2(v[4], v[5]), pack_h2(v[6], v[7]));
  d4[1] = make_uint4(pack_h2(v[8], v[9]), pack_h2(v[10], v[11]), pack_h2(v[12], v[13]), pack_h2(v[14], v[15]));
}

// Rows of Swin blocks change their order where a block's windows lie differently from those before: a LayerNorm stage writes row `row` to
// the place that its token has in the order it leaves in (Stage::tok_grid), so that all products and the attention stage have rows that
// are adjacent.  (When the products permuted, an epilogue took 1.9 k cycles per 32 columns, and windows of 49 tokens took 64 rows of
// the projection.)  The divisors are host constants, so a quotient is one multiply-high.
__device__ __forceinline__ int ln_out_row(const Stage& st, int row) {
  const int R = st.tok_grid;
  if (!R) return row;
  const int win = st.win, nwr = st.nwr, n_tok = win * win;
  int img, ty, tx;
  if (st.shift < 0) {                      // rows come in the order of the tokens
    img = st.mg_seq2 ? (int)__umulhi((uint32_t)row, st.mg_seq2) : row / (R * R);
    const int t = row - img * R * R;
    ty = (int)fast_div((uint32_t)t, (uint32_t)R, st.mg_seq);
    tx = t - ty * R;
  } else {
    const int wg = (int)fast_div((uint32_t)row, (uint32_t)n_tok, st.mg_tok), pos = row - wg * n_tok;
    img = (int)fast_div((uint32_t)wg, (uint32_t)(nwr * nwr), st.mg_nwr2);
    const int w = wg - img * nwr * nwr, wy = (int)fast_div((uint32_t)w, (uint32_t)nwr, st.mg_nwr);
    const int py = (int)fast_div((uint32_t)pos, (uint32_t)win, st.mg_win);
    ty = wy * win + py + st.shift;
    tx = (w - wy * nwr) * win + (pos - py * win) + st.shift;
    if (ty >= R) ty -= R;
    if (tx >= R) tx -= R;
  }
  if (st.to_shift < 0) return (img * R + ty) * R + tx;
  int sy = ty - st.to_shift, sx = tx - st.to_shift;
  if (sy < 0) sy += R;
  if (sx < 0) sx += R;
  const int wy = (int)fast_div((uint32_t)sy, (uint32_t)win, st.mg_win), wx = (int)fast_div((uint32_t)sx, (uint32_t)win, st.mg_win);
  return ((img * nwr + wy) * nwr + wx) * n_tok + (sy - wy * win) * win + (sx - wx * win);
}

// LayerNorm in the epilogue of a product whose K is not cut: out = LayerNorm(acc + bias + residual) without a plane in memory and
// without a stage of its own.  A row's columns lie in tiles_n tiles of as many CTAs (or pairs), all of which are running or have run:
// items are dealt out in order, every CTA takes its own in order, and a CTA has at most one tile of a row block (the host checks that
// tiles_n is not larger than the grid), so the tile of the lowest number that has not been published never waits for another.
//   0. The residual is added by the tensor core: behind the last step along K come steps of 64 columns of it times a unit matrix
//      (exact products, fp32 sums).  Read by the epilogue warps, 16 bytes of a row at a time, it cost 1.5 k cycles per 32 columns.
//   1. A thread adds the bias to its row's columns, puts the sum back into tensor memory and forms (mean, squared deviations
//      from it); sets of columns are merged as in ln_shared_rows.
//   2. The tile's pair is published as a RowStat per row: value and tag in one 64-bit word, so neither a fence in front of the store
//      nor a flag behind it is needed, and who finds the tags has the values.
//   3. A thread reads the pairs of all of its row's tiles (bounded), normalises the sums and stores fp16 rows as boxes.
// Out of line: its registers are not charged to the other stages.  Few arguments: they have to live beside the caller's values.
// `acc_bits`: see RoleState; bit 31: the stage's record is the second one.
// kSwin: the sum leaves as well, rounded to fp16, which is then what gets normalised (or leaves alone: eps < 0), and rows may leave in
// another order; such stores are plain ones.
template <bool kPair, bool kSwin>
__device__ __forceinline__ uint32_t gemm_ln_epilogue_of(const CallArgs& ca, uint32_t acc_bits) {
  SmemCtl& cs = *reinterpret_cast<SmemCtl*>(smem_raw);
  const Stage& st = cs.stage[acc_bits >> 31];
  acc_bits &= 7u;
  const WaitCtl& ctl = cs.wait;
  uint8_t* boxes = smem_raw + kCtlBytes + kRingBytes;
  const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
  const MegaParams& p = ca.p;
  const int q = epi_quarter(warp), cpar = epi_part(warp), my_col = (int)threadIdx.x - 64;
  const int bn = st.bn, chunks = bn >> 5, tiles_n = st.tiles_n, nh = kPair ? 1 : st.bm >> 7, M = st.M;
  const uint32_t rank = kPair ? cluster_cta_rank() : 0u;
  const int first_item = kPair ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, item_step = kPair ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const uint32_t tfull0 = smem_u32(&cs.tmem_full[0]), tempty0 = smem_u32(&cs.tmem_empty[0]);
  const uint32_t tmem = cs.tmem_base + ((uint32_t)(q * 32) << 16);
  const CUtensorMap* tm_out = map_ptr(ca, st.tm_out);
  const bool sum_only = kSwin && st.eps < 0.0f;
  // plain stores: offset of output row row0 + lane; a lane's rows of the staged pieces are other lanes' (see staged_store_64B)
  auto out_row = [&](int row0) -> uint32_t { return row0 + lane < M ? (uint32_t)ln_out_row(st, row0 + lane) * (uint32_t)st.ldo : kNoRow; };
  auto store_rows = [&](uint8_t* sbuf, __half* to, uint32_t own, int col, const uint32_t (&w)[16]) {
    uint32_t so[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) so[i] = __shfl_sync(0xffffffffu, own, 8 * i + (lane >> 2));
    uint8_t* rowptr[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) rowptr[i] = so[i] != kNoRow ? reinterpret_cast<uint8_t*>(to + (so[i] + (uint32_t)col)) : nullptr;
    staged_store_64B(sbuf, w, rowptr, lane);
  };
  const uint32_t tag = cs.epoch | st.ordinal;
  const float inv_n = 1.0f / (float)st.N;
  const bool prof = p.prof != nullptr, affine = st.gamma != nullptr;
  float* bias_s = cs.bias[0];
  __half* gamma_s = reinterpret_cast<__half*>(cs.bias[1]);          // gamma of the tile's columns, then beta
  // Statistics that part 1 of these rows hands to part 0, in part 1's own second box: its copies have left it before the tile begins, and
  // the next ones go into it once all tiles of the row have been published, which for this one part 0 does with what it has read here
  // (plain stores pass through the first box).
  float2* other = reinterpret_cast<float2*>(boxes + ln_stats_box(q) * kStageWarp);
  StoreBoxes sb;
  sb.base = boxes + epi_box(warp) * kStageWarp;
  sb.box = 0;
  sb.n = 2;
  bool ok = true;            // a warp that has given up goes through the remaining tiles, whose barriers the others wait in
#pragma unroll 1
  for (int item = first_item; item < st.items; item += item_step) {
    const int mt = (int)fast_div((uint32_t)item, (uint32_t)tiles_n, st.mg_tiles_n), nt = item - mt * tiles_n;
    const int colbase = nt * bn;
    float b = 0.0f;
    __half gm = __ushort_as_half(0), bt = gm;
    if (my_col < bn) {
      if (st.bias) b = __half2float(__ldg(reinterpret_cast<const __half*>(st.bias) + colbase + my_col));
      if (affine) {
        gm = __ldg(reinterpret_cast<const __half*>(st.gamma) + colbase + my_col);
        bt = __ldg(reinterpret_cast<const __half*>(st.beta) + colbase + my_col);
      }
    }
    named_barrier_sync(1, kEpiThreads);                              // the tile before has been read
    bias_s[my_col] = b;
    gamma_s[my_col] = gm;
    gamma_s[256 + my_col] = bt;
    if (elect_one()) bulk_wait_group_read<0>();
    named_barrier_sync(1, kEpiThreads);
    if (item + item_step >= st.items) {                              // boxes inside the operand ring, see StoreBoxes
      sb.base = boxes - kRingBytes + (warp - 2) * kRingBoxes * kStageWarp;
      sb.box = 0;
      sb.n = kRingBoxes;
    }
    const uint32_t acc0 = nh == 2 ? 0u : acc_bits >> 2;
#pragma unroll 1
    for (int h = 0; h < nh; ++h) {
      const uint32_t acc = acc0 + (uint32_t)h, t0 = tmem + acc * kAccStride;
      const int row0 = mt * st.bm + (kPair ? (int)rank : h) * 128 + q * 32;
      ok = ok && mbar_wait_warp(tfull0 + 8 * acc, (acc_bits >> acc) & 1u, ctl, 400 + (int)acc, lane);
      tc_fence_after_sync();
      if (prof && item == first_item && h == 0 && warp == 2 && lane == 0)
        p.prof[((size_t)st.position * gridDim.x + blockIdx.x) * kProfSlots + 14] = clock64();
      float mean = 0.0f, dev = 0.0f, sets = 0.0f;                    // of `sets` chunks of 32 columns
      const uint32_t own = kSwin ? out_row(row0) : 0u;
#pragma unroll 1
      for (int c = cpar; c < chunks; c += 2) {
        uint32_t r[32];
        tmem_ld32(t0 + c * 32, r);
        tmem_ld_wait(r);
        float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        const float4* b4 = reinterpret_cast<const float4*>(bias_s + c * 32);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 bb = b4[i];
          const float z0 = __uint_as_float(r[4 * i]) + bb.x, z1 = __uint_as_float(r[4 * i + 1]) + bb.y;
          const float z2 = __uint_as_float(r[4 * i + 2]) + bb.z, z3 = __uint_as_float(r[4 * i + 3]) + bb.w;
          if constexpr (!kSwin) { sum[0] += z0; sum[1] += z1; sum[2] += z2; sum[3] += z3; }
          r[4 * i] = __float_as_uint(z0); r[4 * i + 1] = __float_as_uint(z1);
          r[4 * i + 2] = __float_as_uint(z2); r[4 * i + 3] = __float_as_uint(z3);
        }
        if constexpr (kSwin) {
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = pack_h2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
          if (ok) store_rows(sb.base, reinterpret_cast<__half*>(sum_only ? const_cast<void*>(sel_ptr(st.out_sel, st.out, p)) : st.sum_out), own, colbase + c * 32, w);
          if (sum_only) continue;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
            r[2 * i] = __float_as_uint(f.x);
            r[2 * i + 1] = __float_as_uint(f.y);
            sum[i & 3] += f.x + f.y;
          }
        }
        tmem_st32(t0 + c * 32, r);
        const float cm = ((sum[0] + sum[1]) + (sum[2] + sum[3])) * (1.0f / 32.0f);
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float d = __uint_as_float(r[i]) - cm;
          v[i & 3] = fmaf(d, d, v[i & 3]);
        }
        const float w = 1.0f / (sets + 1.0f), d = cm - mean;
        dev += ((v[0] + v[1]) + (v[2] + v[3])) + d * d * (32.0f * sets * w);
        mean = fmaf(d, w, mean);
        sets += 1.0f;
      }
      if (sum_only) continue;
      tmem_st_wait();
      if (chunks > 1) {
        if (cpar == 1) other[h * 32 + lane] = make_float2(mean, dev);
        named_barrier_sync(4 + q, 64);
        if (cpar == 0) {
          const float2 o = other[h * 32 + lane];
          const float os = (float)(chunks >> 1), w = os / (sets + os), d = o.x - mean;
          dev += o.y + d * d * (32.0f * sets * w);
          mean = fmaf(d, w, mean);
        }
      }
      if (cpar == 0 && ok)
        st_relaxed_2x64(st.stats + ((size_t)(row0 >> 5) * tiles_n + nt) * 32 + lane, (uint64_t)__float_as_uint(mean) | ((uint64_t)tag << 32),
                        (uint64_t)__float_as_uint(dev) | ((uint64_t)tag << 32));
    }
    // (one half's statistics have been read before they are published, and so before part 1 gets past its wait for them; with two halves
    // the second one's may not have been)
    if (nh == 2) named_barrier_sync(4 + q, 64);
#pragma unroll 1
    for (int h = 0; h < nh; ++h) {
      const uint32_t acc = acc0 + (uint32_t)h, t0 = tmem + acc * kAccStride;
      const int row0 = mt * st.bm + (kPair ? (int)rank : h) * 128 + q * 32;
      float mean = 0.0f, dev = 0.0f;
      const uint32_t own = kSwin && st.tok_grid ? out_row(row0) : 0u;
      const RowStat* from = st.stats + (size_t)(row0 >> 5) * tiles_n * 32 + lane;
      uint32_t spins = 0;
#pragma unroll 1
      for (int s0 = 0; ok && !sum_only && s0 < tiles_n;) {
        constexpr int kG = kSwin ? 2 : 4;                            // tiles whose pairs are on their way at once (more would spill)
        uint64_t a[kG], v[kG];
        bool there = true;
#pragma unroll
        for (int i = 0; i < kG; ++i)
          if (s0 + i < tiles_n) ld_relaxed_2x64(from + (s0 + i) * 32, a[i], v[i]);
#pragma unroll
        for (int i = 0; i < kG; ++i)
          if (s0 + i < tiles_n) there = there && (uint32_t)(a[i] >> 32) == tag && (uint32_t)(v[i] >> 32) == tag;
        if (!__all_sync(0xffffffffu, there)) {
          if (((++spins) & 0x3F) == 0) {
            int give_up = 0;
            if (lane == 0) {
              give_up = *ctl.abort_smem;
              if (!give_up && globaltimer_ns() > ctl.deadline_ns + kWaitGraceNs) {
                record_timeout(ctl, DEV_TIMEOUT_FLAG, 750);
                give_up = 1;
              }
            }
            if (__shfl_sync(0xffffffffu, give_up, 0)) ok = false;
          }
          continue;
        }
        // sets of bn columns each: those of this round among themselves, then with the rounds before
        const int n = tiles_n - s0 < kG ? tiles_n - s0 : kG;
        float m = 0.0f, e = 0.0f, sq = 0.0f;
#pragma unroll
        for (int i = 0; i < kG; ++i) m += i < n ? __uint_as_float((uint32_t)a[i]) : 0.0f;
        m *= 1.0f / (float)n;
#pragma unroll
        for (int i = 0; i < kG; ++i)
          if (i < n) {
            const float d = __uint_as_float((uint32_t)a[i]) - m;
            e += __uint_as_float((uint32_t)v[i]);
            sq = fmaf(d, d, sq);
          }
        const float w = (float)n / (float)(s0 + n), d = m - mean;
        dev += e + (float)bn * (sq + d * d * ((float)s0 * w));
        mean = fmaf(d, w, mean);
        s0 += kG;
      }
      const float rstd = rsqrtf(dev * inv_n + st.eps), nm = -mean * rstd;
#pragma unroll 1
      for (int c = cpar; ok && !sum_only && c < chunks; c += 2) {
        uint32_t r[32], w[16];
        tmem_ld32(t0 + c * 32, r);
        tmem_ld_wait(r);
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = pack_h2(fmaf(__uint_as_float(r[2 * i]), rstd, nm), fmaf(__uint_as_float(r[2 * i + 1]), rstd, nm));
        if (affine) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 ug = *(reinterpret_cast<const uint4*>(gamma_s + c * 32) + i), ub = *(reinterpret_cast<const uint4*>(gamma_s + 256 + c * 32) + i);
            const uint32_t g4[4] = {ug.x, ug.y, ug.z, ug.w}, b4[4] = {ub.x, ub.y, ub.z, ub.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const __half2 y = __hfma2(*reinterpret_cast<const __half2*>(&w[4 * i + j]), *reinterpret_cast<const __half2*>(&g4[j]),
                                        *reinterpret_cast<const __half2*>(&b4[j]));
              w[4 * i + j] = *reinterpret_cast<const uint32_t*>(&y);
            }
          }
        }
        if (kSwin && st.tok_grid) {
          store_rows(sb.base, reinterpret_cast<__half*>(st.out), own, colbase + c * 32, w);
        } else {
          store_box(sb, w, lane, [&](uint32_t buf) {
            if (row0 < M) tma_store_2d(tm_out, buf, colbase + c * 32, row0);
          });
        }
      }
      tc_fence_before_sync();
      if constexpr (kPair) {
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(map_shared_rank(tempty0 + 8 * acc, 0));
      } else {
        mbar_arrive(tempty0 + 8 * acc);
      }
      acc_bits ^= 1u << acc;
    }
    if (nh == 1) acc_bits ^= 4u;
  }
  if (elect_one()) {                      // the stores are complete before the CTA reports the stage done
    bulk_wait_group_all();
    fence_proxy_async_global();
  }
  __syncwarp();
  if (prof && warp == 2 && lane == 0) p.prof[((size_t)st.position * gridDim.x + blockIdx.x) * kProfSlots + 15] = clock64();
  return acc_bits;
}

// The Swin build's, with sums and reordered rows.
__device__ __noinline__ uint32_t gemm_swin_ln(const CallArgs& ca, uint32_t acc_bits) { return gemm_ln_epilogue_of<false, true>(ca, acc_bits); }
template <bool kPair>
__device__ __noinline__ uint32_t gemm_ln_epilogue(const CallArgs& ca, uint32_t acc_bits) { return gemm_ln_epilogue_of<kPair, false>(ca, acc_bits); }

// Tiles are bm x bn with bm = 128 (two accumulators used alternately, so the epilogue of one tile
// overlaps the main loop of the next) or bm = 256 (two 128-row halves share every B tile, which
// halves the B traffic per FLOP; each half has its own accumulator and hand-shake).
// kPair: the two CTAs of a cluster work on one 256 x bn tile with pair MMAs (see sm100_ptx.cuh).  CTA r loads rows
// 128 r .. 128 r + 127 of the A tile and rows bn/2 * r .. of the B tile (the weights' output columns) into its own
// shared memory -- half the B traffic per FLOP of the single-CTA form -- with every copy's completion counted on the
// leader's full barrier; the leader's MMA lane issues for both and its commits arrive on the barriers of both CTAs;
// each CTA's epilogue warps drain their own 128 rows and report to the leader's accumulator-free barrier.
template <bool kPair = false, bool kLnEpi = false, bool kSwin = false>
__device__ __forceinline__ void gemm_stage(const Stage& st, const CallArgs& ca, SmemCtl& ctl_s, uint32_t ring, __half* vec_s,
                           uint8_t* stage_s, RoleState& rs, const WaitCtl& ctl, int warp_id, int lane) {
  const int warp = uniform_warp(warp_id);
  const MegaParams& p = ca.p;
  GemmGeom g = gemm_geom(st);
  if constexpr (kPair) g.nh = 1;                                       // per CTA: one 128-row half of the pair's tile
  if (rs.slot >= (uint32_t)g.nslots) rs.slot = 0;
  const uint32_t full0 = smem_u32(&ctl_s.full[0]), empty0 = smem_u32(&ctl_s.empty[0]);
  const uint32_t tfull0 = smem_u32(&ctl_s.tmem_full[0]), tempty0 = smem_u32(&ctl_s.tmem_empty[0]);
  const uint32_t a_bytes = (uint32_t)(g.nh * kATileBytes);
  const uint32_t sub_bytes = (uint32_t)g.slot_bytes >> (g.kper - 1);       // a slot holds one or two K steps of 64, each its A tile and its B tile
  const uint32_t rank = kPair ? cluster_cta_rank() : 0u;               // 0 = the pair's leader
  const int first_item = kPair ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int item_step = kPair ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  // CTAs start at different K chunks so they do not all pull the same A tile at once
  auto first_chunk = [&](int item) {
    const uint32_t rot = (uint32_t)first_item + (uint32_t)item;
    return (int)(rot - fast_div(rot, (uint32_t)g.kchunks, st.mg_kchunks) * (uint32_t)g.kchunks);
  };
  if (warp == 0) {
    // ---------------- feeder: activation tiles, behind the grid barrier ----------------
    if (elect_one()) {
      const CUtensorMap* tmA = map_ptr(ca, st.tm_a);
      unsigned t_wait = 0;
      const bool prof = p.prof != nullptr;
      uint32_t s = rs.slot, bits = rs.slot_bits;
      int mt, nt, ks;
      gemm_item(st, first_item, mt, nt, ks);
      int kk = first_chunk(first_item);
      bool ok = grid_wait(p, ctl, st);
      const long long t_first = prof ? clock64() : 0;
      if (ok && st.dead_bytes[0]) publish_go(ctl_s, st.ordinal);
      for (int item = first_item; ok && item < g.items;) {
        const int m0 = mt * g.bm + (int)rank * 128, kbase = ks * g.kchunks;
        for (int kc = 0; kc < g.kchunks; ++kc) {
          const long long tw = prof ? clock64() : 0;
          if (!mbar_wait_hot(empty0 + 8 * s, ((bits >> s) & 1u) ^ 1u, ctl, 100 + (int)s)) { ok = false; break; }
          if (prof) t_wait += (unsigned)(clock64() - tw);
          const uint32_t fb = full0 + 8 * s, dst = ring + s * g.slot_bytes;
          const int k0 = (kbase + kk) * g.kper * 64;
          if constexpr (kPair) {
            // both CTAs' bytes are counted on the leader's barrier, which only the leader arms
            if (rank == 0) mbar_expect_tx(fb, 2u * a_bytes);
            tma_load_2d_pair(dst, tmA, map_shared_rank(fb, 0), k0, m0);      // box rows = 128: this CTA's half of the rows
          } else {
            mbar_expect_tx(fb, a_bytes * (uint32_t)g.kper);
            tma_load_2d(dst, tmA, fb, k0, m0);      // box rows = bm: both halves in one copy
            if (g.kper == 2) tma_load_2d(dst + sub_bytes, tmA, fb, k0 + 64, m0);
          }
          bits ^= 1u << s;
          s = (s + 1 == (uint32_t)g.nslots) ? 0 : s + 1;
          kk = (kk + 1 == g.kchunks) ? 0 : kk + 1;
        }
        if constexpr (kLnEpi) {          // the tile's residual, one step of 64 columns per slot (see gemm_ln_epilogue)
          const int steps = st.epi == EPI_LN ? (g.bn + 63) >> 6 : 0;
          for (int i = 0; ok && i < steps; ++i) {
            if (!mbar_wait_hot(empty0 + 8 * s, ((bits >> s) & 1u) ^ 1u, ctl, 120 + (int)s)) { ok = false; break; }
            const uint32_t fb = full0 + 8 * s, dst = ring + s * g.slot_bytes;
            const CUtensorMap* tmR = map_ptr(ca, st.tm_resid);
            if constexpr (kPair) {
              if (rank == 0) mbar_expect_tx(fb, 2u * a_bytes);
              tma_load_2d_pair(dst, tmR, map_shared_rank(fb, 0), nt * g.bn + i * 64, m0);
            } else {
              mbar_expect_tx(fb, a_bytes);
              tma_load_2d(dst, tmR, fb, nt * g.bn + i * 64, m0);
            }
            bits ^= 1u << s;
            s = (s + 1 == (uint32_t)g.nslots) ? 0 : s + 1;
          }
        }
        item += item_step;
        gemm_item(st, item, mt, nt, ks);
        kk = first_chunk(item);
      }
      rs.slot = s;
      rs.slot_bits = bits;
      if (p.prof) {
        long long* pr = p.prof + ((size_t)st.position * gridDim.x + blockIdx.x) * kProfSlots;
        pr[5] = t_wait;
        pr[11] = t_first;
      }
    }
    __syncwarp();
  } else if (warp == kWeightWarp) {
    // ---------------- weight tiles: no stage writes them, so they are requested as soon as there are slots ----------------
    // (a lane of its own: a copy takes the issuing thread 100 cycles and more, which behind the barrier is the stage's latency)
    if (elect_one()) {
      const CUtensorMap* tmB = map_ptr(ca, st.tm_b);
      uint32_t s = rs.slot, bits = rs.slot_bits;
      const bool b_mn = st.b_mn_major != 0;
      const uint32_t b_bytes = sub_bytes - a_bytes;
      bool ok = wait_arrived(ctl_s, st.ordinal, ctl);
      for (int item = first_item; ok && item < g.items; item += item_step) {
        int mt, nt, ks;
        gemm_item(st, item, mt, nt, ks);
        const int n0 = nt * g.bn + (int)rank * (g.bn >> 1), kbase = ks * g.kchunks;
        int kk = first_chunk(item);
        for (int kc = 0; kc < g.kchunks; ++kc) {
          if (!mbar_wait_hot(empty0 + 8 * s, ((bits >> s) & 1u) ^ 1u, ctl, 110 + (int)s)) { ok = false; break; }
          const int k0 = (kbase + kk) * g.kper * 64;
          const uint32_t fb = full0 + 8 * s, dst = ring + s * g.slot_bytes + a_bytes;
          if constexpr (kPair) {
            if (rank == 0) mbar_expect_tx(fb, 2u * b_bytes);
            if (!b_mn) {
              tma_load_2d_pair(dst, tmB, map_shared_rank(fb, 0), k0, n0);          // box rows = bn / 2: this CTA's half of the columns
            } else {
              for (int j = 0; j < g.bn / 128; ++j) tma_load_2d_pair(dst + j * 8192, tmB, map_shared_rank(fb, 0), n0 + j * 64, k0);
            }
          } else {
            mbar_expect_tx(fb, b_bytes * (uint32_t)g.kper);
            for (int sub = 0; sub < g.kper; ++sub) {
              const uint32_t to = dst + (uint32_t)sub * sub_bytes;
              if (!b_mn) {
                tma_load_2d(to, tmB, fb, k0 + sub * 64, n0);
              } else {
                for (int j = 0; j < g.bn / 64; ++j) tma_load_2d(to + j * 8192, tmB, fb, n0 + j * 64, k0 + sub * 64);
              }
            }
          }
          bits ^= 1u << s;
          s = (s + 1 == (uint32_t)g.nslots) ? 0 : s + 1;
          kk = (kk + 1 == g.kchunks) ? 0 : kk + 1;
        }
        if constexpr (kLnEpi) {          // unit matrices for the residual
          const int steps = st.epi == EPI_LN ? (g.bn + 63) >> 6 : 0;
          for (int i = 0; ok && i < steps; ++i) {
            if (!mbar_wait_hot(empty0 + 8 * s, ((bits >> s) & 1u) ^ 1u, ctl, 130 + (int)s)) { ok = false; break; }
            const uint32_t fb = full0 + 8 * s, dst = ring + s * g.slot_bytes + a_bytes;
            const CUtensorMap* tmU = map_ptr(ca, st.tm_unit);
            if constexpr (kPair) {
              if (rank == 0) mbar_expect_tx(fb, 2u * kUnitBytes / 2u);
              const int n = g.bn - 64 * i < 64 ? g.bn - 64 * i : 64;      // the pair MMA's columns: each CTA has half of them
              tma_load_2d_pair(dst, tmU, map_shared_rank(fb, 0), 0, (int)rank * (n >> 1));
            } else {
              mbar_expect_tx(fb, kUnitBytes);
              tma_load_2d(dst, tmU, fb, 0, 0);
            }
            bits ^= 1u << s;
            s = (s + 1 == (uint32_t)g.nslots) ? 0 : s + 1;
          }
        }
      }
      rs.slot = s;
      rs.slot_bits = bits;
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer (of a pair: the leader's) ----------------
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = kPair ? umma_idesc_f16_pair((uint32_t)g.bn, (uint32_t)st.b_mn_major)
                                   : umma_idesc_f16((uint32_t)g.bn, (uint32_t)st.b_mn_major);
      const uint32_t tmem = ctl_s.tmem_base;
      // descriptor low words of slot 0; a slot further on adds slot_bytes/16 to both
      const uint32_t a_lo0 = umma_desc_lo(ring, 16);
      const uint32_t b_lo0 = umma_desc_lo(ring + a_bytes, st.b_mn_major ? 8192u : 16u);
      const uint32_t slot16 = (uint32_t)g.slot_bytes >> 4;
      const uint32_t bstep = st.b_mn_major ? 128u : 2u;       // 16 K-rows = 2048 B, or 16 halves = 32 B
      const bool prof = p.prof != nullptr;
      bool ok = true;
      // in registers: `rs` may live in memory
      uint32_t s = rs.slot, bits = rs.slot_bits, acc_next = rs.acc_bits >> 2, acc_bits = rs.acc_bits & 3u;
      unsigned t_full = 0, t_acc = 0;
      long long t_first = 0, t_last = 0;
      for (int item = first_item; ok && item < g.items; item += item_step) {
        const uint32_t acc0 = g.nh == 2 ? 0u : acc_next;       // accumulator of half 0; half 1 uses buffer 1
        const uint32_t d0 = tmem + acc0 * kAccStride, d1 = d0 + kAccStride;
        {                                                      // the epilogue must have drained the buffers
          const long long ta = prof ? clock64() : 0;
          for (int h = 0; h < g.nh; ++h) {
            const uint32_t acc = acc0 + (uint32_t)h;
            if (!mbar_wait_hot(tempty0 + 8 * acc, ((acc_bits >> acc) & 1u) ^ 1u, ctl, 200 + (int)acc)) { ok = false; break; }
          }
          tc_fence_after_sync();
          if (prof) t_acc += (unsigned)(clock64() - ta);
        }
        for (int kc = 0; ok && kc < g.kchunks; ++kc) {
          const long long tw = prof ? clock64() : 0;
          if (!mbar_wait_hot(full0 + 8 * s, (bits >> s) & 1u, ctl, 300 + (int)s)) { ok = false; break; }
          if (prof) {
            const long long tn = clock64();
            t_full += (unsigned)(tn - tw);
            if (!t_first) t_first = tn;
          }
          tc_fence_after_sync();
          const uint32_t a_lo = a_lo0 + s * slot16, b_lo = b_lo0 + s * slot16;
          if constexpr (kPair) {
            umma_f16_k64_pair(d0, a_lo, b_lo, bstep, idesc, (uint32_t)(kc != 0));
            umma_commit_pair(empty0 + 8 * s);
          } else {
            if (g.nh == 2) umma_f16_k64_x2(d0, d1, a_lo, b_lo, bstep, idesc, (uint32_t)(kc != 0));
            else umma_f16_k64(d0, a_lo, b_lo, bstep, idesc, (uint32_t)(kc != 0));
            if (g.kper == 2) umma_f16_k64(d0, a_lo + (sub_bytes >> 4), b_lo + (sub_bytes >> 4), bstep, idesc, 1u);
            umma_commit(empty0 + 8 * s);
          }
          bits ^= 1u << s;
          s = (s + 1 == (uint32_t)g.nslots) ? 0 : s + 1;
        }
        if constexpr (kLnEpi) {          // + residual x unit matrix, 64 columns at a time
          const int steps = st.epi == EPI_LN ? (g.bn + 63) >> 6 : 0;
          for (int i = 0; ok && i < steps; ++i) {
            const uint32_t n = g.bn - 64 * i < 64 ? (uint32_t)(g.bn - 64 * i) : 64u;
            if (!mbar_wait_hot(full0 + 8 * s, (bits >> s) & 1u, ctl, 310 + (int)s)) { ok = false; break; }
            tc_fence_after_sync();
            const uint32_t a_lo = a_lo0 + s * slot16, b_lo = b_lo0 + s * slot16, d = d0 + 64u * (uint32_t)i;
            if constexpr (kPair) {
              umma_f16_k64_pair(d, a_lo, b_lo, 2u, umma_idesc_f16_pair(n, 0u), 1u);
              umma_commit_pair(empty0 + 8 * s);
            } else {
              if (g.nh == 2) umma_f16_k64_x2(d, d + kAccStride, a_lo, b_lo, 2u, umma_idesc_f16(n, 0u), 1u);
              else umma_f16_k64(d, a_lo, b_lo, 2u, umma_idesc_f16(n, 0u), 1u);
              umma_commit(empty0 + 8 * s);
            }
            bits ^= 1u << s;
            s = (s + 1 == (uint32_t)g.nslots) ? 0 : s + 1;
          }
        }
        if (!ok) break;
        for (int h = 0; h < g.nh; ++h) {
          const uint32_t acc = acc0 + (uint32_t)h;
          if constexpr (kPair) umma_commit_pair(tfull0 + 8 * acc);
          else umma_commit(tfull0 + 8 * acc);
          acc_bits ^= 1u << acc;
        }
        if (prof) t_last = clock64();
        if (g.nh == 1) acc_next ^= 1u;
      }
      rs.slot = s;
      rs.slot_bits = bits;
      rs.acc_bits = acc_bits | (acc_next << 2);
      if (p.prof) {
        long long* pr = p.prof + ((size_t)st.position * gridDim.x + blockIdx.x) * kProfSlots;
        pr[3] = t_full;
        pr[4] = t_acc;
        pr[12] = t_first;
        pr[13] = t_last;
      }
    }
    __syncwarp();
  } else if (warp < 2 + kEpiWarps) {
    // ---------------- epilogue: TMEM -> registers -> global (8 warps: lane quarter x column parity) --
    const int q = epi_quarter(warp), cpar = epi_part(warp);
    const uint32_t tmem = ctl_s.tmem_base + ((uint32_t)(q * 32) << 16);
    const int full_chunks = g.bn >> 5;
    if (kLnEpi && st.epi == EPI_LN) {
      const uint32_t which = (uint32_t)(&st == &ctl_s.stage[1]) << 31;
      if constexpr (kSwin) rs.acc_bits = gemm_swin_ln(ca, rs.acc_bits | which);
      else rs.acc_bits = gemm_ln_epilogue<kPair>(ca, rs.acc_bits | which);
    } else {
    EpiCtx e;
    e.epi = st.epi; e.act = st.act; e.M = st.M; e.N = st.N; e.ldo = st.ldo;
    e.out = reinterpret_cast<__half*>(const_cast<void*>(sel_ptr(st.out_sel, st.out, p)));
    e.partial = st.partial;
    e.tm_out = map_ptr(ca, st.tm_out);
    const bool prof = p.prof != nullptr;
    e.prof = prof;
    // cycle totals of the profile go straight to its record (no registers held for them over the tiles)
    auto note = [&](int slot, unsigned cycles) {
      if (warp == 2 && lane == 0)
        atomicAdd(reinterpret_cast<unsigned long long*>(p.prof + ((size_t)st.position * gridDim.x + blockIdx.x) * kProfSlots + slot),
                  (unsigned long long)cycles);
    };
    if (prof && warp == 2 && lane == 0)
      for (int i = 6; i < 11; ++i) p.prof[((size_t)st.position * gridDim.x + blockIdx.x) * kProfSlots + i] = 0;
    StoreBoxes sb;
    sb.base = reinterpret_cast<uint8_t*>(vec_s) + epi_box(warp) * kStageWarp;
    sb.box = 0;
    sb.n = 2;
    // The bias of a tile's columns goes to shared memory as fp32 in front of the tile: a thread loads one column's (0 where there is
    // none) while the tile before is being stored, and one barrier per tile separates the two buffers' uses.
    const int my_col = (int)threadIdx.x - 64;
    const __half* bias = e.epi != EPI_PARTIAL ? reinterpret_cast<const __half*>(st.bias) : nullptr;
    auto load_bias = [&](int nt) -> float { return bias && my_col < g.bn && nt * g.bn + my_col < e.N ? __half2float(__ldg(bias + nt * g.bn + my_col)) : 0.0f; };
    int mt, nt, ks;
    gemm_item(st, first_item, mt, nt, ks);
    float next_bias = first_item < g.items ? load_bias(nt) : 0.0f;
    uint32_t turn = 0;
    // The warps look at the wait limit one by one and meet in a barrier per tile: one that has given up goes through the remaining
    // tiles without waiting again and without storing.
    bool ok = true;
#pragma unroll 1
    for (int item = first_item; item < g.items; item += item_step, turn ^= 1u) {
      const uint32_t acc0 = g.nh == 2 ? 0u : rs.acc_bits >> 2;
      const int row_tile = mt * g.bm, colbase = nt * g.bn, plane = ks;
      const int left = (e.N - colbase) >> 5, chunks = left < full_chunks ? left : full_chunks;
      const float* bias_t = ctl_s.bias[turn];
      if (e.epi != EPI_PARTIAL) {
        ctl_s.bias[turn][my_col] = next_bias;
        named_barrier_sync(1, kEpiThreads);
      }
      // TMA-store boxes of the CTA's last tile live in the operand ring: once its accumulator is complete every operand
      // tile of the stage has been consumed, and nothing is loaded before the next stage
      if (item + item_step >= g.items) {
        sb.base = stage_s - kVecBytes - kRingBytes + (warp - 2) * kRingBoxes * kStageWarp;
        sb.box = 0;
        sb.n = kRingBoxes;
      } else {
        gemm_item(st, item + item_step, mt, nt, ks);
        next_bias = load_bias(nt);
      }
      for (int h = 0; h < g.nh; ++h) {
        const uint32_t acc = acc0 + (uint32_t)h;
        // output rows first: worked out while the accumulator is still being filled
        const int row0 = row_tile + (kPair ? (int)rank : h) * 128 + q * 32;
        const uint32_t own = epi_row_offset(st, e, row0 + lane, plane);
        // head-split stores: rows of the [3 B heads S][64] view at which the block's two halves of 16 rows begin
        uint32_t tok0 = 0, tok1 = 0;
        if (e.epi == EPI_QKV) {
          tok0 = __shfl_sync(0xffffffffu, own, 0) >> 6;
          tok1 = __shfl_sync(0xffffffffu, own, 16);
          tok1 = tok1 == kNoRow ? kNoRow : tok1 >> 6;
        }
        const unsigned tw = prof ? (unsigned)clock64() : 0u;
        ok = ok && mbar_wait_warp(tfull0 + 8 * acc, (rs.acc_bits >> acc) & 1u, ctl, 400 + (int)acc, lane);
        if (!ok) break;
        unsigned tb = 0;
        if (prof) {
          const long long now = clock64();
          tb = (unsigned)now;
          note(6, tb - tw);
          if (item == first_item && h == 0 && warp == 2 && lane == 0)
            p.prof[((size_t)st.position * gridDim.x + blockIdx.x) * kProfSlots + 14] = now;
        }
        tc_fence_after_sync();
        const uint32_t t0 = tmem + acc * kAccStride;
        // this warp takes chunks cpar, cpar+2, ... (its partner warp on the same lane quarter the others)
        // and a last tile that is wider than what is left of the matrix (a multiple of 64 columns) ends with it
        for (int c = cpar; c < chunks; c += 2) {
          uint32_t r[32];
          const unsigned tl = prof ? (unsigned)clock64() : 0u;
          tmem_ld32(t0 + c * 32, r);
          tmem_ld_wait(r);
          unsigned tm = 0, tmid = 0;
          if (prof) {
            tm = (unsigned)clock64();
            note(8, tm - tl);
          }
          const int col = colbase + c * 32;
          if (e.epi == EPI_PARTIAL) {
            // fp32 planes: two boxes of 16 columns.  (Storing each thread's own 128-byte row segment directly measured twice as
            // slow: an instruction's cost grows with the lines it touches.)
            if (prof) tmid = (unsigned)clock64();
#pragma unroll
            for (int half = 0; half < 2; ++half)
              store_box(sb, r + 16 * half, lane, [&](uint32_t buf) {
                if (row0 < e.M) tma_store_3d(e.tm_out, buf, col + 16 * half, row0, plane);
              });
          } else {
            uint32_t w[16];
            epilogue_values32(e, r, bias_t + c * 32, w);
            if (prof) tmid = (unsigned)clock64();
            store_box(sb, w, lane, [&](uint32_t buf) {
              if (row0 < e.M) {
                if (e.epi == EPI_QKV) {
                  const uint32_t gq = (uint32_t)col >> 6, which = fast_div(gq, (uint32_t)st.heads, st.mg_heads), hh = gq - which * (uint32_t)st.heads;
                  const uint32_t head_row = (which * (uint32_t)(st.batch * st.heads) + hh) * (uint32_t)st.seq;
                  tma_store_2d(e.tm_out, buf, col & 63, (int)(head_row + tok0));
                  if (st.out_stores == 2 && tok1 != kNoRow) tma_store_2d(e.tm_out, buf + 16 * kStageRow, col & 63, (int)(head_row + tok1));
                } else {
                  tma_store_2d(e.tm_out, buf, col, row0);
                }
              }
            });
          }
          if (prof) {
            note(9, tmid - tm);
            note(10, (unsigned)clock64() - tmid);
          }
        }
        if ((g.bn & 16) && (full_chunks & 1) == cpar) {
          uint32_t r[16];
          tmem_ld16(t0 + full_chunks * 32, r);
          tmem_ld_wait(r);
          epilogue_chunk16(st, e, r, bias_t + full_chunks * 32, own, colbase + full_chunks * 32);
        }
        tc_fence_before_sync();
        if constexpr (kPair) {                      // one arrival per warp on the leader's barrier (16 in all)
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_relaxed(map_shared_rank(tempty0 + 8 * acc, 0));
        } else {
          mbar_arrive(tempty0 + 8 * acc);
        }
        rs.acc_bits ^= 1u << acc;
        if (prof) note(7, (unsigned)clock64() - tb);
      }
      if (g.nh == 1) rs.acc_bits ^= 4u;
    }
    if (elect_one()) {        // the stores are complete before the CTA reports the stage done
      bulk_wait_group_all();
      fence_proxy_async_global();
    }
    __syncwarp();
    if (prof && warp == 2 && lane == 0)
      p.prof[((size_t)st.position * gridDim.x + blockIdx.x) * kProfSlots + 15] = clock64();
    }
  }
}

// Parity output of the attention stages: normalised probabilities of one query row per thread, recomputed from the
// scores in TMEM.  Out of line: only the parity configurations call them, and inlined their registers would be charged
// to every attention item.
// Tile form (the cooperative attention stage): the unnormalised probabilities already sit in shared memory as the
// fp16 A-operand tiles of P.V ([128 rows][64 keys] per tile, 128-byte rows with the 16-byte pieces XOR-swizzled by
// row & 7); the 256 softmax threads copy them out scaled by 1 / rowsum: eight threads per row, 32 rows per pass, so a
// store instruction writes four rows of 128 contiguous bytes.  An item has `qrows` query rows, each in 128 / qrows copies
// (see attn_stage); `sums` = the partial row sums [2][copies][qrows].
__device__ __noinline__ void attn_copy_probs_tiles(const uint8_t* ptiles, const float* sums, __half* mat, int S, int qrows, int rows, int t8) {
  const int sub = t8 & 7, rsub = t8 >> 3, copies = 128 / qrows;
  for (int r = rsub; r < rows; r += 32) {
    float sum = 0.0f;
    for (int i = r; i < 256; i += qrows) sum += sums[i];
    const float inv = 1.0f / sum;
    __half* dst = mat + (size_t)r * S + sub * 8;
    for (int tile = 0; tile * 64 + sub * 8 + 8 <= S; ++tile) {
      const int prow = ((tile * 4 + (sub >> 1)) & (copies - 1)) * qrows + r;       // the copy that holds these keys
      const uint4 v = *reinterpret_cast<const uint4*>(ptiles + tile * kATileBytes + prow * 128 + ((sub ^ (prow & 7)) << 4));
      const uint32_t in[4] = {v.x, v.y, v.z, v.w};
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&in[i]));
        w[i] = pack_h2(f.x * inv, f.y * inv);
      }
      *reinterpret_cast<uint4*>(dst + tile * 64) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// Staged form (S <= 128, a warp owns rows row0 .. row0 + 31 of the [S][S] matrix at `mat`): whole 64-byte row pieces
// go through the warp's staging buffer, so that a store instruction writes eight rows of 64 contiguous bytes.
__device__ __noinline__ void attn_store_probs_staged(uint32_t ts, uint8_t* sbuf, __half* mat, int row0, int S, int kv_len,
                                                     float sl2, float mask_l2, float mx, float inv, int lane) {
  for (int c = 0; c * 32 < S; ++c) {
    uint32_t r[32];
    tmem_ld32(ts + c * 32, r);
    tmem_ld_wait(r);
    uint32_t w[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int key = c * 32 + 2 * i;
      const float ta = __uint_as_float(r[2 * i]) * sl2 + (key >= kv_len ? mask_l2 : 0.0f);
      const float tb = __uint_as_float(r[2 * i + 1]) * sl2 + (key + 1 >= kv_len ? mask_l2 : 0.0f);
      w[i] = pack_h2(ex2_fast(ta - mx) * inv, ex2_fast(tb - mx) * inv);
    }
    if (c * 32 + 32 <= S) {
      uint8_t* rowptr[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int rr = row0 + 8 * i + (lane >> 2);
        rowptr[i] = rr < S ? reinterpret_cast<uint8_t*>(mat + (size_t)rr * S + c * 32) : nullptr;
      }
      staged_store_64B(sbuf, w, rowptr, lane);
    } else if (row0 + lane < S) {                     // the last 16 keys of a row (S is a multiple of 16)
      uint4* dst = reinterpret_cast<uint4*>(mat + (size_t)(row0 + lane) * S + c * 32);
      dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
      dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
  }
}

// ------------------------------------------------------------------------------------
// attention stage: one work item = (sequence, head, query tile); S <= 384, head_dim 64
//
// A tile has st.bm = 128, 64 or 32 query rows (the smallest for which every CTA has one item at most), and the MMA has 128: a
// tile of fewer rows is loaded 128 / bm times, one copy below the other, and every copy takes its own share of the keys.  A copy
// leaves 0 where another copy's keys are, so P.V gives each copy's part of the output, and the parts are added up at the end.
// So all eight softmax warps have work, and one sequence's attention lies on four times as many CTAs: a layer of one sequence
// (bm = 32 against 128, the lone lanes' loops as they are) 36.0 -> 34.8 us at 128 tokens, the stage 9.7 k -> 7.2 k cycles; at 384
// tokens 16.4 k -> 10.3 k.  What is left is latency: 2.7 k until the scores are there, 0.4 k for the maxima, 0.5 k for their
// exchange, 0.7 k for the exponentials, 0.9 k for P.V, 1.1 k for the output.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void attn_stage(const Stage& st, const CallArgs& ca, SmemCtl& ctl_s, uint32_t ring, uint8_t* ring_ptr,
                                           uint8_t* stage_s, RoleState& rs, const WaitCtl& ctl, int warp, int lane) {
  const MegaParams& p = ca.p;
  const int S = st.seq, B = st.batch, H = st.heads;
  const int qrows = st.bm, copies = 128 / qrows, n_qt = (S + qrows - 1) / qrows;
  const int n_kb = (S + 127) / 128;
  const int items = B * H * n_qt;
  const uint32_t q_off = 0, k_off = kATileBytes, v_off = k_off + n_kb * kATileBytes,
                 p_off = v_off + n_kb * kATileBytes;
  const uint32_t qk_full = smem_u32(&ctl_s.qk_full), qk_empty = smem_u32(&ctl_s.qk_empty);
  const uint32_t v_full = smem_u32(&ctl_s.v_full), v_empty = smem_u32(&ctl_s.v_empty);
  const uint32_t s_full = smem_u32(&ctl_s.s_full), p_full = smem_u32(&ctl_s.p_full),
                 o_full = smem_u32(&ctl_s.o_full);
  const CUtensorMap* tm = map_ptr(ca, st.tm_qkv);

  if (warp == 0) {
    if (elect_one()) {
      const CUtensorMap* tmq = map_ptr(ca, st.tm_a);
      uint32_t bit = rs.attn_bit;
      int qt = (int)blockIdx.x % n_qt, bh = (int)blockIdx.x / n_qt;          // in front of the wait: divisions
      const bool ok = grid_wait(p, ctl, st);
      if (ok && st.dead_bytes[0]) publish_go(ctl_s, st.ordinal);
      for (int item = blockIdx.x; ok && item < items;) {
        const int rq = bh * S, rk = (B * H + bh) * S, rv = (2 * B * H + bh) * S;
        if (!mbar_wait_hot(qk_empty, bit ^ 1u, ctl, 500)) break;
        mbar_expect_tx(qk_full, (uint32_t)(kATileBytes * (1 + n_kb)));
#pragma unroll 1
        for (int c = 0; c < copies; ++c) tma_load_2d(ring + q_off + c * qrows * 128, tmq, qk_full, 0, rq + qt * qrows);
#pragma unroll 1
        for (int kb = 0; kb < n_kb; ++kb) tma_load_2d(ring + k_off + kb * kATileBytes, tm, qk_full, 0, rk + kb * 128);
        if (!mbar_wait_hot(v_empty, bit ^ 1u, ctl, 501)) break;
        mbar_expect_tx(v_full, (uint32_t)(kATileBytes * n_kb));
#pragma unroll 1
        for (int kb = 0; kb < n_kb; ++kb) tma_load_2d(ring + v_off + kb * kATileBytes, tm, v_full, 0, rv + kb * 128);
        bit ^= 1u;
        item += gridDim.x;
        qt = item % n_qt;
        bh = item / n_qt;
      }
      rs.attn_bit = bit;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc_s = umma_idesc_f16(128u, 0u);
      const uint32_t idesc_o = umma_idesc_f16(64u, 1u);
      const uint32_t tmem = ctl_s.tmem_base;
      const uint32_t q_lo = umma_desc_lo(ring + q_off, 16), k_lo = umma_desc_lo(ring + k_off, 16), p_lo = umma_desc_lo(ring + p_off, 16),
                     v_lo = umma_desc_lo(ring + v_off, 8192);
      uint32_t bit = rs.attn_bit;
      for (int item = blockIdx.x; item < items; item += gridDim.x) {
        if (!mbar_wait_hot(qk_full, bit, ctl, 510)) break;
        tc_fence_after_sync();
#pragma unroll 1
        for (int kb = 0; kb < n_kb; ++kb) umma_f16_k64(tmem + kb * 128, q_lo, k_lo + kb * (kATileBytes >> 4), 2u, idesc_s, 0u);
        umma_commit(s_full);
        umma_commit(qk_empty);
        if (!mbar_wait_hot(v_full, bit, ctl, 512)) break;
        if (!mbar_wait_hot(p_full, bit, ctl, 511)) break;
        tc_fence_after_sync();
        // 64 keys per chunk: a tile of P, half a tile of V
#pragma unroll 1
        for (int c = 0; c < 2 * n_kb; ++c)
          umma_f16_k64(tmem + kOCol, p_lo + c * (kATileBytes >> 4), v_lo + c * (8192 >> 4), 128u, idesc_o, (uint32_t)(c != 0));
        umma_commit(o_full);
        umma_commit(v_empty);
        bit ^= 1u;
      }
      rs.attn_bit = bit;
    }
    __syncwarp();
  } else if (warp < 2 + kEpiWarps) {
    // Both groups of four warps work on the same item.  Of the 16-key blocks, copy c takes numbers c, c + copies, ...,
    // group 0 and group 1 in turn (a thread of each group owns row r_in); row maxima and row sums are exchanged through
    // shared memory around two 256-thread barriers.  The output columns are split 32 / 32 between the groups.
    const int grp = (warp - 2) >> 2, q = warp & 3;
    const int r_in = q * 32 + lane;
    const int copy = r_in / qrows, row = r_in & (qrows - 1);
    const int blk0 = copy + grp * copies, stepb = 2 * copies;
    const uint32_t tmem = ctl_s.tmem_base + ((uint32_t)(q * 32) << 16);
    const float sl2 = st.scale * 1.4426950408889634f;
    const int* lens = p.lens;
    __half* ctx = reinterpret_cast<__half*>(st.out);
    __half* probs = reinterpret_cast<__half*>(st.probs);
    const int hidden = H * st.head_dim;
    // At S = 384 the tiles of this stage (Q, 3 K, 3 V, 6 P = 208 KB) run past the 192 KB ring into the vector and
    // staging areas behind it, which no one else uses during attention; the exchange buffer sits at their very end.
    static_assert(13 * kATileBytes <= kRingBytes + kVecBytes + kStageBytes - 2048, "attention tiles overlap the exchange buffer");
    float* red = reinterpret_cast<float*>(stage_s + kStageBytes - 2048);   // [2 groups][128 rows] maxima, then [2][128] sums
    // The warps look at the wait limit one by one and meet in barriers, so none leaves the loop early: one that has given up goes
    // through the remaining items without waiting again and without storing.
    bool ok = true;
    uint8_t* pbase = ring_ptr + p_off + r_in * 128;
    auto zero16 = [&](int blk) {
      uint8_t* base = pbase + (blk >> 2) * kATileBytes;
      const int j = (blk & 3) * 2;
      *reinterpret_cast<uint4*>(base + ((j ^ (r_in & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(base + (((j + 1) ^ (r_in & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
    };
    const int nb_all = n_kb * 8;
    if (copies > 1 && (int)blockIdx.x < items) {               // the other copies' keys, while nothing has arrived yet; there is one item
#pragma unroll 1
      for (int blk = grp; blk < nb_all; blk += 2)
        if ((blk & (copies - 1)) != copy) zero16(blk);
    }
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const int qt = item % n_qt, h = (item / n_qt) % H, b = item / (n_qt * H);
      const int kv_len = lens ? lens[b] : S;
      ok = ok && mbar_wait_warp(s_full, rs.attn_bit, ctl, 520, lane);
      tc_fence_after_sync();
      // Keys >= kv_len carry the additive -1e4 mask: probability 0 in fp32, never the maximum -> only the blocks
      // with valid keys are visited; the other P blocks are written as zeros.
      const int kvl = kv_len < 1 ? 1 : (kv_len > S ? S : kv_len);
      const int nb = (kvl + 15) >> 4;
      uint32_t ra[16];                     // (one block at a time: two in flight would spill in this build)
      // ---- pass 1: maximum of the raw scores of the valid keys (the scale is positive) ----
      float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
      auto max16 = [&](const uint32_t (&r)[16], int blk) {
        const int key0 = blk * 16;
        if (key0 + 16 <= kvl) {
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            m0 = fmaxf(m0, __uint_as_float(r[i])); m1 = fmaxf(m1, __uint_as_float(r[i + 1]));
            m2 = fmaxf(m2, __uint_as_float(r[i + 2])); m3 = fmaxf(m3, __uint_as_float(r[i + 3]));
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) m0 = fmaxf(m0, key0 + i < kvl ? __uint_as_float(r[i]) : -INFINITY);
        }
      };
      for (int blk = blk0; blk < nb; blk += stepb) {
        tmem_ld16(tmem + blk * 16, ra);
        tmem_ld_wait(ra);
        max16(ra, blk);
      }
      red[grp * 128 + r_in] = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
      named_barrier_sync(3, 256);
      float mx = red[row];
#pragma unroll 1
      for (int i = row + qrows; i < 256; i += qrows) mx = fmaxf(mx, red[i]);
      mx *= sl2;
      // ---- pass 2: unnormalised probabilities -> fp16 A-operand tiles (128B-swizzled rows, 64 keys per tile) ----
      float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
      auto exp16 = [&](const uint32_t (&r)[16], int blk) {
        const int key0 = blk * 16;
        uint32_t w[8];
        if (key0 + 16 <= kvl) {
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const float p0 = ex2_fast(fmaf(__uint_as_float(r[i]), sl2, -mx)), p1 = ex2_fast(fmaf(__uint_as_float(r[i + 1]), sl2, -mx));
            const float p2 = ex2_fast(fmaf(__uint_as_float(r[i + 2]), sl2, -mx)), p3 = ex2_fast(fmaf(__uint_as_float(r[i + 3]), sl2, -mx));
            s0 += p0; s1 += p1; s2 += p2; s3 += p3;
            w[i >> 1] = pack_h2(p0, p1);
            w[(i >> 1) + 1] = pack_h2(p2, p3);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const float p0 = key0 + i < kvl ? ex2_fast(fmaf(__uint_as_float(r[i]), sl2, -mx)) : 0.f;
            const float p1 = key0 + i + 1 < kvl ? ex2_fast(fmaf(__uint_as_float(r[i + 1]), sl2, -mx)) : 0.f;
            s0 += p0; s1 += p1;
            w[i >> 1] = pack_h2(p0, p1);
          }
        }
        uint8_t* base = pbase + (blk >> 2) * kATileBytes;
        const int j = (blk & 3) * 2;
        *reinterpret_cast<uint4*>(base + ((j ^ (r_in & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(base + (((j + 1) ^ (r_in & 7)) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
      };
      for (int blk = blk0; blk < nb; blk += stepb) {
        tmem_ld16(tmem + blk * 16, ra);
        tmem_ld_wait(ra);
        exp16(ra, blk);
      }
#pragma unroll 1
      for (int blk = blk0; blk < nb_all; blk += stepb)        // keys past the valid ones: probability 0
        if (blk >= nb) zero16(blk);
      red[256 + grp * 128 + r_in] = (s0 + s1) + (s2 + s3);
      fence_proxy_async_smem();                               // this thread's P rows -> visible to the MMA
      named_barrier_sync(3, 256);
      float sum = 0.0f;
#pragma unroll 1
      for (int i = row; i < 256; i += qrows) sum += red[256 + i];
      const float inv = 1.0f / sum;
      const int row0 = qt * qrows;
      tc_fence_before_sync();
      if (grp == 0) mbar_arrive(p_full);                      // 128 arrivals: group 1's rows are behind the barrier above
      if (probs) {
        // parity output: normalised probabilities [B*heads][S][S], copied from the P tiles while P.V runs; nobody may
        // start the next item's P rows or row sums before every thread has copied
        attn_copy_probs_tiles(ring_ptr + p_off, red + 256, probs + ((size_t)(b * H + h) * S + row0) * S, S, qrows,
                              S - row0 < qrows ? S - row0 : qrows, (int)threadIdx.x - 64);
        named_barrier_sync(3, 256);
      }
      ok = ok && mbar_wait_warp(o_full, rs.attn_bit, ctl, 521, lane);
      tc_fence_after_sync();
      {
        // This group's 32 of the 64 output columns.  The P tiles have been consumed: a warp hands its rows over through 4 KB of
        // them (16-byte pieces XOR-swizzled by the row), and a thread adds up the copies of eight columns of a row, so that a store
        // instruction writes eight rows of 64 contiguous bytes.
        uint32_t r0[32];
        tmem_ld32(tmem + kOCol + grp * 32, r0);
        tmem_ld_wait(r0);
        uint8_t* part = ring_ptr + p_off + grp * kATileBytes;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<float4*>(part + r_in * 128 + ((i ^ (r_in & 7)) << 4)) =
              make_float4(__uint_as_float(r0[4 * i]) * inv, __uint_as_float(r0[4 * i + 1]) * inv, __uint_as_float(r0[4 * i + 2]) * inv,
                          __uint_as_float(r0[4 * i + 3]) * inv);
        if (copies > 1) named_barrier_sync(4 + grp, 128);      // a copy's rows lie with other warps
        else __syncwarp();
        // threads 4 r .. 4 r + 3 of the group (of the warp, where it owns its rows alone): columns 8 j .. 8 j + 7
        const int j = lane & 3;
        for (int rr = q * 8 + (lane >> 2) + (copies > 1 ? 0 : q * 24); rr < (copies > 1 ? qrows : q * 32 + 32); rr += copies > 1 ? 32 : 8) {
          float o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = 0.0f;
#pragma unroll 1
          for (int pr = rr; pr < 128; pr += qrows) {
            const float4 u0 = *reinterpret_cast<const float4*>(part + pr * 128 + (((2 * j) ^ (pr & 7)) << 4));
            const float4 u1 = *reinterpret_cast<const float4*>(part + pr * 128 + (((2 * j + 1) ^ (pr & 7)) << 4));
            o[0] += u0.x; o[1] += u0.y; o[2] += u0.z; o[3] += u0.w; o[4] += u1.x; o[5] += u1.y; o[6] += u1.z; o[7] += u1.w;
          }
          if (ok && row0 + rr < S)
            *reinterpret_cast<uint4*>(ctx + ((size_t)b * S + row0 + rr) * hidden + h * st.head_dim + grp * 32 + j * 8) =
                make_uint4(pack_h2(o[0], o[1]), pack_h2(o[2], o[3]), pack_h2(o[4], o[5]), pack_h2(o[6], o[7]));
        }
      }
      // (the next item's P rows go over the parts just read, but behind the barrier of its maxima)
      tc_fence_before_sync();
      rs.attn_bit ^= 1u;
    }
  }
}

// ------------------------------------------------------------------------------------
// attention stage for S <= 128: two independent pipelines ("ping" and "pong").  The CTA's work items
// alternate between them; each pipeline has its own Q/K/V/P tiles in shared memory, its own score and
// output accumulators in TMEM, its own barriers and its own group of four softmax warps (warps 2..5
// and 6..9).  While one group runs the softmax of item i, the tensor core already holds the scores of
// item i+1 for the other group, and the loads of item i+2 are in flight.
// ------------------------------------------------------------------------------------
enum AttnBar : int { AB_QK_FULL = 0, AB_QK_EMPTY, AB_V_FULL, AB_V_EMPTY, AB_S_FULL, AB_P_FULL, AB_O_FULL };
constexpr int kPipeBytes = 5 * kATileBytes;      // Q 16 KiB, K 16, V 16, P 32
constexpr int kPipeOCol = 256;                   // TMEM: scores at 0 / 128, outputs at 256 / 320

template <bool kPair>
__device__ __forceinline__ void attn_stage_pp(const Stage& st, const CallArgs& ca, SmemCtl& ctl_s, uint32_t ring, uint8_t* ring_ptr,
                              uint8_t* boxes, RoleState& rs, const WaitCtl& ctl, int warp, int lane) {
  const MegaParams& p = ca.p;
  const int S = st.seq, B = st.batch, H = st.heads;
  // kPair: the two CTAs of a pair take the two heads 2c, 2c + 1 of one sequence (same valid length) and the leader
  // issues ONE pair MMA for both: A = [Q_0; Q_1] (M = 256), B = [K_0; K_1] (N = 256), so CTA r finds Q_r K_r^T in
  // columns 128 r .. of its accumulator (the off-diagonal blocks are waste the tensor core has time for); then
  // A = [P_0; P_1], B = [V_0 | V_1] (N = 128) leaves O_r in columns 64 r ...  Every CTA loads exactly its own Q, K, V.
  // The output accumulator re-uses the columns of the scores (512 columns hold two pipelines of 256), so the scores
  // of a pipeline's next item wait until its output has been read (o_empty).
  const uint32_t rank = kPair ? cluster_cta_rank() : 0u;
  const int units = kPair ? (B * H) >> 1 : B * H;                      // couples of heads, or single (sequence, head) items
  const int first = kPair ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, step = kPair ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int my_items = units > first ? (units - 1 - first) / step + 1 : 0;
  auto item_of = [&](int k) -> int { const int u = first + k * step; return kPair ? 2 * u + (int)rank : u; };
  auto seq_of = [&](int item) -> int { return (int)fast_div((uint32_t)item, (uint32_t)H, st.mg_heads); };
  const uint32_t bar0 = smem_u32(&ctl_s.qk_full), bar1 = smem_u32(&ctl_s.attn1[0]);
  auto bar = [&](int g, int which) -> uint32_t { return (g ? bar1 : bar0) + 8u * (uint32_t)which; };
  const uint32_t oempty0 = smem_u32(&ctl_s.o_empty[0]);
  const CUtensorMap* tm = map_ptr(ca, st.tm_qkv);

  if (warp == 0) {
    if (elect_one()) {
      uint32_t bits = rs.attn_bit | (rs.attn_bit1 << 1);
      const bool ok = grid_wait(p, ctl, st);
      if (ok && st.dead_bytes[0]) publish_go(ctl_s, st.ordinal);
      for (int k = 0; ok && k < my_items; ++k) {
        const int item = item_of(k), g = k & 1;
        const int rq = item * S, rk = (B * H + item) * S, rv = (2 * B * H + item) * S;
        const uint32_t base = ring + g * kPipeBytes, bit = (bits >> g) & 1u;
        if (!mbar_wait_hot(bar(g, AB_QK_EMPTY), bit ^ 1u, ctl, 500 + g)) break;
        if constexpr (kPair) {            // both CTAs' tiles are counted on the leader's barriers
          if (rank == 0) mbar_expect_tx(bar(g, AB_QK_FULL), 4u * kATileBytes);
          const uint32_t fl = map_shared_rank(bar(g, AB_QK_FULL), 0);
          tma_load_2d_pair(base, tm, fl, 0, rq);
          tma_load_2d_pair(base + kATileBytes, tm, fl, 0, rk);
        } else {
          mbar_expect_tx(bar(g, AB_QK_FULL), 2u * kATileBytes);
          tma_load_2d(base, tm, bar(g, AB_QK_FULL), 0, rq);
          tma_load_2d(base + kATileBytes, tm, bar(g, AB_QK_FULL), 0, rk);
        }
        if (!mbar_wait_hot(bar(g, AB_V_EMPTY), bit ^ 1u, ctl, 502 + g)) break;
        if constexpr (kPair) {
          if (rank == 0) mbar_expect_tx(bar(g, AB_V_FULL), 2u * kATileBytes);
          tma_load_2d_pair(base + 2 * kATileBytes, tm, map_shared_rank(bar(g, AB_V_FULL), 0), 0, rv);
        } else {
          mbar_expect_tx(bar(g, AB_V_FULL), (uint32_t)kATileBytes);
          tma_load_2d(base + 2 * kATileBytes, tm, bar(g, AB_V_FULL), 0, rv);
        }
        bits ^= 1u << g;
      }
      rs.attn_bit = bits & 1u;
      rs.attn_bit1 = (bits >> 1) & 1u;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      const uint32_t idesc_s = kPair ? umma_idesc_f16_pair(256u, 0u) : umma_idesc_f16(128u, 0u);
      const uint32_t idesc_o = kPair ? umma_idesc_f16_pair(128u, 1u) : umma_idesc_f16(64u, 1u);
      const uint32_t tmem = ctl_s.tmem_base;
      uint32_t bits = rs.attn_bit | (rs.attn_bit1 << 1);
      uint32_t obits = rs.o_bits;                              // pair form: phase bit of the o_empty barrier of each pipeline
      bool ok = true;
      auto issue_s = [&](int k) {                              // scores of item k: S = Q K^T
        const int g = k & 1;
        const uint32_t base = ring + g * kPipeBytes;
        if (!mbar_wait_hot(bar(g, AB_QK_FULL), (bits >> g) & 1u, ctl, 510 + g)) { ok = false; return; }
        tc_fence_after_sync();
        if constexpr (kPair) {
          umma_f16_k64_pair(tmem + g * 256, umma_desc_lo(base, 16), umma_desc_lo(base + kATileBytes, 16), 2u, idesc_s, 0u);
          umma_commit_pair(bar(g, AB_S_FULL));
          umma_commit_pair(bar(g, AB_QK_EMPTY));
        } else {
          umma_f16_k64(tmem + g * 128, umma_desc_lo(base, 16), umma_desc_lo(base + kATileBytes, 16), 2u, idesc_s, 0u);
          umma_commit(bar(g, AB_S_FULL));
          umma_commit(bar(g, AB_QK_EMPTY));
        }
      };
      if (my_items > 0) issue_s(0);
      if (ok && my_items > 1) issue_s(1);
      for (int k = 0; ok && k < my_items; ++k) {
        const int g = k & 1;
        const uint32_t base = ring + g * kPipeBytes, bit = (bits >> g) & 1u;
        if constexpr (kPair) {            // rows of P that warps of the other CTA have written
          if (!mbar_wait_cluster(bar(g, AB_P_FULL), bit, ctl, 512 + g)) break;
        } else {
          if (!mbar_wait_hot(bar(g, AB_P_FULL), bit, ctl, 512 + g)) break;
        }
        if (!mbar_wait_hot(bar(g, AB_V_FULL), bit, ctl, 514 + g)) break;
        tc_fence_after_sync();
        // O = P V: K = 128 keys = two chunks of 64; V is an MN-major B operand (16 keys = 2048 B per step)
        if constexpr (kPair) {
          const uint32_t d = tmem + g * 256;                   // over the scores, which the softmax has consumed
          umma_f16_k64_pair(d, umma_desc_lo(base + 3 * kATileBytes, 16), umma_desc_lo(base + 2 * kATileBytes, 8192), 128u, idesc_o, 0u);
          umma_f16_k64_pair(d, umma_desc_lo(base + 4 * kATileBytes, 16), umma_desc_lo(base + 2 * kATileBytes + 8192, 8192), 128u,
                            idesc_o, 1u);
          umma_commit_pair(bar(g, AB_O_FULL));
          umma_commit_pair(bar(g, AB_V_EMPTY));
        } else {
          const uint32_t d = tmem + kPipeOCol + g * 64;
          umma_f16_k64(d, umma_desc_lo(base + 3 * kATileBytes, 16), umma_desc_lo(base + 2 * kATileBytes, 8192), 128u, idesc_o, 0u);
          umma_f16_k64(d, umma_desc_lo(base + 4 * kATileBytes, 16), umma_desc_lo(base + 2 * kATileBytes + 8192, 8192), 128u,
                       idesc_o, 1u);
          umma_commit(bar(g, AB_O_FULL));
          umma_commit(bar(g, AB_V_EMPTY));
        }
        bits ^= 1u << g;
        if (k + 2 < my_items) {
          if constexpr (kPair) {          // the next scores of this pipeline overwrite the output just issued: wait for its readers
            if (!mbar_wait_hot(oempty0 + 8 * g, (obits >> g) & 1u, ctl, 516 + g)) break;
            tc_fence_after_sync();
          }
          issue_s(k + 2);
        }
        obits ^= 1u << g;                 // one phase of o_empty per item, waited for or not
      }
      rs.attn_bit = bits & 1u;
      rs.attn_bit1 = (bits >> 1) & 1u;
      rs.o_bits = obits;
    }
    __syncwarp();
  } else if (warp < 2 + kEpiWarps) {
    const int g = (warp - 2) >> 2, q = warp & 3;
    const int r_in = q * 32 + lane;
    const uint32_t tmem = ctl_s.tmem_base + ((uint32_t)(q * 32) << 16);
    const float sl2 = st.scale * 1.4426950408889634f;
    const float mask_l2 = -10000.0f * 1.4426950408889634f;
    const int* lens = p.lens;
    __half* probs = reinterpret_cast<__half*>(st.probs);
    const CUtensorMap* tm_out = map_ptr(ca, st.tm_out);
    StoreBoxes sb;                                            // a row's 64 columns are two boxes
    sb.base = boxes + epi_box(warp) * kStageWarp;
    sb.box = 0;
    sb.n = 2;
    uint8_t* pbase = ring_ptr + g * kPipeBytes + 3 * kATileBytes + r_in * 128;
    uint32_t bit = g ? rs.attn_bit1 : rs.attn_bit;
    const bool prof = p.prof != nullptr;
    long long t_ws = 0, t_sm = 0, t_wo = 0, t_ep = 0, t_p1 = 0;
    for (int k = g; k < my_items; k += 2) {
      const int item = item_of(k);
      const int b = seq_of(item), h = item - b * H;
      const int kv_len = lens ? lens[b] : S;
      const long long c0 = prof ? clock64() : 0;
      if (!mbar_wait_warp(bar(g, AB_S_FULL), bit, ctl, 520 + g, lane)) break;
      const long long c1 = prof ? clock64() : 0;
      tc_fence_after_sync();
      const uint32_t ts = kPair ? tmem + g * 256 + rank * 128 : tmem + g * 128;
      // Masked keys (>= kv_len) get -10000 added, which underflows to probability 0 in fp32 and never wins
      // the maximum, so both passes only visit the 32-column blocks that hold valid keys.  The next block is requested as soon
      // as this one's values have been used (16 columns at a time left the exponentials waiting for one another: softmax of
      // 64 x 128 4.0 k cycles an item).
      const int kvl = kv_len < 1 ? 1 : (kv_len > S ? S : kv_len);
      const int nb = (kvl + 31) >> 5;
      uint32_t r[32];
      // ---- pass 1: row maximum of the raw scores of the valid keys (the scale is positive) ----
      float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
      auto max32 = [&](int blk) {
        const int left = kvl - blk * 32;
        if (left >= 32) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            m0 = fmaxf(m0, fmaxf(__uint_as_float(r[i]), __uint_as_float(r[i + 4])));
            m1 = fmaxf(m1, fmaxf(__uint_as_float(r[i + 1]), __uint_as_float(r[i + 5])));
            m2 = fmaxf(m2, fmaxf(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 6])));
            m3 = fmaxf(m3, fmaxf(__uint_as_float(r[i + 3]), __uint_as_float(r[i + 7])));
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            m0 = fmaxf(m0, i < left ? __uint_as_float(r[i]) : -INFINITY);
            m1 = fmaxf(m1, i + 1 < left ? __uint_as_float(r[i + 1]) : -INFINITY);
          }
        }
        if (left > 32) tmem_ld32(ts + (blk + 1) * 32, r);
      };
      tmem_ld32(ts, r);
#pragma unroll 1
      for (int blk = 0; blk < nb; ++blk) {
        tmem_ld_wait(r);
        max32(blk);
      }
      const float mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3)) * sl2;
      const long long c1a = prof ? clock64() : 0;
      // ---- pass 2: unnormalised probabilities -> fp16 A-operand tile (128B-swizzled rows) ----
      float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
      auto exp32 = [&](int blk) {
        const int left = kvl - blk * 32;
        uint32_t w[16];
        if (left >= 32) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float p0 = ex2_fast(fmaf(__uint_as_float(r[i]), sl2, -mx)), p1 = ex2_fast(fmaf(__uint_as_float(r[i + 1]), sl2, -mx));
            const float p2 = ex2_fast(fmaf(__uint_as_float(r[i + 2]), sl2, -mx)), p3 = ex2_fast(fmaf(__uint_as_float(r[i + 3]), sl2, -mx));
            s0 += p0; s1 += p1; s2 += p2; s3 += p3;
            w[i >> 1] = pack_h2(p0, p1);
            w[(i >> 1) + 1] = pack_h2(p2, p3);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float p0 = i < left ? ex2_fast(fmaf(__uint_as_float(r[i]), sl2, -mx)) : 0.f;
            const float p1 = i + 1 < left ? ex2_fast(fmaf(__uint_as_float(r[i + 1]), sl2, -mx)) : 0.f;
            s0 += p0; s1 += p1;
            w[i >> 1] = pack_h2(p0, p1);
          }
        }
        if (left > 32) tmem_ld32(ts + (blk + 1) * 32, r);
        uint8_t* base = pbase + (blk >> 1) * kATileBytes;
        const int j = (blk & 1) * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(base + (((j + i) ^ (r_in & 7)) << 4)) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
      };
      tmem_ld32(ts, r);
#pragma unroll 1
      for (int blk = 0; blk < nb; ++blk) {
        tmem_ld_wait(r);
        exp32(blk);
      }
      for (int blk = nb; blk < 4; ++blk) {                    // keys past the valid ones: probability 0
        uint8_t* base = pbase + (blk >> 1) * kATileBytes;
        const int j = (blk & 1) * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(base + (((j + i) ^ (r_in & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
      }
      const float inv = 1.0f / ((s0 + s1) + (s2 + s3));
      if (probs) {                                            // parity output: normalised probabilities
        attn_store_probs_staged(ts, sb.base, probs + (size_t)(b * H + h) * S * S, q * 32, S, kv_len, sl2, mask_l2, mx, inv, lane);
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      if constexpr (kPair) {                                  // one arrival per warp on the leader's barrier (8 in all)
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_shared_rank(bar(g, AB_P_FULL), 0));
      } else {
        mbar_arrive(bar(g, AB_P_FULL));
      }
      const long long c2 = prof ? clock64() : 0;
      if (!mbar_wait_warp(bar(g, AB_O_FULL), bit, ctl, 522 + g, lane)) break;
      const long long c3 = prof ? clock64() : 0;
      tc_fence_after_sync();
#pragma unroll
      for (int half = 0; half < 2; ++half) {                  // (no plain stores: a pair's arrivals would wait for them)
        uint32_t w[16];
        tmem_ld32((kPair ? tmem + g * 256 + rank * 64 : tmem + kPipeOCol + g * 64) + half * 32, r);
        tmem_ld_wait(r);
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = pack_h2(__uint_as_float(r[2 * i]) * inv, __uint_as_float(r[2 * i + 1]) * inv);
        store_box(sb, w, lane, [&](uint32_t buf) {
          // 16 rows of the block where the sequence ends inside it
          const int row0 = q * 32, y = b * S + row0, x = h * 64 + half * 32;
          if (row0 < S) tma_store_2d(tm_out, buf, x, y);
          if (st.out_stores == 2 && row0 + 16 < S) tma_store_2d(tm_out, buf + 16 * kStageRow, x, y + 16);
        });
      }
      tc_fence_before_sync();
      if constexpr (kPair) {                                  // this warp has read its rows of the output accumulator
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(map_shared_rank(oempty0 + 8 * g, 0));
      }
      bit ^= 1u;
      if (prof) { const long long c4 = clock64(); t_ws += c1 - c0; t_sm += c2 - c1; t_wo += c3 - c2; t_ep += c4 - c3; t_p1 += c1a - c1; }
    }
    if (prof && warp == 2 && lane == 0) {  // [3] waiting for scores, [4] softmax, [5] waiting for P.V, [6] output
      long long* pr = p.prof + ((size_t)st.position * gridDim.x + blockIdx.x) * kProfSlots;
      pr[3] = t_ws; pr[4] = t_sm; pr[5] = t_wo; pr[6] = t_ep; pr[7] = t_p1;
    }
    if (elect_one()) {                     // the stores are complete before the CTA reports the stage done
      bulk_wait_group_all();
      fence_proxy_async_global();
    }
    __syncwarp();
    if (g) rs.attn_bit1 = bit; else rs.attn_bit = bit;
    // the other pipeline's bit advances with that pipeline's item count
    const int n_other = (my_items + (g ? 1 : 0)) >> 1;        // items handled by pipeline 1-g
    if (g) rs.attn_bit ^= (uint32_t)(n_other & 1); else rs.attn_bit1 ^= (uint32_t)(n_other & 1);
  }
}

// ------------------------------------------------------------------------------------
// Swin window attention.  The rows of Q, K and V, side by side in [tokens][3 C], and of the output are in the order of the block's
// windows, win * win rows each, with the heads side by side in C.  Seen as [windows][win * win][columns], a box of 64 rows of one window x 64
// columns of a PAIR of 32-wide heads is a tile whose rows past the window read as zero and are not written.  A work item is n
// consecutive windows x n heads:
// n = 2  group g of four softmax warps takes head 2 c + g; its upper 64 rows are the first window, the lower 64 the second,
//        and every product is issued once per window (the rows of the other window in it are dropped), so all eight warps
//        have rows of their own and a CTA has four (window, head) problems in flight;
// n = 1  one (window, head): half of group 0's rows are padding and group 1 is idle, but no warp waits for another head.
// The host takes n = 1 while that gives every CTA one item at most.  Two blocks and a merge, n = 1 -> 2: 16 x 28 x 28 x 256
// (2048 problems) 281 -> 238 us, 4 x 56 x 56 x 128 (1024) 185 -> 166, 18 blocks of 4 x 14 x 14 x 512 (256) 860 -> 831; below
// one item per CTA the other way round: 6 blocks of 5 x 7 x 7 x 768 (120) 262 against 280, 2 of 14 x 14 x 512 (64) 79 against 82.
// The MMAs of head h read their half of every 128-byte row (K-major operands: descriptor start +64 B for odd heads)
// or their half of the output columns (P.V is computed for the pair, the other half is dropped).
// Scores get the relative-position bias of the (query, key) offset and, for shifted windows, -100 where
// query and key come from different sides of the wrap-around.  Slots >= win*win are padding.
// ------------------------------------------------------------------------------------
// Softmax of one query row of a WS x WS window (thread = row, `r_in` = row of the window, `live` = the window exists):
// reads the 64 score columns from TMEM, adds bias and shift mask, writes the unnormalised probabilities as an fp16
// A-operand row (128B swizzle) and returns their sum.  Rows and keys >= WS*WS are padding (probability 0).
template <int WS>
__device__ __forceinline__ float swin_softmax_row(uint32_t tmem, const float* bias_s, uint8_t* prow, int r_in, bool live, int wy, int wx,
                                                  int R, int shift, float sl2) {
  constexpr int NT = WS * WS, TBL = 2 * WS - 1;
  const bool rowok = live && r_in < NT;
  const int qy = rowok ? r_in / WS : 0, qx = rowok ? r_in - qy * WS : 0;
  // region of a shifted coordinate along one axis: 0 | 1 | 2 (only the last window row/column mixes regions)
  int regy[WS], regx[WS];
#pragma unroll
  for (int i = 0; i < WS; ++i) {
    const int sy = wy + i, sx = wx + i;
    regy[i] = shift ? (sy < R - WS ? 0 : (sy < R - shift ? 1 : 2)) : 0;
    regx[i] = shift ? (sx < R - WS ? 0 : (sx < R - shift ? 1 : 2)) : 0;
  }
  int qreg = 0;
#pragma unroll
  for (int i = 0; i < WS; ++i) {
    if (i == qy) qreg += regy[i] * 3;
    if (i == qx) qreg += regx[i];
  }
  const float* brow = bias_s + (qy + WS - 1) * TBL + (qx + WS - 1);   // bias index = brow[-(ky*TBL + kx)]
  const float mask = -100.0f * 1.4426950408889634f;
  uint32_t r0[32], r1[32];
  tmem_ld32(tmem, r0);
  tmem_ld32(tmem + 32, r1);
  tmem_ld_wait(r0);
  tmem_ld_wait(r1);
  float mx = -INFINITY;
#pragma unroll
  for (int k = 0; k < 64; ++k) {
    if (k < NT) {
      constexpr int dummy = 0; (void)dummy;
      const int ky = k / WS, kx = k % WS;
      float v = __uint_as_float(k < 32 ? r0[k & 31] : r1[k & 31]) * sl2 + brow[-(ky * TBL + kx)];
      if (regy[ky] * 3 + regx[kx] != qreg) v += mask;
      if (k < 32) r0[k & 31] = __float_as_uint(v); else r1[k & 31] = __float_as_uint(v);
      mx = fmaxf(mx, v);
    }
  }
  float sum = 0.f;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint32_t wv[16];
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const int k = half * 32 + i;
      const float p0 = (k < NT && rowok) ? ex2_fast(__uint_as_float(half ? r1[i] : r0[i]) - mx) : 0.f;
      const float p1 = (k + 1 < NT && rowok) ? ex2_fast(__uint_as_float(half ? r1[i + 1] : r0[i + 1]) - mx) : 0.f;
      sum += p0 + p1;
      wv[i >> 1] = pack_h2(p0, p1);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<uint4*>(prow + (((half * 4 + j) ^ (r_in & 7)) << 4)) = make_uint4(wv[4 * j], wv[4 * j + 1], wv[4 * j + 2], wv[4 * j + 3]);
  }
  return rowok ? sum : 1.0f;
}

__device__ __noinline__ uint32_t attn_swin_stage(const Stage& st, const CallArgs& ca, SmemCtl& ctl_s, uint32_t ring, uint8_t* ring_ptr,
                                uint8_t* boxes, uint32_t state, const WaitCtl& ctl, int warp, int lane) {
  RoleState rs = RoleState::unpack(state);
  const int R = st.seq, ws = st.win, shift = st.shift, H = st.heads, C = st.ldo;
  const int nwr = st.nwr, nw_img = nwr * nwr, n_windows = st.batch * nw_img, n_tok = ws * ws;
  const uint32_t n = (uint32_t)st.bn;                                // windows and heads per item: 1 or 2
  const int item_h = H / (int)n, items = (n_windows + (int)n - 1) / (int)n * item_h;
  auto wp_of = [&](int item) -> int { return (int)fast_div((uint32_t)item, (uint32_t)item_h, st.mg_heads); };
  // scores, probabilities and output have barriers per head (bar(g, ...)), the loads one set; all phases advance once per item
  const uint32_t bar0 = smem_u32(&ctl_s.qk_full), bar1 = smem_u32(&ctl_s.attn1[0]);
  auto bar = [&](int g, int which) -> uint32_t { return (g ? bar1 : bar0) + 8u * (uint32_t)which; };
  const uint32_t qk_full = bar(0, AB_QK_FULL), qk_empty = bar(0, AB_QK_EMPTY), v_full = bar(0, AB_V_FULL), v_empty = bar(0, AB_V_EMPTY);
  // shared memory: Q 16 KiB | K 16 KiB | V 16 KiB | P of head 0 16 KiB | P of head 1 16 KiB | bias tables
  // TMEM: scores of (head g, window j) at column 64 (2 g + j), outputs 256 further on
  if (warp == 0) {
    if (elect_one()) {
      const CUtensorMap* tm = map_ptr(ca, st.tm_qkv);
      uint32_t bit = rs.attn_bit;
      int wp = wp_of((int)blockIdx.x), col = (((int)blockIdx.x - wp * item_h) * (int)n >> 1) * 64;
      const bool ok = grid_wait(ca.p, ctl, st);
      if (ok && st.dead_bytes[0]) publish_go(ctl_s, st.ordinal);
      for (int item = blockIdx.x; ok && item < items;) {
        if (!mbar_wait_hot(qk_empty, bit ^ 1u, ctl, 530)) break;
        mbar_expect_tx(qk_full, n * kATileBytes);                    // two tiles of n windows of 64 rows
        tma_load_3d(ring, tm, qk_full, col, 0, wp * (int)n);
        tma_load_3d(ring + kATileBytes, tm, qk_full, C + col, 0, wp * (int)n);
        if (!mbar_wait_hot(v_empty, bit ^ 1u, ctl, 531)) break;
        mbar_expect_tx(v_full, n * (kATileBytes / 2));
        tma_load_3d(ring + 2 * kATileBytes, tm, v_full, 2 * C + col, 0, wp * (int)n);
        bit ^= 1u;
        item += gridDim.x;
        wp = wp_of(item);
        col = ((item - wp * item_h) * (int)n >> 1) * 64;
      }
      rs.attn_bit = bit;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc_s = umma_idesc_f16(64u, 0u), idesc_o = umma_idesc_f16(64u, 1u);
      const uint32_t tmem = ctl_s.tmem_base, q_lo = umma_desc_lo(ring, 16), k_lo = umma_desc_lo(ring + kATileBytes, 16);
      const uint64_t hi = (uint64_t)kDescHiSw128 << 32;
      uint32_t bit = rs.attn_bit;
      for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const uint32_t odd = n == 1 ? (uint32_t)(item - wp_of(item) * item_h) & 1u : 0u;       // a single head may be the pair's second
        if (!mbar_wait_hot(qk_full, bit, ctl, 532)) break;
        tc_fence_after_sync();
#pragma unroll 1
        for (uint32_t g = 0; g < n; ++g) {
          // S[128 x 64] = Q_h K_h^T per window, K = 32: two K=16 steps; head g starts 64 bytes into every row, window j
          // 64 rows (8 KiB) into the K tile
          const uint64_t qd = hi | (q_lo + 4u * (g + odd));
#pragma unroll 1
          for (uint32_t j = 0; j < n; ++j) {
            const uint64_t kd = hi | (k_lo + j * (8192u >> 4) + 4u * (g + odd));
            const uint32_t d = tmem + (2u * g + j) * 64u;
            umma_f16(d, qd, kd, idesc_s, 0u);
            umma_f16(d, qd + 2u, kd + 2u, idesc_s, 1u);
          }
          umma_commit(bar((int)g, AB_S_FULL));
        }
        umma_commit(qk_empty);
        if (!mbar_wait_hot(v_full, bit, ctl, 534)) break;
        bool ok = true;
#pragma unroll 1
        for (uint32_t g = 0; g < n; ++g) {
          ok = mbar_wait_hot(bar((int)g, AB_P_FULL), bit, ctl, 533);
          if (!ok) break;
          tc_fence_after_sync();
          // O[128 x 64] = P[128 x 64 keys] V_pair[64 keys x 64] per window: one K chunk of 64
#pragma unroll 1
          for (uint32_t j = 0; j < n; ++j)
            umma_f16_k64(tmem + 256u + (2u * g + j) * 64u, umma_desc_lo(ring + (3u + g) * kATileBytes, 16),
                         umma_desc_lo(ring + 2 * kATileBytes + j * 8192u, 8192), 128u, idesc_o, 0u);
          umma_commit(bar((int)g, AB_O_FULL));
        }
        if (!ok) break;
        umma_commit(v_empty);
        bit ^= 1u;
      }
      rs.attn_bit = bit;
    }
    __syncwarp();
  } else if (warp < 2 + (int)n * 4) {
    const int grp = (warp - 2) >> 2, q = warp & 3, r_in = q * 32 + lane;
    const int j = q >> 1, row = r_in & 63;                           // window of the item, row of the window
    const uint32_t tmem = ctl_s.tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(2 * grp + j) * 64u;
    const float sl2 = st.scale * 1.4426950408889634f, l2e = 1.4426950408889634f;
    const __half* table = reinterpret_cast<const __half*>(st.rel_bias);
    const CUtensorMap* tm_out = map_ptr(ca, st.tm_out);
    const int tbl2 = (2 * ws - 1) * (2 * ws - 1);                    // at most 225
    float* bias_s = reinterpret_cast<float*>(ring_ptr + 5 * kATileBytes) + grp * 256;      // this head's column of the bias table (x log2 e)
    uint8_t* prow = ring_ptr + (3 + grp) * kATileBytes + r_in * 128;
    StoreBoxes sb;
    sb.base = boxes + epi_box(warp) * kStageWarp;
    sb.box = 0;
    sb.n = 2;
    // the table's column of the next item is requested while this one is worked on
    auto load_bias = [&](int i, int h) -> float { return i < tbl2 ? __half2float(__ldg(table + i * H + h)) * l2e : 0.0f; };
    int wp = wp_of((int)blockIdx.x), h = (int)n * ((int)blockIdx.x - wp * item_h) + grp;
    float b0 = 0.0f, b1 = 0.0f;
    if ((int)blockIdx.x < items) { b0 = load_bias(r_in, h); b1 = load_bias(r_in + 128, h); }
    bool ok = true;                                                  // false: given up, see attn_stage
#pragma unroll 1
    for (int item = blockIdx.x; item < items;) {
      const int wg = (int)n * wp + j;
      const int w = wg - (int)fast_div((uint32_t)wg, (uint32_t)nw_img, st.mg_nwr2) * nw_img;
      const bool live = j < (int)n && wg < n_windows;                // an odd number of windows: the last item has one
      const int wrow = (int)fast_div((uint32_t)w, (uint32_t)nwr, st.mg_nwr), wy = wrow * ws, wx = (w - wrow * nwr) * ws;
      named_barrier_sync(2 + grp, 128);                              // previous item's readers are done with bias_s
      bias_s[r_in] = b0;
      bias_s[r_in + 128] = b1;
      named_barrier_sync(2 + grp, 128);
      const int this_h = h;
      item += gridDim.x;
      wp = wp_of(item);
      h = (int)n * (item - wp * item_h) + grp;
      if (item < items) { b0 = load_bias(r_in, h); b1 = load_bias(r_in + 128, h); }
      ok = ok && mbar_wait_warp(bar(grp, AB_S_FULL), rs.attn_bit, ctl, 535, lane);
      tc_fence_after_sync();
      float sum = 1.0f;
      if (ws == 7) sum = swin_softmax_row<7>(tmem, bias_s, prow, row, live, wy, wx, R, shift, sl2);
      else sum = swin_softmax_row<8>(tmem, bias_s, prow, row, live, wy, wx, R, shift, sl2);
      const float inv = 1.0f / sum;
      fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive(bar(grp, AB_P_FULL));
      ok = ok && mbar_wait_warp(bar(grp, AB_O_FULL), rs.attn_bit, ctl, 536, lane);
      tc_fence_after_sync();
      {
        uint32_t o[32], wv[16];
        tmem_ld32(tmem + 256u + (uint32_t)(this_h & 1) * 32u, o);
        tmem_ld_wait(o);
#pragma unroll
        for (int i = 0; i < 16; ++i) wv[i] = pack_h2(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv);
        store_box(sb, wv, lane, [&](uint32_t buf) {                   // (rows past the window are outside the map's extent)
          if (ok && live && (q & 1) * 32 < n_tok) tma_store_3d(tm_out, buf, this_h * 32, (q & 1) * 32, wg);
        });
      }
      tc_fence_before_sync();
      rs.attn_bit ^= 1u;
    }
    if (elect_one()) {                     // the stores are complete before the CTA reports the stage done
      bulk_wait_group_all();
      fence_proxy_async_global();
    }
    __syncwarp();
  }
  return rs.pack();
}

// Intermediates that the previous stage read for the last time (the barrier behind it has been passed by every CTA):
// this CTA's share of their lines is dropped from L2 before anything evicts them to DRAM.  Out of line: a few
// instructions per thread and stage, whose registers are not charged to the stages.
// Threads tid0 .. tid0 + nthr - 1 of every CTA share the work: all of them in a LayerNorm stage, a spare warp in the other
// stages.
__device__ __noinline__ void drop_dead_buffers(const Stage& st, int tid0, int nthr) {
  const int tid = (int)threadIdx.x - tid0;
#pragma unroll 1
  for (int b = 0; b < 2; ++b) {
    const uint32_t lines = st.dead_bytes[b] >> 7;
    if (!lines) continue;
    const char* base = reinterpret_cast<const char*>(st.dead_ptr[b]);
    for (uint32_t i = blockIdx.x * nthr + tid; i < lines; i += gridDim.x * nthr) discard_l2_128(base + ((size_t)i << 7));
  }
}

// ------------------------------------------------------------------------------------
// LayerNorm stages: z = sum of planes + bias + residual, two-pass statistics (or their merged equivalent) in fp32, fp16 output.
// Rows are read straight from L2, except the patch-merging form (ln_stage_ool), whose rows are gathered from four tokens each by
// bulk copies into a ring of batches in shared memory.
// ------------------------------------------------------------------------------------
// Two gathered rows per call (the second optional): their instruction streams interleave, which hides the
// shared-memory, shuffle and MUFU latencies a single row's dependent chain exposes.
template <int NJ>
__device__ __forceinline__ void ln_rows2(const __half* row0, const __half* row1, const __half* gamma, const __half* beta, float eps,
                                         __half* out0, __half* out1, int lane) {
  const bool two = out1 != nullptr;
  float z[2][NJ][4];
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint2 u = r == 0 || two ? *reinterpret_cast<const uint2*>((r ? row1 : row0) + (lane + 32 * j) * 4) : make_uint2(0u, 0u);
      const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
      const float2 f1 = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
      z[r][j][0] = f0.x; z[r][j][1] = f0.y; z[r][j][2] = f1.x; z[r][j][3] = f1.y;
    }
  const float inv_n = 1.0f / (float)(NJ * 128);
  float sa = 0.0f, sb = 0.0f;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    sa += (z[0][j][0] + z[0][j][1]) + (z[0][j][2] + z[0][j][3]);
    sb += (z[1][j][0] + z[1][j][1]) + (z[1][j][2] + z[1][j][3]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sa += __shfl_xor_sync(0xffffffffu, sa, o);
    sb += __shfl_xor_sync(0xffffffffu, sb, o);
  }
  const float mean0 = sa * inv_n, mean1 = sb * inv_n;
  float va = 0.0f, vb = 0.0f;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float d0 = z[0][j][i] - mean0, d1 = z[1][j][i] - mean1;
      va = fmaf(d0, d0, va);
      vb = fmaf(d1, d1, vb);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    va += __shfl_xor_sync(0xffffffffu, va, o);
    vb += __shfl_xor_sync(0xffffffffu, vb, o);
  }
  const float rstd0 = rsqrtf(va * inv_n + eps), rstd1 = rsqrtf(vb * inv_n + eps);
  // (z - mean) * rstd in fp32 (one FMA), rounded to fp16 pairs; gamma and beta are applied on the pairs (one packed
  // FMA per two elements, no conversions).  With gamma = 1, beta = 0 that last step is exact.
  const float nm0 = -mean0 * rstd0, nm1 = -mean1 * rstd1;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    uint2 ug = make_uint2(0u, 0u), ub = make_uint2(0u, 0u);
    if (gamma) {
      ug = *reinterpret_cast<const uint2*>(gamma + (lane + 32 * j) * 4);
      ub = *reinterpret_cast<const uint2*>(beta + (lane + 32 * j) * 4);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (r == 1 && !two) break;
      const float rs_ = r ? rstd1 : rstd0, nm = r ? nm1 : nm0;
      uint32_t w0 = pack_h2(fmaf(z[r][j][0], rs_, nm), fmaf(z[r][j][1], rs_, nm));
      uint32_t w1 = pack_h2(fmaf(z[r][j][2], rs_, nm), fmaf(z[r][j][3], rs_, nm));
      if (gamma) {
        const __half2 y0 = __hfma2(*reinterpret_cast<const __half2*>(&w0), *reinterpret_cast<const __half2*>(&ug.x),
                                   *reinterpret_cast<const __half2*>(&ub.x));
        const __half2 y1 = __hfma2(*reinterpret_cast<const __half2*>(&w1), *reinterpret_cast<const __half2*>(&ug.y),
                                   *reinterpret_cast<const __half2*>(&ub.y));
        w0 = *reinterpret_cast<const uint32_t*>(&y0);
        w1 = *reinterpret_cast<const uint32_t*>(&y1);
      }
      *reinterpret_cast<uint2*>((r ? out1 : out0) + (lane + 32 * j) * 4) = make_uint2(w0, w1);
    }
  }
}

// Patch-merging gather (one lane): row (img, h, w) of the merged matrix = tokens (2h, 2w), (2h+1, 2w), (2h, 2w+1),
// (2h+1, 2w+1) of a [batch][R][R][N/4] fp16 grid side by side, one bulk copy each.
__device__ __noinline__ void ln_gather_rows(uint32_t dst, const __half* src, int row0, int rows, int N, int R, uint32_t bar) {
  const int R2 = R >> 1, Cq = N >> 2;
  for (int r = 0; r < rows; ++r) {
    const int gr = row0 + r, img = gr / (R2 * R2), rem = gr - img * R2 * R2, h2 = rem / R2, w2 = rem - h2 * R2;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const size_t token = (size_t)img * R * R + (size_t)(2 * h2 + (q & 1)) * R + (2 * w2 + (q >> 1));
      bulk_load(dst + (uint32_t)(r * N + q * Cq) * 2u, src + token * Cq, (uint32_t)(Cq * 2), bar);
    }
  }
}

// LayerNorm of one fp16 row of 2048 columns held in shared memory (the merged rows of a C = 512 stage): too wide
// for the two-rows-per-warp routine's registers.  Same arithmetic: two-pass fp32 statistics, packed-half affine.
__device__ __noinline__ void ln_row_wide(const __half* row, const __half* gamma, const __half* beta, float eps, __half* out, int lane) {
  constexpr int NJ = 16;
  float z[NJ][4];
  float sa = 0.0f;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const uint2 u = *reinterpret_cast<const uint2*>(row + (lane + 32 * j) * 4);
    const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
    const float2 f1 = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
    z[j][0] = f0.x; z[j][1] = f0.y; z[j][2] = f1.x; z[j][3] = f1.y;
    sa += (f0.x + f0.y) + (f1.x + f1.y);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sa += __shfl_xor_sync(0xffffffffu, sa, o);
  const float inv_n = 1.0f / (float)(NJ * 128), mean = sa * inv_n;
  float va = 0.0f;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float d0 = z[j][i] - mean;
      va = fmaf(d0, d0, va);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) va += __shfl_xor_sync(0xffffffffu, va, o);
  const float rstd = rsqrtf(va * inv_n + eps), nm = -mean * rstd;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    uint32_t w0 = pack_h2(fmaf(z[j][0], rstd, nm), fmaf(z[j][1], rstd, nm));
    uint32_t w1 = pack_h2(fmaf(z[j][2], rstd, nm), fmaf(z[j][3], rstd, nm));
    if (gamma) {
      // plain loads: the vectors may have been staged in shared memory by the caller
      const uint2 ug = *reinterpret_cast<const uint2*>(gamma + (lane + 32 * j) * 4);
      const uint2 ub = *reinterpret_cast<const uint2*>(beta + (lane + 32 * j) * 4);
      const __half2 y0 = __hfma2(*reinterpret_cast<const __half2*>(&w0), *reinterpret_cast<const __half2*>(&ug.x),
                                 *reinterpret_cast<const __half2*>(&ub.x));
      const __half2 y1 = __hfma2(*reinterpret_cast<const __half2*>(&w1), *reinterpret_cast<const __half2*>(&ug.y),
                                 *reinterpret_cast<const __half2*>(&ub.y));
      w0 = *reinterpret_cast<const uint32_t*>(&y0);
      w1 = *reinterpret_cast<const uint32_t*>(&y1);
    }
    *reinterpret_cast<uint2*>(out + (lane + 32 * j) * 4) = make_uint2(w0, w1);
  }
}

// Rows read straight from L2.  W = N / 256 warps share a row (one for a row of 128 columns): lane l of part w holds columns
// 256 w + 4 l .. + 3 and those 128 further on.  So 12 / W rows are in flight per CTA, dealt out over the CTAs first.  What a row
// costs is latency: one L2 round trip for its planes, then a dependent chain in code that is cold when a CTA has one row, and
// both the chain and the code grow with the columns a lane holds; with fewer columns than eight the shuffles of all the warps
// cost more than they save.  The next row's loads are issued as soon as this row's sum is formed, and bias, gamma and beta are
// loaded once per stage, in front of the wait for the stage's start.  Sets of columns are merged as (mean, squared deviations
// from it), which is as exact as a second pass over the row (Chan, Golub, LeVeque) and needs one chain of shuffles and one
// exchange between the parts.
// `red`: 192 bytes of shared memory.
template <bool kPermute>
__device__ __forceinline__ void ln_shared_rows(const Stage& st, const MegaParams& p, SmemCtl& cs, float2* red, const WaitCtl& ctl, int warp, int lane) {
  constexpr int NJ = 2, kG = 2;                           // blocks of 128 columns per warp, planes in flight at once
  const int N = st.N, M = st.M, P = st.n_partial, W = st.splitk, G = (kThreads / 32) / W;
  const int grp = (int)fast_div((uint32_t)warp, (uint32_t)W, st.mg_splitk), part = warp - grp * W;
  const int col = part * NJ * 128 + lane * 4;
  const bool both = N > 128;
  const size_t plane = (size_t)M * N;
  const float* planes = st.partial + col;
  const __half* resid = reinterpret_cast<const __half*>(sel_ptr(st.resid_sel, st.resid, p));
  __half* out = reinterpret_cast<__half*>(const_cast<void*>(sel_ptr(st.out_sel, st.out, p))) + col;
  __half* sum_out = st.sum_out ? reinterpret_cast<__half*>(st.sum_out) + col : nullptr;
  const float eps = st.eps;
  const int step = (int)gridDim.x * G;
  int row = grp < G ? grp * (int)gridDim.x + (int)blockIdx.x : M;
  uint2 ub[NJ], ug[NJ], ubt[NJ], ur[NJ];
  float4 v[kG][NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const __half *bias = reinterpret_cast<const __half*>(st.bias), *gamma = reinterpret_cast<const __half*>(st.gamma),
                 *beta = reinterpret_cast<const __half*>(st.beta);
    ub[j] = bias && (j == 0 || both) ? __ldg(reinterpret_cast<const uint2*>(bias + col + 128 * j)) : make_uint2(0u, 0u);
    ug[j] = gamma && (j == 0 || both) ? __ldg(reinterpret_cast<const uint2*>(gamma + col + 128 * j)) : make_uint2(0u, 0u);
    ubt[j] = gamma && (j == 0 || both) ? __ldg(reinterpret_cast<const uint2*>(beta + col + 128 * j)) : make_uint2(0u, 0u);
  }
  const bool affine = st.gamma != nullptr;
  const float inv_n = 1.0f / (float)N;
  red += grp * W;
  if (!stage_go(p, cs, st, ctl, warp, lane)) return;
  auto load_planes = [&](int r, int g0) {
    const float* src = planes + (size_t)r * N + (size_t)g0 * plane;
#pragma unroll
    for (int g = 0; g < kG; ++g, src += plane)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        v[g][j] = g0 + g < P && (j == 0 || both) ? __ldcg(reinterpret_cast<const float4*>(src + 128 * j)) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  auto load_row = [&](int r) {
    load_planes(r, 0);
#pragma unroll
    for (int j = 0; j < NJ; ++j)
      ur[j] = resid && (j == 0 || both) ? __ldcg(reinterpret_cast<const uint2*>(resid + (size_t)r * N + col + 128 * j)) : make_uint2(0u, 0u);
  };
  if (row < M) load_row(row);
  if (st.dead_bytes[0]) drop_dead_buffers(st, 0, kThreads);       // while the first rows are on their way
#pragma unroll 1
  for (uint32_t turn = 0; row < M; row += step, turn ^= 1u) {
    float z[NJ][4];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const float2 b0 = __half22float2(*reinterpret_cast<const __half2*>(&ub[j].x)), b1 = __half22float2(*reinterpret_cast<const __half2*>(&ub[j].y));
      const float2 r0 = __half22float2(*reinterpret_cast<const __half2*>(&ur[j].x)), r1 = __half22float2(*reinterpret_cast<const __half2*>(&ur[j].y));
      z[j][0] = b0.x + r0.x; z[j][1] = b0.y + r0.y; z[j][2] = b1.x + r1.x; z[j][3] = b1.y + r1.y;
    }
#pragma unroll 1
    for (int g0 = 0;;) {                                  // deep splits: further rounds
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int g = 0; g < kG; ++g) { z[j][0] += v[g][j].x; z[j][1] += v[g][j].y; z[j][2] += v[g][j].z; z[j][3] += v[g][j].w; }
      g0 += kG;
      if (g0 >= P) break;
      load_planes(row, g0);
    }
    if (row + step < M) load_row(row + step);
    const size_t to = (size_t)(kPermute ? ln_out_row(st, row) : row) * N;
    __half* o = out + to;
    if (eps < 0.0f || sum_out) {        // the sum itself, as fp16; what is normalised below is the rounded value
      __half* so = eps < 0.0f ? o : sum_out + to;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const uint2 w = make_uint2(pack_h2(z[j][0], z[j][1]), pack_h2(z[j][2], z[j][3]));
        if (j == 0 || both) *reinterpret_cast<uint2*>(so + 128 * j) = w;
        const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), f1 = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
        z[j][0] = f0.x; z[j][1] = f0.y; z[j][2] = f1.x; z[j][3] = f1.y;
      }
      if (eps < 0.0f) continue;         // sum only
    }
    // (mean, sum of squared deviations from it) of the lane's columns, then of twice as many with every step: a pair of
    // equally large sets has the mean of the means, and its deviations grow by (difference of the means)^2 n / 2
    float row_mean = 0.0f, va = 0.0f;
#pragma unroll
    for (int j = 0; j < NJ; ++j) row_mean += (z[j][0] + z[j][1]) + (z[j][2] + z[j][3]);
    row_mean *= both ? 0.125f : 0.25f;
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float d = z[j][i] - row_mean;
        if (j == 0 || both) va = fmaf(d, d, va);
      }
    const float half_n = both ? 4.0f : 2.0f;
#pragma unroll
    for (int o2 = 1; o2 < 32; o2 <<= 1) {
      const float m2 = __shfl_xor_sync(0xffffffffu, row_mean, o2), v2 = __shfl_xor_sync(0xffffffffu, va, o2);
      const float d = m2 - row_mean;
      va = fmaf(d * d, half_n * (float)o2, va + v2);
      row_mean = 0.5f * (row_mean + m2);
    }
    if (W > 1) {
      float2* slot = red + turn * (kThreads / 32);        // two sets, used by alternate rows: one barrier per row is enough
      if (lane == 0) slot[part] = make_float2(row_mean, va);
      named_barrier_sync(4 + grp, W * 32);
      float2 t[8];                                        // W <= 8
      float total = 0.0f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        t[i] = i < W ? slot[i] : make_float2(0.f, 0.f);
        total += t[i].x;
      }
      row_mean = total * ((float)(NJ * 128) * inv_n);
      va = 0.0f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float d = i < W ? t[i].x - row_mean : 0.0f;
        va += fmaf(d * d, (float)(NJ * 128), t[i].y);
      }
    }
    const float rstd = rsqrtf(va * inv_n + eps), nm = -row_mean * rstd;
    // (z - mean) * rstd in fp32 (one FMA), rounded to fp16 pairs; gamma and beta are applied on the pairs (one packed
    // FMA per two elements, no conversions).  With gamma = 1, beta = 0 that last step is exact.
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      uint32_t w0 = pack_h2(fmaf(z[j][0], rstd, nm), fmaf(z[j][1], rstd, nm));
      uint32_t w1 = pack_h2(fmaf(z[j][2], rstd, nm), fmaf(z[j][3], rstd, nm));
      if (affine) {
        const __half2 y0 = __hfma2(*reinterpret_cast<const __half2*>(&w0), *reinterpret_cast<const __half2*>(&ug[j].x),
                                   *reinterpret_cast<const __half2*>(&ubt[j].x));
        const __half2 y1 = __hfma2(*reinterpret_cast<const __half2*>(&w1), *reinterpret_cast<const __half2*>(&ug[j].y),
                                   *reinterpret_cast<const __half2*>(&ubt[j].y));
        w0 = *reinterpret_cast<const uint32_t*>(&y0);
        w1 = *reinterpret_cast<const uint32_t*>(&y1);
      }
      if (j == 0 || both) *reinterpret_cast<uint2*>(o + 128 * j) = make_uint2(w0, w1);
    }
  }
}

// The same for many rows per CTA: a warp per row, nothing exchanged between warps, twelve rows in flight (the form above has four of
// 768 columns and is bound by its chain: 64 sequences 21.2 k cycles a stage against 16.3 k).  Every round trip costs ~800 cycles,
// so the loads are issued in as few dependent rounds as the registers allow: bias, residual and the first planes
// together, further planes kG at a time, gamma and beta just before the statistics (they land while the shuffles run).
// With the loads strung one behind the other a row of six planes took 6.2 k cycles.
template <int NJ>
__device__ __forceinline__ void ln_row_alone(const float* pl, int n_partial, size_t plane_stride, const __half* res,
                                              const __half* bias, const __half* gamma, const __half* beta, float eps,
                                              __half* out, __half* sum_out, int lane) {
  constexpr int kG = NJ <= 4 ? 4 : (NJ <= 6 ? 3 : 2);      // planes in flight at once
  float z[NJ][4];
  {
    uint2 ub[NJ], ur[NJ];
    float4 v[kG][NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      ub[j] = bias ? __ldg(reinterpret_cast<const uint2*>(bias + (lane + 32 * j) * 4)) : make_uint2(0u, 0u);
      ur[j] = res ? __ldcg(reinterpret_cast<const uint2*>(res + (lane + 32 * j) * 4)) : make_uint2(0u, 0u);
    }
#pragma unroll
    for (int g = 0; g < kG; ++g)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        v[g][j] = g < n_partial ? __ldcg(reinterpret_cast<const float4*>(pl + (size_t)g * plane_stride + (lane + 32 * j) * 4))
                                : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const float2 b0 = __half22float2(*reinterpret_cast<const __half2*>(&ub[j].x)), b1 = __half22float2(*reinterpret_cast<const __half2*>(&ub[j].y));
      const float2 r0 = __half22float2(*reinterpret_cast<const __half2*>(&ur[j].x)), r1 = __half22float2(*reinterpret_cast<const __half2*>(&ur[j].y));
      z[j][0] = b0.x + r0.x; z[j][1] = b0.y + r0.y; z[j][2] = b1.x + r1.x; z[j][3] = b1.y + r1.y;
#pragma unroll
      for (int g = 0; g < kG; ++g) { z[j][0] += v[g][j].x; z[j][1] += v[g][j].y; z[j][2] += v[g][j].z; z[j][3] += v[g][j].w; }
    }
    for (int p0 = kG; p0 < n_partial; p0 += kG) {
#pragma unroll
      for (int g = 0; g < kG; ++g)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          v[g][j] = p0 + g < n_partial ? __ldcg(reinterpret_cast<const float4*>(pl + (size_t)(p0 + g) * plane_stride + (lane + 32 * j) * 4))
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int g = 0; g < kG; ++g) { z[j][0] += v[g][j].x; z[j][1] += v[g][j].y; z[j][2] += v[g][j].z; z[j][3] += v[g][j].w; }
    }
  }
  if (sum_out) {                        // the sum itself, as fp16; what is normalised below is the rounded value
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const uint2 w = make_uint2(pack_h2(z[j][0], z[j][1]), pack_h2(z[j][2], z[j][3]));
      *reinterpret_cast<uint2*>(sum_out + (lane + 32 * j) * 4) = w;
      const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), f1 = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
      z[j][0] = f0.x; z[j][1] = f0.y; z[j][2] = f1.x; z[j][3] = f1.y;
    }
    if (eps < 0.0f) return;             // sum only
  }
  uint2 ug[NJ], ubt[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    ug[j] = gamma ? __ldg(reinterpret_cast<const uint2*>(gamma + (lane + 32 * j) * 4)) : make_uint2(0u, 0u);
    ubt[j] = gamma ? __ldg(reinterpret_cast<const uint2*>(beta + (lane + 32 * j) * 4)) : make_uint2(0u, 0u);
  }
  const float inv_n = 1.0f / (float)(NJ * 128);
  float sa = 0.0f;
#pragma unroll
  for (int j = 0; j < NJ; ++j) sa += (z[j][0] + z[j][1]) + (z[j][2] + z[j][3]);
  sa = warp_sum(sa);
  const float mean = sa * inv_n;
  float va = 0.0f;
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float d0 = z[j][i] - mean;
      va = fmaf(d0, d0, va);
    }
  va = warp_sum(va);
  const float rstd = rsqrtf(va * inv_n + eps), nm = -mean * rstd;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    uint32_t w0 = pack_h2(fmaf(z[j][0], rstd, nm), fmaf(z[j][1], rstd, nm));
    uint32_t w1 = pack_h2(fmaf(z[j][2], rstd, nm), fmaf(z[j][3], rstd, nm));
    if (gamma) {
      const __half2 y0 = __hfma2(*reinterpret_cast<const __half2*>(&w0), *reinterpret_cast<const __half2*>(&ug[j].x),
                                 *reinterpret_cast<const __half2*>(&ubt[j].x));
      const __half2 y1 = __hfma2(*reinterpret_cast<const __half2*>(&w1), *reinterpret_cast<const __half2*>(&ug[j].y),
                                 *reinterpret_cast<const __half2*>(&ubt[j].y));
      w0 = *reinterpret_cast<const uint32_t*>(&y0);
      w1 = *reinterpret_cast<const uint32_t*>(&y1);
    }
    *reinterpret_cast<uint2*>(out + (lane + 32 * j) * 4) = make_uint2(w0, w1);
  }
}

// kNJ: the row's blocks of 128 columns, or 0: any.
template <int kNJ>
__device__ __forceinline__ void ln_lone_rows(const Stage& st, const MegaParams& p, SmemCtl& cs, const WaitCtl& ctl, int warp, int lane) {
  const int N = st.N, M = st.M, P = st.n_partial;
  const size_t plane = (size_t)M * N;
  const __half* resid = reinterpret_cast<const __half*>(sel_ptr(st.resid_sel, st.resid, p));
  __half* out = reinterpret_cast<__half*>(const_cast<void*>(sel_ptr(st.out_sel, st.out, p)));
  const __half* bias = reinterpret_cast<const __half*>(st.bias);
  const __half* gamma = reinterpret_cast<const __half*>(st.gamma);
  const __half* beta = reinterpret_cast<const __half*>(st.beta);
  if (!stage_go(p, cs, st, ctl, warp, lane)) return;
  if (st.dead_bytes[0]) drop_dead_buffers(st, 0, kThreads);
  for (int row = warp * (int)gridDim.x + (int)blockIdx.x; row < M; row += (int)gridDim.x * (kThreads / 32)) {
    const float* pl0 = st.partial + (size_t)row * N;
    const __half* ra = resid ? resid + (size_t)row * N : nullptr;
    __half* o0 = out + (size_t)row * N;
    __half* so = st.eps < 0.0f ? o0 : st.sum_out ? reinterpret_cast<__half*>(st.sum_out) + (size_t)row * N : nullptr;
    if constexpr (kNJ > 0) {
      ln_row_alone<kNJ>(pl0, P, plane, ra, bias, gamma, beta, st.eps, o0, so, lane);
      continue;
    }
    switch (N >> 7) {
      case 1: ln_row_alone<1>(pl0, P, plane, ra, bias, gamma, beta, st.eps, o0, so, lane); break;
      case 2: ln_row_alone<2>(pl0, P, plane, ra, bias, gamma, beta, st.eps, o0, so, lane); break;
      case 4: ln_row_alone<4>(pl0, P, plane, ra, bias, gamma, beta, st.eps, o0, so, lane); break;
      case 6: ln_row_alone<6>(pl0, P, plane, ra, bias, gamma, beta, st.eps, o0, so, lane); break;
      default: ln_row_alone<8>(pl0, P, plane, ra, bias, gamma, beta, st.eps, o0, so, lane); break;
    }
  }
}

// The LayerNorm stages of the builds, out of line: their registers are not charged to the stage interpreter.
__device__ __noinline__ void ln_stage_direct(const Stage& st, const MegaParams& p, SmemCtl& cs, float2* red, const WaitCtl& ctl, int warp, int lane) {
  ln_shared_rows<true>(st, p, cs, red, ctl, warp, lane);
}
__device__ __noinline__ void ln_stage_many(const Stage& st, const MegaParams& p, SmemCtl& cs, const WaitCtl& ctl, int warp, int lane) {
  ln_lone_rows<0>(st, p, cs, ctl, warp, lane);
}
// Both forms, for the build that runs long sequences as well as small batches.  Rows of 768 columns, which leave the shared form
// four in flight, go one to a warp where a CTA has more than 16 of them (layers of 256 tokens: at 13 rows per CTA 277.6 us shared,
// 277.8 alone, at 27 395.3 / 389.1, at 69 854.0 / 830.0, at 110 1358 / 1296); narrower rows and rows of 1024 columns are
// faster shared at any number (512 columns, 110 per CTA: 737.7 / 740.4; 256: 360.2 / 390.4; 1024: 2149 / 2197).  The
// lone form for all widths would spill here.
__device__ __noinline__ void ln_stage_either(const Stage& st, const MegaParams& p, SmemCtl& cs, float2* red, const WaitCtl& ctl, int warp, int lane) {
  if (st.N == 768 && st.M > 16 * (int)gridDim.x) ln_lone_rows<6>(st, p, cs, ctl, warp, lane);
  else ln_shared_rows<false>(st, p, cs, red, ctl, warp, lane);
}

// The patch-merging form (Swin, python/models/swin_transformer/swin_patch_merge.py:1-17): the fp16 input is a
// [batch][R][R][N/4] token grid (R = st.seq), and row (b, h, w) of the normalised matrix is the concatenation of tokens
// (2h, 2w), (2h+1, 2w), (2h, 2w+1), (2h+1, 2w+1), fetched as four bulk copies.  N = 512, 1024 or 2048; rows of 2048
// columns are normalised one per warp and call.
__device__ __noinline__ uint32_t ln_stage_ool(const Stage& st, const MegaParams& p, SmemCtl& cs, uint32_t ring, uint8_t* ring_ptr,
                                              __half* vec_s, uint32_t state, const WaitCtl& ctl, int warp, int lane) {
  RoleState rs = RoleState::unpack(state);
  const int N = st.N, M = st.M;
  const __half* src = reinterpret_cast<const __half*>(sel_ptr(st.resid_sel, st.resid, p));
  __half* out = reinterpret_cast<__half*>(const_cast<void*>(sel_ptr(st.out_sel, st.out, p)));
  const __half* gamma = reinterpret_cast<const __half*>(st.gamma);
  const __half* beta = reinterpret_cast<const __half*>(st.beta);
  // Warp 0 only feeds the ring (issuing a bulk copy of tens of KB stalls the issuing thread until the copy
  // engine has taken the previous ones); the other warps normalise rows, two per warp and round.
  constexpr int kComp = kThreads / 32 - 1;
  // batch geometry from the host (finalize_stage)
  const int rb = st.bm, batch_bytes = st.slot_bytes, nbuf = st.nslots, n_batches = st.items;
  const int my_batches = n_batches > (int)blockIdx.x ? (n_batches - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const uint32_t full0 = smem_u32(&cs.ln_full[0]), empty0 = smem_u32(&cs.ln_empty[0]);
  uint32_t bits = rs.ln_bits;

  if (warp == 0) {
    if (lane == 0) {
      const bool go = grid_wait(p, ctl, st);
      int buf = 0;
      for (int k = 0; go && k < my_batches; ++k) {
        const int batch = blockIdx.x + k * gridDim.x;
        if (!mbar_wait(empty0 + 8 * buf, ((bits >> buf) & 1u) ^ 1u, ctl, 610 + buf)) break;
        const int row0 = batch * rb;
        const int rows = (M - row0) < rb ? (M - row0) : rb;
        const uint32_t bar = full0 + 8 * buf;
        mbar_expect_tx(bar, (uint32_t)(rows * N * 2));
        ln_gather_rows(ring + buf * batch_bytes, src, row0, rows, N, st.seq, bar);
        bits ^= 1u << buf;
        buf = buf + 1 == nbuf ? 0 : buf + 1;
      }
    }
    __syncwarp();
  } else {
    const int cw = warp - 1;
    // gamma and beta go to shared memory once (while the first batches are in flight): read from global
    // memory inside the row loop, a miss in the small L1 costs an L2 round trip in the middle of every row
    if (gamma) {
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const uint2* from = reinterpret_cast<const uint2*>(v ? beta : gamma);
        uint2* to = reinterpret_cast<uint2*>(vec_s + v * N);
        for (int i = threadIdx.x - 32; i < N / 4; i += kThreads - 32) to[i] = __ldg(from + i);
      }
      named_barrier_sync(2, kThreads - 32);
      gamma = vec_s;
      beta = vec_s + N;
    }
    int buf = 0;
    for (int k = 0; k < my_batches; ++k) {
      const int batch = blockIdx.x + k * gridDim.x;
      const bool ok = mbar_wait_warp(full0 + 8 * buf, (bits >> buf) & 1u, ctl, 600 + buf, lane);
      bits ^= 1u << buf;
      if (!ok) break;
      const int row0 = batch * rb;
      const int rows = (M - row0) < rb ? (M - row0) : rb;
      const __half* base = reinterpret_cast<const __half*>(ring_ptr + buf * batch_bytes);
      for (int r = cw; r < rows; r += 2 * kComp) {
        const int r2 = r + kComp;
        const bool two = r2 < rows;
        const __half* a = base + (size_t)r * N;
        const __half* b = two ? base + (size_t)r2 * N : nullptr;
        __half* o0 = out + (size_t)(row0 + r) * N;
        __half* o1 = two ? out + (size_t)(row0 + r2) * N : nullptr;
        switch (N >> 7) {
          case 4: ln_rows2<4>(a, b, gamma, beta, st.eps, o0, o1, lane); break;
          case 8: ln_rows2<8>(a, b, gamma, beta, st.eps, o0, o1, lane); break;
          default:
            ln_row_wide(a, gamma, beta, st.eps, o0, lane);
            if (two) ln_row_wide(b, gamma, beta, st.eps, o1, lane);
            break;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty0 + 8 * buf);    // this warp is done with the buffer
      buf = buf + 1 == nbuf ? 0 : buf + 1;
    }
  }
  // every thread leaves with the same view of the buffers' phase bits
  {
    const int q = my_batches / nbuf, rem = my_batches - q * nbuf;     // buffers 0..rem-1 were used q+1 times
    uint32_t flip = (q & 1) ? (1u << nbuf) - 1u : 0u;
    if (rem) flip ^= (1u << rem) - 1u;
    rs.ln_bits ^= flip;
  }
  return rs.pack();
}

// ------------------------------------------------------------------------------------
// the kernel
// ------------------------------------------------------------------------------------
// 384 threads leave 168 registers per thread (the register file is handed out per four warps, so ten warps would
// leave no more); the epilogue is written to stay below that without spilling.
// The kernel exists in four builds, so that each fits 168 registers with its stages inlined where that matters:
//   kFamilyBert      BERT layers whose attention items outnumber the CTAs (two-pipeline attention), plain GEMMs,
//                    LayerNorm; every stage inlined into one register allocation (fastest).
//   kFamilyBertCoop  the same with the attention stage in which all eight softmax warps share one item: S up to
//                    384, and short sequences at small batch, where a CTA has at most one item anyway.
//   kFamilySwin      GEMM stages, whose LayerNorm epilogue can also store the sum and change the order of the rows, the
//                    window-attention stage and the LayerNorm stages that sum, permute and merge; GEMM stages but for that
//                    epilogue are inlined, the others stay out of line (the allocation would no longer fit).
//   kFamilyBertPair  kFamilyBert on CTA pairs: a cluster of two CTAs shares every MMA (cta_group::2), which halves the
//                    weight-tile traffic per FLOP of the GEMM stages; the attention stage takes two heads per pair.
//                    Launched with a cluster dimension of two.
constexpr int kFamilyBert = 0, kFamilyBertCoop = 1, kFamilySwin = 2, kFamilyBertPair = 3;
// One warp copies a stage record to shared memory.
__device__ __forceinline__ void copy_record(Stage* to, const Stage* from, int lane) {
  static_assert(sizeof(Stage) % 16 == 0, "records are copied 16 bytes at a time");
  for (int i = lane; i < (int)(sizeof(Stage) / 16); i += 32) reinterpret_cast<uint4*>(to)[i] = reinterpret_cast<const uint4*>(from)[i];
}

template <int kFamily>
__global__ void __launch_bounds__(kThreads, 1)
souffle_megakernel(const __grid_constant__ CallArgs ca) {
  const MegaParams& p = ca.p;
  if (p.prof && threadIdx.x == 0) {
    long long* pr = p.prof + ((size_t)p.n_stages * gridDim.x + blockIdx.x) * kProfSlots;
    pr[0] = clock64();
    pr[3] = (long long)globaltimer_ns();        // wall clock shared by all SMs: launch skew between CTAs
  }
  // The same for all CTAs of a launch: nobody waits for those that leave here.  (Test hook -1: an alignment that no base has.)
  if (smem_u32(smem_raw) & ((p.skip_arrival == -1 ? 1u << 20 : kSmemAlign) - 1u)) {
    if (threadIdx.x == 0) {
      p.status[0] = DEV_SMEM_BASE;
      if (p.expired) *p.expired = 1;
    }
    return;
  }
  SmemCtl& cs = *reinterpret_cast<SmemCtl*>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kMaxSlots; ++i) {
      mbar_init(smem_u32(&cs.full[i]), 2);        // armed by the feeder and by the weight warp
      mbar_init(smem_u32(&cs.empty[i]), 1);
    }
    constexpr bool kPairK = kFamily == kFamilyBertPair;
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&cs.tmem_full[i]), 1);
      // arrivals of the epilogue: every thread, or (pairs) one per epilogue warp of both CTAs on the leader's barrier
      mbar_init(smem_u32(&cs.tmem_empty[i]), kPairK ? 2 * kEpiWarps : kEpiThreads);
      mbar_init(smem_u32(&cs.o_empty[i]), 8);
    }
    mbar_init(smem_u32(&cs.qk_full), 1);
    mbar_init(smem_u32(&cs.qk_empty), 1);
    mbar_init(smem_u32(&cs.v_full), 1);
    mbar_init(smem_u32(&cs.v_empty), 1);
    mbar_init(smem_u32(&cs.s_full), 1);
    mbar_init(smem_u32(&cs.p_full), kPairK ? 8 : 128);         // softmax threads, or (pairs) the softmax warps of both CTAs
    mbar_init(smem_u32(&cs.o_full), 1);
    for (int i = 0; i < 7; ++i) mbar_init(smem_u32(&cs.attn1[i]), i == 5 ? (kPairK ? 8 : 128) : 1);
    for (int i = 0; i < 4; ++i) {
      mbar_init(smem_u32(&cs.ln_full[i]), 1);
      mbar_init(smem_u32(&cs.ln_empty[i]), kThreads / 32 - 1);
    }
    cs.abort = 0;
    cs.leave[0] = cs.leave[1] = 0;
    cs.go = cs.arrived = 0u;
    cs.epoch = p.epoch ? *const_cast<volatile unsigned*>(p.epoch) & ~(kLaunchSteps - 1u) : 0u;
    cs.wait.abort_smem = &cs.abort;
    cs.wait.status_g = p.status;
    cs.wait.deadline_ns = globaltimer_ns() + p.timeout_ns;      // read once per CTA
    fence_mbar_init();
    if (blockIdx.x == 0) {          // the other launch parity's barrier words start clean
      p.sync_next[0] = 0u;
      p.sync_next[1] = 0u;
    }
  }
  if constexpr (kFamily == kFamilyBertPair) {
    if (warp == 1) tmem_alloc_pair(smem_u32(&cs.tmem_base), kTmemCols);
  } else {
    if (warp == 1) tmem_alloc(smem_u32(&cs.tmem_base), kTmemCols);
  }
  if (warp == 0) copy_record(&cs.stage[0], p.stages ? p.stages : &ca.inline_stages[0], lane);
  if (warp >= 2 && p.maps) {               // warm the descriptor cache while the CTA sets up
    for (int i = (int)threadIdx.x - 64; i < p.n_maps; i += kThreads - 64) tma_prefetch_desc(p.maps + i);
  }
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (kFamily == kFamilyBertPair) cluster_sync_all();     // the peer's barriers exist before anything arrives on them
  tc_fence_after_sync();

  if (p.prof && threadIdx.x == 0) {          // one record past the stages: kernel entry, prologue done, ...
    long long* pr = p.prof + ((size_t)p.n_stages * gridDim.x + blockIdx.x) * kProfSlots;
    pr[1] = clock64();
  }

  uint32_t state = RoleState().pack();
  for (int si = 0, ord = 0, next; si < p.n_stages; si = next, ++ord) {
    // Addresses and the warp's role are worked out anew for every stage, the roles' state is packed between them: the compiler would
    // keep what follows from them in registers over all stages, and the stages that need most of them would spill.
    {
      uint32_t off = 0, tid = threadIdx.x;
      asm volatile("" : "+r"(off), "+r"(tid));
      SmemCtl& cs = *reinterpret_cast<SmemCtl*>(smem_raw + off);
      const WaitCtl& ctl = cs.wait;
      uint8_t* ring_ptr = smem_raw + off + kCtlBytes;
      __half* vec_s = reinterpret_cast<__half*>(ring_ptr + kRingBytes);
      uint8_t* stage_s = ring_ptr + kRingBytes + kVecBytes;
      const uint32_t ring = smem_u32(smem_raw) + off + kCtlBytes;
      const int warp = (int)(tid >> 5), lane = (int)(tid & 31u);
      const Stage& st = cs.stage[ord & 1];
      next = st.next;
      // The spare warps' part, in front of anything that waits: the next stage's record (constant since the launch: plan-owned
      // programs lie in global memory, the stages of the plan-less entry points in the launch parameters) goes to shared
      // memory, and this CTA's slice of the next stage's weights to L2 (they come from HBM when the program's weights exceed
      // L2; without this every GEMM stage starts with all CTAs waiting on the same DRAM rows).
      if (warp == kWeightWarp && next < p.n_stages) copy_record(&cs.stage[(ord + 1) & 1], p.stages ? p.stages + next : &ca.inline_stages[next], lane);
      if (warp == kSpareWarp && lane == 0) {
        const uint32_t pf_bytes = st.pf_bytes;
        if (pf_bytes) {
          const uint32_t per = ((pf_bytes + gridDim.x - 1) / gridDim.x + 15u) & ~15u, off = blockIdx.x * per;
          if (off < pf_bytes)
            bulk_prefetch_l2(reinterpret_cast<const char*>(st.pf_ptr) + off, off + per <= pf_bytes ? per : pf_bytes - off);
        }
      }
      __syncwarp();
      if (st.type != STAGE_LN && warp == kSpareWarp && st.dead_bytes[0]) {
        if (wait_go(cs, ord, ctl)) drop_dead_buffers(st, warp * 32, 32);
      }
      if constexpr (kFamily == kFamilySwin) {
        if (st.type == STAGE_GEMM) {
          RoleState rs = RoleState::unpack(state);
          gemm_stage<false, true, true>(st, ca, cs, ring, vec_s, stage_s, rs, ctl, warp, lane);
          state = rs.pack();
        }
        else if (st.type == STAGE_ATTN_SWIN) state = attn_swin_stage(st, ca, cs, ring, ring_ptr, reinterpret_cast<uint8_t*>(vec_s), state, ctl, warp, lane);
        else if (st.type == STAGE_LN && st.nslots == 0) ln_stage_direct(st, p, cs, reinterpret_cast<float2*>(vec_s), ctl, warp, lane);
        else if (st.type == STAGE_LN) state = ln_stage_ool(st, p, cs, ring, ring_ptr, vec_s, state, ctl, warp, lane);
      } else {
        if (st.type == STAGE_GEMM) {
          RoleState rs = RoleState::unpack(state);
          gemm_stage<kFamily == kFamilyBertPair, kFamily != kFamilyBertCoop>(st, ca, cs, ring, vec_s, stage_s, rs, ctl, warp, lane);
          state = rs.pack();
        } else if (st.type == STAGE_ATTN) {
          RoleState rs = RoleState::unpack(state);
          if constexpr (kFamily == kFamilyBert) attn_stage_pp<false>(st, ca, cs, ring, ring_ptr, reinterpret_cast<uint8_t*>(vec_s), rs, ctl, warp, lane);
          else if constexpr (kFamily == kFamilyBertPair) attn_stage_pp<true>(st, ca, cs, ring, ring_ptr, reinterpret_cast<uint8_t*>(vec_s), rs, ctl, warp, lane);
          else attn_stage(st, ca, cs, ring, ring_ptr, stage_s, rs, ctl, warp, lane);
          state = rs.pack();
        } else if (st.type == STAGE_LN) {
          if constexpr (kFamily == kFamilyBertCoop) ln_stage_either(st, p, cs, reinterpret_cast<float2*>(vec_s), ctl, warp, lane);
          else ln_stage_many(st, p, cs, ctl, warp, lane);
        }
      }
    }
    // Every thread comes by here once per stage, whatever became of its waits, and all leave the loop together.
    uint32_t off = 0, tid = threadIdx.x;
    asm volatile("" : "+r"(off), "+r"(tid));
    SmemCtl& cs = *reinterpret_cast<SmemCtl*>(smem_raw + off);
    const WaitCtl& ctl = cs.wait;
    fence_proxy_async_smem();             // this thread's accesses to shared memory before the next stage's copies into it
    if (*ctl.abort_smem) cs.leave[ord & 1] = 1;       // two words in turn: the next stage's is not written before all have read this one
    __syncthreads();
    if (*const_cast<volatile int*>(&cs.leave[ord & 1])) break;
    if (tid == kSpareWarp * 32) {
      if (p.prof) p.prof[((size_t)si * gridDim.x + blockIdx.x) * kProfSlots + 1] = clock_now();
      if (next < p.n_stages) {
        if (p.skip_arrival > 0 && si == p.skip_arrival >> 16 && (int)blockIdx.x == (p.skip_arrival & 0xFFFF) - 1) *ctl.abort_smem = 1;      // test hook
        else red_add_release_u32(p.sync, 1u);
        st_release_cta_shared_u32(smem_u32(&cs.arrived), (uint32_t)ord + 1u);
      } else if (p.prof) {
        p.prof[((size_t)si * gridDim.x + blockIdx.x) * kProfSlots + 2] = clock_now();
      }
    }
  }

  __syncthreads();
  if (p.epoch && threadIdx.x == 0) atomicAdd(p.epoch, launch_step(blockIdx.x, gridDim.x));
  if (p.prof && threadIdx.x == 0) {
    long long* pr = p.prof + ((size_t)p.n_stages * gridDim.x + blockIdx.x) * kProfSlots;
    pr[2] = clock64();
    pr[4] = (long long)globaltimer_ns();
  }
  if (cs.abort) {
    if (threadIdx.x == 0 && p.expired) *p.expired = 1;
    // let copies that were already issued land before the CTA's shared memory is released
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (kFamily == kFamilyBertPair) {
    cluster_sync_all();                    // both CTAs are done with the pair's tensor memory and with each other's barriers
    if (warp == 1) tmem_dealloc_pair(cs.tmem_base, kTmemCols);
  } else {
    if (warp == 1) tmem_dealloc(cs.tmem_base, kTmemCols);
  }
}

}  // namespace souffle
