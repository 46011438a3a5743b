// Stage program: the host-built description a persistent megakernel interprets.
//
// The reference fuses an encoder layer into one cooperative launch whose stages are separated
// by grid.sync() (cpp/bert/kernels/fused_sqq_bert.cu:34-2305: nine stages, compile-time shapes
// from cpp/bert/kernels/bert.h:8-52).  Here the stage list is data: every stage is a record in
// global memory, shapes are runtime values, and the same kernel runs a BERT layer, a chain of
// layers, the Swin MLP pair or a single GEMM.
#pragma once
#include <stdint.h>

namespace souffle {

enum StageType : int {
  STAGE_GEMM = 0,   // C = A . B with a fused epilogue
  STAGE_ATTN = 1,   // per (sequence, head, query tile): softmax(Q K^T * scale + mask) V
  STAGE_LN = 2,     // z = sum_p partial[p] + bias + resid ; y = LayerNorm(z)
  STAGE_ATTN_SWIN = 3,  // per (window, head): softmax(Q K^T * scale + relative-position bias + shift mask) V
};

enum EpilogueKind : int {
  EPI_F16 = 0,      // out[row, col] = f16(act(acc + bias))
  EPI_QKV = 1,      // like EPI_F16 but scattered head-split to [3][B][heads][S][d]
  EPI_PARTIAL = 2,  // raw fp32 accumulators to partial[split][row][col]
  EPI_LN = 3,       // f16(LayerNorm(acc + bias + resid)): the row's statistics come from all tiles that share it; sum_out, eps < 0 and
                    // tok_grid as in a LayerNorm stage (Swin build)
};

enum Activation : int { ACT_NONE = 0, ACT_RELU = 1, ACT_GELU = 2 };

// Pointer selectors: a stage either carries a plan-owned pointer or names a per-call argument.
enum PtrSel : int { PTR_PLAN = 0, PTR_CALL_X = 1, PTR_CALL_Y = 2 };

// Mean and sum of squared deviations of a row's columns in one tile, each beside a tag that tells when it was written: a word of
// 64 bits is written as a whole, so a reader that finds the tag has the value.
struct alignas(16) RowStat {
  float mean;
  uint32_t tag0;
  float dev;
  uint32_t tag1;
};

struct alignas(16) Stage {      // 16-byte multiples: records are copied 16 bytes at a time
  int type;
  // ---- GEMM ----
  int tm_a;          // tensor-map index of the A operand ([M][K], box 64 x bm; STAGE_ATTN: of Q); negative = per-call map
  int tm_b;          // tensor-map index of the B operand
  int tm_out;        // with out_stores: tensor-map index of the output, 64B swizzle.  EPI_PARTIAL: the fp32 planes as
                     // [splitk][M][N], box 16 columns x 32 rows x 1 plane; EPI_F16: [M][N], box 32 x 32; EPI_QKV: [3 B heads S][d],
                     // box 32 columns x 32 / out_stores rows
  int out_stores;    // copies per box of 32 rows (2 where a sequence ends inside one)
  int M, N, K;
  int bm;            // tile height: 128, or 256 (two 128-row halves that share each B tile); STAGE_ATTN: query rows per item
  int bn;            // tile width in N (multiple of 16, <= 256; N may end inside the last tile, see ragged_width)
  int splitk;        // K is cut into this many independent partial products (STAGE_LN: warps that may share a row)
  int b_mn_major;    // 0: B stored [N][K] (K contiguous); 1: B stored [K][N] (N contiguous, bn % 64 == 0)
  int epi;           // EpilogueKind
  int act;           // Activation
  int out_sel;       // PtrSel for `out`
  int resid_sel;     // PtrSel for `resid`
  int ldo;           // leading dimension of out / resid (elements)
  const void* bias;  // fp16 [N] or null
  const void* resid; // fp16 [M][ldo] or null
  void* out;         // fp16 output
  union {
    float* partial;  // fp32 [splitk][M][N] (EPI_PARTIAL and STAGE_LN)
    RowStat* stats;  // EPI_LN: [blocks of 32 rows][tiles_n][32]
  };
  // ---- attention / head split ----
  union {
    struct { int batch, heads, seq, head_dim; };
    struct { int tm_resid, tm_unit; };  // EPI_LN: tensor maps of the residual ([M][N], box 64 x bm) and of the unit matrix ([64][64])
  };
  union {
    float scale;     // softmax scale applied to Q.K
    int to_shift;    // STAGE_LN and EPI_LN of a Swin block, see tok_grid
  };
  union {
    int tm_qkv;      // tensor map over the head-split buffer viewed as [3*B*heads*S][d], box 64 x 128; Swin: see attn_swin_stage
    int tok_grid;    // STAGE_LN, EPI_LN: 0, or the side of the token grid whose rows leave in another order than they come in: in the order of the
  };                 // windows of `win` x `win` tokens after a shift, to_shift and `shift`, or in that of the tokens (-1)
  int win, shift;    // Swin: window size (7) and cyclic shift; `seq` is then the side of the token grid
  const void* rel_bias;  // Swin: fp16 [(2*win-1)^2][heads] relative-position bias table
  void* probs;       // optional fp16 [B*heads][S][S] normalised probabilities (debug / parity output)
  // ---- layer norm ----
  const void* gamma; // fp16 [N] or null
  const void* beta;  // fp16 [N] or null
  float eps;         // < 0: no normalisation, the sum goes to `out`
  void* sum_out;     // fp16 [M][N] or null: the sum (rounded to fp16, which is then what gets normalised) is stored here as well
  uint8_t n_partial; // number of fp32 partial planes to sum
  // ---- order, set by the host.  A LayerNorm stage that the GEMM stage in front of it does in its epilogue keeps its place in the
  //      program, but nothing runs there ----
  uint8_t fused;     // STAGE_LN: done by the stage before
  uint8_t position;  // of this stage in the program
  uint8_t prev, next;// positions of the stages that run before and after it (the number of stages: none)
  uint8_t ordinal;   // stages that run before it: the grid barrier counts arrivals against it
  // ---- weight prefetch: the B matrix of the next stage, a GEMM, pulled into L2 by all CTAs at the start of this one
  //      (weights never depend on an earlier stage) ----
  uint32_t pf_bytes;
  const void* pf_ptr;
  // ---- buffers whose last reader was the stage before this one (multiples of 128 bytes, 128-byte aligned), where a layer's
  //      intermediates take much of L2 (see upload_program): their lines are dropped from it at the start of this stage ----
  uint32_t dead_bytes[2];
  const void* dead_ptr[2];
  // ---- derived on the host by finalize_stage(): the kernel's lone producer / MMA lanes would otherwise
  //      spend a few thousand cycles per stage in integer divisions ----
  int tiles_n, kchunks, kper, items, slot_bytes, nslots;   // a K chunk: kper steps of 64
  uint32_t mg_splitk, mg_tiles_n, mg_kchunks;   // magic multipliers, see fast_div()
  uint32_t mg_seq, mg_head_dim, mg_heads;
  // Swin row maps: windows per side of the grid, and the multipliers of the divisors grid * grid (0: divide plainly), win, nwr,
  // nwr * nwr and win * win
  int nwr;
  uint32_t mg_seq2, mg_win, mg_nwr, mg_nwr2, mg_tok;
};

#ifdef __CUDACC__
#define SOUFFLE_HOST_DEVICE __host__ __device__
#else
#define SOUFFLE_HOST_DEVICE
#endif

// The eight epilogue warps of a CTA, numbers 2..9.  The hardware lets a warp read one quarter of tensor memory's lanes, by its number
// modulo four; the two warps of a quarter have the same rows and take every other 32 columns, the one of part 0 the first.
SOUFFLE_HOST_DEVICE constexpr int epi_quarter(int warp) { return warp & 3; }
SOUFFLE_HOST_DEVICE constexpr int epi_part(int warp) { return (warp - 2) >> 2; }
SOUFFLE_HOST_DEVICE constexpr int epi_warp(int quarter, int part) { return 2 + 4 * part + ((quarter + 2) & 3); }
// Each has two boxes for its stores; number of a warp's first one.
SOUFFLE_HOST_DEVICE constexpr int epi_box(int warp) { return (warp - 2) * 2; }
// The box through which the warps of a quarter exchange the statistics of their rows: the second one of its own part 1.
SOUFFLE_HOST_DEVICE constexpr int ln_stats_box(int quarter) { return epi_box(epi_warp(quarter, 1)) + 1; }

// Launches on one scratch are told apart by a counter in it: a launch's number is the counter / kLaunchSteps.  A CTA reads it when it
// starts, and its step is added when it leaves.  The steps of a launch make kLaunchSteps together, so until the last CTA has read it the
// number stays: a CTA that starts after others have given up and gone still marks its words as this launch's, not as the next one's.
constexpr uint32_t kLaunchSteps = 256;      // CTAs of a launch at most
SOUFFLE_HOST_DEVICE constexpr uint32_t launch_step(uint32_t cta, uint32_t ctas) { return cta == 0 ? kLaunchSteps - (ctas - 1) : 1u; }

// q = n / d for n * d < 2^32 as one multiply-high: mg = ceil(2^32 / d); d == 1 has no 32-bit multiplier.
inline uint32_t fast_div_magic(uint32_t d) { return d <= 1 ? 0u : (uint32_t)((0x100000000ull + d - 1) / d); }

constexpr int kMaxTensorMaps = 96;
constexpr int kMaxStages = 160;   // positions fit a byte
constexpr int kProfSlots = 16;   // int64 words per (stage, CTA) record of the in-kernel profile

}  // namespace souffle
