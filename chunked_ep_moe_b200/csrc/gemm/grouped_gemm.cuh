// Parameters of the grouped tcgen05 GEMM kernels: row_gemm.cu (row-wise modes), grouped_gemm_pair.cu (weight gradients).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <atomic>

#include "../common/status.cuh"
#include "../plan/plan_tables.cuh"

namespace cem {

// Per CTA of a pair: 128 x (up to) 256 accumulator (fp32 in TMEM, double buffered = all 512 columns), K step 64 bf16 =
// one 128-byte swizzle span.
constexpr int kBlockM = 128;
constexpr int kBlockN = 256;
constexpr int kBlockK = 64;
constexpr int kUmmaK = 16;
constexpr int kSmemAlignSlack = 512;  // the kernels check at run time that the 1024-byte aligned layout fits
constexpr int kSmemTailBytes = 256;   // barriers, TMEM slot, flags
constexpr int kCombineCols = kBlockM; // columns of one returned row piece (what the returned-piece counters count)

enum GemmMode : int {
  kModeSwiglu = 0,   // act = w * silu(x Wg) * (x Wu) from striped w_up; optional h      (replaces gmm_swiglu)
  kModeDownFwd = 1,  // y = act Wd, rows stored to their source rank                         (gmm + combine)
  // (2 is not used: the slot numbering of the pipeline counters is public)
  kModeDswiglu = 3,  // d_act = w * (g Wd^T); epilogue SwiGLU' with h -> dh, d_weight partials (gmm_dswiglu)
  kModeDx = 4,       // dx = dh Wu^T; rows stored to their source rank                      (gmm^T + combine)
  kModeTgmm = 5,     // dW[g] = lhs[rows_g]^T rhs[rows_g], fp32 carry across slices         (tgmm + accumulate)
};

// Per-CTA pipeline counters (SM cycles unless noted). They say which side of the operand ring waits for the other.
enum ProfSlot : int {
  kProfLoopCycles = 0,   // MMA warp: first tile started -> last MMA issued
  kProfLoopNs = 1,       // the same span in nanoseconds of the global timer (cycles / ns = SM clock in GHz)
  kProfEmptyWait = 2,    // producer: waiting for a free stage (the MMAs are the slower side)
  kProfFullWait = 3,     // MMA warp: waiting for a filled stage (the loads are the slower side)
  kProfAccWait = 4,      // MMA warp: waiting for the epilogue to hand an accumulator back
  kProfKBlocks = 5,      // k-blocks issued
  kProfEpiWait = 6,      // first epilogue warp: waiting for a finished accumulator
  kProfTiles = 7,        // tiles
  kProfSlots = 8,
};

struct GemmParams {
  // --- schedule ---------------------------------------------------------------------------
  const int* plan;   // per-pass plan buffer (see plan_tables.cuh)
  PlanLayout lay;
  int slice;         // slice index inside the pass
  // The tiles of experts [first, last) only; last = 0: of all. (Weight gradients: in the tables of a pass that is one slice, where
  // every expert has a group.)
  int first_expert, last_expert;
  int n_tiles;       // 256-column tiles of the weights (row-wise modes) or of the gradient (tgmm)
  int unit_cols, row_units;  // tgmm: column tiles that a pair takes together of experts of few rows, and how many such units a row of
                             // tiles has (set by the launcher)
  int m_tiles;       // tgmm: M / 128 (row tiles of the weight gradient); unused otherwise
  int k_blocks;      // gmm modes: K / 64
  int b_group_rows;  // rows one expert occupies in the flattened 2-D weight tensor map
  int me;            // this rank
  int stripe;        // SwiGLU stripe width (swiglu / dswiglu)
  uint32_t spin_limit;   // polls of a cross-GPU flag before giving up
  uint32_t mbar_limit;   // microseconds a pipeline barrier may take before giving up
  StatusBlock* status;
  // Optional pipeline counters of this mode, [grid][kProfSlots] summed over launches; null = not counted.
  unsigned long long* prof;
  // --- arrival flags (swiglu and dswiglu: the first consumer of a slice's rows) -----------------------------------------------------
  const uint32_t* arrive;     // [P*L] cumulative rows received per (source, local expert); null = no wait
  const uint32_t* pass_base;  // [P*L] value of `arrive` when this pass began
  // fp8 wire: rows are usable once the expansion kernel has released them, per local expert (replaces `arrive`)
  const uint32_t* ready;       // [L] cumulative rows expanded per local expert; null = not used
  const uint32_t* ready_base;  // [L] value of `ready` when this pass began
  // --- row-wise outputs / inputs (leading dims in elements) -----------------------------------
  __nv_bfloat16* out0;        // swiglu: act [S,F]; dswiglu: dh [S,2F]
  __nv_bfloat16* out1;        // swiglu: h [S,2F] or null
  const __nv_bfloat16* in0;   // dswiglu: h [S,2F]
  const __nv_bfloat16* in1;   // dswiglu: w * act [S,F], leading dimension ld1 (with dwp)
  const float* row_w;         // router weight per slice row [S]; swiglu / dswiglu: null = 1
  float* dwp;                 // dswiglu: shares of the router weights' gradients (times the weight, see `weight_divides`), one per
                              // 32 columns [S, dwp_tiles], or null
  int dwp_tiles;
  int ld0, ld1;
  // --- gathered rows (`launch_gather_swiglu`): row r of the slice is row tokens[r] of `gather` --------------------------------
  const __nv_bfloat16* gather;  // [tokens, 64 k_blocks]
  const int* tokens;
  // `launch_few_swiglu`: [num_ids] expert ids and router weights by flat index t * top_k + k, in place of `tokens` and `row_w`
  const int* ids;
  const float* w_flat;
  int num_ids, top_k;
  // --- combine targets (down_fwd, dx) --------------------------------------------------------
  __nv_bfloat16* const* peer_rows;   // [P] base of each source rank's [T*K, ld] return buffer; null: rows go to out0
  uint32_t* const* peer_count;       // [P] each source rank's returned-row counter; null: nobody waits for the rows
  // --- kernel-level entry points: rows of an output past the groups' last one (up to S) are set to zero -----------
  __nv_bfloat16* tail[2];            // base of an output, or null
  int tail_cols[2];
  // --- tgmm ---------------------------------------------------------------------------------
  const float* carry_in;   // [M, N] fp32 partial of the expert that straddles the previous slice boundary
  float* carry_out;        // [M, N] fp32 partial of the expert that straddles the next slice boundary
  __nv_bfloat16* grad_out; // [L, M, N] final gradient
};

// Activation operand of the row-wise modes, [S, cols] bf16: `by_width[i]` has boxes of 16 (i + 1) rows, what each CTA of a
// pair loads for a tile of 32 (i + 1) rows.
struct alignas(64) TokenMaps {
  CUtensorMap by_width[8];
};

// Row-wise modes (everything but kModeTgmm). `map_a`: the weights, for the modes that read them with K along rows the
// chunked description with boxes of 64 rows x 2 chunks (1 chunk for SwiGLU with stripes of 128), else boxes of 128 rows.
// `grid` is rounded down to an even number and clamped to what is resident at once. `behind`: the kernel may become resident in
// its predecessor's tail (programmatic dependent launch). Only where nothing else wants the SMs meanwhile: a waiting CTA holds
// one, which two slices in flight would miss, and which a kernel that the PREDECESSOR waits for (the expansion of the fp8
// wire, a put to this rank) may need. So: one rank, one stream (one-slice forwards: one token 46.3 -> 43.1 us, 64 tokens at
// D=7168 497 -> 487 us, 2000 tokens at D=2048 153 -> 147 us; a kernel-level forward + backward gained nothing, 248 against 251 and, with
// the weight gradients too, 251 against 254). And in one-range backwards, on the caller's stream and the auxiliary one, whose kernels
// wait for nothing that comes behind them: see `FusedRank::backward_whole`.
void launch_row_gemm(int mode, const GemmParams& p, const CUtensorMap& map_a, const TokenMaps& maps_b, int grid,
                     cudaStream_t stream, bool behind = false);

// kModeSwiglu on all experts' rows, gathered: no map of them.
void launch_gather_swiglu(const GemmParams& p, const CUtensorMap& map_a, int grid, cudaStream_t stream, bool behind = false);

// The same as the first kernel of a pass of at most 32 expert ids, without a plan: what the kernels behind it need of one goes to `plan`.
struct FewPlan {
  int* plan;          // header, tiles and their number, the last entry of tile_start, and of experts with rows tile_start (their own
                      // and the next expert's), in_start, in_size and src_send_start; nothing else
  int* order;         // [num_ids]
  int* inv_order;
  int32_t* host_out;  // as in `PlanKernelParams`
  uint32_t host_seq;
};
constexpr int kFewIds = 32;
void launch_few_swiglu(const GemmParams& p, const CUtensorMap& map_a, const FewPlan& plan, int grid, cudaStream_t stream,
                       bool behind = false);

// Weight gradients (kModeTgmm). `map_a`, `map_b`: chunked descriptions with boxes of 64 rows x 2 chunks; `map_c`: the bf16
// gradient [L*M, N] with boxes of 32 rows x 64 columns (tiled stores). `rows`: of the slice, or what it can hold.
void launch_weight_grad(const GemmParams& p, const CUtensorMap& map_a, const CUtensorMap& map_b, const CUtensorMap& map_c, int grid,
                        int64_t rows, cudaStream_t stream, bool behind = false);

int weight_grad_unit_cols(int rows_of_tiles, int n_tiles, int pairs);  // (the launcher's choice of `unit_cols`)
int row_gemm_smem_bytes();    // dynamic shared memory of a row-wise GEMM CTA
extern std::atomic<int> g_pair_grid_used;  // grid of the last GEMM launch, for diagnostics (passes of several workspaces store it)

}  // namespace cem
