// Per-rank executor of the fused NVLink path: owns the scratch buffers, the peer pointer tables,
// the TMA descriptors, the comm stream and the slice sequence counter, and launches the kernels
// of one slice at a time.
//
// The step methods (begin_*, put, compute_*, finish_*) are what a pass is made of:
//
//     begin_forward -> put(0) -> for j: put(j+1); compute_forward(j) -> finish_forward
//
// One process drives one rank per GPU that way. A test harness may instead drive several
// ranks that live on ONE device in lockstep (all puts of a slice, then all computes); then
// every flag a kernel looks at has already been set when it starts and nothing ever spins.
#pragma once

#include <torch/extension.h>

#include <cuda.h>
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <algorithm>
#include <exception>
#include <string>
#include <tuple>
#include <vector>

#include "../comm/comm_kernels.cuh"
#include "../gemm/grouped_gemm.cuh"
#include "../plan/plan_kernel.cuh"

namespace cem {

// Byte offsets inside one rank's symmetric arena (identical on every rank).
struct ArenaLayout {
  size_t xbuf, gbuf, wbuf, xq, gq, xs, gs, ret, dw_rows, arrive, credit, ret_count, traffic, traffic_flags, total;
};

ArenaLayout make_arena_layout(int P, int L, int S, int D, int tk_cap, bool fp8);

// Text of a recorded status block {code, kernel, mode, slice, detail, expected, seen, block} (what check_status raises).
std::string format_status(const std::vector<int64_t>& status, int rank);

// Rows of a slice x D x F from which a training forward keeps h and w * act. Measured, forward + backward, keeping against
// recomputing: 16384-row slices at D=1024, F=512 (2^33) 1026 against 1072 us, 7996 rows at D=2048, F=1024 (2^34) 503 against
// 530 us; 1024-row slices at D=2048, F=1024 (2^31) 1133 against 1126 us (the GEMM it saves runs in the shadow of the next
// put there), 1024 rows at D=F=512 204 us both ways (a kernel takes 8 us however little it does, and two allocations and a
// slice's tensor maps cost the host what its launch does).
constexpr int64_t kKeepWork = int64_t{1} << 32;

// Slices of a training forward that a rank among several keeps h and w * act of: those that its own stream reached in the pass
// before (`stream_rows`), at most the `guess` it launches. Every rank loops as often as the fullest one, but a rank only has
// memory reserved for about the rows that come to it; slices past them hold none, and one that does after all is recomputed.
inline int64_t slices_to_keep(int64_t guess, int64_t stream_rows, int64_t slice_rows) {
  return std::min<int64_t>(guess, (stream_rows + slice_rows - 1) / slice_rows);
}

// What a forward that ran as one slice (`FusedRank::runs_whole`) gives as its slice count.
constexpr int64_t kWholePass = -1;
// Ranges of whole experts in which such a pass runs (equal numbers of experts each, whatever their rows): one, except where hiding
// the puts and finding in L2 what the GEMM before wrote is worth more than every range's launches and tails, that is for large
// experts with rows enough. There, as many as have four waves of their first GEMM's tiles each under even routing, at most eight.
// Forward + backward, and forward alone, in ms, one range -> eight in both directions:
//   D=7168, F=2048  12,288 rows  3.60 -> 3.72   1.18 -> 1.18       D=5120, F=2048  36,000 rows  6.57 -> 6.50   2.18 -> 2.13
//                   16,384       4.65 -> 4.69   1.58 -> 1.52       D=4096, F=2048  65,536       8.74 -> 8.79   2.87 -> 2.88
//      64 experts   16,384       5.46 -> 5.60                      D=5120, F=1536  49,152       6.17 -> 6.34
//                   24,000       6.55 -> 6.20   2.16 -> 2.06       D=7168, F=1024  65,536       8.42 -> 8.46
//                   32,768       8.54 -> 8.13   2.90 -> 2.72       D=2048, F=2048  65,536       4.53 -> 4.69
//                   65,536      16.28 -> 15.62  5.35 -> 5.23       D=2048, F=1024  49,152       1.95 -> 2.13   0.64 -> 0.69
// (24,000 rows have four waves in six ranges of the forward and three of the backward: 6.18 ms, with Zipf routing 6.34 as in eight.
// The runs of one side differ by 3-5 %, under the power cap.)
constexpr int kRanges = 8;
constexpr int64_t kRangesExpert = int64_t{9} << 20;                            // least D x F
constexpr int64_t kRangesTraining = int64_t{300} * 1000 * 1000 * 1000;         // least rows x D x F
constexpr int64_t kRangesForward = int64_t{220} * 1000 * 1000 * 1000;          // without autograd
constexpr int64_t kRangeTiles = 4 * 74;
inline int64_t whole_ranges(int64_t rows, int64_t L, int64_t D, int64_t F, bool training, bool backward) {
  if (L < kRanges || D * F < kRangesExpert || rows * D * F < (training ? kRangesTraining : kRangesForward)) return 1;
  const int64_t tiles = (rows + 191) / 192 * ((backward ? F : 2 * F) / kBlockN);
  return std::max<int64_t>(1, std::min<int64_t>(kRanges, tiles / kRangeTiles));
}

class FusedRank {
  using Turn = std::lock_guard<std::recursive_mutex>;

 public:
  FusedRank(int P, int L, int me, int S, int D, int F, int K, int stripe, int tk_cap, int max_slices, int num_sms,
            bool fp8, int64_t arena, std::vector<int64_t> peer_arenas, bool use_comm_stream, int64_t spin_limit,
            int put_blocks);
  ~FusedRank();

  // Forward pass set-up: sort, traffic exchange, plan tables, arrival targets. `plan`, `order`,
  // `inv_order` are caller-owned int32 tensors (they are what the backward needs again).
  // With `counts_prefilled` the [P,P,L] traffic matrix in `counts` is taken as is (lockstep harness).
  // Returns the number of slices (this synchronises the host with the plan kernel once).
  int64_t begin_forward(torch::Tensor expert_ids, torch::Tensor plan, torch::Tensor order, torch::Tensor inv_order,
                        torch::Tensor counts, bool counts_prefilled);
  // The same set-up without waiting for the device: the plan kernel stores the plan header and the status block to pinned
  // host memory, their sequence number last. Returns the slice count of this workspace's previous
  // forward pass (-1 if there was none) as a GUESS; the caller may launch that many slices at once, then calls
  // `resolve_slices()` for the real count, launches what is still missing and reports what it launched with
  // `set_pass_slices()`. Slices past the real count find empty tables and do nothing, on every rank alike.
  int64_t begin_forward_async(torch::Tensor expert_ids, torch::Tensor plan, torch::Tensor order,
                              torch::Tensor inv_order, torch::Tensor counts, bool counts_prefilled);
  // Polls for that sequence number (does not wait for the stream), raises a recorded kernel error, returns the real slice count.
  int64_t resolve_slices();
  void set_pass_slices(int64_t launched);
  // Microseconds a pipeline barrier inside a GEMM may take before the kernel gives up (default 20 s).
  void set_mbar_limit_us(int64_t us);
  // Lockstep harness only: sort + histogram without the exchange (fills order, inv_order, my row of counts).
  void sort_only(torch::Tensor expert_ids, torch::Tensor order, torch::Tensor inv_order, torch::Tensor my_counts);
  // `known_slices`, `known_rows` (T*K): what the forward of the same plan returned / was given; when both are >= 0
  // the plan header is not read back and the stream is not synchronised.
  int64_t begin_backward(torch::Tensor plan, int64_t known_slices = -1, int64_t known_rows = -1);

  void put(int64_t j, torch::Tensor plan, torch::Tensor order, torch::Tensor x, c10::optional<torch::Tensor> g,
           torch::Tensor w_flat);
  void compute_forward(int64_t j, torch::Tensor plan, torch::Tensor w_up, torch::Tensor w_down);
  void compute_backward(int64_t j, torch::Tensor plan, torch::Tensor w_up, torch::Tensor w_down, torch::Tensor dw_up,
                        torch::Tensor dw_down);
  // Behind begin_*: the pass keeps (forward) or finds (backward) h and w * act of its first `slices` slices in `h` [rows, 2F] and
  // `act` [rows, F]. Lasts until the pass is finished.
  void keep_rows(torch::Tensor h, torch::Tensor act, int64_t slices);
  void finish_forward(torch::Tensor inv_order, torch::Tensor out);
  void finish_backward(torch::Tensor inv_order, torch::Tensor dx, torch::Tensor d_weights) {
    const Turn turn(pass_mutex_);
    reduce_backward(inv_order, dx, d_weights, nullptr);
  }

  // The two passes as one call each (what `chunked_moe` runs). Forward: ([out, plan, order, inv_order] and, when a
  // `training` pass keeps them, [h, w * act]; slice count; slices kept); it throws a recorded kernel error. Nothing is kept
  // under saved-tensor hooks: what is saved may then not depend on how much memory is free (activation checkpointing wants
  // the same tensors from the recomputation) and may be on its way to the host. Backward:
  // (dx, d_weights, dw_up, dw_down). Tensors are contiguous CUDA tensors of the workspace's geometry: x, g [T, D] bf16,
  // expert_ids [T, K] int32, w_flat [T*K] fp32. A forward whose plan is not wanted (no backward follows) may give `out` alone.
  std::tuple<std::vector<torch::Tensor>, int64_t, int64_t> forward_pass(
      torch::Tensor x, torch::Tensor expert_ids, torch::Tensor w_flat, torch::Tensor w_up, torch::Tensor w_down,
      bool training, bool plan_wanted = true);
  std::tuple<torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor> backward_pass(
      torch::Tensor x, torch::Tensor g, torch::Tensor w_flat, torch::Tensor w_up, torch::Tensor w_down,
      torch::Tensor plan, torch::Tensor order, torch::Tensor inv_order, int64_t known_slices,
      const std::vector<torch::Tensor>& kept, int64_t kept_slices);

  // The arena is about to go. Waits for the pass under way on another thread and for the device; whatever comes later is refused
  // behind the same lock, before it launches anything. Gives the scratch back.
  void release();

  // Reads the status block (synchronises); throws std::runtime_error describing the first recorded error.
  void check_status();
  std::vector<int64_t> plan_header() const {
    const Turn turn(pass_mutex_);
    std::vector<int64_t> header(host_header_, host_header_ + 16);
    if (header_whole_) header[0] = (header[2] + S_ - 1) / S_;  // in slices of the configured size
    return header;
  }
  int64_t plan_ints() const { return lay_.total; }
  // Whether passes of a rank on its own may run as one slice (default). Off: slice by slice, also the backward of a forward that
  // ran as one.
  void set_whole_passes(bool on) {
    const Turn turn(pass_mutex_);
    whole_passes_ = on;
  }
  int64_t launches() const {
    const Turn turn(pass_mutex_);
    return launches_;
  }
  // Turns the GEMM kernels' pipeline counters on: `counters` is a zeroed int64 CUDA tensor [6 modes, num_sms, 8]
  // (slots: ProfSlot in gemm/grouped_gemm.cuh) that every later GEMM launch adds to. An undefined tensor turns
  // them off again. Waits for the last pass, whose kernels still add to the counters before. Diagnostics only: the counting costs a
  // few clock reads per k-block.
  void set_pipeline_counters(c10::optional<torch::Tensor> counters);
  // Debug views of the local scratch (tests compare them with the torch reference).
  torch::Tensor act() const {
    const Turn turn(pass_mutex_);
    return act_[0];
  }
  torch::Tensor h() const {
    const Turn turn(pass_mutex_);
    return h_[0];
  }
  torch::Tensor dh() const {
    const Turn turn(pass_mutex_);
    return dh_[0];
  }

 private:
  // Common start of a pass: counter targets on the device, what the pass will receive back (`pieces_per_row` of T*K rows).
  void begin_pass(const torch::Tensor& plan, int64_t slices, int64_t rows, int pieces_per_row,
                  bool targets_set = false);
  void enter_pass();
  void expect_arena(const char* what) const;
  // `after`: an event that the caller's stream waits for behind the pass's last kernel, or null.
  void reduce_backward(torch::Tensor inv_order, torch::Tensor dx, torch::Tensor d_weights, cudaEvent_t after);
  void end_pass(int64_t n_slices);
  void wait_header();
  void quiesce() const;
  // Declared behind the tensors that a pass uses on the rank's streams: they are not released under it by an exception.
  struct QuiesceOnError {
    const FusedRank* rank;
    const int before = std::uncaught_exceptions();
    ~QuiesceOnError() {
      if (std::uncaught_exceptions() > before) rank->quiesce();
    }
  };
  void release_kept();
  std::vector<torch::Tensor> allocate_kept(int64_t rows, int64_t slice_rows, const torch::TensorOptions& bf16) const;
  __nv_bfloat16* kept_h(int64_t j) const {
    return reinterpret_cast<__nv_bfloat16*>(kept_h_.data_ptr()) + static_cast<size_t>(j) * S_ * 2 * F_;
  }
  __nv_bfloat16* kept_act(int64_t j) const {
    return reinterpret_cast<__nv_bfloat16*>(kept_act_.data_ptr()) + static_cast<size_t>(j) * S_ * F_;
  }
  uint64_t kept_slice_rows(int64_t j) const { return std::min<int64_t>(S_, kept_act_.size(0) - j * S_); }
  // fp8 wire among several ranks: rows arrive as e4m3 and an expansion kernel turns them into the bf16 the GEMMs read. On one
  // rank the put kernel stores the expanded values at once (32 experts of 1024 rows,
  // D=7168, F=2048, forward + backward: 11.1 -> 9.06 ms).
  bool expands() const { return fp8_ && P_ > 1; }
  // Slices are what ranks exchange. A rank on its own exchanges nothing, so its passes run as ONE slice, the large ones in ranges of
  // whole experts (`whole_ranges`): no tail of a GEMM per slice (1024 rows at F=1024 are 0.2-0.8 waves of tiles), no fp32 carry of
  // the experts that straddle slices (176 MB written and read per boundary at D=7168, F=2048), no put that waits for a buffer. Rows
  // are still put into expert order; with ranges, range by range, each beside the GEMMs of the range before: only the first is waited
  // for; and a range's GEMMs follow one another, so that what one writes the next finds in L2. (The whole pass GEMM by GEMM, with
  // ranges for the first one only: 15.72 ms at 32 experts x 2048 rows, D=7168, F=2048, where slices of 8192 rows took 15.63; range by
  // range 15.41 against 16.04.) Forward + backward, slices -> one slice: 8 x 1024 rows at D=2048, F=1024 0.955 -> 0.430 ms, Zipf
  // routing in 12 slices of 2048 rows at D=7168 7.50 -> 6.21, 3 x 16384 rows at D=1024, F=512 0.895 -> 0.792. The buffers are the
  // pass's own, from the caching allocator, while live tensors and arenas stay within half of the device; otherwise slice by slice.
  bool runs_whole(int64_t rows, bool training) const;
  bool runs_brief(int64_t tokens, int64_t rows, bool training) const;
  void expect_pass(const torch::Tensor& x, const torch::Tensor& expert_ids, const torch::Tensor& w_flat, const torch::Tensor& w_up,
                   const torch::Tensor& w_down) const;
  std::tuple<std::vector<torch::Tensor>, int64_t, int64_t> forward_brief(torch::Tensor x, torch::Tensor expert_ids, torch::Tensor w_flat,
                                                                         torch::Tensor w_up, torch::Tensor w_down, bool plan_wanted);
  bool within_half(size_t bytes, int share = 2) const;  // (or another share of the device)
  GemmParams range_params(const int* plan, int64_t first, int64_t last) const;
  template <typename Part>
  void run_parts(int64_t parts, Part&& part);
  std::tuple<std::vector<torch::Tensor>, int64_t, int64_t> forward_whole(
      torch::Tensor x, torch::Tensor expert_ids, torch::Tensor w_flat, torch::Tensor w_up, torch::Tensor w_down,
      const std::vector<torch::Tensor>& kept, const std::vector<torch::Tensor>& buffers, bool training);
  void backward_whole(torch::Tensor x, torch::Tensor g, torch::Tensor w_flat, torch::Tensor w_up, torch::Tensor w_down,
                      torch::Tensor plan, torch::Tensor inv_order, const std::vector<torch::Tensor>& kept, const torch::Tensor& kept_x,
                      const std::vector<torch::Tensor>& buffers, torch::Tensor dw_up, torch::Tensor dw_down);
  void put_whole(const torch::Tensor& plan, const torch::Tensor& inv_order, const torch::Tensor& x, const torch::Tensor* g,
                 const torch::Tensor& w_flat, __nv_bfloat16* to_x, __nv_bfloat16* to_g, float* to_w, int64_t first, int64_t last,
                 cudaStream_t st, bool behind, bool beside);
  bool overlapped() const { return use_comm_stream_ && !inline_; }
  void join_streams(bool backward);
  GemmParams base_params(const int* plan, int j) const;
  // `chunks` > 0: the MN-major description (64-column chunks, `chunks` of them per copy); 0: plain 2-D boxes.
  const CUtensorMap& weight_map(const torch::Tensor& w, uint32_t box_rows, uint32_t chunks = 0);
  void dequant(const int* plan, int j, int b, bool with_g, cudaStream_t st);
  const CUtensorMap& up_map(const torch::Tensor& w_up);  // w_up as the SwiGLU mode reads it
  void count_pipeline(int mode, GemmParams* p);
  void row_gemm(int mode, const GemmParams& p, const CUtensorMap& weights, const TokenMaps& rows, cudaStream_t st,
                int spare_sms = 0);
  void weight_grad(const GemmParams& p, const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& out,
                   cudaStream_t st);

  int P_, L_, me_, S_, D_, F_, K_, stripe_, tk_cap_, max_slices_, num_sms_, put_blocks_;
  bool fp8_, use_comm_stream_;
  uint32_t spin_limit_, mbar_limit_;
  PlanLayout lay_;
  PlanLayout whole_lay_{};      // one slice of tk_cap rows
  bool whole_passes_ = true;
  bool header_whole_ = false;   // the forward that filled the header ran as one slice
  ArenaLayout arena_lay_;
  uint8_t* arena_;
  std::vector<uint8_t*> peers_;

  // local scratch (torch-owned)
  torch::Tensor act_[2], h_[2], dh_[2], dwp_[2];
  torch::Tensor kept_h_, kept_act_;  // of the current pass: [rows, 2F], [rows, F] of its first kept_slices_ slices
  int64_t kept_slices_ = 0;
  int device_ = 0;
  size_t device_bytes_ = 0;
  bool keep_activations_ = true;  // CEM_KEEP_ACTIVATIONS=0: always recompute (least memory)
  torch::Tensor carry_up_, carry_down_, pass_base_, expected_total_, status_, tables_,
      sort_scratch_, my_counts_;
  torch::Tensor brief_tokens_;  // tokens by row of a pass that `runs_brief`
  torch::Tensor ready_, ready_base_, ready_total_;  // fp8 wire: per-expert "rows expanded" counter, its base, its target
  // device pointer tables, rows of `tables_`
  enum Table { kTabX, kTabG, kTabW, kTabXq, kTabGq, kTabXs, kTabGs, kTabArrive, kTabRet, kTabDw, kTabCount,
               kTabCredit, kTabTraffic0, kTabTraffic1, kTabTflags0, kTabTflags1, kNumTables };
  template <typename T>
  T* const* table(int t) const { return reinterpret_cast<T* const*>(tables_.data_ptr<int64_t>() + t * P_); }

  TokenMaps map_x_[2], map_g_[2], map_act_[2], map_dh_[2];
  CUtensorMap map_x_mn_[2], map_g_mn_[2], map_act_mn_[2], map_dh_mn_[2];
  std::map<std::tuple<const void*, uint32_t, int64_t, int64_t>, CUtensorMap> weight_maps_;

  // One public call at a time: a forward on the caller's thread, a backward on the autograd engine's and whoever asks for a header or a
  // count share all of the above and the counters below, and none of them holds the interpreter's lock meanwhile.
  mutable std::recursive_mutex pass_mutex_;
  bool released_ = false;
  cudaStream_t comm_stream_ = nullptr, aux_stream_ = nullptr, chain_[2] = {};
  cudaStream_t expand_stream_ = nullptr;  // fp8 wire: the expansion kernels run here, beside the GEMM chains
  cudaEvent_t ev_expand_[4] = {};  // expansion of slice j (mod 4) has finished
  cudaEvent_t ev_down_[2] = {}, ev_up_[2] = {}, ev_ds_[2] = {}, ev_dx_[2] = {}, ev_tgd_[2] = {}, ev_tgu_[2] = {};
  cudaEvent_t ev_pass_ = nullptr, ev_put_[4] = {}, ev_done_[4] = {};
  cudaEvent_t ev_end_ = nullptr;           // the last pass's final kernel
  unsigned long long pass_stream_ = 0;     // id of the stream that pass came on (ids are never used again, handles are)
  bool passed_ = false;                    // there was one
  int64_t last_slices_ = -1;  // slice count of the previous forward pass (the next pass's guess)
  int64_t last_rows_ = 0;     // rows that came to this rank in it
  int32_t* host_header_ = nullptr;  // pinned: 16 plan header ints + 8 status ints + their sequence number, see the .cpp
  uint32_t host_seq_ = 0;     // headers asked for so far
  bool short_pass_ = false;   // an inline pass without autograd: fewer, larger kernels
  bool inline_ = false;       // the current pass runs on the caller's stream alone

  uint32_t seq_ = 0;          // global slice sequence number of the next pass's first slice
  uint32_t fwd_epoch_ = 0;    // forward passes started (traffic exchange epoch)
  uint32_t ret_target_ = 0;   // value the returned-row counter reaches at the end of the current pass
  int64_t cur_slices_ = 0;
  int64_t cur_rows_ = 0;      // T*K of the current pass
  int64_t launches_ = 0;
  torch::Tensor prof_;
};

// Symmetric arena helpers (cudaMalloc + CUDA IPC), one arena per rank.
int64_t arena_alloc(int64_t bytes);
void arena_free(int64_t ptr);
py::bytes arena_export(int64_t ptr);
int64_t arena_import(py::bytes handle);
void arena_close(int64_t ptr);
// Bytes of this process's arenas on the current device (the caching allocator's statistics do not know them).
int64_t arenas_allocated();
void arena_zero(int64_t ptr, int64_t bytes);
void arena_fill(int64_t ptr, int64_t bytes, int value);
// Synchronises the device and copies `count` int32 values at `ptr + offset_bytes` to a CPU tensor (tests read counters).
torch::Tensor arena_read_i32(int64_t ptr, int64_t offset_bytes, int64_t count);

}  // namespace cem
