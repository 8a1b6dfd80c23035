#include "fused_rank.h"

#include <ATen/SavedTensorHooks.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <nvtx3/nvToolsExt.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <stdexcept>

#include "../common/aligned.h"
#include "tensor_map.h"

namespace cem {

namespace {

constexpr int kPutAloneBlocks = 592;  // of a put that has the device to itself: four blocks on each SM
constexpr int kBriefTokens = 96;      // see `runs_brief`
constexpr int kExpandSms = 12;  // SMs the up-projection GEMM leaves to the fp8 expansion kernel
// Pinned words: 16 of the plan header, 8 of the status block and their sequence number (written by the plan kernel), then
// a second status block for `check_status`.
constexpr int kHostSeq = kPlanHeaderInts + 8, kHostStatus = 32, kHostInts = 40;

struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  NvtxRange(const char* name, int64_t j) {
    char buf[48];
    std::snprintf(buf, sizeof(buf), "%s %lld", name, static_cast<long long>(j));
    nvtxRangePushA(buf);
  }
  ~NvtxRange() { nvtxRangePop(); }
};

inline void cuda_check(cudaError_t err, const char* what) {
  if (err != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(err));
}

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

inline cudaStream_t current_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

// (A macro: the message of a check that holds is never put together.)
#define expect(cond, msg)                            \
  do {                                               \
    if (!(cond)) throw std::runtime_error(msg);      \
  } while (0)

void expect_at_16(const torch::Tensor& t, const char* name) {
  expect(at_16_bytes(t), std::string(name) + " must be at an address of 16 bytes");
}

void expect_bf16_2d(const torch::Tensor& t, int64_t cols, const char* name) {
  expect(t.is_cuda() && t.scalar_type() == torch::kBFloat16 && t.dim() == 2 && t.size(1) == cols && t.is_contiguous(),
         std::string(name) + " must be a contiguous CUDA bf16 matrix with " + std::to_string(cols) + " columns");
  expect_at_16(t, name);
}

void expect_i32(const torch::Tensor& t, int64_t min_numel, const char* name) {
  expect(t.is_cuda() && t.scalar_type() == torch::kInt32 && t.is_contiguous() && t.numel() >= min_numel,
         std::string(name) + " must be a contiguous CUDA int32 tensor with at least " + std::to_string(min_numel) +
             " elements");
}

const char* status_name(int code) {
  switch (code) {
    case kStatusMbarTimeout: return "pipeline barrier timed out";
    case kStatusArrivalTimeout: return "dispatched rows never arrived";
    case kStatusCreditTimeout: return "a receiver never released its slice buffer";
    case kStatusReturnTimeout: return "combined rows never came back";
    case kStatusBadIndex: return "index check failed";
    case kStatusTrafficTimeout: return "a peer's traffic-matrix row never arrived";
    default: return "unknown";
  }
}

}  // namespace

ArenaLayout make_arena_layout(int P, int L, int S, int D, int tk_cap, bool fp8) {
  fp8 = fp8 && P > 1;  // a rank on its own receives nothing over the wire (`FusedRank::expands`)
  ArenaLayout a{};
  size_t o = 0;
  auto take = [&](size_t bytes) { size_t at = o; o = align_up(o + bytes, 1024); return at; };
  a.xbuf = take(2ull * S * D * 2);
  a.gbuf = take(2ull * S * D * 2);
  a.wbuf = take(2ull * S * 4);
  a.xq = take(fp8 ? 2ull * S * D : 0);
  a.gq = take(fp8 ? 2ull * S * D : 0);
  a.xs = take(fp8 ? 2ull * S * (D / 128) * 4 : 0);
  a.gs = take(fp8 ? 2ull * S * (D / 128) * 4 : 0);
  a.ret = take(static_cast<size_t>(tk_cap) * D * 2);
  a.dw_rows = take(static_cast<size_t>(tk_cap) * 4);
  a.arrive = take(static_cast<size_t>(P) * L * 4);
  a.credit = take(static_cast<size_t>(P) * 4);
  a.ret_count = take(4);
  a.traffic = take(2ull * P * P * L * 4);
  a.traffic_flags = take(2ull * P * 4);
  a.total = o;
  return a;
}

FusedRank::FusedRank(int P, int L, int me, int S, int D, int F, int K, int stripe, int tk_cap, int max_slices,
                     int num_sms, bool fp8, int64_t arena, std::vector<int64_t> peer_arenas, bool use_comm_stream,
                     int64_t spin_limit, int put_blocks)
    : P_(P), L_(L), me_(me), S_(S), D_(D), F_(F), K_(K), stripe_(stripe), tk_cap_(tk_cap), max_slices_(max_slices),
      num_sms_(num_sms), put_blocks_(put_blocks), fp8_(fp8), use_comm_stream_(use_comm_stream) {
  expect(P >= 1 && L >= 1 && me >= 0 && me < P, "bad rank geometry");
  expect(static_cast<int>(peer_arenas.size()) == P, "need one arena pointer per rank");
  expect(P <= 32, "at most 32 expert-parallel ranks (one warp lane watches one source)");
  expect(P * L <= 1024, "at most 1024 experts");
  expect(tk_cap < (1 << 27), "at most 2^27 token copies per rank (a returned row's position has 27 bits)");
  expect(D % 256 == 0, "fused kernels need D % 256 == 0");
  expect(F % 256 == 0, "fused kernels need F % 256 == 0");
  expect(stripe == 32 || stripe == 64 || stripe == 128, "fused kernels need stripe_width in {32, 64, 128}");
  expect(S % 8 == 0 && S >= 8, "fused kernels need slice_size % 8 == 0");
  expect(!fp8 || D % 128 == 0, "fp8 wire needs D % 128 == 0");
  spin_limit_ = static_cast<uint32_t>(spin_limit);
  mbar_limit_ = 20u * 1000u * 1000u;  // microseconds: longer than any legitimate wait on another rank
  lay_ = make_plan_layout(P, L, S, max_slices);
  whole_lay_ = make_plan_layout(P, L, std::max(8, (tk_cap + 7) / 8 * 8), 1);
  arena_lay_ = make_arena_layout(P, L, S, D, tk_cap, fp8);
  arena_ = reinterpret_cast<uint8_t*>(arena);
  cudaDeviceProp prop;
  cuda_check(cudaGetDevice(&device_), "device");
  cuda_check(cudaGetDeviceProperties(&prop, device_), "device properties");
  device_bytes_ = prop.totalGlobalMem;
  if (const char* v = std::getenv("CEM_KEEP_ACTIVATIONS")) keep_activations_ = std::atoi(v) != 0;
  for (int64_t p : peer_arenas) peers_.push_back(reinterpret_cast<uint8_t*>(p));

  auto bf16 = torch::TensorOptions().device(torch::kCUDA).dtype(torch::kBFloat16);
  auto f32 = torch::TensorOptions().device(torch::kCUDA).dtype(torch::kFloat32);
  auto i32 = torch::TensorOptions().device(torch::kCUDA).dtype(torch::kInt32);
  for (int q = 0; q < 2; ++q) {  // double buffered by slice parity: two slices are in flight at a time
    act_[q] = torch::zeros({S, F}, bf16);
    h_[q] = torch::zeros({S, 2 * F}, bf16);
    dh_[q] = torch::zeros({S, 2 * F}, bf16);
    dwp_[q] = torch::zeros({S, F / 32}, f32);
  }
  carry_up_ = torch::zeros({2, D, 2 * F}, f32);
  carry_down_ = torch::zeros({2, F, D}, f32);
  pass_base_ = torch::zeros({P * L}, i32);
  ready_ = torch::zeros({L}, i32);
  ready_base_ = torch::zeros({L}, i32);
  ready_total_ = torch::zeros({L}, i32);
  brief_tokens_ = torch::zeros({kPlanSmallIds}, i32);
  expected_total_ = torch::zeros({P * L}, i32);
  status_ = torch::zeros({8}, i32);
  my_counts_ = torch::zeros({P * L}, i32);
  sort_scratch_ = torch::zeros({static_cast<int64_t>(expert_sort_scratch_ints(tk_cap, P * L))}, i32);

  // Pointer tables: row t holds, for every rank r, the address of buffer t inside r's arena.
  std::vector<int64_t> host(static_cast<size_t>(kNumTables) * P);
  const size_t traffic_half = static_cast<size_t>(P) * P * L * 4, flags_half = static_cast<size_t>(P) * 4;
  for (int r = 0; r < P; ++r) {
    auto at = [&](size_t off) { return reinterpret_cast<int64_t>(peers_[r] + off); };
    host[kTabX * P + r] = at(arena_lay_.xbuf);
    host[kTabG * P + r] = at(arena_lay_.gbuf);
    host[kTabW * P + r] = at(arena_lay_.wbuf);
    host[kTabXq * P + r] = at(arena_lay_.xq);
    host[kTabGq * P + r] = at(arena_lay_.gq);
    host[kTabXs * P + r] = at(arena_lay_.xs);
    host[kTabGs * P + r] = at(arena_lay_.gs);
    host[kTabArrive * P + r] = at(arena_lay_.arrive);
    host[kTabRet * P + r] = at(arena_lay_.ret);
    host[kTabDw * P + r] = at(arena_lay_.dw_rows);
    host[kTabCount * P + r] = at(arena_lay_.ret_count);
    host[kTabCredit * P + r] = at(arena_lay_.credit);
    host[kTabTraffic0 * P + r] = at(arena_lay_.traffic);
    host[kTabTraffic1 * P + r] = at(arena_lay_.traffic + traffic_half);
    host[kTabTflags0 * P + r] = at(arena_lay_.traffic_flags);
    host[kTabTflags1 * P + r] = at(arena_lay_.traffic_flags + flags_half);
  }
  tables_ = torch::from_blob(host.data(), {static_cast<int64_t>(kNumTables), P}, torch::kInt64).clone().to(torch::kCUDA);

  // TMA descriptors of the local buffers: row-wise operands by tile width, weight-gradient operands as 64 rows of two
  // 64-column chunks brought by one 3-D copy (what each CTA of a pair loads).
  for (int b = 0; b < 2; ++b) {
    const void* xb = arena_ + arena_lay_.xbuf + static_cast<size_t>(b) * S * D * 2;
    const void* gb = arena_ + arena_lay_.gbuf + static_cast<size_t>(b) * S * D * 2;
    map_x_[b] = make_token_maps(xb, S, D);
    map_x_mn_[b] = make_bf16_map_chunked(xb, S, D, 64, 2);
    map_g_[b] = make_token_maps(gb, S, D);
    map_g_mn_[b] = make_bf16_map_chunked(gb, S, D, 64, 2);
  }
  for (int q = 0; q < 2; ++q) {
    map_act_[q] = make_token_maps(act_[q].data_ptr(), S, F);
    map_act_mn_[q] = make_bf16_map_chunked(act_[q].data_ptr(), S, F, 64, 2);
    map_dh_[q] = make_token_maps(dh_[q].data_ptr(), S, 2 * F);
    map_dh_mn_[q] = make_bf16_map_chunked(dh_[q].data_ptr(), S, 2 * F, 64, 2);
  }

  if (use_comm_stream_) {
    // The put and expansion kernels feed kernels that wait for them: their blocks go first when SMs free up.
    int prio_low = 0, prio_high = 0;
    cuda_check(cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high), "stream priority range");
    if (const char* v = std::getenv("CEM_COMM_PRIORITY")) {
      if (std::atoi(v) == 0) prio_high = prio_low;  // measurement knob: comm streams at the default priority
    }
    cuda_check(cudaStreamCreateWithPriority(&comm_stream_, cudaStreamNonBlocking, prio_high), "comm stream");
    cuda_check(cudaStreamCreateWithFlags(&aux_stream_, cudaStreamNonBlocking), "aux stream");
    for (int q = 0; q < 2; ++q) cuda_check(cudaStreamCreateWithFlags(&chain_[q], cudaStreamNonBlocking), "chain stream");
    if (expands()) cuda_check(cudaStreamCreateWithPriority(&expand_stream_, cudaStreamNonBlocking, prio_high), "expand stream");
  }
  for (int i = 0; i < 4; ++i) cuda_check(cudaEventCreateWithFlags(&ev_expand_[i], cudaEventDisableTiming), "event");
  for (int q = 0; q < 2; ++q)
    for (cudaEvent_t* e : {&ev_down_[q], &ev_up_[q], &ev_ds_[q], &ev_dx_[q], &ev_tgd_[q], &ev_tgu_[q]})
      cuda_check(cudaEventCreateWithFlags(e, cudaEventDisableTiming), "event");
  cuda_check(cudaEventCreateWithFlags(&ev_pass_, cudaEventDisableTiming), "event");
  cuda_check(cudaEventCreateWithFlags(&ev_end_, cudaEventDisableTiming), "event");
  for (int i = 0; i < 4; ++i) {
    cuda_check(cudaEventCreateWithFlags(&ev_put_[i], cudaEventDisableTiming), "event");
    cuda_check(cudaEventCreateWithFlags(&ev_done_[i], cudaEventDisableTiming), "event");
  }
  cuda_check(cudaMallocHost(reinterpret_cast<void**>(&host_header_), kHostInts * sizeof(int32_t)), "pinned header");
  std::memset(host_header_, 0, kHostInts * sizeof(int32_t));
}

FusedRank::~FusedRank() {
  if (comm_stream_) cudaStreamDestroy(comm_stream_);
  if (aux_stream_) cudaStreamDestroy(aux_stream_);
  if (expand_stream_) cudaStreamDestroy(expand_stream_);
  for (int i = 0; i < 4; ++i)
    if (ev_expand_[i]) cudaEventDestroy(ev_expand_[i]);
  for (int q = 0; q < 2; ++q) {
    if (chain_[q]) cudaStreamDestroy(chain_[q]);
    for (cudaEvent_t e : {ev_down_[q], ev_up_[q], ev_ds_[q], ev_dx_[q], ev_tgd_[q], ev_tgu_[q]})
      if (e) cudaEventDestroy(e);
  }
  if (ev_pass_) cudaEventDestroy(ev_pass_);
  if (ev_end_) cudaEventDestroy(ev_end_);
  for (int i = 0; i < 4; ++i) {
    if (ev_put_[i]) cudaEventDestroy(ev_put_[i]);
    if (ev_done_[i]) cudaEventDestroy(ev_done_[i]);
  }
  if (host_header_) cudaFreeHost(host_header_);
}

void FusedRank::release() {
  const Turn turn(pass_mutex_);
  released_ = true;
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device_));
  cudaDeviceSynchronize();  // (an error of the device is raised by whoever frees the arena)
  // Nodes of graphs that are still alive hold the rank, but they have no use for its scratch any more.
  for (auto* scratch : {&act_, &h_, &dh_, &dwp_})
    for (torch::Tensor& t : *scratch) t = torch::Tensor();
  carry_up_ = carry_down_ = sort_scratch_ = prof_ = torch::Tensor();
  release_kept();
}

void FusedRank::expect_arena(const char* what) const {
  expect(!released_, std::string("chunked_moe fused path: the workspace of this pass was released before its ") + what);
}

void FusedRank::check_status() {
  const Turn turn(pass_mutex_);
  cudaStream_t st = current_stream();
  cuda_check(cudaMemcpyAsync(host_header_ + kHostStatus, status_.data_ptr(), 8 * sizeof(int32_t),
                             cudaMemcpyDeviceToHost, st),
             "status copy");
  cuda_check(cudaStreamSynchronize(st), "status sync");
  const int32_t* s = host_header_ + kHostStatus;
  if (s[0] != 0) {
    const std::string message = format_status(std::vector<int64_t>(s, s + 8), me_);
    cuda_check(cudaMemsetAsync(status_.data_ptr(), 0, 8 * sizeof(int32_t), st), "status clear");
    cuda_check(cudaStreamSynchronize(st), "status clear sync");
    throw std::runtime_error(message);
  }
}

std::string format_status(const std::vector<int64_t>& s, int rank) {
  if (s.size() < 8) return "chunked_moe fused path: malformed status block";
  char buf[512];
  std::snprintf(buf, sizeof(buf),
                "chunked_moe fused path: %s (code %lld, kernel %lld, mode %lld, slice/tile %lld, detail %lld, "
                "expected %llu, seen %llu, block %lld, rank %d)",
                status_name(static_cast<int>(s[0])), static_cast<long long>(s[0]), static_cast<long long>(s[1]),
                static_cast<long long>(s[2]), static_cast<long long>(s[3]), static_cast<long long>(s[4]),
                static_cast<unsigned long long>(static_cast<uint32_t>(s[5])),
                static_cast<unsigned long long>(static_cast<uint32_t>(s[6])), static_cast<long long>(s[7]), rank);
  return std::string(buf);
}

void FusedRank::sort_only(torch::Tensor expert_ids, torch::Tensor order, torch::Tensor inv_order,
                          torch::Tensor my_counts) {
  const Turn turn(pass_mutex_);
  expect_arena("step");
  const int64_t tk = expert_ids.numel();
  expect(tk <= tk_cap_, "T*K exceeds the workspace capacity");
  expect_i32(expert_ids, tk, "expert_ids");
  expect_i32(order, tk, "order");
  expect_i32(inv_order, tk, "inv_order");
  expect_i32(my_counts, P_ * L_, "my_counts");
  launch_expert_sort(expert_ids.data_ptr<int>(), static_cast<int>(tk), P_ * L_, order.data_ptr<int>(),
                     inv_order.data_ptr<int>(), my_counts.data_ptr<int>(), sort_scratch_.data_ptr<int>(),
                     current_stream(), reinterpret_cast<StatusBlock*>(status_.data_ptr()));
  launches_ += 3;
}

int64_t FusedRank::begin_forward_async(torch::Tensor expert_ids, torch::Tensor plan, torch::Tensor order,
                                       torch::Tensor inv_order, torch::Tensor counts, bool counts_prefilled) {
  const Turn turn(pass_mutex_);
  expect_arena("step");
  cudaStream_t st = current_stream();
  const int64_t tk = expert_ids.numel();
  expect(tk <= tk_cap_, "T*K exceeds the workspace capacity");
  expect_i32(plan, lay_.total, "plan");
  expect_at_16(plan, "plan");
  enter_pass();
  header_whole_ = false;
  PlanKernelParams pp{};
  pp.lay = lay_;
  pp.me = me_;
  pp.plan = plan.data_ptr<int>();
  pp.spin_limit = spin_limit_;
  pp.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
  pp.host_out = host_header_;
  pp.host_seq = ++host_seq_;
  if (short_pass_ && tk <= kPlanSmallIds && L_ <= kPlanSmallExperts) {
    expect_i32(expert_ids, tk, "expert_ids");
    expect_i32(order, tk, "order");
    expect_i32(inv_order, tk, "inv_order");
    launch_plan_small(pp, expert_ids.data_ptr<int>(), static_cast<int>(tk), order.data_ptr<int>(),
                      inv_order.data_ptr<int>(), reinterpret_cast<uint32_t*>(expected_total_.data_ptr()),
                      reinterpret_cast<uint32_t*>(pass_base_.data_ptr()), RowTable{}, st);
    ++launches_;
    begin_pass(plan, max_slices_, tk, D_ / kCombineCols, /*targets_set=*/true);
    return last_slices_;
  }
  if (counts_prefilled) {
    expect_i32(counts, static_cast<int64_t>(P_) * P_ * L_, "counts");
    pp.counts = counts.data_ptr<int>();
    pp.my_counts = counts.data_ptr<int>() + static_cast<size_t>(me_) * P_ * L_;
    pp.peer_counts = nullptr;
    pp.peer_flags = nullptr;
    pp.flags = nullptr;
    pp.epoch = 0;
  } else {
    sort_only(expert_ids, order, inv_order, my_counts_);
    const uint32_t epoch = ++fwd_epoch_;
    const int parity = static_cast<int>(epoch & 1u);
    pp.my_counts = my_counts_.data_ptr<int>();
    pp.counts = reinterpret_cast<int*>(arena_ + arena_lay_.traffic + static_cast<size_t>(parity) * P_ * P_ * L_ * 4);
    pp.peer_counts = table<int>(parity ? kTabTraffic1 : kTabTraffic0);
    pp.peer_flags = table<uint32_t>(parity ? kTabTflags1 : kTabTflags0);
    pp.flags = reinterpret_cast<const uint32_t*>(arena_ + arena_lay_.traffic_flags + static_cast<size_t>(parity) * P_ * 4);
    pp.epoch = epoch;
  }
  // The plan kernel itself stores header and status to the pinned words as soon as it knows them; nobody waits here.
  launch_plan_build(pp, st);
  ++launches_;
  // any slice below the workspace's capacity may be launched until resolved; D/128 pieces per row come back
  begin_pass(plan, max_slices_, tk, D_ / kCombineCols);
  return last_slices_ < 0 ? -1 : std::min<int64_t>(last_slices_, max_slices_);
}

// Waits for the plan kernel's stores to the pinned words. Polling memory notices them in well under a microsecond (a
// blocking event wait and the two copies it followed took 25-40 us on the way of a one-token decode); a wait that turns
// out long, behind a stream full of earlier work, sleeps between polls.
void FusedRank::wait_header() {
  const volatile uint32_t* seq = reinterpret_cast<const volatile uint32_t*>(host_header_ + kHostSeq);
  cudaStream_t st = current_stream();
  const auto arrived = [&]() { return *seq == host_seq_; };
  const auto spin = [&](bool sleeping) {  // true: arrived, false: the time for busy polling is over
    const auto t0 = std::chrono::steady_clock::now();
    for (uint32_t i = 1; !arrived(); ++i) {
      if (sleeping) {
        usleep(20);
      } else if (i % 256 != 0) {
        continue;
      }
      // A stream that has failed, or is done without the store having become visible, ends the wait.
      const cudaError_t state = cudaStreamQuery(st);
      if (state == cudaSuccess && !arrived()) throw std::runtime_error("plan header wait: the plan kernel did not report");
      if (state != cudaSuccess && state != cudaErrorNotReady) cuda_check(state, "plan header wait");
      if (!sleeping && std::chrono::steady_clock::now() - t0 > std::chrono::microseconds(150)) return false;
    }
    return true;
  };
  if (!spin(false)) spin(true);
  std::atomic_thread_fence(std::memory_order_acquire);
}

// Waits until nothing that was launched for a pass runs any more: behind an error the pass's tensors are about to be released
// and the status block, which makes its remaining kernels return at once, to be cleared. (Every wait in a kernel is bounded.)
void FusedRank::quiesce() const {
  for (cudaStream_t s : {comm_stream_, expand_stream_, chain_[0], chain_[1], aux_stream_})
    if (s != nullptr) cudaStreamSynchronize(s);
  cudaStreamSynchronize(current_stream());
}

int64_t FusedRank::resolve_slices() {
  const Turn turn(pass_mutex_);
  wait_header();
  std::string message;
  const int32_t* st = host_header_ + 16;
  if (st[0] != 0) message = format_status(std::vector<int64_t>(st, st + 8), me_);
  else if (host_header_[4] != 0) message = "routing needs more slices than the workspace was sized for (max_slices)";
  else if (host_header_[5] != cur_rows_) message = "the routing plan does not account for every token copy";
  if (!message.empty()) {
    quiesce();  // what was launched on the guess ends (at once, if an error is recorded) before anything is cleared
    if (st[0] != 0) {
      cuda_check(cudaMemsetAsync(status_.data_ptr(), 0, 8 * sizeof(int32_t), current_stream()), "status clear");
      cuda_check(cudaStreamSynchronize(current_stream()), "status clear sync");
    }
    throw std::runtime_error(message);
  }
  last_slices_ = host_header_[0];
  last_rows_ = host_header_[1];
  return last_slices_;
}

void FusedRank::set_pass_slices(int64_t launched) {
  const Turn turn(pass_mutex_);
  expect(launched >= 0 && launched <= max_slices_, "slice count exceeds the workspace");
  cur_slices_ = launched;
}

void FusedRank::set_mbar_limit_us(int64_t us) {
  const Turn turn(pass_mutex_);
  expect(us > 0 && us <= 600ll * 1000 * 1000, "barrier limit must be between 1 us and 600 s");
  mbar_limit_ = static_cast<uint32_t>(us);
}

int64_t FusedRank::begin_forward(torch::Tensor expert_ids, torch::Tensor plan, torch::Tensor order,
                                 torch::Tensor inv_order, torch::Tensor counts, bool counts_prefilled) {
  const Turn turn(pass_mutex_);
  begin_forward_async(expert_ids, plan, order, inv_order, counts, counts_prefilled);
  const int64_t n = resolve_slices();
  set_pass_slices(n);
  return n;
}


int64_t FusedRank::begin_backward(torch::Tensor plan, int64_t known_slices, int64_t known_rows) {
  const Turn turn(pass_mutex_);
  expect_arena("step");
  cudaStream_t st = current_stream();
  expect_i32(plan, lay_.total, "plan");
  expect_at_16(plan, "plan");
  enter_pass();
  if (known_slices >= 0 && known_rows >= 0) {
    // The caller kept what the forward of this plan read back: no device-to-host copy, no synchronisation, so the
    // host keeps running ahead of the device through the whole backward. (A recorded kernel error then surfaces at
    // the next synchronising call: the next forward, or `check_status`.)
    expect(known_slices <= max_slices_, "slice count exceeds the workspace");
    cur_slices_ = known_slices;
    cur_rows_ = known_rows;
  } else {
    cuda_check(cudaMemcpyAsync(host_header_, plan.data_ptr(), 16 * sizeof(int32_t), cudaMemcpyDeviceToHost, st),
               "plan header copy");
    check_status();  // synchronises the stream: header and status are both on the host now
    expect(host_header_[4] == 0, "routing needs more slices than the workspace was sized for (max_slices)");
    cur_slices_ = host_header_[0];
    cur_rows_ = host_header_[5];
  }
  begin_pass(plan, cur_slices_, cur_rows_, D_ / kCombineCols + 1);  // per row: the pieces of dx and the d_weight scalar
  return cur_slices_;
}

// Passes of a workspace share its scratch, its return buffer and its counters, whatever streams they come on: a pass on
// another stream than the one before waits there for that one's end. (One event record per pass; nothing else as long as the
// stream stays the same.)
void FusedRank::enter_pass() {
  cudaStream_t st = current_stream();
  unsigned long long id = 0;
  cuda_check(cudaStreamGetId(st, &id), "stream id");
  if (passed_ && id != pass_stream_) cuda_check(cudaStreamWaitEvent(st, ev_end_, 0), "wait for the last pass");
  pass_stream_ = id;
}

void FusedRank::begin_pass(const torch::Tensor& plan, int64_t slices, int64_t rows, int pieces_per_row,
                           bool targets_set) {
  cudaStream_t st = current_stream();
  cur_slices_ = slices;
  cur_rows_ = rows;
  if (!targets_set) {
    launch_pass_begin(plan.data_ptr<int>(), lay_, reinterpret_cast<uint32_t*>(expected_total_.data_ptr()),
                      reinterpret_cast<uint32_t*>(pass_base_.data_ptr()),
                      expands() ? reinterpret_cast<uint32_t*>(ready_total_.data_ptr()) : nullptr,
                      expands() ? reinterpret_cast<uint32_t*>(ready_base_.data_ptr()) : nullptr, st);
    ++launches_;
  }
  ret_target_ += static_cast<uint32_t>(cur_rows_) * static_cast<uint32_t>(pieces_per_row);
  if (overlapped()) cuda_check(cudaEventRecord(ev_pass_, st), "event record");
}

void FusedRank::put(int64_t j, torch::Tensor plan, torch::Tensor order, torch::Tensor x,
                    c10::optional<torch::Tensor> g, torch::Tensor w_flat) {
  const Turn turn(pass_mutex_);
  expect_arena("step");
  expect(j >= 0 && j < cur_slices_, "slice index out of range");
  expect_bf16_2d(x, D_, "x");
  if (g.has_value()) expect_bf16_2d(*g, D_, "g");
  expect(w_flat.is_cuda() && w_flat.scalar_type() == torch::kFloat32 && w_flat.is_contiguous() &&
             w_flat.numel() == cur_rows_,
         "router weights must be a contiguous CUDA fp32 tensor of T*K elements");
  expect_i32(order, cur_rows_, "order");
  cudaStream_t st = overlapped() ? comm_stream_ : current_stream();
  if (overlapped()) {
    if (j == 0) cuda_check(cudaStreamWaitEvent(comm_stream_, ev_pass_, 0), "wait pass event");
    if (j >= 2) cuda_check(cudaStreamWaitEvent(comm_stream_, ev_done_[(j - 2) % 4], 0), "wait slice event");
  }
  PutParams p{};
  p.plan = plan.data_ptr<int>();
  p.lay = lay_;
  p.slice = static_cast<int>(j);
  p.seq = seq_ + static_cast<uint32_t>(j);
  p.me = me_;
  p.top_k = K_;
  p.hidden = D_;
  p.order = order.data_ptr<int>();
  p.x = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr());
  p.g = g.has_value() ? reinterpret_cast<const __nv_bfloat16*>(g->data_ptr()) : nullptr;
  p.w_flat = w_flat.data_ptr<float>();
  p.num_tokens = static_cast<int>(x.size(0));
  p.peer_x = table<__nv_bfloat16>(kTabX);
  p.peer_g = table<__nv_bfloat16>(kTabG);
  p.peer_w = table<float>(kTabW);
  p.peer_arrive = table<uint32_t>(kTabArrive);
  p.credit = reinterpret_cast<const uint32_t*>(arena_ + arena_lay_.credit);
  p.spin_limit = spin_limit_;
  p.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
  p.round_fp8 = fp8_ && !expands();
  if (expands()) {
    p.peer_xq = table<uint8_t>(kTabXq);
    p.peer_gq = table<uint8_t>(kTabGq);
    p.peer_xs = table<float>(kTabXs);
    p.peer_gs = table<float>(kTabGs);
  }
  launch_dispatch_put(p, put_blocks_, st, inline_);
  ++launches_;
  if (overlapped()) cuda_check(cudaEventRecord(ev_put_[j % 4], comm_stream_), "event record");
  if (expands() && overlapped()) {
    // The expansion of slice j is issued together with its put, one slice ahead of the GEMMs: it waits for arrivals
    // expert by expert while slice j-1 computes. It may overwrite the bf16 slice buffer once slice j-2 is done with it.
    if (j == 0) cuda_check(cudaStreamWaitEvent(expand_stream_, ev_pass_, 0), "wait pass event");
    if (j >= 2) cuda_check(cudaStreamWaitEvent(expand_stream_, ev_done_[(j - 2) % 4], 0), "wait slice event");
    dequant(plan.data_ptr<int>(), static_cast<int>(j), static_cast<int>(p.seq & 1u), g.has_value(), expand_stream_);
    cuda_check(cudaEventRecord(ev_expand_[j % 4], expand_stream_), "event record");
  }
}

GemmParams FusedRank::base_params(const int* plan, int j) const {
  GemmParams p{};
  p.plan = plan;
  p.lay = lay_;
  p.slice = j;
  p.me = me_;
  p.stripe = stripe_;
  p.spin_limit = spin_limit_;
  p.mbar_limit = mbar_limit_;
  p.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
  return p;
}

const CUtensorMap& FusedRank::weight_map(const torch::Tensor& w, uint32_t box_rows, uint32_t chunks) {
  // Keyed by address AND geometry: a freed tensor's address can come back with another shape.
  auto key = std::make_tuple(static_cast<const void*>(w.data_ptr()), box_rows | (chunks << 16),
                             static_cast<int64_t>(w.size(0)) * w.size(1), static_cast<int64_t>(w.size(2)));
  auto it = weight_maps_.find(key);
  if (it == weight_maps_.end()) {
    if (weight_maps_.size() > 4096) weight_maps_.clear();
    // [L, R, C] viewed as the 2-D matrix [L*R, C]; tiles never straddle experts because R % box_rows == 0.
    const uint64_t rows = static_cast<uint64_t>(w.size(0)) * w.size(1), cols = static_cast<uint64_t>(w.size(2));
    it = weight_maps_.emplace(key, chunks ? make_bf16_map_chunked(w.data_ptr(), rows, cols, box_rows, chunks)
                                          : make_bf16_map_2d(w.data_ptr(), rows, cols, box_rows)).first;
  }
  return it->second;
}

const CUtensorMap& FusedRank::up_map(const torch::Tensor& w_up) { return weight_map(w_up, 64, stripe_ == 128 ? 1 : 2); }

void FusedRank::dequant(const int* plan, int j, int b, bool with_g, cudaStream_t st) {
  // Rows arrived as e4m3 + block scales: expand them into the bf16 slice buffers the GEMMs read.
  DequantParams d{};
  d.plan = plan;
  d.lay = lay_;
  d.slice = j;
  d.hidden = D_;
  d.arrive = reinterpret_cast<const uint32_t*>(arena_ + arena_lay_.arrive);
  d.pass_base = reinterpret_cast<const uint32_t*>(pass_base_.data_ptr());
  const size_t rows_off = static_cast<size_t>(b) * S_;
  d.xq = arena_ + arena_lay_.xq + rows_off * D_;
  d.xs = reinterpret_cast<const float*>(arena_ + arena_lay_.xs) + rows_off * (D_ / 128);
  d.x = reinterpret_cast<__nv_bfloat16*>(arena_ + arena_lay_.xbuf) + rows_off * D_;
  if (with_g) {
    d.gq = arena_ + arena_lay_.gq + rows_off * D_;
    d.gs = reinterpret_cast<const float*>(arena_ + arena_lay_.gs) + rows_off * (D_ / 128);
    d.g = reinterpret_cast<__nv_bfloat16*>(arena_ + arena_lay_.gbuf) + rows_off * D_;
  }
  d.ready = reinterpret_cast<uint32_t*>(ready_.data_ptr());
  d.spin_limit = spin_limit_;
  d.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
  launch_dequant_slice(d, st);
  ++launches_;
}

void FusedRank::set_pipeline_counters(c10::optional<torch::Tensor> counters) {
  const Turn turn(pass_mutex_);
  if (passed_) cuda_check(cudaEventSynchronize(ev_end_), "wait for the last pass");
  quiesce();  // (and for whatever has filled the new counters)
  if (!counters.has_value()) {
    prof_ = torch::Tensor();
    return;
  }
  const torch::Tensor& t = *counters;
  expect(t.is_cuda() && t.scalar_type() == torch::kInt64 && t.is_contiguous() && t.dim() == 3 && t.size(0) == 6 &&
             t.size(1) >= num_sms_ && t.size(2) == kProfSlots,
         "pipeline counters must be a contiguous CUDA int64 [6, >= num_sms, 8] tensor");
  prof_ = t;
}

void FusedRank::count_pipeline(int mode, GemmParams* p) {
  if (prof_.defined())
    p->prof = reinterpret_cast<unsigned long long*>(prof_.data_ptr<int64_t>()) +
              static_cast<size_t>(mode) * prof_.size(1) * kProfSlots;
}

void FusedRank::row_gemm(int mode, const GemmParams& p0, const CUtensorMap& weights, const TokenMaps& rows,
                         cudaStream_t st, int spare_sms) {
  GemmParams p = p0;
  count_pipeline(mode, &p);
  launch_row_gemm(mode, p, weights, rows, std::max(2, num_sms_ - spare_sms), st, inline_);
  ++launches_;
}

void FusedRank::weight_grad(const GemmParams& p0, const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& out,
                            cudaStream_t st) {
  GemmParams p = p0;
  count_pipeline(kModeTgmm, &p);
  // (Slice by slice the rows are cut as they come: how many an expert has of them is anything up to a slice.)
  launch_weight_grad(p, a, b, out, std::max(2, num_sms_), p0.lay.S == whole_lay_.S ? cur_rows_ : S_, st, inline_);
  ++launches_;
}

namespace {
void expect_weights(const torch::Tensor& w_up, const torch::Tensor& w_down, int L, int D, int F) {
  expect(w_up.is_cuda() && w_up.scalar_type() == torch::kBFloat16 && w_up.is_contiguous() && w_up.dim() == 3 &&
             w_up.size(0) == L && w_up.size(1) == D && w_up.size(2) == 2 * F,
         "w_up must be a contiguous CUDA bf16 [L, D, 2F] tensor");
  expect(w_down.is_cuda() && w_down.scalar_type() == torch::kBFloat16 && w_down.is_contiguous() && w_down.dim() == 3 &&
             w_down.size(0) == L && w_down.size(1) == F && w_down.size(2) == D,
         "w_down must be a contiguous CUDA bf16 [L, F, D] tensor");
}
}  // namespace

// Two slices are in flight at a time. Even and odd slices run their kernel chains on two streams with their own
// scratch buffers, the weight-gradient GEMMs and the in-order credit release run on an auxiliary stream, the puts on
// the comm stream. A persistent GEMM kernel needs a whole SM per CTA, so two ready kernels do not share SMs: the
// later one's CTAs start as the earlier one's CTAs finish, i.e. every kernel fills the idle tail of the previous
// (independent) one instead of waiting for it. Scratch reuse and the carry chain are ordered by events.
void FusedRank::compute_forward(int64_t j, torch::Tensor plan, torch::Tensor w_up, torch::Tensor w_down) {
  const Turn turn(pass_mutex_);
  expect_arena("step");
  expect(j >= 0 && j < cur_slices_, "slice index out of range");
  expect_weights(w_up, w_down, L_, D_, F_);
  const bool async = overlapped();
  const int q = static_cast<int>(j & 1);
  cudaStream_t st = async ? chain_[q] : current_stream();
  cudaStream_t aux = async ? aux_stream_ : st;
  if (async) {
    cuda_check(cudaStreamWaitEvent(st, ev_put_[j % 4], 0), "wait put event");  // (behind the pass event)
  }
  const uint32_t seq = seq_ + static_cast<uint32_t>(j);
  const int b = static_cast<int>(seq & 1u);
  const int* pl = plan.data_ptr<int>();
  const bool keep = j < kept_slices_;
  if (expands() && !async) dequant(pl, static_cast<int>(j), b, /*with_g=*/false, st);  // lockstep: every put is done
  {
    GemmParams p = base_params(pl, static_cast<int>(j));
    p.n_tiles = 2 * F_ / kBlockN;
    p.k_blocks = D_ / kBlockK;
    p.b_group_rows = D_;
    p.arrive = expands() ? nullptr : reinterpret_cast<const uint32_t*>(arena_ + arena_lay_.arrive);
    p.pass_base = reinterpret_cast<const uint32_t*>(pass_base_.data_ptr());
    p.ready = expands() ? reinterpret_cast<const uint32_t*>(ready_.data_ptr()) : nullptr;
    p.ready_base = reinterpret_cast<const uint32_t*>(ready_base_.data_ptr());
    p.row_w = reinterpret_cast<const float*>(arena_ + arena_lay_.wbuf) + static_cast<size_t>(b) * S_;
    p.out0 = keep ? kept_act(j) : reinterpret_cast<__nv_bfloat16*>(act_[q].data_ptr());
    p.ld0 = F_;
    p.out1 = keep ? kept_h(j) : nullptr;
    p.ld1 = 2 * F_;
    // fp8 wire: this kernel waits (in its producer warp) for the expansion kernel of the same slice. A persistent CTA
    // takes all of an SM's shared memory, so nothing else can start beside it: the kernel leaves a few SMs free for the
    // expansion kernel, and it only starts once the expansion of the PREVIOUS slice has finished, so that at most one
    // kernel is ever waiting for an expansion that still needs SMs.
    if (expands() && async && j >= 1) cuda_check(cudaStreamWaitEvent(st, ev_expand_[(j - 1) % 4], 0), "wait expansion");
    row_gemm(kModeSwiglu, p, up_map(w_up), map_x_[b], st, expands() && async ? kExpandSms : 0);
  }
  {
    GemmParams p = base_params(pl, static_cast<int>(j));
    p.n_tiles = D_ / kBlockN;
    p.k_blocks = F_ / kBlockK;
    p.b_group_rows = F_;
    p.peer_rows = table<__nv_bfloat16>(kTabRet);
    p.peer_count = table<uint32_t>(kTabCount);
    p.ld0 = D_;
    row_gemm(kModeDownFwd, p, weight_map(w_down, 64, 2),
             keep ? make_token_maps(kept_act(j), kept_slice_rows(j), F_) : map_act_[q], st);
  }
  if (async) {
    cuda_check(cudaEventRecord(ev_down_[q], st), "event record");
    cuda_check(cudaStreamWaitEvent(aux, ev_down_[q], 0), "wait down event");
  }
  if (!short_pass_) {  // (else the combine kernel gives the credit)
    launch_slice_done(table<uint32_t>(kTabCredit), P_, me_, seq, aux);  // credits leave in slice order
    ++launches_;
  }
  if (async) cuda_check(cudaEventRecord(ev_done_[j % 4], aux), "event record");
}

void FusedRank::compute_backward(int64_t j, torch::Tensor plan, torch::Tensor w_up, torch::Tensor w_down,
                                 torch::Tensor dw_up, torch::Tensor dw_down) {
  const Turn turn(pass_mutex_);
  expect_arena("step");
  expect(j >= 0 && j < cur_slices_, "slice index out of range");
  expect_weights(w_up, w_down, L_, D_, F_);
  expect_weights(dw_up, dw_down, L_, D_, F_);
  const bool async = overlapped();
  const int q = static_cast<int>(j & 1);
  cudaStream_t st = async ? chain_[q] : current_stream();
  cudaStream_t aux = async ? aux_stream_ : st;
  const bool keep = j < kept_slices_;
  if (async) {
    cuda_check(cudaStreamWaitEvent(st, ev_put_[j % 4], 0), "wait put event");  // (behind the pass event)
    if (!keep && j >= 2) cuda_check(cudaStreamWaitEvent(st, ev_tgd_[q], 0), "wait dW_down event");  // act of slice j-2
  }
  const uint32_t seq = seq_ + static_cast<uint32_t>(j);
  const int b = static_cast<int>(seq & 1u);
  const int* pl = plan.data_ptr<int>();
  const int par = static_cast<int>(j & 1);
  const int dwp_tiles = F_ / 32;
  if (expands() && !async) dequant(pl, static_cast<int>(j), b, /*with_g=*/true, st);  // lockstep: every put is done
  // fp8 wire: the slice's first GEMM waits (in its producer warp) for the expansion kernel of the same slice. A persistent
  // CTA takes all of an SM's shared memory, so nothing else can start beside it: that GEMM leaves a few SMs free for the
  // expansion kernel, and it only starts once the expansion of the PREVIOUS slice has finished, so that at most one kernel
  // is ever waiting for an expansion that still needs SMs.
  if (expands() && async && j >= 1) cuda_check(cudaStreamWaitEvent(st, ev_expand_[(j - 1) % 4], 0), "wait expansion");
  const int spare = expands() && async ? kExpandSms : 0;
  auto wait_for_rows = [&](GemmParams* p) {
    p->arrive = expands() ? nullptr : reinterpret_cast<const uint32_t*>(arena_ + arena_lay_.arrive);
    p->pass_base = reinterpret_cast<const uint32_t*>(pass_base_.data_ptr());
    p->ready = expands() ? reinterpret_cast<const uint32_t*>(ready_.data_ptr()) : nullptr;
    p->ready_base = reinterpret_cast<const uint32_t*>(ready_base_.data_ptr());
  };
  // Unless the forward kept them: h and w * act again. y is not recomputed: d_weight = <g, act Wd> = <g Wd^T, act> is a
  // by-product of the next GEMM, so the down-projection GEMM that used to form <g, y> and w * g here (8 % of a step's FLOPs, 230 us per 8192-row slice at
  // D=7168, F=2048) and the w * g matrix are gone: 23.1 -> 21.4 ms per forward + backward at 32 experts, 65,536 rows.
  if (!keep) {
    GemmParams p = base_params(pl, static_cast<int>(j));
    p.row_w = reinterpret_cast<const float*>(arena_ + arena_lay_.wbuf) + static_cast<size_t>(b) * S_;
    p.n_tiles = 2 * F_ / kBlockN;
    p.k_blocks = D_ / kBlockK;
    p.b_group_rows = D_;
    wait_for_rows(&p);
    p.out0 = reinterpret_cast<__nv_bfloat16*>(act_[q].data_ptr());
    p.ld0 = F_;
    p.out1 = reinterpret_cast<__nv_bfloat16*>(h_[q].data_ptr());
    p.ld1 = 2 * F_;
    row_gemm(kModeSwiglu, p, up_map(w_up), map_x_[b], st, spare);
    if (async) cuda_check(cudaEventRecord(ev_up_[q], st), "event record");
  }
  if (async && j >= 2) cuda_check(cudaStreamWaitEvent(st, ev_tgu_[q], 0), "wait dW_up event");  // dh, d_weight shares of slice j-2
  {  // acc = g Wd^T; dh = SwiGLU'(h) * (w * acc), d_weight shares <acc, w * act>
    GemmParams p = base_params(pl, static_cast<int>(j));
    p.n_tiles = F_ / kBlockN;
    p.k_blocks = D_ / kBlockK;
    p.b_group_rows = F_;
    p.row_w = reinterpret_cast<const float*>(arena_ + arena_lay_.wbuf) + static_cast<size_t>(b) * S_;
    if (keep) wait_for_rows(&p);
    p.in0 = keep ? kept_h(j) : reinterpret_cast<const __nv_bfloat16*>(h_[q].data_ptr());
    p.in1 = keep ? kept_act(j) : reinterpret_cast<const __nv_bfloat16*>(act_[q].data_ptr());
    p.ld1 = F_;
    p.out0 = reinterpret_cast<__nv_bfloat16*>(dh_[q].data_ptr());
    p.ld0 = 2 * F_;
    p.dwp = dwp_[q].data_ptr<float>();
    p.dwp_tiles = dwp_tiles;
    row_gemm(kModeDswiglu, p, weight_map(w_down, 128), map_g_[b], st, keep ? spare : 0);
  }
  if (async) {
    cuda_check(cudaEventRecord(ev_ds_[q], st), "event record");
    // (The first GEMM of the slice saw every row arrive.)
    cuda_check(cudaStreamWaitEvent(aux, keep ? ev_ds_[q] : ev_up_[q], 0), "wait for the first GEMM");
  }
  {  // dW_down[g] = (w act)^T g   (auxiliary stream; the fp32 carry chains slice to slice there)
    GemmParams p = base_params(pl, static_cast<int>(j));
    p.m_tiles = F_ / kBlockM;
    p.n_tiles = D_ / kBlockN;
    p.carry_in = carry_down_.data_ptr<float>() + static_cast<size_t>(par ^ 1) * F_ * D_;
    p.carry_out = carry_down_.data_ptr<float>() + static_cast<size_t>(par) * F_ * D_;
    p.grad_out = reinterpret_cast<__nv_bfloat16*>(dw_down.data_ptr());
    weight_grad(p, keep ? make_bf16_map_chunked(kept_act(j), kept_slice_rows(j), F_, 64, 2) : map_act_mn_[q],
                map_g_mn_[b], weight_map(dw_down, 32), aux);
  }
  if (async && !keep) {
    cuda_check(cudaEventRecord(ev_tgd_[q], aux), "event record");
    cuda_check(cudaStreamWaitEvent(aux, ev_ds_[q], 0), "wait dswiglu event");
  }
  {  // d_weight of every row goes back to its source rank
    ReturnDwParams r{};
    r.plan = pl;
    r.lay = lay_;
    r.slice = static_cast<int>(j);
    r.dwp = dwp_[q].data_ptr<float>();
    r.row_w = reinterpret_cast<const float*>(arena_ + arena_lay_.wbuf) + static_cast<size_t>(b) * S_;
    r.parts = dwp_tiles;
    r.peer_dw = table<float>(kTabDw);
    r.peer_count = table<uint32_t>(kTabCount);
    r.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
    launch_return_dw(r, aux);
    ++launches_;
  }
  {  // dx = dh Wu^T, rows go back to their source rank
    GemmParams p = base_params(pl, static_cast<int>(j));
    p.n_tiles = D_ / kBlockN;
    p.k_blocks = 2 * F_ / kBlockK;
    p.b_group_rows = D_;
    p.peer_rows = table<__nv_bfloat16>(kTabRet);
    p.peer_count = table<uint32_t>(kTabCount);
    p.ld0 = D_;
    row_gemm(kModeDx, p, weight_map(w_up, 128), map_dh_[q], st);
  }
  if (async) cuda_check(cudaEventRecord(ev_dx_[q], st), "event record");
  {  // dW_up[g] = x^T dh
    GemmParams p = base_params(pl, static_cast<int>(j));
    p.m_tiles = D_ / kBlockM;
    p.n_tiles = 2 * F_ / kBlockN;
    p.carry_in = carry_up_.data_ptr<float>() + static_cast<size_t>(par ^ 1) * D_ * 2 * F_;
    p.carry_out = carry_up_.data_ptr<float>() + static_cast<size_t>(par) * D_ * 2 * F_;
    p.grad_out = reinterpret_cast<__nv_bfloat16*>(dw_up.data_ptr());
    weight_grad(p, map_x_mn_[b], map_dh_mn_[q], weight_map(dw_up, 32), aux);
  }
  if (async) cuda_check(cudaEventRecord(ev_tgu_[q], aux), "event record");
  launch_slice_done(table<uint32_t>(kTabCredit), P_, me_, seq, aux);
  ++launches_;
  if (async) cuda_check(cudaEventRecord(ev_done_[j % 4], aux), "event record");
}

// Makes the caller's stream wait for everything the pass issued on the chain and auxiliary streams.
void FusedRank::join_streams(bool backward) {
  if (!overlapped() || cur_slices_ <= 0) return;
  cudaStream_t st = current_stream();
  cuda_check(cudaStreamWaitEvent(st, ev_done_[(cur_slices_ - 1) % 4], 0), "join aux stream");
  if (expands()) cuda_check(cudaStreamWaitEvent(st, ev_expand_[(cur_slices_ - 1) % 4], 0), "join expand stream");
  if (backward) {
    cuda_check(cudaStreamWaitEvent(st, ev_dx_[(cur_slices_ - 1) & 1], 0), "join chain stream");
    if (cur_slices_ >= 2) cuda_check(cudaStreamWaitEvent(st, ev_dx_[cur_slices_ & 1], 0), "join chain stream");
  }
}

void FusedRank::end_pass(int64_t n_slices) {
  cuda_check(cudaEventRecord(ev_end_, current_stream()), "event record");
  passed_ = true;
  seq_ += static_cast<uint32_t>(n_slices);
  cur_slices_ = 0;
  inline_ = short_pass_ = false;
  release_kept();
}

// What a training forward keeps for its backward: h and w * act of its first `kept_slices_` slices (12 KB a row at F = 2048),
// so that the backward starts from them instead of running the up-projection GEMM again (4 of its 16 D x F products per
// row). Results do not change by it: the backward recomputes the same bits when it has to. Forward + backward, D=7168,
// F=2048: 64 experts of 256 rows 7.10 -> 6.09 ms, Zipf routing in slices of 2048 rows 9.05 -> 7.67 ms, 32 experts of 1024
// rows on the fp8 wire 12.0 -> 10.9 ms.
void FusedRank::keep_rows(torch::Tensor h, torch::Tensor act, int64_t slices) {
  const Turn turn(pass_mutex_);
  expect(h.is_cuda() && h.is_contiguous() && h.scalar_type() == torch::kBFloat16 && h.dim() == 2 && h.size(1) == 2 * F_ &&
             act.is_cuda() && act.is_contiguous() && act.scalar_type() == torch::kBFloat16 && act.dim() == 2 &&
             act.size(1) == F_ && act.size(0) == h.size(0) && act.size(0) > (slices - 1) * S_,
         "kept activations must be contiguous CUDA bf16 [rows, 2F] and [rows, F] matrices that reach into every slice");
  expect_at_16(h, "kept h");
  expect_at_16(act, "kept w * act");
  kept_h_ = h;
  kept_act_ = act;
  kept_slices_ = slices;
}

void FusedRank::release_kept() {
  kept_h_ = torch::Tensor();
  kept_act_ = torch::Tensor();
  kept_slices_ = 0;
}

// Keeping pays once the GEMM that it saves is longer than a launch, and only while there is memory to spare: live tensors
// and all of the process's arenas, these included, stay within half of the device, else (or when the allocation fails) the
// backward recomputes.
// (What the caching allocator knows, not `cudaMemGetInfo`: that call takes 2 ms with a busy device.)
std::vector<torch::Tensor> FusedRank::allocate_kept(int64_t rows, int64_t slice_rows, const torch::TensorOptions& bf16) const {
  if (std::min<int64_t>(rows, slice_rows) * D_ * F_ < kKeepWork || !keep_activations_) return {};
  if (!within_half(static_cast<size_t>(rows) * 3 * F_ * 2)) return {};
  try {
    return {torch::empty({rows, 2 * F_}, bf16), torch::empty({rows, F_}, bf16)};
  } catch (const c10::Error&) {  // no memory for them after all
    return {};
  }
}

void FusedRank::finish_forward(torch::Tensor inv_order, torch::Tensor out) {
  const Turn turn(pass_mutex_);
  expect_arena("step");
  expect_bf16_2d(out, D_, "out");
  expect(out.size(0) * K_ == cur_rows_, "out rows do not match the pass");
  expect_i32(inv_order, cur_rows_, "inv_order");
  join_streams(/*backward=*/false);
  CombineParams c{};
  c.rows = reinterpret_cast<const __nv_bfloat16*>(arena_ + arena_lay_.ret);
  c.inv_order = inv_order.data_ptr<int>();
  c.out = reinterpret_cast<__nv_bfloat16*>(out.data_ptr());
  c.num_tokens = static_cast<int>(out.size(0));
  c.top_k = K_;
  c.hidden = D_;
  c.count = reinterpret_cast<const uint32_t*>(arena_ + arena_lay_.ret_count);
  c.target = ret_target_;
  if (short_pass_) {
    c.credit = reinterpret_cast<uint32_t*>(arena_ + arena_lay_.credit);
    c.credit_value = seq_ + 1;
  }
  c.spin_limit = spin_limit_;
  c.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
  launch_combine_reduce(c, current_stream(), inline_);
  ++launches_;
  end_pass(cur_slices_);
}

void FusedRank::reduce_backward(torch::Tensor inv_order, torch::Tensor dx, torch::Tensor d_weights, cudaEvent_t after) {
  expect_arena("step");
  expect_bf16_2d(dx, D_, "dx");
  expect(dx.size(0) * K_ == cur_rows_, "dx rows do not match the pass");
  expect(d_weights.is_cuda() && d_weights.scalar_type() == torch::kFloat32 && d_weights.is_contiguous() &&
             d_weights.numel() == cur_rows_,
         "d_weights must be a contiguous CUDA fp32 tensor of T*K elements");
  expect_i32(inv_order, cur_rows_, "inv_order");
  join_streams(/*backward=*/true);
  CombineParams c{};
  c.rows = reinterpret_cast<const __nv_bfloat16*>(arena_ + arena_lay_.ret);
  c.inv_order = inv_order.data_ptr<int>();
  c.out = reinterpret_cast<__nv_bfloat16*>(dx.data_ptr());
  c.dw_rows = reinterpret_cast<const float*>(arena_ + arena_lay_.dw_rows);
  c.d_weights = d_weights.data_ptr<float>();
  c.num_tokens = static_cast<int>(dx.size(0));
  c.top_k = K_;
  c.hidden = D_;
  c.count = reinterpret_cast<const uint32_t*>(arena_ + arena_lay_.ret_count);
  c.target = ret_target_;
  c.spin_limit = spin_limit_;
  c.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
  launch_combine_reduce(c, current_stream(), inline_);
  ++launches_;
  // (of a pass that runs as one slice: its weight gradients; the sum of dx has run beside them)
  if (after != nullptr) cuda_check(cudaStreamWaitEvent(current_stream(), after, 0), "join aux stream");
  end_pass(cur_slices_);
}

// ---------------------------------------------------------------------------------------------
// passes of a rank on its own, as one slice
// ---------------------------------------------------------------------------------------------
bool FusedRank::within_half(size_t bytes, int share) const {
  try {
    const auto pool = c10::cuda::CUDACachingAllocator::getDeviceStats(c10::cuda::current_device());
    const size_t live = static_cast<size_t>(pool.allocated_bytes[0].current) + static_cast<size_t>(arenas_allocated());
    return live + bytes <= device_bytes_ / share;
  } catch (const c10::Error&) {  // an allocator that keeps no statistics
    return false;
  }
}

// Whatever the rows and slices: forward + backward as one slice against one / two / three slices of the same rows takes 192 rows
// at D=1024, F=512 237 against 262 / 322 / 383 us, 12,288 rows there 308 against 342 / 433 / 502, 12,288 at D=2048, F=1024 589
// against 619 / 658 / 723, 12,288 at D=7168, F=2048 3.60 against 3.59 / 3.82 / 3.93 ms. Only a forward of one slice without autograd
// has a shorter pass of its own up to 2048 ids (`plan_small_kernel`).
bool FusedRank::runs_whole(int64_t rows, bool training) const {
  if (P_ != 1 || !whole_passes_ || !use_comm_stream_ || rows == 0) return false;
  if (rows <= S_ && !training && rows <= kPlanSmallIds) return false;
  // x, act (and h, and in the backward g and dh), 2 bytes each
  return within_half(static_cast<size_t>(rows) * 2 * (training ? 2 * D_ + 5 * F_ : D_ + F_));
}

GemmParams FusedRank::range_params(const int* plan, int64_t first, int64_t last) const {
  GemmParams p = base_params(plan, 0);
  p.lay = whole_lay_;
  if (last - first < L_) {  // (all experts: the tables as they are)
    p.first_expert = static_cast<int>(first);
    p.last_expert = static_cast<int>(last);
  }
  return p;
}

// Runs `part(first expert, last expert, put stream, GEMM stream)` range by range: the puts one behind the other, the GEMMs in turn
// on two streams (each fills the other's tail). The caller's stream then waits for all of them. One range: everything on the
// caller's stream.
template <typename Part>
void FusedRank::run_parts(int64_t parts, Part&& part) {
  cudaStream_t st = current_stream();
  if (parts == 1) {
    part(0, L_, st, st);
    return;
  }
  cuda_check(cudaEventRecord(ev_pass_, st), "event record");
  cuda_check(cudaStreamWaitEvent(comm_stream_, ev_pass_, 0), "wait pass event");
  for (int64_t k = 0; k < parts; ++k) part(L_ * k / parts, L_ * (k + 1) / parts, comm_stream_, chain_[k & 1]);
  for (int q = 0; q < 2; ++q) {
    cuda_check(cudaEventRecord(ev_up_[q], chain_[q]), "event record");
    cuda_check(cudaStreamWaitEvent(st, ev_up_[q], 0), "join chain stream");
  }
}

// `beside`: GEMMs run at the same time.
void FusedRank::put_whole(const torch::Tensor& plan, const torch::Tensor& inv_order, const torch::Tensor& x, const torch::Tensor* g,
                          const torch::Tensor& w_flat, __nv_bfloat16* to_x, __nv_bfloat16* to_g, float* to_w, int64_t first,
                          int64_t last, cudaStream_t st, bool behind, bool beside) {
  WholePutParams p{};
  p.plan = plan.data_ptr<int>();
  p.lay = whole_lay_;
  p.first_expert = static_cast<int>(first);
  p.last_expert = static_cast<int>(last);
  p.top_k = K_;
  p.hidden = D_;
  p.num_tokens = static_cast<int>(x.size(0));
  p.inv_order = inv_order.data_ptr<int>();
  p.w_flat = w_flat.data_ptr<float>();
  p.x = to_x != nullptr ? reinterpret_cast<const __nv_bfloat16*>(x.data_ptr()) : nullptr;
  p.g = to_g != nullptr ? reinterpret_cast<const __nv_bfloat16*>(g->data_ptr()) : nullptr;
  p.rows_x = to_x;
  p.rows_g = to_g;
  p.rows_w = to_w;
  p.round_fp8 = fp8_;
  p.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
  launch_whole_put(p, beside ? put_blocks_ : kPutAloneBlocks, st, behind);
  ++launches_;
}

void FusedRank::expect_pass(const torch::Tensor& x, const torch::Tensor& expert_ids, const torch::Tensor& w_flat,
                            const torch::Tensor& w_up, const torch::Tensor& w_down) const {
  const int64_t tk = expert_ids.numel();
  expect_bf16_2d(x, D_, "x");
  expect_weights(w_up, w_down, L_, D_, F_);
  expect_i32(expert_ids, tk, "expert_ids");
  expect(x.size(0) * K_ == tk && w_flat.is_cuda() && w_flat.scalar_type() == torch::kFloat32 && w_flat.is_contiguous() &&
             w_flat.numel() == tk,
         "router weights must be a contiguous CUDA fp32 tensor of T*K elements");
}

// `kept`: h and w * act, or nothing. `buffers`: x by rows, router weights by rows and, where nothing is kept, w * act.
std::tuple<std::vector<torch::Tensor>, int64_t, int64_t> FusedRank::forward_whole(
    torch::Tensor x, torch::Tensor expert_ids, torch::Tensor w_flat, torch::Tensor w_up, torch::Tensor w_down,
    const std::vector<torch::Tensor>& kept, const std::vector<torch::Tensor>& buffers, bool training) {
  cudaStream_t st = current_stream();
  const int64_t tk = expert_ids.numel();
  auto i32 = torch::TensorOptions().device(x.device()).dtype(torch::kInt32);
  torch::Tensor plan = torch::empty({whole_lay_.total}, i32), order = torch::empty({tk}, i32),
                inv_order = torch::empty({tk}, i32), out = torch::empty_like(x);
  const torch::Tensor &rows_x = buffers[0], &rows_w = buffers[1], &act = kept.empty() ? buffers[2] : kept[1];
  const QuiesceOnError guard{this};
  enter_pass();
  header_whole_ = true;
  cur_slices_ = 0;  // (no streams of slices to join)
  {
    NvtxRange range("chunked_moe/plan");
    PlanKernelParams pp{};
    pp.lay = whole_lay_;
    pp.plan = plan.data_ptr<int>();
    pp.spin_limit = spin_limit_;
    pp.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
    pp.host_out = host_header_;
    pp.host_seq = ++host_seq_;
    if (tk <= kPlanSmallIds && L_ <= kPlanSmallExperts) {
      // (Sort and tables as one kernel: 192 x 2 ids, forward + backward 162 -> 156 us, the host's wait for the header among them.)
      launch_plan_small(pp, expert_ids.data_ptr<int>(), static_cast<int>(tk), order.data_ptr<int>(), inv_order.data_ptr<int>(), nullptr,
                        nullptr, RowTable{}, st);
      ++launches_;
    } else {
      launch_sort_and_plan(pp, expert_ids.data_ptr<int>(), static_cast<int>(tk), order.data_ptr<int>(),
                           inv_order.data_ptr<int>(), my_counts_.data_ptr<int>(), sort_scratch_.data_ptr<int>(), st);
      launches_ += 3;
    }
  }
  cur_rows_ = tk;
  ret_target_ += static_cast<uint32_t>(tk) * static_cast<uint32_t>(D_ / kCombineCols);
  const int* pl = plan.data_ptr<int>();
  const int64_t parts = whole_ranges(tk, L_, D_, F_, training, /*backward=*/false);
  inline_ = parts == 1;
  const TokenMaps x_map = make_token_maps(rows_x.data_ptr(), tk, D_), act_map = make_token_maps(act.data_ptr(), tk, F_);
  run_parts(parts, [&](int64_t first, int64_t last, cudaStream_t put_stream, cudaStream_t gemm_stream) {
    NvtxRange range("chunked_moe/fwd experts from", first);
    put_whole(plan, inv_order, x, nullptr, w_flat, reinterpret_cast<__nv_bfloat16*>(rows_x.data_ptr()), nullptr,
              rows_w.data_ptr<float>(), first, last, put_stream, inline_, first > 0);
    if (put_stream != gemm_stream) {
      cuda_check(cudaEventRecord(ev_put_[0], put_stream), "event record");
      cuda_check(cudaStreamWaitEvent(gemm_stream, ev_put_[0], 0), "wait put event");
    }
    {
      GemmParams p = range_params(pl, first, last);
      p.n_tiles = 2 * F_ / kBlockN;
      p.k_blocks = D_ / kBlockK;
      p.b_group_rows = D_;
      p.row_w = rows_w.data_ptr<float>();
      p.out0 = reinterpret_cast<__nv_bfloat16*>(act.data_ptr());
      p.ld0 = F_;
      p.out1 = kept.empty() ? nullptr : reinterpret_cast<__nv_bfloat16*>(kept[0].data_ptr());
      p.ld1 = 2 * F_;
      row_gemm(kModeSwiglu, p, up_map(w_up), x_map, gemm_stream);
    }
    GemmParams p = range_params(pl, first, last);
    p.n_tiles = D_ / kBlockN;
    p.k_blocks = F_ / kBlockK;
    p.b_group_rows = F_;
    p.peer_rows = table<__nv_bfloat16>(kTabRet);
    p.peer_count = table<uint32_t>(kTabCount);
    p.ld0 = D_;
    row_gemm(kModeDownFwd, p, weight_map(w_down, 64, 2), act_map, gemm_stream);
  });
  {
    NvtxRange range("chunked_moe/combine");
    finish_forward(inv_order, out);
  }
  resolve_slices();  // raises what the pass's kernels had recorded by the time the plan was made
  std::vector<torch::Tensor> result{out, plan, order, inv_order};
  result.insert(result.end(), kept.begin(), kept.end());
  // x by rows stays for the backward of a pass of one range as well, while what lives stays within a quarter of the device
  // (activations, which save a GEMM, come first: they have the half). Its put then moves g alone: forward + backward of 8192 x 6
  // rows at D=1024 711 -> 693 us, 1999 x 4 at D=2048 410 -> 400 us, 2048 x 8 at D=7168 5.67 -> 5.60 ms.
  if (training && parts == 1 && keep_activations_ && within_half(0, 4)) result.push_back(rows_x);
  return std::make_tuple(result, kWholePass, kept.empty() ? 0 : 1);
}

// `buffers`: x by rows, g by rows, router weights by rows, dh, d_weight shares and, where nothing was kept, h and w * act.
// On the caller's stream put, [up-projection,] SwiGLU', dx, d_weight and the sum of dx, in a pass of one range each launched behind the
// one before; the weight gradients on the auxiliary stream. The sum of dx needs none of them and runs beside them (between them and
// the end of the pass it took 12 us of 430 at 1999 x 4 rows of D=2048 and 32 of 730 at 8192 x 6 of D=1024, the d_weight kernel
// between the two weight gradients 9 and 10). Forward + backward there 431 -> 410 and 732 -> 713 us; 4096 x 8 rows at D=7168 on the fp8
// wire 8.39 -> 8.11 ms, Zipf routing 6.20 -> 6.14, many small or very large experts unchanged (power: what runs side by side draws more).
void FusedRank::backward_whole(torch::Tensor x, torch::Tensor g, torch::Tensor w_flat, torch::Tensor w_up,
                               torch::Tensor w_down, torch::Tensor plan, torch::Tensor inv_order,
                               const std::vector<torch::Tensor>& kept, const torch::Tensor& kept_x,
                               const std::vector<torch::Tensor>& buffers, torch::Tensor dw_up, torch::Tensor dw_down) {
  cudaStream_t st = current_stream();
  const int64_t tk = inv_order.numel();
  if (!kept.empty()) {
    expect_bf16_2d(kept[0], 2 * F_, "kept h");
    expect_bf16_2d(kept[1], F_, "kept w * act");
    expect(kept[0].size(0) == tk && kept[1].size(0) == tk, "kept rows do not match the pass");
  }
  enter_pass();
  cur_slices_ = 0;
  cur_rows_ = tk;
  ret_target_ += static_cast<uint32_t>(tk) * static_cast<uint32_t>(D_ / kCombineCols + 1);
  const bool keep = !kept.empty();
  auto bf16 = [](const torch::Tensor& t) { return reinterpret_cast<__nv_bfloat16*>(t.data_ptr()); };
  const torch::Tensor &rows_x = kept_x.defined() ? kept_x : buffers[0], &rows_g = buffers[1], &rows_w = buffers[2],
                      &dh = buffers[3], &dwp = buffers[4], &h = keep ? kept[0] : buffers[5], &act = keep ? kept[1] : buffers[6];
  const int* pl = plan.data_ptr<int>();
  const int dwp_tiles = F_ / 32;
  const TokenMaps x_map = keep ? TokenMaps{} : make_token_maps(rows_x.data_ptr(), tk, D_);
  const TokenMaps g_map = make_token_maps(rows_g.data_ptr(), tk, D_), dh_map = make_token_maps(dh.data_ptr(), tk, 2 * F_);
  const CUtensorMap x_mn = make_bf16_map_chunked(rows_x.data_ptr(), tk, D_, 64, 2),
                    g_mn = make_bf16_map_chunked(rows_g.data_ptr(), tk, D_, 64, 2),
                    act_mn = make_bf16_map_chunked(act.data_ptr(), tk, F_, 64, 2),
                    dh_mn = make_bf16_map_chunked(dh.data_ptr(), tk, 2 * F_, 64, 2);
  // d_act = w * (g Wd^T) needs g's rows; x's, where nothing has to be recomputed from them, follow beside that GEMM.
  const int64_t parts = whole_ranges(tk, L_, D_, F_, /*training=*/true, /*backward=*/true);
  const bool x_later = keep && parts > 1 && !kept_x.defined();
  inline_ = parts == 1;
  run_parts(parts, [&](int64_t first, int64_t last, cudaStream_t put_stream, cudaStream_t gemm_stream) {
    NvtxRange range("chunked_moe/bwd experts from", first);
    put_whole(plan, inv_order, x, &g, w_flat, x_later || kept_x.defined() ? nullptr : bf16(rows_x), bf16(rows_g),
              rows_w.data_ptr<float>(), first, last, put_stream, inline_, first > 0);
    if (put_stream != gemm_stream) {
      cuda_check(cudaEventRecord(ev_put_[0], put_stream), "event record");
      cuda_check(cudaStreamWaitEvent(gemm_stream, ev_put_[0], 0), "wait put event");
    }
    if (x_later) {
      put_whole(plan, inv_order, x, nullptr, w_flat, bf16(rows_x), nullptr, nullptr, first, last, put_stream, false, true);
      cuda_check(cudaEventRecord(ev_put_[1], put_stream), "event record");
    }
    if (!keep) {
      GemmParams p = range_params(pl, first, last);
      p.n_tiles = 2 * F_ / kBlockN;
      p.k_blocks = D_ / kBlockK;
      p.b_group_rows = D_;
      p.row_w = rows_w.data_ptr<float>();
      p.out0 = bf16(act);
      p.ld0 = F_;
      p.out1 = bf16(h);
      p.ld1 = 2 * F_;
      row_gemm(kModeSwiglu, p, up_map(w_up), x_map, gemm_stream);
      cuda_check(cudaEventRecord(ev_tgd_[0], gemm_stream), "event record");
    }
    {  // acc = g Wd^T; dh = SwiGLU'(h) * (w * acc), d_weight shares <acc, w * act>
      GemmParams p = range_params(pl, first, last);
      p.n_tiles = F_ / kBlockN;
      p.k_blocks = D_ / kBlockK;
      p.b_group_rows = F_;
      p.row_w = rows_w.data_ptr<float>();
      p.in0 = bf16(h);
      p.in1 = bf16(act);
      p.ld1 = F_;
      p.out0 = bf16(dh);
      p.ld0 = 2 * F_;
      p.dwp = dwp.data_ptr<float>();
      p.dwp_tiles = dwp_tiles;
      row_gemm(kModeDswiglu, p, weight_map(w_down, 128), g_map, gemm_stream);
    }
    cuda_check(cudaEventRecord(ev_ds_[0], gemm_stream), "event record");
    // dW_down needs w * act and g's rows: where the up-projection has just made the former it fills the tail of the SwiGLU' GEMM
    // instead of following it, as slice by slice (experts of many rows, whose weight gradients are few tiles: 8 x 6144 rows at
    // D=F=256, forward + backward 442 -> 398 us; slice by slice 418).
    cuda_check(cudaStreamWaitEvent(aux_stream_, keep ? ev_ds_[0] : ev_tgd_[0], 0), "wait for the first GEMM");
    {  // dW_down[g] = (w act)^T g   (auxiliary stream)
      GemmParams p = range_params(pl, first, last);
      p.m_tiles = F_ / kBlockM;
      p.n_tiles = D_ / kBlockN;
      p.grad_out = bf16(dw_down);
      weight_grad(p, act_mn, g_mn, weight_map(dw_down, 32), aux_stream_);
    }
    if (!keep) cuda_check(cudaStreamWaitEvent(aux_stream_, ev_ds_[0], 0), "wait dswiglu event");
    {  // dx = dh Wu^T
      GemmParams p = range_params(pl, first, last);
      p.n_tiles = D_ / kBlockN;
      p.k_blocks = 2 * F_ / kBlockK;
      p.b_group_rows = D_;
      p.peer_rows = table<__nv_bfloat16>(kTabRet);
      p.peer_count = table<uint32_t>(kTabCount);
      p.ld0 = D_;
      row_gemm(kModeDx, p, weight_map(w_up, 128), dh_map, gemm_stream);
    }
    if (x_later) cuda_check(cudaStreamWaitEvent(aux_stream_, ev_put_[1], 0), "wait put event");
    {  // dW_up[g] = x^T dh
      GemmParams p = range_params(pl, first, last);
      p.m_tiles = D_ / kBlockM;
      p.n_tiles = 2 * F_ / kBlockN;
      p.grad_out = bf16(dw_up);
      weight_grad(p, x_mn, dh_mn, weight_map(dw_up, 32), aux_stream_);
    }
  });
  cuda_check(cudaEventRecord(ev_tgu_[0], aux_stream_), "event record");
  ReturnDwParams r{};  // d_weight of every row
  r.plan = pl;
  r.lay = whole_lay_;
  r.dwp = dwp.data_ptr<float>();
  r.row_w = rows_w.data_ptr<float>();
  r.parts = dwp_tiles;
  r.peer_dw = table<float>(kTabDw);
  r.peer_count = table<uint32_t>(kTabCount);
  r.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
  launch_return_dw(r, st, inline_);
  ++launches_;
}

// A forward of few tokens without autograd, on the caller's stream: plan, up-projection with its rows gathered, down-projection,
// sum of the K rows a token. No put, no buffer of a slice and no arrival is involved, and up to 32 ids no plan kernel
// (`launch_few_swiglu`) where nobody wants the plan: what that kernel leaves of one is enough for the two behind it, not for a
// backward. With the put, a launch and 5 us of latency between plan and first GEMM, -> without: 64 tokens at D=7168 495 -> 481 us, one
// token at D=1024 45.5 -> 42.9. Up to 96 tokens the gather keeps up with the tensor cores, whatever the routing (gemm/row_gemm.cuh).
bool FusedRank::runs_brief(int64_t tokens, int64_t rows, bool training) const {
  return P_ == 1 && whole_passes_ && use_comm_stream_ && !training && !fp8_ && tokens > 0 && tokens <= kBriefTokens && rows <= S_ &&
         rows <= kPlanSmallIds && L_ <= kPlanSmallExperts;
}

std::tuple<std::vector<torch::Tensor>, int64_t, int64_t> FusedRank::forward_brief(torch::Tensor x, torch::Tensor expert_ids,
                                                                                  torch::Tensor w_flat, torch::Tensor w_up,
                                                                                  torch::Tensor w_down,
                                                                                  bool plan_wanted) {
  cudaStream_t st = current_stream();
  const int64_t tk = expert_ids.numel();
  auto i32 = torch::TensorOptions().device(x.device()).dtype(torch::kInt32);
  torch::Tensor plan = torch::empty({whole_lay_.total}, i32), order = torch::empty({tk}, i32),
                inv_order = torch::empty({tk}, i32), out = torch::empty_like(x);
  const QuiesceOnError guard{this};
  enter_pass();
  header_whole_ = true;
  cur_slices_ = 0;
  inline_ = true;
  const bool few = tk <= kFewIds && !plan_wanted;
  RowTable rows;
  rows.tokens = brief_tokens_.data_ptr<int>();
  rows.weights = reinterpret_cast<float*>(arena_ + arena_lay_.wbuf);
  rows.w_flat = w_flat.data_ptr<float>();
  rows.top_k = K_;
  ++host_seq_;
  if (!few) {
    NvtxRange range("chunked_moe/plan");
    PlanKernelParams pp{};
    pp.lay = whole_lay_;
    pp.plan = plan.data_ptr<int>();
    pp.spin_limit = spin_limit_;
    pp.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
    pp.host_out = host_header_;
    pp.host_seq = host_seq_;
    launch_plan_small(pp, expert_ids.data_ptr<int>(), static_cast<int>(tk), order.data_ptr<int>(), inv_order.data_ptr<int>(), nullptr,
                      nullptr, rows, st);
    ++launches_;
  }
  cur_rows_ = tk;
  ret_target_ += static_cast<uint32_t>(tk) * static_cast<uint32_t>(D_ / kCombineCols);
  {
    GemmParams p = range_params(plan.data_ptr<int>(), 0, L_);
    p.n_tiles = 2 * F_ / kBlockN;
    p.k_blocks = D_ / kBlockK;
    p.b_group_rows = D_;
    p.row_w = rows.weights;
    p.out0 = reinterpret_cast<__nv_bfloat16*>(act_[0].data_ptr());
    p.ld0 = F_;
    p.gather = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr());
    p.tokens = rows.tokens;
    count_pipeline(kModeSwiglu, &p);
    if (few) {
      p.ids = expert_ids.data_ptr<int>();
      p.w_flat = rows.w_flat;
      p.num_ids = static_cast<int>(tk);
      p.top_k = K_;
      const FewPlan made{plan.data_ptr<int>(), order.data_ptr<int>(), inv_order.data_ptr<int>(), host_header_, host_seq_};
      launch_few_swiglu(p, up_map(w_up), made, std::max(2, num_sms_), st, /*behind=*/true);
    } else {
      launch_gather_swiglu(p, up_map(w_up), std::max(2, num_sms_), st, /*behind=*/true);
    }
    ++launches_;
  }
  {
    GemmParams p = range_params(plan.data_ptr<int>(), 0, L_);
    p.n_tiles = D_ / kBlockN;
    p.k_blocks = F_ / kBlockK;
    p.b_group_rows = F_;
    p.peer_rows = table<__nv_bfloat16>(kTabRet);
    p.peer_count = table<uint32_t>(kTabCount);
    p.ld0 = D_;
    row_gemm(kModeDownFwd, p, weight_map(w_down, 64, 2), map_act_[0], st);
  }
  {
    NvtxRange range("chunked_moe/combine");
    finish_forward(inv_order, out);
  }
  resolve_slices();
  if (few) return std::make_tuple(std::vector<torch::Tensor>{out}, kWholePass, 0);
  return std::make_tuple(std::vector<torch::Tensor>{out, plan, order, inv_order}, kWholePass, 0);
}

// ---------------------------------------------------------------------------------------------
// passes as one call each
// ---------------------------------------------------------------------------------------------
std::tuple<std::vector<torch::Tensor>, int64_t, int64_t> FusedRank::forward_pass(
    torch::Tensor x, torch::Tensor expert_ids, torch::Tensor w_flat, torch::Tensor w_up, torch::Tensor w_down,
    bool training, bool plan_wanted) {
  const Turn turn(pass_mutex_);
  expect_arena("forward");
  const int64_t tk = expert_ids.numel();
  release_kept();  // (of a pass that threw)
  short_pass_ = false;
  expect(tk <= tk_cap_, "T*K exceeds the workspace capacity");
  expect_pass(x, expert_ids, w_flat, w_up, w_down);
  if (runs_brief(x.size(0), tk, training)) return forward_brief(x, expert_ids, w_flat, w_up, w_down, plan_wanted);
  // Under saved-tensor hooks a pass keeps nothing and runs slice by slice: whether it may do otherwise depends on the free memory,
  // and its backward may get the plan of a recomputation.
  const bool hooks = training && at::SavedTensorDefaultHooks::get_hooks().has_value();
  if (!hooks && runs_whole(tk, training)) {
    std::vector<torch::Tensor> kept, buffers;
    if (training) kept = allocate_kept(tk, tk, x.options());
    try {
      buffers = {torch::empty({tk, D_}, x.options()), torch::empty({tk}, x.options().dtype(torch::kFloat32))};
      if (kept.empty()) buffers.push_back(torch::empty({tk, F_}, x.options()));
    } catch (const c10::Error&) {  // no memory for it after all
      buffers.clear();
    }
    if (!buffers.empty()) return forward_whole(x, expert_ids, w_flat, w_up, w_down, kept, buffers, training);
  }
  auto i32 = torch::TensorOptions().device(x.device()).dtype(torch::kInt32);
  // (The send order needs no initial values: an id the sort leaves out is recorded in the status block first, and with
  // that set every kernel that would read the order returns at once.)
  torch::Tensor plan = torch::empty({lay_.total}, i32), order = torch::empty({tk}, i32),
                inv_order = torch::empty({tk}, i32), out = torch::empty_like(x);
  std::vector<torch::Tensor> kept;
  const QuiesceOnError guard{this};
  auto run_slices = [&](int64_t lo, int64_t hi) {
    if (hi <= lo) return;
    put(lo, plan, order, x, c10::nullopt, w_flat);
    for (int64_t j = lo; j < hi; ++j) {
      NvtxRange range("chunked_moe/fwd slice", j);
      if (j + 1 < hi) put(j + 1, plan, order, x, c10::nullopt, w_flat);  // slice j+1 is in flight while slice j computes
      compute_forward(j, plan, w_up, w_down);
    }
  };
  // The slice count is a device value (it depends on the routing of every rank). The host does not wait for it: it
  // launches as many slices as the previous pass of this workspace needed, THEN reads the real count (by then long on
  // the host) and launches what is missing. Too many is harmless: a slice past the real count finds empty tables on
  // every rank. Every rank guesses and learns the same numbers, so all ranks loop alike. One rank on its own receives
  // exactly its own T*K copies and knows the count beforehand.
  const int64_t known = P_ == 1 ? (tk + S_ - 1) / S_ : -1;
  // A single slice of one rank: put, GEMMs and combine only follow one another, so they go to the caller's stream and the
  // events that tie the streams together are saved (one-token decode 82 -> 77 us, 2000 tokens at D=2048 195 -> 190 us).
  // The backward keeps its streams: its weight gradients fill the other GEMMs' tails (same layer 542 us, else 558 us).
  inline_ = use_comm_stream_ && known == 1;
  // Without autograd such a pass is also launched with as few kernels as it can do with: sort, plan and arrival targets as one
  // (few ids), the slice's credit from the combine kernel. (Training passes keep the launches that `expected_launches` counts;
  // a training step's forty launches hide what these five cost.) 61 -> 46 us for one token.
  short_pass_ = inline_ && !training;
  int64_t guess;
  {
    NvtxRange range("chunked_moe/plan");
    guess = std::max<int64_t>(0, begin_forward_async(expert_ids, plan, order, inv_order, plan, false));
  }
  if (known >= 0) guess = std::min<int64_t>(known, max_slices_);
  int64_t kept_slices = 0;
  if (training && !hooks) {
    const int64_t slices = known >= 0 ? guess : slices_to_keep(guess, last_rows_, S_);  // the others are recomputed
    if (slices > 0) kept = allocate_kept(known >= 0 ? tk : slices * S_, S_, x.options());
    if (!kept.empty()) {
      kept_slices = slices;
      keep_rows(kept[0], kept[1], kept_slices);
    }
  }
  run_slices(0, guess);
  int64_t n = known;
  if (known >= 0) {
    set_pass_slices(guess);
  } else {
    n = resolve_slices();  // throws here if an earlier kernel recorded an error (bad expert id, timed-out wait)
    run_slices(guess, n);
    set_pass_slices(std::max(guess, n));
  }
  {
    NvtxRange range("chunked_moe/combine");
    finish_forward(inv_order, out);
  }
  if (known >= 0) n = resolve_slices();  // the same checks, with all of the pass on its way to the device
  std::vector<torch::Tensor> result{out, plan, order, inv_order};
  result.insert(result.end(), kept.begin(), kept.end());
  return std::make_tuple(result, n, kept_slices);
}

std::tuple<torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor> FusedRank::backward_pass(
    torch::Tensor x, torch::Tensor g, torch::Tensor w_flat, torch::Tensor w_up, torch::Tensor w_down,
    torch::Tensor plan, torch::Tensor order, torch::Tensor inv_order, int64_t known_slices,
    const std::vector<torch::Tensor>& saved, int64_t kept_slices) {
  const Turn turn(pass_mutex_);
  expect_arena("backward");
  inline_ = short_pass_ = false;  // (also behind a forward that threw)
  release_kept();
  const int64_t rows = order.numel();
  expect_bf16_2d(x, D_, "x");
  expect_bf16_2d(g, D_, "g");
  expect(g.size(0) == x.size(0) && x.size(0) * K_ == rows, "x and g rows do not match the pass");
  expect_weights(w_up, w_down, L_, D_, F_);
  expect_i32(inv_order, rows, "inv_order");
  expect_i32(plan, known_slices == kWholePass ? whole_lay_.total : lay_.total, "plan");
  expect_at_16(plan, "plan");
  // Saved: h and w * act, x by rows, both or neither.
  const std::vector<torch::Tensor> kept(saved.begin(), saved.size() >= 2 ? saved.begin() + 2 : saved.begin());
  const torch::Tensor kept_x = saved.size() % 2 == 1 ? saved.back() : torch::Tensor();
  expect(!kept_x.defined() || (kept_x.is_cuda() && kept_x.is_contiguous() && kept_x.scalar_type() == torch::kBFloat16 &&
                               kept_x.dim() == 2 && kept_x.size(0) == rows && kept_x.size(1) == D_),
         "x by rows must be a contiguous CUDA bf16 [T*K, D] matrix");
  torch::Tensor dw_up = torch::empty_like(w_up), dw_down = torch::empty_like(w_down), dx = torch::empty_like(x);
  torch::Tensor d_weights = torch::empty({w_flat.numel()}, w_flat.options());
  std::vector<torch::Tensor> buffers;
  // (g, dh by rows, router weights and d_weight shares; x, h and w * act unless they were kept and live already. What lives by now is not
  // what lived when the forward decided: a model's later layers have saved theirs.)
  const int64_t columns = (kept_x.defined() ? 1 : 2) * D_ + (kept.size() == 2 ? 2 : 5) * F_;
  if (known_slices == kWholePass && whole_passes_ && within_half(static_cast<size_t>(rows) * (2 * columns + F_ / 8 + 4))) {
    const auto f32 = x.options().dtype(torch::kFloat32);
    try {
      buffers = {kept_x.defined() ? torch::Tensor() : torch::empty({rows, D_}, x.options()),
                 torch::empty({rows, D_}, x.options()), torch::empty({rows}, f32),
                 torch::empty({rows, 2 * F_}, x.options()), torch::empty({rows, F_ / 32}, f32)};
      if (kept.size() != 2) {
        buffers.push_back(torch::empty({rows, 2 * F_}, x.options()));
        buffers.push_back(torch::empty({rows, F_}, x.options()));
      }
    } catch (const c10::Error&) {  // no memory for it: slice by slice
      buffers.clear();
    }
  }
  const QuiesceOnError guard{this};
  if (!buffers.empty()) {
    backward_whole(x, g, w_flat, w_up, w_down, plan, inv_order, kept, kept_x, buffers, dw_up, dw_down);
    // (dx and d_weight need nothing of the weight gradients, which are still running on the auxiliary stream)
    reduce_backward(inv_order, dx, d_weights, ev_tgu_[0]);
    return std::make_tuple(dx, d_weights, dw_up, dw_down);
  }
  if (known_slices == kWholePass) {
    // The workspace's slices after all, with tables made of the row counts in the forward's.
    torch::Tensor sliced = torch::empty({lay_.total}, plan.options());
    PlanKernelParams pp{};
    pp.lay = lay_;
    pp.me = me_;
    pp.plan = sliced.data_ptr<int>();
    pp.counts = plan.data_ptr<int>() + whole_lay_.off_in_size;
    pp.my_counts = pp.counts;
    pp.spin_limit = spin_limit_;
    pp.status = reinterpret_cast<StatusBlock*>(status_.data_ptr());
    launch_plan_build(pp, current_stream());
    ++launches_;
    plan = sliced;
    known_slices = (rows + S_ - 1) / S_;
    if (kept.size() == 2) kept_slices = known_slices;
  }
  if (kept.size() == 2) keep_rows(kept[0], kept[1], kept_slices);
  // The slice count is the forward's: nothing is read back, the host never waits for the device here.
  const int64_t n = begin_backward(plan, known_slices, rows);
  if (n > 0) {
    put(0, plan, order, x, g, w_flat);
  } else {
    dw_up.zero_();
    dw_down.zero_();
  }
  for (int64_t j = 0; j < n; ++j) {
    NvtxRange range("chunked_moe/bwd slice", j);
    if (j + 1 < n) put(j + 1, plan, order, x, g, w_flat);
    compute_backward(j, plan, w_up, w_down, dw_up, dw_down);
  }
  finish_backward(inv_order, dx, d_weights);
  return std::make_tuple(dx, d_weights, dw_up, dw_down);
}

// ---------------------------------------------------------------------------------------------
// symmetric arena: cudaMalloc + CUDA IPC handles
// ---------------------------------------------------------------------------------------------
namespace {
std::mutex g_arena_mutex;
std::map<int64_t, std::pair<int, int64_t>> g_arenas;  // address -> (device, bytes)

int current_device() {
  int device = 0;
  cuda_check(cudaGetDevice(&device), "device");
  return device;
}
}  // namespace

int64_t arena_alloc(int64_t bytes) {
  void* p = nullptr;
  cuda_check(cudaMalloc(&p, static_cast<size_t>(bytes)), "arena cudaMalloc");
  const int64_t ptr = reinterpret_cast<int64_t>(p);
  {
    std::lock_guard<std::mutex> lock(g_arena_mutex);
    g_arenas[ptr] = {current_device(), bytes};
  }
  cuda_check(cudaMemset(p, 0, static_cast<size_t>(bytes)), "arena memset");
  cuda_check(cudaDeviceSynchronize(), "arena sync");
  return ptr;
}

void arena_free(int64_t ptr) {
  {
    std::lock_guard<std::mutex> lock(g_arena_mutex);
    g_arenas.erase(ptr);
  }
  cudaFree(reinterpret_cast<void*>(ptr));
}

int64_t arenas_allocated() {
  const int device = current_device();
  int64_t total = 0;
  std::lock_guard<std::mutex> lock(g_arena_mutex);
  for (const auto& [ptr, at] : g_arenas)
    if (at.first == device) total += at.second;
  return total;
}

py::bytes arena_export(int64_t ptr) {
  cudaIpcMemHandle_t h;
  cuda_check(cudaIpcGetMemHandle(&h, reinterpret_cast<void*>(ptr)), "cudaIpcGetMemHandle");
  return py::bytes(reinterpret_cast<const char*>(&h), sizeof(h));
}

int64_t arena_import(py::bytes handle) {
  std::string s = handle;
  expect(s.size() == sizeof(cudaIpcMemHandle_t), "bad IPC handle size");
  cudaIpcMemHandle_t h;
  std::memcpy(&h, s.data(), sizeof(h));
  void* p = nullptr;
  cuda_check(cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess), "cudaIpcOpenMemHandle");
  return reinterpret_cast<int64_t>(p);
}

void arena_close(int64_t ptr) { cudaIpcCloseMemHandle(reinterpret_cast<void*>(ptr)); }

void arena_zero(int64_t ptr, int64_t bytes) {
  cuda_check(cudaMemset(reinterpret_cast<void*>(ptr), 0, static_cast<size_t>(bytes)), "arena memset");
  cuda_check(cudaDeviceSynchronize(), "arena sync");
}

torch::Tensor arena_read_i32(int64_t ptr, int64_t offset_bytes, int64_t count) {
  expect(ptr != 0 && offset_bytes >= 0 && offset_bytes % 4 == 0 && count >= 0, "bad arena range");
  torch::Tensor out = torch::empty({count}, torch::kInt32);
  cuda_check(cudaDeviceSynchronize(), "arena sync");
  cuda_check(cudaMemcpy(out.data_ptr(), reinterpret_cast<const uint8_t*>(ptr) + offset_bytes,
                        static_cast<size_t>(count) * 4, cudaMemcpyDeviceToHost),
             "arena read");
  return out;
}

void arena_fill(int64_t ptr, int64_t bytes, int value) {
  cuda_check(cudaMemset(reinterpret_cast<void*>(ptr), value, static_cast<size_t>(bytes)), "arena memset");
  cuda_check(cudaDeviceSynchronize(), "arena sync");
}

}  // namespace cem
