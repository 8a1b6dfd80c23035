// Device-side plan construction: traffic-matrix exchange over NVLink + table build in one kernel,
// and the stable counting sort of token copies by expert.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../common/status.cuh"
#include "plan_tables.cuh"

namespace cem {

struct PlanKernelParams {
  PlanLayout lay;
  int me;
  const int* my_counts;            // [P*L] this rank's histogram (global expert order = receiver-major)
  int* counts;                     // [P*P*L] this rank's copy of the traffic matrix for this parity
  int* const* peer_counts;         // [P] every rank's traffic buffer for this parity (null when P == 1 and local)
  uint32_t* const* peer_flags;     // [P] every rank's [P] "row s has landed" epoch flags for this parity
  const uint32_t* flags;           // this rank's flags for this parity
  uint32_t epoch;                  // forward-pass counter; flags reach it when a row has landed
  int* plan;                       // output tables
  uint32_t spin_limit;
  StatusBlock* status;
  int32_t* host_out = nullptr;     // pinned host words: header (16), status block (8), sequence number; or null
  uint32_t host_seq = 0;           // stored last: the host polls for it
  int use_smem = 0;                // set by the launcher: the tables are built from a shared-memory copy of the matrix
};

// Exchanges the [P, L] histograms (each rank stores its row into every peer and releases a flag),
// waits for all rows, then builds the per-pass tables. Replaces the reference's all_gather +
// prefix sums + per-slice argument builders (src/chunked_moe/plan.py:77-163).
void launch_plan_build(const PlanKernelParams& p, cudaStream_t stream);

// What a GEMM that gathers its rows (gemm/row_gemm.cuh) knows about them, by sorted position: the token and the router weight.
struct RowTable {
  int* tokens = nullptr;           // [T*K], or null: no table
  float* weights = nullptr;        // [T*K]
  const float* w_flat = nullptr;   // [T*K] router weights by flat index
  int top_k = 1;
};

// Everything that starts a pass of ONE rank with few ids, as one kernel: the stable sort (order, inv_order), the tables, header
// and status to the host, and the arrival targets (`expected_total`, `pass_base`: as in `launch_pass_begin`; null where rows are
// gathered by `rows` and none arrive). `p.counts`,
// `p.my_counts` and the exchange's fields are not used. At most kPlanSmallIds ids and kPlanSmallExperts experts.
constexpr int kPlanSmallIds = 2048, kPlanSmallExperts = 512;
void launch_plan_small(const PlanKernelParams& p, const int* expert_ids, int n, int* order, int* inv_order,
                       uint32_t* expected_total, uint32_t* pass_base, const RowTable& rows, cudaStream_t stream);

// The start of a pass of ONE rank that runs as one slice, whatever the number of ids (three kernels): the sort, the tables and the
// header. At most 1024 experts. `counts` [L] and `scratch` (`expert_sort_scratch_ints`) are written.
void launch_sort_and_plan(const PlanKernelParams& p, const int* expert_ids, int n, int* order, int* inv_order, int* counts,
                          int* scratch, cudaStream_t stream);

// Host restatement of the table build, for CPU tests of the shared arithmetic.
void plan_build_host(const int* counts, int* plan, const PlanLayout& lay, int me);

// Stable counting sort of the T*K expert ids: order (send order -> flat index), inverse, histogram.
// Replaces argsort + scatter-add bincount (src/chunked_moe/plan.py:74-76). Ids outside [0, num_experts) take no part
// in the sort (their `inv_order` entry and the tail of `order` are left untouched); with a status block the first one
// is recorded as kStatusBadIndex (detail = its position, expected = num_experts, seen = the id).
void launch_expert_sort(const int* expert_ids, int n, int num_experts, int* order, int* inv_order, int* counts,
                        int* scratch, cudaStream_t stream, StatusBlock* status = nullptr);
size_t expert_sort_scratch_ints(int n, int num_experts);

}  // namespace cem
