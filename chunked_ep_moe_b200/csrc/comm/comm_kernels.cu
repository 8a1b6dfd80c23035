// Dispatch put, credits, combine reduce.
//
// dispatch_put replaces three things of the reference at once: the send-order gather
// (src/chunked_moe/moe.py:91-93), the wire quantisation (moe.py:56-63) and the slice exchange
// (transport/nvshmem.py:125-177 / ragged_all_to_all). A warp takes a chunk of up to
// kPutChunkRows rows of one (receiver, expert) segment, reads each row straight from x[token]
// (no [T*K, D] send buffer is ever materialised), stores it with 16-byte vector stores into the
// expert-major position of the receiver's S-row slice buffer over NVLink, and then releases
// the row count to the receiver's per-(source, expert) arrival counter. Receivers never take
// part in the transfer; their GEMM producer warps acquire the counters.
//
// What bounds the put is the chain of dependent accesses in front of each copy (segment, send order, row), 0.6 us each with
// 128 blocks on the device: the warp searches the segments 32 at a time, fetches its rows' send-order entries together and
// keeps eight 16-byte loads per lane in flight. 1024 rows of x (and, in the backward, g) at D=2048, beside GEMMs: 25 -> 14.5 us
// on average; forward + backward of eight such slices 1133 -> 977 us, 8192 tokens at D=1024 1026 -> 894 us.
//
// Protocol invariants:
//   * arrival counters only grow (cumulative rows per (source, expert)); a pass's targets are
//     base + rows expected so far, so nothing is ever reset and stale values are detectable;
//   * slice buffers are double buffered by the global slice sequence number; before writing
//     sequence q a sender waits until the receiver's credit says q-2 has been consumed;
//   * every wait is bounded and reports through the status block.
#include "comm_kernels.cuh"

#include <cuda_fp8.h>

#include <algorithm>

#include "../common/pdl.cuh"
#include "../common/umma.cuh"

namespace cem {

namespace {

constexpr int kPutThreads = 256;  // with 64 registers each it fits beside a GEMM CTA (see row_gemm.cu)

// Last segment whose chunk prefix is <= chunk (empty segments share a prefix with their successor), for the whole warp: 32
// prefixes at a time, two rounds for up to 1024 segments. (The first prefix is 0 and prefixes ascend.)
__device__ __forceinline__ int find_segment(const int4* put, int n, int chunk, int lane) {
  int lo = 0, len = n;
  while (len > 1) {
    const int step = (len + 31) >> 5, at = lane * step;
    const unsigned below = __ballot_sync(0xffffffffu, at < len && put[lo + at].w <= chunk);
    const int k = (31 - __clz(below)) * step;
    lo += k;
    len = len - k < step ? len - k : step;
  }
  return lo;
}

// Eight bf16 columns to e4m3 with one scale per 128 columns (the 16 lanes that share a block); all lanes take part.
__device__ __forceinline__ uint2 quantise_e4m3(const int4& raw, float* scale_out) {
  const uint32_t wds[4] = {static_cast<uint32_t>(raw.x), static_cast<uint32_t>(raw.y), static_cast<uint32_t>(raw.z),
                           static_cast<uint32_t>(raw.w)};
  float v[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) { v[2 * i] = bf16_lo(wds[i]); v[2 * i + 1] = bf16_hi(wds[i]); }
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
  for (int o = 8; o >= 1; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float scale = fmaxf(amax, 1e-12f) * (1.0f / 448.0f);
  const float inv = 1.0f / scale;
  uint32_t lo = 0, hi = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t b0 = __nv_cvt_float_to_fp8(v[i] * inv, __NV_SATFINITE, __NV_E4M3);
    const uint32_t b1 = __nv_cvt_float_to_fp8(v[4 + i] * inv, __NV_SATFINITE, __NV_E4M3);
    lo |= b0 << (8 * i);
    hi |= b1 << (8 * i);
  }
  *scale_out = scale;
  return make_uint2(lo, hi);
}

__device__ __forceinline__ int4 expand_e4m3(const uint2& raw, float scale) {
  float v[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half_raw h0 = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>((raw.x >> (8 * i)) & 0xFF), __NV_E4M3);
    const __half_raw h1 = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>((raw.y >> (8 * i)) & 0xFF), __NV_E4M3);
    v[i] = __half2float(*reinterpret_cast<const __half*>(&h0)) * scale;
    v[4 + i] = __half2float(*reinterpret_cast<const __half*>(&h1)) * scale;
  }
  return make_int4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}

// Copies a chunk's rows to consecutive rows at `dst`, two rows side by side, eight 16-byte loads per lane in flight. Lane r
// holds the token of row r, or -1 for a row that is left out.
__device__ __forceinline__ void copy_rows(const __nv_bfloat16* src, __nv_bfloat16* dst, int lane_token, int rows,
                                          int hidden, int lane) {
  constexpr int kAhead = 4;
  const int units = hidden >> 3;  // 16-byte units of a row, a multiple of 32
#pragma unroll 1
  for (int r = 0; r < rows; r += 2) {
    const int t0 = __shfl_sync(0xffffffffu, lane_token, r), t1 = __shfl_sync(0xffffffffu, lane_token, r + 1);
    const bool live0 = t0 >= 0, live1 = t1 >= 0;  // (lanes past `rows` hold -1)
    const int4* s0 = reinterpret_cast<const int4*>(src + static_cast<size_t>(live0 ? t0 : 0) * hidden);
    const int4* s1 = reinterpret_cast<const int4*>(src + static_cast<size_t>(live1 ? t1 : 0) * hidden);
    int4* d = reinterpret_cast<int4*>(dst) + r * units;
#pragma unroll 1
    for (int u = lane; u < units; u += 32 * kAhead) {
      int4 v0[kAhead], v1[kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        if (u + 32 * k < units) {
          if (live0) v0[k] = ld_nc_v4(s0 + u + 32 * k);
          if (live1) v1[k] = ld_nc_v4(s1 + u + 32 * k);
        }
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        if (u + 32 * k < units) {
          if (live0) d[u + 32 * k] = v0[k];
          if (live1) d[units + u + 32 * k] = v1[k];
        }
      }
    }
  }
}

// Quantises one row to e4m3 with a scale per 128 columns.
__device__ __forceinline__ void put_row_fp8(const __nv_bfloat16* src, uint8_t* dq, float* ds, int hidden, int lane) {
  const int units = hidden >> 3;  // a multiple of 32
  const int4* s = reinterpret_cast<const int4*>(src);
  for (int u = lane; u < units; u += 32) {
    float scale;
    const uint2 q = quantise_e4m3(ld_nc_v4(s + u), &scale);
    *reinterpret_cast<uint2*>(dq + static_cast<size_t>(u) * 8) = q;
    if ((lane & 15) == 0) ds[u >> 4] = scale;
  }
}

// One row over the fp8 wire without leaving this GPU: quantised and expanded again.
__device__ __forceinline__ void put_row_rounded(const __nv_bfloat16* src, __nv_bfloat16* dst, int hidden, int lane) {
  const int units = hidden >> 3;  // a multiple of 32
  const int4* s = reinterpret_cast<const int4*>(src);
  int4* d = reinterpret_cast<int4*>(dst);
  for (int u = lane; u < units; u += 128) {
    int4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (u + 32 * k < units) v[k] = ld_nc_v4(s + u + 32 * k);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (u + 32 * k < units) {  // (the same in all lanes)
        float scale;
        const uint2 q = quantise_e4m3(v[k], &scale);
        d[u + 32 * k] = expand_e4m3(q, scale);
      }
    }
  }
}

enum Wire { kWireBf16, kWireFp8, kWireRounded };

template <int WIRE>
__global__ void __launch_bounds__(kPutThreads, 4) dispatch_put_kernel(const PutParams p) {
  __shared__ int s_abort;
  release_successor();
  wait_predecessor();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_seg = p.lay.P * p.lay.L;
  if (threadIdx.x == 0) s_abort = (p.status != nullptr && p.status->code != 0) ? 1 : 0;
  __syncthreads();
  if (s_abort) return;  // an earlier kernel of this pass already gave up
  // Buffer reuse: sequence q overwrites what sequence q-2 used on every receiver.
  if (p.seq >= 2 && threadIdx.x < p.lay.P) {
    uint32_t seen = 0;
    if (!spin_until_reached(p.credit + threadIdx.x, p.seq - 1, p.spin_limit, &seen)) {
      report_status(p.status, kStatusCreditTimeout, kKernelPut, 0, static_cast<int>(p.seq), threadIdx.x, p.seq - 1, seen);
      s_abort = 1;
    }
  }
  __syncthreads();
  if (s_abort) return;

  const int4* put = reinterpret_cast<const int4*>(p.plan + p.lay.off_put + 4 * n_seg * p.slice);
  const int num_chunks = p.plan[p.lay.off_num_chunks + p.slice];
  const int buf = static_cast<int>(p.seq & 1u);
  const int S = p.lay.S, D = p.hidden;
  const int warps_total = gridDim.x * (kPutThreads / 32);
  // Arrival releases are batched: a system-scope fence drains this warp's stores over NVLink, so one fence covers
  // up to kPendingSignals chunks instead of one (lane i of the warp keeps pending signal i).
  constexpr int kPendingSignals = 8;
  uint32_t* pend_ptr = nullptr;
  uint32_t pend_cnt = 0;
  int pending = 0;
  auto flush = [&]() {
    __syncwarp();
    if (lane < pending) release_count(pend_ptr, pend_cnt, p.lay.P);
    pending = 0;
  };
  for (int c = blockIdx.x * (kPutThreads / 32) + warp; c < num_chunks; c += warps_total) {
    const int seg = find_segment(put, n_seg, c, lane);
    const int4 e = put[seg];  // {send-order offset, rows, dest row, chunk prefix}
    const int r = seg / p.lay.L, l = seg - r * p.lay.L;
    const int first = (c - e.w) * kPutChunkRows;
    const int rows = min(kPutChunkRows, e.y - first);
    const size_t drow = static_cast<size_t>(buf) * S + e.z + first;
    int token = -1;  // of row `lane`
    if (lane < rows) {
      const int at = e.x + first + lane, row = e.z + first + lane;
      const int flat = at >= 0 && at < p.num_tokens * p.top_k ? p.order[at] : -1;
      token = flat / p.top_k;
      // Index check: a segment outside the send order, an entry outside the token range or a destination row outside the slice
      // buffer is recorded and the row is skipped, never dereferenced. The arrival is still signalled, so nothing waits for the
      // row; the recorded status tells the host that the pass is invalid.
      if (flat < 0 || token >= p.num_tokens || row < 0 || row >= S) {
        report_status(p.status, kStatusBadIndex, kKernelPut, 0, p.slice, at, static_cast<uint32_t>(p.num_tokens),
                      static_cast<uint32_t>(token));
        token = -1;
      } else {
        p.peer_w[r][drow + lane] = p.w_flat[flat];
      }
    }
    __syncwarp();
    if constexpr (WIRE == kWireBf16) {
#pragma unroll 1
      for (int what = 0; what < 2; ++what) {  // (one copy of the loop: it fills the registers)
        const __nv_bfloat16* from = what ? p.g : p.x;
        if (from == nullptr) continue;
        copy_rows(from, (what ? p.peer_g[r] : p.peer_x[r]) + drow * D, token, rows, D, lane);
      }
    } else {
      for (int rr = 0; rr < rows; ++rr) {
        const int t = __shfl_sync(0xffffffffu, token, rr);
        if (t < 0) continue;
        const size_t to = drow + rr;
        if constexpr (WIRE == kWireFp8) {
          const __nv_bfloat16* x = p.x + static_cast<size_t>(t) * D;
          const __nv_bfloat16* g = p.g != nullptr ? p.g + static_cast<size_t>(t) * D : nullptr;
          put_row_fp8(x, p.peer_xq[r] + to * D, p.peer_xs[r] + to * (D >> 7), D, lane);
          if (g != nullptr) put_row_fp8(g, p.peer_gq[r] + to * D, p.peer_gs[r] + to * (D >> 7), D, lane);
        } else {
#pragma unroll 1
          for (int what = 0; what < 2; ++what) {
            const __nv_bfloat16* from = what ? p.g : p.x;
            if (from == nullptr) continue;
            put_row_rounded(from + static_cast<size_t>(t) * D, (what ? p.peer_g[r] : p.peer_x[r]) + to * D, D, lane);
          }
        }
      }
    }
    if (lane == pending) {
      pend_ptr = p.peer_arrive[r] + p.me * p.lay.L + l;
      pend_cnt = static_cast<uint32_t>(rows);
    }
    if (++pending == kPendingSignals) flush();
  }
  flush();
}

// The put of a rank on its own is a plain scatter: its stream is in send order, so `inv_order` says where a token's rows are. A warp
// takes up to 256 16-byte units of one token's row, all of them in flight together, and stores them to each of the token's rows: x
// is read (and rounded for the fp8 wire) once a token and range instead of once a copy, and no copy waits for a search of the segments
// and a send-order entry first, which is what bounded the dispatch put here (1.9 TB/s of stores from 128 blocks). Bound by its stores:
// 8192 tokens x 6 copies at D=1024 x 34 us (of x alone, 100 MB) and 41 us (x and g; 85 by the dispatch put), 2048 x 8 at D=7168 103 us
// (x and g, 470 MB; 247), first range of 4096 x 8 rounded tokens at D=7168 33 us (116). Forward + backward at those sizes, dispatch put
// and this one in turn on one GPU: 790 -> 721 us, 5.49 -> 5.43 ms, 8.47 -> 8.19 ms; 1999 x 4 at D=2048 429 -> 418 us. Beside GEMMs (ranges) it keeps to the dispatch put's 128 blocks.
constexpr int kWholeAhead = 8;

template <bool ROUND>
__global__ void __launch_bounds__(kPutThreads, 4) whole_put_kernel(const WholePutParams p) {
  __shared__ int s_abort;
  release_successor();
  wait_predecessor();
  if (threadIdx.x == 0) s_abort = (p.status != nullptr && p.status->code != 0) ? 1 : 0;
  __syncthreads();
  if (s_abort) return;  // an earlier kernel of this pass already gave up
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int all = p.plan[1], L = p.lay.L;
  const int* expert_start = p.plan + p.lay.off_expert_start;
  const int begin = p.first_expert > 0 ? expert_start[p.first_expert] : 0;
  const int end = p.last_expert < L ? expert_start[p.last_expert] : all;
  const int units = p.hidden >> 3;  // of a row, a multiple of 32
  const int parts = (units + 32 * kWholeAhead - 1) / (32 * kWholeAhead);
  const int tasks = p.num_tokens * parts;
  for (int task = blockIdx.x * (kPutThreads / 32) + warp; task < tasks; task += gridDim.x * (kPutThreads / 32)) {
    const int t = task / parts, part = task - t * parts;
    const int u0 = part * 32 * kWholeAhead + lane;
    for (int k0 = 0; k0 < p.top_k; k0 += 32) {
      int row = -1;  // of copy k0 + lane
      if (k0 + lane < p.top_k) {
        const int flat = t * p.top_k + k0 + lane, at = p.inv_order[flat];
        // Index check: a row outside the stream is recorded and skipped, never written.
        if (at < 0 || at >= all) {
          report_status(p.status, kStatusBadIndex, kKernelPut, 0, 0, flat, static_cast<uint32_t>(all), static_cast<uint32_t>(at));
        } else if (at >= begin && at < end) {
          row = at;
          if (part == 0 && p.rows_w != nullptr) p.rows_w[row] = p.w_flat[flat];
        }
      }
      const unsigned copies = __ballot_sync(0xffffffffu, row >= 0);
      if (copies == 0) continue;
#pragma unroll 1
      for (int what = 0; what < 2; ++what) {
        const __nv_bfloat16* from = what ? p.g : p.x;
        if (from == nullptr) continue;
        const int4* s = reinterpret_cast<const int4*>(from + static_cast<size_t>(t) * p.hidden) + u0;
        int4* d = reinterpret_cast<int4*>(what ? p.rows_g : p.rows_x) + u0;
        int4 v[kWholeAhead];
#pragma unroll
        for (int i = 0; i < kWholeAhead; ++i)
          if (u0 + 32 * i < units) v[i] = ld_nc_v4(s + 32 * i);
        if constexpr (ROUND) {
#pragma unroll
          for (int i = 0; i < kWholeAhead; ++i) {
            if (u0 + 32 * i < units) {  // (the same in all lanes)
              float scale;
              const uint2 q = quantise_e4m3(v[i], &scale);
              v[i] = expand_e4m3(q, scale);
            }
          }
        }
        for (unsigned left = copies; left != 0; left &= left - 1) {
          const int r = __shfl_sync(0xffffffffu, row, __ffs(left) - 1);
          int4* to = d + static_cast<size_t>(r) * units;
#pragma unroll
          for (int i = 0; i < kWholeAhead; ++i)
            if (u0 + 32 * i < units) to[32 * i] = v[i];
        }
      }
    }
  }
}

__global__ void slice_done_kernel(uint32_t* const* peer_credit, int num_ranks, int me, uint32_t seq) {
  if (threadIdx.x < num_ranks) st_release_sys(peer_credit[threadIdx.x] + me, seq + 1);
}

__global__ void pass_begin_kernel(const int* plan, PlanLayout lay, uint32_t* expected_total, uint32_t* pass_base,
                                  uint32_t* ready_total, uint32_t* ready_base) {
  wait_predecessor();
  const int n = lay.P * lay.L;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const uint32_t base = expected_total[i];
    pass_base[i] = base;
    expected_total[i] = base + static_cast<uint32_t>(plan[lay.off_in_size + i]);
  }
  if (ready_total != nullptr) {
    for (int l = threadIdx.x; l < lay.L; l += blockDim.x) {
      const uint32_t base = ready_total[l];
      ready_base[l] = base;
      ready_total[l] = base + static_cast<uint32_t>(plan[lay.off_expert_rows + l]);
    }
  }
}

// One thread per slice row: the row's expert by bisection of the experts' starts in the stream, its source among the P
// segments of that expert. (The up-projection gradient's GEMM follows on the same stream; this is a few us beside the
// chain's GEMMs, where summing inside the dX epilogue kept one column tile's warps busy with strided reads.)
__global__ void __launch_bounds__(256) return_dw_kernel(const ReturnDwParams p) {
  release_successor();
  wait_predecessor();
  if (p.status != nullptr && p.status->code != 0) return;  // an earlier kernel of this pass already gave up
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * blockDim.x + threadIdx.x, at = p.slice * p.lay.S + row;  // slice row, stream row
  const int* expert_start = p.plan + p.lay.off_expert_start;
  int src = -1;
  if (row < p.lay.S && at < p.plan[1]) {  // plan[1]: rows of this rank's stream
    int lo = 0, hi = p.lay.L - 1;
    while (lo < hi) {  // last expert that starts at or before the row (empty experts share the next one's start)
      const int mid = (lo + hi + 1) >> 1;
      if (expert_start[mid] <= at) lo = mid; else hi = mid - 1;
    }
    float sum = 0.0f;
    const float w = p.row_w[row];
    const float4* parts = reinterpret_cast<const float4*>(p.dwp + static_cast<size_t>(row) * p.parts);
    for (int q = 0; q < p.parts / 4; ++q) {  // F / 32 of them: a multiple of eight
      const float4 v = parts[q];
      sum += (v.x + v.y) + (v.z + v.w);
    }
    if (weight_divides(w)) sum /= w;
    for (int s = 0; s < p.lay.P; ++s) {
      const int i = s * p.lay.L + lo, off = at - p.plan[p.lay.off_in_start + i];
      if (off >= 0 && off < p.plan[p.lay.off_in_size + i]) {
        src = s;
        p.peer_dw[s][p.plan[p.lay.off_src_send_start + i] + off] = sum;
      }
    }
  }
  uint32_t sent = 0;  // lane s: rows this warp has stored to source s
  for (int s = 0; s < p.lay.P; ++s) {
    const uint32_t cnt = __popc(__ballot_sync(0xffffffffu, src == s));
    if (lane == s) sent = cnt;
  }
  __syncwarp();
  if (sent > 0) release_count(p.peer_count[lane], sent, p.lay.P);
}

__global__ void __launch_bounds__(256) combine_reduce_kernel(const CombineParams p) {
  __shared__ int s_abort;
  wait_predecessor();
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0 && p.credit != nullptr) st_release_sys(p.credit, p.credit_value);  // (behind the GEMMs on this stream)
    s_abort = (p.status != nullptr && p.status->code != 0) ? 1 : 0;
    uint32_t seen = 0;
    if (!s_abort && !spin_until_reached(p.count, p.target, p.spin_limit, &seen)) {
      report_status(p.status, kStatusReturnTimeout, kKernelCombineReduce, 0, 0, 0, p.target, seen);
      s_abort = 1;
    }
  }
  __syncthreads();
  if (s_abort) return;
  const int units = p.hidden >> 3;
  for (int t = blockIdx.x; t < p.num_tokens; t += gridDim.x) {
    for (int u = threadIdx.x; u < units; u += blockDim.x) {
      float acc[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
      for (int k = 0; k < p.top_k; ++k) {  // fixed k order: bitwise reproducible
        const int pos = p.inv_order[t * p.top_k + k];
        const int4 raw = *reinterpret_cast<const int4*>(p.rows + static_cast<size_t>(pos) * p.hidden + u * 8);
        const uint32_t wds[4] = {static_cast<uint32_t>(raw.x), static_cast<uint32_t>(raw.y),
                                 static_cast<uint32_t>(raw.z), static_cast<uint32_t>(raw.w)};
#pragma unroll
        for (int i = 0; i < 4; ++i) { acc[2 * i] += bf16_lo(wds[i]); acc[2 * i + 1] += bf16_hi(wds[i]); }
      }
      *reinterpret_cast<int4*>(p.out + static_cast<size_t>(t) * p.hidden + u * 8) =
          make_int4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]),
                    pack_bf16(acc[6], acc[7]));
    }
    if (p.d_weights != nullptr && threadIdx.x < p.top_k) {
      const int flat = t * p.top_k + threadIdx.x;
      p.d_weights[flat] = p.dw_rows[p.inv_order[flat]];
    }
  }
}

// Expands one e4m3 row with its 1x128 block scales into bf16; the CTA's threads stride over 8-value units.
__device__ __forceinline__ void dequant_row(const uint8_t* q, const float* scales, __nv_bfloat16* out, int row,
                                            int hidden) {
  const int units = hidden >> 3;
  const uint8_t* qrow = q + static_cast<size_t>(row) * hidden;
  const float* srow = scales + static_cast<size_t>(row) * (hidden >> 7);
  __nv_bfloat16* orow = out + static_cast<size_t>(row) * hidden;
  for (int u = threadIdx.x; u < units; u += blockDim.x) {
    const uint2 raw = *reinterpret_cast<const uint2*>(qrow + static_cast<size_t>(u) * 8);
    *reinterpret_cast<int4*>(orow + static_cast<size_t>(u) * 8) = expand_e4m3(raw, srow[u >> 4]);
  }
}

__global__ void __launch_bounds__(256) dequant_slice_kernel(const DequantParams p) {
  __shared__ int s_abort;
  if (threadIdx.x == 0) s_abort = (p.status != nullptr && p.status->code != 0) ? 1 : 0;
  __syncthreads();
  if (s_abort) return;
  const int lo = p.slice * p.lay.S, hi = lo + p.lay.S;
  for (int l = 0; l < p.lay.L; ++l) {
    const int es = p.plan[p.lay.off_expert_start + l], er = p.plan[p.lay.off_expert_rows + l];
    const int first = plan_clip(lo, es, es + er), last = plan_clip(hi, es, es + er);
    if (last <= first) continue;
    // This expert's rows of the slice have arrived from every source (thread s watches source s).
    if (threadIdx.x < p.lay.P) {
      const int i = threadIdx.x * p.lay.L + l;
      const int through = plan_clip(hi - p.plan[p.lay.off_in_start + i], 0, p.plan[p.lay.off_in_size + i]);
      const uint32_t target = p.pass_base[i] + static_cast<uint32_t>(through);
      uint32_t seen = 0;
      if (!spin_until_reached(p.arrive + i, target, p.spin_limit, &seen)) {
        report_status(p.status, kStatusArrivalTimeout, kKernelPut, 1, p.slice, i, target, seen);
        s_abort = 1;
      }
    }
    __syncthreads();
    if (s_abort) return;
    // Slice rows [first - lo, last - lo); this CTA takes every gridDim.x-th of them.
    uint32_t mine = 0;
    for (int r = first - lo + blockIdx.x; r < last - lo; r += gridDim.x, ++mine) {
      dequant_row(p.xq, p.xs, p.x, r, p.hidden);
      if (p.gq != nullptr) dequant_row(p.gq, p.gs, p.g, r, p.hidden);
    }
    __syncthreads();  // all of this CTA's stores for the expert are issued before one thread releases them
    if (threadIdx.x == 0 && mine > 0) {
      __threadfence();
      atomicAdd(p.ready + l, mine);
    }
  }
}

__global__ void wait_probe_kernel(const uint32_t* flag, uint32_t target, uint32_t spin_limit, StatusBlock* status) {
  uint32_t seen = 0;
  if (!spin_until_reached(flag, target, spin_limit, &seen))
    report_status(status, kStatusArrivalTimeout, kKernelWaitProbe, 0, 0, 0, target, seen);
}

}  // namespace

void launch_dispatch_put(const PutParams& p, int grid, cudaStream_t stream, bool behind) {
  if (p.peer_xq != nullptr) launch_maybe_behind(behind, dispatch_put_kernel<kWireFp8>, grid, kPutThreads, 0, stream, p);
  else if (p.round_fp8) launch_maybe_behind(behind, dispatch_put_kernel<kWireRounded>, grid, kPutThreads, 0, stream, p);
  else launch_maybe_behind(behind, dispatch_put_kernel<kWireBf16>, grid, kPutThreads, 0, stream, p);
}

void launch_whole_put(const WholePutParams& p, int grid, cudaStream_t stream, bool behind) {
  const int parts = (p.hidden / 8 + 32 * kWholeAhead - 1) / (32 * kWholeAhead);
  grid = std::max(1, std::min(grid, (p.num_tokens * parts + kPutThreads / 32 - 1) / (kPutThreads / 32)));
  if (p.round_fp8) launch_maybe_behind(behind, whole_put_kernel<true>, grid, kPutThreads, 0, stream, p);
  else launch_maybe_behind(behind, whole_put_kernel<false>, grid, kPutThreads, 0, stream, p);
}

void launch_slice_done(uint32_t* const* peer_credit, int num_ranks, int me, uint32_t seq, cudaStream_t stream) {
  slice_done_kernel<<<1, 32, 0, stream>>>(peer_credit, num_ranks, me, seq);
}

void launch_pass_begin(const int* plan, PlanLayout lay, uint32_t* expected_total, uint32_t* pass_base,
                       uint32_t* ready_total, uint32_t* ready_base, cudaStream_t stream) {
  launch_behind(pass_begin_kernel, 1, 256, 0, stream, plan, lay, expected_total, pass_base, ready_total, ready_base);
}

void launch_return_dw(const ReturnDwParams& p, cudaStream_t stream, bool behind) {
  launch_maybe_behind(behind, return_dw_kernel, (p.lay.S + 255) / 256, 256, 0, stream, p);
}

void launch_combine_reduce(const CombineParams& p, cudaStream_t stream, bool behind) {
  int grid = p.num_tokens < 1184 ? p.num_tokens : 1184;  // 8 CTAs per SM on 148 SMs
  if (grid < 1) grid = 1;
  launch_maybe_behind(behind, combine_reduce_kernel, grid, 256, 0, stream, p);
}

void launch_dequant_slice(const DequantParams& p, cudaStream_t stream) {
  // Every CTA visits every expert of the slice and waits for its arrival, so ALL CTAs must be resident at once for
  // an expert's rows to be released while later experts are still arriving: 72 CTAs of 256 threads fit on the dozen
  // SMs the up-projection GEMM leaves free on the fp8 wire (8 such CTAs per SM).
  dequant_slice_kernel<<<72, 256, 0, stream>>>(p);
}

void launch_wait_probe(const uint32_t* flag, uint32_t target, uint32_t spin_limit, StatusBlock* status,
                       cudaStream_t stream) {
  wait_probe_kernel<<<1, 1, 0, stream>>>(flag, target, spin_limit, status);
}

}  // namespace cem
