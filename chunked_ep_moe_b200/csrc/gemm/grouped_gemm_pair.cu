// Weight-gradient GEMM (dW[g] = lhs[rows_g]^T rhs[rows_g]) on CTA pairs: two CTAs of one cluster drive ONE 256 x 256 x 16
// tcgen05.mma (cta_group::2). Each CTA stages only its own 128 columns of A and its own 128 columns of B (32 KB per
// k-block instead of 48 KB): what bounds this mode, and any 128 x 256 tile per CTA, is the port between an SM and the
// crossbar to L2, one request per 128-byte line loaded and 32 bytes of store data per cycle.
//
//   both CTAs   warp 0      TMA producer for the CTA's own columns
//   leader      warp 1      waits for both halves of a stage, issues the pair MMAs, commits to both CTAs' empty barriers
//                           and both accumulator-full barriers.
//   peer        warp 1      for a tile's ragged last k-block it waits for its own loads, zero-fills the rows past the
//                           group and forwards the arrival to the leader.
//   both CTAs   warps 2-5   epilogue of the CTA's own 128 x 256 accumulator half, then arrive on the leader's
//                           accumulator-empty barrier.
//
// The pair splits the dense feature dimension, so it costs no token padding. Every wait is bounded; a CTA that gives up
// records a status and unwinds, and its partner then runs into its own limits.
#include "../common/pdl.cuh"
#include "gemm_common.cuh"

#include <type_traits>

namespace cem {

namespace {

constexpr int kPairStages = 6;
constexpr int kPairStageBytesA = kBlockM * kBlockK * 2;        // 16 KB: this CTA's 128 rows
constexpr int kPairStageBytesB = (kBlockN / 2) * kBlockK * 2;  // 16 KB: this CTA's 128 columns
constexpr int kPairStageBytes = kPairStageBytesA + kPairStageBytesB;
constexpr int kPairThreads = 192;
constexpr int kPairStagingBytes = 4 * 8192;  // two swizzled 4 KB blocks per epilogue warp
constexpr int kPairTailBytes = 512;  // barriers, TMEM slot, flags
constexpr int kPairSmemBytes = kSmemAlignSlack + kPairStages * kPairStageBytes + kPairStagingBytes + kPairTailBytes;
static_assert(kPairSmemBytes + 1024 + 1024 + 16 <= 233472, "no room for a second, small CTA on the SM");

// Experts of few rows: the A operand of a row of output tiles (an expert's rows x this CTA's 128 columns, up to five k-blocks) stays in
// shared memory while the pair walks `p.unit_cols` tiles along that row, and a k-block loads 16 KB instead of 32. Their tiles are a few
// k-blocks of MMA work for 64 KB of output, and the port that both have to cross is what bounds them. 256 rows of 64 experts at D=7168,
// F=2048: 880 -> 785 cycles per k-block, forward + backward (with the registers below) 5.61 -> 5.35 ms; of 256 experts 22.05 -> 21.32.
constexpr int kResidentBlocks = 5;                        // 16 KB slots of the panel; the ring's other seven hold B
constexpr int kResidentRing = 2 * kPairStages - kResidentBlocks;

// What a pair takes at a time, as seen by CTA `rank`: column tiles [n, n_end) of one row of tiles. One tile, unless the panel stays.
struct Unit {
  int g;      // local expert
  int row0;   // first slice row of the group
  int nrows;  // rows of the group
  int flags;  // kGroupFirst | kGroupFinal
  int m;      // row tile of the weight gradient (128 rows)
  int n, n_end;  // column tiles (256 columns)
  int kblocks;
  bool resident;
};

// The k-th unit where every unit is one tile.
__device__ __forceinline__ void tile_unit(const GemmParams& p, int t, int rank, Unit* u) {
  const int per_group = (p.m_tiles / 2) * p.n_tiles;
  const int gi = t / per_group, rem = t - gi * per_group;
  const int4 e = reinterpret_cast<const int4*>(p.plan + p.lay.off_gtiles + 4 * p.lay.max_gtiles * p.slice)[p.first_expert + gi];
  const int mp = rem / p.n_tiles;
  u->g = e.x; u->row0 = e.y; u->nrows = e.z; u->flags = e.w;
  u->m = 2 * mp + rank;
  u->n = rem - mp * p.n_tiles;
  u->n_end = u->n + 1;
  u->kblocks = (e.z + kBlockK - 1) / kBlockK;
  u->resident = false;
}

// Walks a pair's units, `step` apart in the order group, row of tiles, columns; a whole warp, which holds 32 groups at a time (one after
// the other, each an access to L2, they took longer than the tiles of small experts).
struct UnitWalk {
  int unit, window, base;  // next unit; first of the groups at hand and its first unit
  int4 e;                  // this lane's group
  int upto;                // units of the groups at hand up to and with this lane's
};

// Whether a unit of this group has `p.unit_cols` column tiles.
__device__ __forceinline__ bool long_units(const GemmParams& p, int rows) {
  return rows > 0 && rows <= kResidentBlocks * kBlockK;
}

__device__ __forceinline__ void load_window(const GemmParams& p, int groups, int lane, UnitWalk* w) {
  const int group = w->window + lane;
  w->e = make_int4(0, 0, 0, 0);
  w->upto = 0;
  if (group < groups) {
    w->e = reinterpret_cast<const int4*>(p.plan + p.lay.off_gtiles + 4 * p.lay.max_gtiles * p.slice)[p.first_expert + group];
    w->upto = (p.m_tiles / 2) * (long_units(p, w->e.z) ? p.row_units : p.n_tiles);
  }
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, w->upto, d);
    if (lane >= d) w->upto += up;
  }
}

template <bool PANEL>
__device__ __forceinline__ UnitWalk first_unit(const GemmParams& p, int groups, int lane, int unit) {
  UnitWalk w;
  w.unit = unit;
  w.window = w.base = 0;
  if constexpr (PANEL) load_window(p, groups, lane, &w);
  return w;
}

// False behind the last unit.
template <bool PANEL>
__device__ __forceinline__ bool next_unit(const GemmParams& p, int groups, int step, int rank, int lane, UnitWalk* w, Unit* u) {
  if constexpr (!PANEL) {
    if (w->unit >= groups * (p.m_tiles / 2) * p.n_tiles) return false;
    tile_unit(p, w->unit, rank, u);
    w->unit += step;
    return true;
  }
  while (w->window < groups) {
    const unsigned beyond = __ballot_sync(0xffffffffu, w->upto > w->unit - w->base);
    if (beyond != 0) {
      const int l = __ffs(beyond) - 1;
      u->g = __shfl_sync(0xffffffffu, w->e.x, l);
      u->row0 = __shfl_sync(0xffffffffu, w->e.y, l);
      u->nrows = __shfl_sync(0xffffffffu, w->e.z, l);
      u->flags = __shfl_sync(0xffffffffu, w->e.w, l);
      u->resident = long_units(p, u->nrows);
      const int per_row = u->resident ? p.row_units : p.n_tiles, cols = u->resident ? p.unit_cols : 1;
      const int rem = w->unit - w->base - __shfl_sync(0xffffffffu, w->upto, l) + (p.m_tiles / 2) * per_row;
      const int mp = rem / per_row;
      u->m = 2 * mp + rank;
      u->n = (rem - mp * per_row) * cols;
      u->n_end = u->n + cols < p.n_tiles ? u->n + cols : p.n_tiles;
      u->kblocks = (u->nrows + kBlockK - 1) / kBlockK;
      w->unit += step;
      return true;
    }
    w->base += __shfl_sync(0xffffffffu, w->upto, 31);
    w->window += 32;
    load_window(p, groups, lane, w);
  }
  return false;
}

// `bar` is the LEADER's full barrier (pair-aware loads credit the leader directly), except for `direct == false`
// (the peer's ragged last k-block): then it is this CTA's own full barrier and the loads are plain ones.
// A and B are both two 64-column chunks.
__device__ __forceinline__ void issue_a_block(const Unit& tl, int kb, const CUtensorMap* map_a, uint32_t sa, uint32_t bar, bool direct) {
  if (direct) tma_load_3d_pair(sa, map_a, bar, tl.row0 + kb * kBlockK, tl.m * (kBlockM / 64));
  else tma_load_3d(sa, map_a, bar, tl.row0 + kb * kBlockK, tl.m * (kBlockM / 64));
}

__device__ __forceinline__ void issue_b_block(const Unit& tl, int n, int kb, int rank, const CUtensorMap* map_b, uint32_t sb, uint32_t bar,
                                              bool direct) {
  const int chunk0 = n * (kBlockN / 64) + rank * (kBlockN / 128);  // this CTA's half of the 256-wide column tile
  if (direct) tma_load_3d_pair(sb, map_b, bar, tl.row0 + kb * kBlockK, chunk0);
  else tma_load_3d(sb, map_b, bar, tl.row0 + kb * kBlockK, chunk0);
}

// Epilogue of this CTA's 128 x 256 accumulator. `tacc` is this warp's TMEM address (lane quarter q, accumulator buffer),
// `stage_gen` the warp's 8 KB staging buffer.
__device__ __forceinline__ void tgmm_epilogue(const GemmParams& p, const Unit& tl, int n, uint32_t tacc, int q, int lane,
                                              uint8_t* stage_gen, const CUtensorMap* map_c) {
  const int row = q * 32 + lane;  // tile row owned by this thread
  uint32_t r[32];
  const size_t m_total = static_cast<size_t>(p.m_tiles) * kBlockM;
  const bool first = (tl.flags & kGroupFirst) != 0, final = (tl.flags & kGroupFinal) != 0;
  // The fp32 carry is private to this epilogue, so it is kept in the layout that suits it: tile by tile, and inside a
  // tile the 16-byte pieces (4 columns) of all 128 rows side by side. One warp load or store then covers 512
  // contiguous bytes (4 lines) instead of 32 rows 1 KB apart (32 requests at the SM's L2 port).
  const size_t tile_base = (static_cast<size_t>(tl.m) * p.n_tiles + n) * (kBlockM * kBlockN);
  auto carry_off = [&](int col) { return tile_base + (static_cast<size_t>(col >> 2) * kBlockM + row) * 4; };
  auto load_chunk = [&](int col) {
    float4 pv[8];
    if (!first) {
#pragma unroll
      for (int i = 0; i < 8; ++i) pv[i] = *reinterpret_cast<const float4*>(p.carry_in + carry_off(col + 4 * i));
    }
    if (tl.kblocks > 0) {
      tmem_ld_32x32(tacc + col, r);
      tmem_ld_wait();
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) r[i] = 0u;
    }
    if (!first) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        r[4 * i] = __float_as_uint(__uint_as_float(r[4 * i]) + pv[i].x);
        r[4 * i + 1] = __float_as_uint(__uint_as_float(r[4 * i + 1]) + pv[i].y);
        r[4 * i + 2] = __float_as_uint(__uint_as_float(r[4 * i + 2]) + pv[i].z);
        r[4 * i + 3] = __float_as_uint(__uint_as_float(r[4 * i + 3]) + pv[i].w);
      }
    }
  };
  if (final) {
    // bf16 gradient: the warp stages 32 rows x 64 columns at a time in the tensor map's swizzled layout (8 KB of
    // staging = two such blocks, so one block is filled while the other is being stored) and one lane hands each
    // block to the TMA as a tiled store: 16 stores of 4 KB per 128 x 256 tile, full lines, nobody waits for them.
    // (One 256-byte bulk store per lane and half tile was measured here and is slower: 256 small copies per tile
    // against ~4 k-blocks of MMA work.)
    const int out_row0 = tl.g * static_cast<int>(m_total) + tl.m * kBlockM + q * 32;  // in the [L*M, N] view
#pragma unroll 1
    for (int ch = 0; ch < kBlockN / 64; ++ch) {
      const int col = ch * 64;
      uint8_t* blk = stage_gen + (ch & 1) * 4096;
      if (lane == 0) bulk_wait_read_but_one();  // the store that last read this block is done with it
      __syncwarp();
      uint32_t r2[32];
      if (first && tl.kblocks > 0) {
        // Common case (the expert lies inside one slice): two TMEM loads per wait.
        tmem_ld_32x32(tacc + col, r);
        tmem_ld_32x32(tacc + col + 32, r2);
        tmem_ld_wait();
      } else {
        load_chunk(col + 32);
#pragma unroll
        for (int i = 0; i < 32; ++i) r2[i] = r[i];
        load_chunk(col);
      }
      uint8_t* my_row = blk + lane * 128;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        *reinterpret_cast<int4*>(my_row + ((i ^ (lane & 7)) << 4)) =
            make_int4(pack_bf16(__uint_as_float(r[8 * i]), __uint_as_float(r[8 * i + 1])),
                      pack_bf16(__uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3])),
                      pack_bf16(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5])),
                      pack_bf16(__uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7])));
        *reinterpret_cast<int4*>(my_row + (((4 + i) ^ (lane & 7)) << 4)) =
            make_int4(pack_bf16(__uint_as_float(r2[8 * i]), __uint_as_float(r2[8 * i + 1])),
                      pack_bf16(__uint_as_float(r2[8 * i + 2]), __uint_as_float(r2[8 * i + 3])),
                      pack_bf16(__uint_as_float(r2[8 * i + 4]), __uint_as_float(r2[8 * i + 5])),
                      pack_bf16(__uint_as_float(r2[8 * i + 6]), __uint_as_float(r2[8 * i + 7])));
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(map_c, smem_u32(blk), n * kBlockN + col, out_row0);
        bulk_commit();
      }
    }
  } else {
#pragma unroll 1
    for (int col = 0; col < kBlockN; col += 32) {
      load_chunk(col);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        *reinterpret_cast<float4*>(p.carry_out + carry_off(col + 4 * i)) =
            make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]),
                        __uint_as_float(r[4 * i + 3]));
    }
  }
}

// 192 registers per thread (at 168 the epilogue spills: expert kernels on 4001 rows of 16 experts at D=2048, F=1024 257.5 -> 253.8 us): two
// warps of 192 leave room in a quarter of the SM for two of the copy CTAs' 64 (the dispatch put, the fp8 expansion), which have to become
// resident BESIDE this kernel for the overlap to happen.
template <bool PANEL>
__global__ void __cluster_dims__(2, 1, 1) __maxnreg__(192)
grouped_gemm_pair_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ CUtensorMap map_a,
                         const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_c) {
  // Every load credits the leader's full barrier directly, with one exception: the last k-block of a weight-gradient
  // tile whose group does not end on a 64-row boundary needs rows zeroed by the CTA that owns them BEFORE the leader
  // may use them. For that k-block the peer loads onto its own full barrier, its warp 1 zero-fills and then makes the
  // arrival on the leader's barrier that the peer's producer makes for every other k-block. (An earlier form relayed
  // EVERY k-block of that mode through the peer's warp 1: one more hop on the critical path of each stage.)
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t staging_base = smem_base + kPairStages * kPairStageBytes;
  uint8_t* staging_gen = smem_gen + kPairStages * kPairStageBytes;
  const uint32_t bar_base = staging_base + kPairStagingBytes;
  // barriers: full[6], empty[6], acc_full[2], acc_empty[2], drain, the resident panel's full and empty, full[7] and empty[7] of the ring
  // beside it; then tmem slot, abort flag, early flag. Stage s of the six: A in slot s, B in slot 6 + s of 16 KB.
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kPairStages + s); };
  auto acc_full_bar = [&](int s) { return bar_base + 8u * (2 * kPairStages + s); };
  auto acc_empty_bar = [&](int s) { return bar_base + 8u * (2 * kPairStages + 2 + s); };
  const uint32_t drain_bar = bar_base + 8u * (2 * kPairStages + 4);
  const uint32_t panel_full = bar_base + 8u * (2 * kPairStages + 5), panel_empty = panel_full + 8;
  auto ring_full = [&](int s) { return panel_full + 16u + 8u * s; };
  auto ring_empty = [&](int s) { return panel_full + 16u + 8u * (kResidentRing + s); };
  constexpr int kSlotOff = 8 * (2 * kPairStages + 7 + 2 * kResidentRing);
  static_assert(kSlotOff + 12 <= kPairTailBytes, "barrier area too small");
  auto slot = [&](int i) { return smem_base + i * kPairStageBytesA; };
  const uint32_t tmem_slot = bar_base + kSlotOff;
  uint8_t* tail_gen = staging_gen + kPairStagingBytes;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(tail_gen + kSlotOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail_gen + kSlotOff + 4);
  volatile int* early_flag = reinterpret_cast<volatile int*>(tail_gen + kSlotOff + 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_cta_rank());
  const bool leader = rank == 0;
  const bool counting = p.prof != nullptr;
  auto prof_add = [&](int slot, long long v) {
    atomicAdd(p.prof + static_cast<size_t>(blockIdx.x) * kProfSlots + slot, static_cast<unsigned long long>(v));
  };

  // A CTA that gives up tells its partner too (the flag sits at the same offset in both CTAs), so the partner's waits
  // end at their next poll instead of running into their own limits.
  const uint32_t partner_abort = map_to_cta(bar_base + kSlotOff + 4, static_cast<uint32_t>(rank ^ 1));
  auto raise_abort = [&]() {
    *abort_flag = 1;
    st_shared_cluster_u32(partner_abort, 1u);
  };

  // The aligned layout must fit into what the launch provided. Both CTAs of a pair see the same offsets, so they
  // leave together.
  if (smem_base - smem_u32(smem_raw) > static_cast<uint32_t>(kSmemAlignSlack)) {
    if (threadIdx.x == 0) report_status(p.status, kStatusBadIndex, kKernelGemm, kModeTgmm, -1, 1, kSmemAlignSlack,
                                        smem_base - smem_u32(smem_raw));
    return;
  }
  release_successor();
  cluster_sync_all();  // both CTAs run

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairStages; ++s) {
      // leader: one arrival from each CTA of the pair; the peer's own barrier only sees its ragged-tail loads
      mbar_init(full_bar(s), leader ? 2 : 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(acc_full_bar(s), 1);
      mbar_init(acc_empty_bar(s), 8);  // four epilogue warps in each CTA of the pair
    }
    for (int s = 0; s < kResidentRing; ++s) {
      mbar_init(ring_full(s), leader ? 2 : 1);
      mbar_init(ring_empty(s), 1);
    }
    mbar_init(panel_full, leader ? 2 : 1);  // leader: its own loads and the peer's warp 1
    mbar_init(panel_empty, 1);
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    mbar_init_fence();
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    tma_prefetch_desc(&map_c);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  // Launched behind its predecessor, the kernel has come this far in that one's tail; global memory from here on.
  wait_predecessor();
  // An earlier kernel of this pass already gave up: neither CTA of the pair does anything (the leader decides).
  if (threadIdx.x == 0 && leader) {
    const uint32_t v = (p.status != nullptr && p.status->code != 0) ? 1u : 0u;
    *early_flag = static_cast<int>(v);
    st_shared_cluster_u32(map_to_cta(bar_base + kSlotOff + 8, 1), v);
  }
  tcgen05_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anyone signals across the pair
  tcgen05_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot_gen;

  int groups = 0;
  if (*early_flag == 0) groups = p.last_expert > 0 ? p.last_expert - p.first_expert : p.plan[p.lay.off_num_gtiles + p.slice];
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

  if (warp == 0) {
    // ================================ TMA producer (both CTAs) ==============================
    // The whole warp walks the k-blocks in step; one elected lane issues the copies.
    uint32_t it = 0, rit = 0, panels = 0;  // uses of the six stages, of the ring beside a panel, of the panel
    // per stage (bits 6 on: the ring): this CTA's own full barrier has been used / parity of its next use
    uint32_t own_used = 0, own_parity = 0;
    long long empty_wait = 0;
    uint32_t ps = 0, pph = 0, rs = 0, rph = 0;
    bool dead = false, was_resident = false;
    int at = 0;  // unit at hand, for the status
    auto fail = [&](int detail) {
      if (lane == 0) {
        report_status(p.status, kStatusMbarTimeout, kKernelGemm, kModeTgmm, at, detail, 0, 0);
        raise_abort();
      }
      dead = true;
    };
    auto wait_free = [&](uint32_t bar, uint32_t parity, int detail) {
      const long long w0 = counting ? clock64() : 0;
      if (!__all_sync(0xffffffffu, mbar_wait(bar, parity, p.mbar_limit, abort_flag))) {
        fail(detail);
        return false;
      }
      if (counting) empty_wait += clock64() - w0;
      return true;
    };
    // Stages and panel share the slots: what the MMAs may still read of one is waited for before the other is filled.
    auto switch_to = [&](bool resident) {
      if (resident == was_resident) return true;
      was_resident = resident;
      bool ok = true;
      if (resident) {
        for (int i = 0; i < kPairStages && ok; ++i)
          ok = wait_free(empty_bar(i), (static_cast<uint32_t>(i) >= ps ? pph : pph ^ 1u) ^ 1u, 1150 + i);
      } else {
        for (int i = 0; i < kResidentRing && ok; ++i)
          ok = wait_free(ring_empty(i), (static_cast<uint32_t>(i) >= rs ? rph : rph ^ 1u) ^ 1u, 1160 + i);
        if (ok) ok = wait_free(panel_empty, (panels & 1u) ^ 1u, 1170);
      }
      return ok;
    };
    // A unit's k-blocks into the six stages, or B's beside the panel. (Two loops: what a k-block costs this warp counts.)
    auto fill = [&](auto resident, const Unit& u, uint32_t& s, uint32_t& ph, uint32_t& used) {
      constexpr bool kResident = decltype(resident)::value;
      constexpr uint32_t kStages = kResident ? kResidentRing : kPairStages;
      constexpr uint32_t kBytes = kResident ? kPairStageBytesB : kPairStageBytes;
      const bool peer_tail = !leader && (u.nrows % kBlockK) != 0;
      for (int n = u.n; n < u.n_end && !dead; ++n) {
        for (int kb = 0; kb < u.kblocks; ++kb) {
          const long long w0 = counting ? clock64() : 0;
          const uint32_t empty = kResident ? ring_empty(s) : empty_bar(s), full = kResident ? ring_full(s) : full_bar(s);
          if (!__all_sync(0xffffffffu, mbar_wait(empty, ph ^ 1u, p.mbar_limit, abort_flag))) {
            fail((kResident ? 1110 : 1100) + s);
            break;
          }
          if (counting) empty_wait += clock64() - w0;
          const bool own = peer_tail && kb == u.kblocks - 1;
          if (own) {
            const uint32_t bit = 1u << (kResident ? kPairStages + s : s);
            own_used |= bit;
            own_parity ^= bit;
          }
          if (elect_one()) {
            const uint32_t fb = own ? full : map_to_cta(full, 0);
            if (own) mbar_expect_tx(fb, kBytes); else mbar_expect_tx_cluster(fb, kBytes);
            if constexpr (!kResident) issue_a_block(u, kb, &map_a, slot(s), fb, !own);
            issue_b_block(u, n, kb, rank, &map_b, slot((kResident ? kResidentBlocks : kPairStages) + s), fb, !own);
          }
          ++used;
          if (++s == kStages) { s = 0; ph ^= 1u; }
        }
      }
    };
    // The next unit is looked up one ahead, so its plan-table loads are in flight while this one runs.
    Unit nxt = {};
    UnitWalk walk = first_unit<PANEL>(p, groups, lane, first);
    bool more = next_unit<PANEL>(p, groups, step, rank, lane, &walk, &nxt);
    while (more && !dead && !*abort_flag) {
      const Unit u = nxt;
      more = next_unit<PANEL>(p, groups, step, rank, lane, &walk, &nxt);
      ++at;
      if constexpr (PANEL) {
        if (!switch_to(u.resident)) break;
      }
      if (PANEL && u.resident) {
        if (!wait_free(panel_empty, (panels & 1u) ^ 1u, 1140)) break;
        ++panels;
        if (elect_one()) {  // each CTA's panel on its own barrier: the peer's warp 1 passes the arrival on
          mbar_expect_tx(panel_full, u.kblocks * kPairStageBytesA);
          for (int kb = 0; kb < u.kblocks; ++kb) issue_a_block(u, kb, &map_a, slot(kb), panel_full, false);
        }
      }
      if (PANEL && u.resident) fill(std::true_type(), u, rs, rph, rit);
      else fill(std::false_type(), u, ps, pph, it);
    }
    __syncwarp();
    if (counting && lane == 0) prof_add(kProfEmptyWait, empty_wait);
    // Unwinding: no exit while a copy may still land in this CTA's shared memory. The leader's barriers see every
    // stage of both CTAs; the peer's own barriers only its ragged-tail loads (their last use has the parity before
    // the next one's). The panel's are each CTA's own.
    if (lane == 0 && *abort_flag) {
      if (PANEL && panels > 0) mbar_wait(panel_full, (panels - 1) & 1u, p.mbar_limit);
      for (uint32_t i = 0; i < kPairStages + (PANEL ? kResidentRing : 0); ++i) {
        const bool ring = i >= kPairStages;
        const uint32_t bar = ring ? ring_full(i - kPairStages) : full_bar(i), stage = ring ? i - kPairStages : i;
        const uint32_t used = ring ? rit : it, stages = ring ? kResidentRing : kPairStages;
        if (leader) {
          if (used > stage) {
            const uint32_t last = used - 1 - ((used - 1 - stage) % stages);
            mbar_wait(bar, (last / stages) & 1u, p.mbar_limit);
          }
        } else if ((own_used >> i) & 1u) {
          mbar_wait(bar, ((own_parity >> i) & 1u) ^ 1u, p.mbar_limit);
        }
      }
    }
  } else if (warp == 1) {
    // ================================ MMA issuer (leader) / stage relay (peer) ==============
    // The whole warp walks the k-blocks in step; one elected lane (always the same one) issues MMAs and commits.
    constexpr uint32_t idesc = make_instr_desc_bf16(2 * kBlockM, kBlockN, true, true);
    constexpr uint32_t kDescStep = 2048u;  // bytes per 16-row k step inside a stage
    const uint32_t peer = static_cast<uint32_t>(rank ^ 1);
    uint32_t it = 0, tcount = 0, panels = 0;
    uint32_t own_phase = 0;  // peer: parity of the next use of its own full barrier, per stage (bits 6 on: the ring)
    long long full_wait = 0, acc_wait = 0;
    const long long loop_c0 = counting ? clock64() : 0;
    const uint64_t loop_n0 = counting ? global_timer_ns() : 0;
    uint32_t cs = 0, cph = 0, rs = 0, rph = 0;
    bool dead = false;
    int at = 0;
    auto fail = [&](int detail) {
      if (lane == 0) {
        report_status(p.status, kStatusMbarTimeout, kKernelGemm, kModeTgmm, at, detail, 0, 0);
        raise_abort();
      }
      dead = true;
    };
    auto wait_all = [&](uint32_t bar, uint32_t parity, int detail) {
      if (__all_sync(0xffffffffu, mbar_wait(bar, parity, p.mbar_limit, abort_flag))) return true;
      fail(detail);
      return false;
    };
    // Zeroes rows [valid, 16 ksteps) of the two 64-column chunks of A (lanes 0-15) and of B (16-31): a k row of a chunk is eight
    // 16-byte pieces, a lane clears one of each row.
    auto zero_rows = [&](uint32_t a, uint32_t b, bool with_a, bool with_b, int valid, int ksteps) {
      uint8_t* piece = smem_gen + ((lane < 16 ? a : b) - smem_base) + ((lane >> 3) & 1) * 8192 + (lane & 7) * 16 + valid * 128;
      const int rows = (lane < 16 ? with_a : with_b) ? ksteps * kUmmaK - valid : 0;
      for (int r = 0; r < rows; ++r, piece += 128) *reinterpret_cast<int4*>(piece) = make_int4(0, 0, 0, 0);
    };
    // A tile's k-blocks out of the six stages, or the panel's and the ring's beside it.
    auto multiply = [&](auto resident, const Unit& u, uint32_t tmem_d, uint32_t& s, uint32_t& ph, int tail_steps, int valid) {
      constexpr bool kResident = decltype(resident)::value;
      constexpr uint32_t kStages = kResident ? kResidentRing : kPairStages;
      const bool ragged = valid != kBlockK;
      auto b_slot = [&]() { return slot((kResident ? kResidentBlocks : kPairStages) + s); };
      auto full = [&]() { return kResident ? ring_full(s) : full_bar(s); };
      auto issue = [&](int kb, int ksteps) {
        const uint64_t da = make_smem_desc(slot(kResident ? kb : s), 8192, 1024), db = make_smem_desc(b_slot(), 8192, 1024);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < kBlockK / kUmmaK; ++k) {
            if (k < ksteps)
              umma_bf16_pair(tmem_d, da + ((k * kDescStep) >> 4), db + ((k * kDescStep) >> 4), idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit_pair_both(kResident ? ring_empty(s) : empty_bar(s));
        }
      };
      auto advance = [&]() {
        ++it;
        if (++s == kStages) { s = 0; ph ^= 1u; }
      };
      const int solo = ragged ? u.kblocks - 1 : u.kblocks;
      for (int kb = 0; kb < solo; ++kb) {
        if (leader) {
          const long long w1 = counting ? clock64() : 0;
          const bool ok = __all_sync(0xffffffffu, mbar_wait(full(), ph, p.mbar_limit, abort_flag));
          if (counting) full_wait += clock64() - w1;
          if (!ok) { fail((kResident ? 1310 : 1300) + s); return; }
          tcgen05_fence_after_sync();
          issue(kb, kBlockK / kUmmaK);
        }
        advance();  // the peer only keeps count of the stages: its loads credit the leader's barrier
      }
      if (!ragged) return;
      // Leader: both halves have landed and the peer has zero-filled its rows. Peer: its own loads have landed.
      const uint32_t bit = kResident ? kPairStages + s : s;
      const uint32_t parity = leader ? ph : (own_phase >> bit) & 1u;
      own_phase ^= 1u << bit;
      if (!wait_all(full(), parity, (kResident ? 1310 : 1300) + s)) return;
      zero_rows(slot(kResident ? 0 : s), b_slot(), !kResident, true, valid, tail_steps);
      fence_proxy_async_smem();
      __syncwarp();
      if (!leader) {
        // the arrival the peer's producer makes for every other k-block, after the rows are clean
        if (elect_one()) mbar_arrive_cluster(map_to_cta(full(), peer));
      } else {
        tcgen05_fence_after_sync();
        issue(u.kblocks - 1, tail_steps);
      }
      advance();
    };
    Unit nxt = {};
    UnitWalk walk = first_unit<PANEL>(p, groups, lane, first);
    bool more = next_unit<PANEL>(p, groups, step, rank, lane, &walk, &nxt);
    while (more && !dead && !*abort_flag) {
      const Unit u = nxt;
      more = next_unit<PANEL>(p, groups, step, rank, lane, &walk, &nxt);
      ++at;
      const int valid = u.kblocks > 0 ? u.nrows - (u.kblocks - 1) * kBlockK : kBlockK;  // rows of the last k-block
      const int tail_steps = (valid + kUmmaK - 1) / kUmmaK;
      if (PANEL && u.resident) {
        if (!wait_all(panel_full, panels & 1u, 1400)) break;
        ++panels;
        if (valid != kBlockK) {
          zero_rows(slot(u.kblocks - 1), 0, true, false, valid, tail_steps);
          fence_proxy_async_smem();
          __syncwarp();
        }
        if (!leader && elect_one()) mbar_arrive_cluster(map_to_cta(panel_full, peer));
        tcgen05_fence_after_sync();
      }
      for (int n = u.n; n < u.n_end && !dead; ++n, ++tcount) {
        const int as = tcount & 1;
        const uint32_t tmem_d = tmem_base + as * kBlockN;
        if (leader) {
          const long long w0 = counting ? clock64() : 0;
          const bool ok = wait_all(acc_empty_bar(as), ((tcount >> 1) & 1u) ^ 1u, 1200 + as);
          if (counting) acc_wait += clock64() - w0;
          if (!ok) break;
          tcgen05_fence_after_sync();
        }
        if (PANEL && u.resident) multiply(std::true_type(), u, tmem_d, rs, rph, tail_steps, valid);
        else multiply(std::false_type(), u, tmem_d, cs, cph, tail_steps, valid);
        if (dead) break;
        if (leader && elect_one()) {
          if ((PANEL && u.resident) && n + 1 == u.n_end) umma_commit_pair_both(panel_empty);
          if (u.kblocks > 0) {
            umma_commit_pair_both(acc_full_bar(as));
          } else {
            mbar_arrive(acc_full_bar(as));  // empty group: both epilogues write zeros
            mbar_arrive_cluster(map_to_cta(acc_full_bar(as), peer));
          }
        }
      }
    }
    __syncwarp();
    if (counting && leader && lane == 0) {
      prof_add(kProfLoopCycles, clock64() - loop_c0);
      prof_add(kProfLoopNs, static_cast<long long>(global_timer_ns() - loop_n0));
      prof_add(kProfFullWait, full_wait);
      prof_add(kProfAccWait, acc_wait);
      prof_add(kProfKBlocks, it);
      prof_add(kProfTiles, tcount);
    }
    if (leader && *abort_flag) {
      __syncwarp();
      if (elect_one()) umma_commit_pair(drain_bar);
      mbar_wait(drain_bar, 0, p.mbar_limit);
    }
  } else {
    // ================================ epilogue (both CTAs) ==================================
    const int q = warp & 3;
    uint8_t* stage_gen = staging_gen + (warp - 2) * 8192;
    const uint32_t leader_acc_empty0 = map_to_cta(acc_empty_bar(0), 0);
    uint32_t tcount = 0;
    bool dead = false;
    int at = 0;
    Unit nxt = {};
    UnitWalk walk = first_unit<PANEL>(p, groups, lane, first);
    bool more = next_unit<PANEL>(p, groups, step, rank, lane, &walk, &nxt);
    while (more && !dead && !*abort_flag) {
      const Unit u = nxt;
      more = next_unit<PANEL>(p, groups, step, rank, lane, &walk, &nxt);
      ++at;
      for (int n = u.n; n < u.n_end && !dead; ++n, ++tcount) {
        const int as = tcount & 1;
        const bool ok = mbar_wait(acc_full_bar(as), (tcount >> 1) & 1u, p.mbar_limit, abort_flag);
        if (!ok) {
          report_status(p.status, kStatusMbarTimeout, kKernelGemm, kModeTgmm, at, 1500 + as, 0, 0);
          raise_abort();
        }
        dead = !__all_sync(0xffffffffu, ok);
        if (dead) break;
        tcgen05_fence_after_sync();
        const uint32_t tacc = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + as * kBlockN;
        tgmm_epilogue(p, u, n, tacc, q, lane, stage_gen, &map_c);
        tcgen05_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(leader_acc_empty0 + 8u * as);
      }
    }
    bulk_wait_all();  // bulk stores of this thread still read the staging rows: no exit before they are done
  }

  // ================================ teardown ================================================
  tcgen05_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // nobody frees TMEM or leaves while its partner may still signal or compute
  if (warp == 1) {
    tcgen05_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace

std::atomic<int> g_pair_grid_used{0};

// Column tiles along which a pair keeps its panel: all of a row, or fewer where the last turn of longer units would leave more pairs
// idle than the loads saved are worth. A tile crosses the port in 2048 cycles of stores and, at 256 rows, 576 of B and 576 of A / the
// unit's tiles. (Were every expert to have few rows; the others' tiles are dealt one by one whatever this says.)
int weight_grad_unit_cols(int rows_of_tiles, int n_tiles, int pairs) {
  int best = 1;
  long long least = 0;
  for (int units = 1; units <= n_tiles; ++units) {  // to a row
    const int cols = (n_tiles + units - 1) / units;
    if (units > 1 && cols == (n_tiles + units - 2) / (units - 1)) continue;
    const long long turns = (static_cast<long long>(rows_of_tiles) * ((n_tiles + cols - 1) / cols) + pairs - 1) / pairs;
    const long long cycles = turns * (cols * (2048ll + 576) + 576);
    if (least == 0 || cycles < least) {
      least = cycles;
      best = cols;
    }
  }
  return best;
}

template <bool PANEL>
static void launch_pair(GemmParams p, const CUtensorMap& map_a, const CUtensorMap& map_b, const CUtensorMap& map_c, int grid, int groups,
                        cudaStream_t stream, bool behind) {
  static const int resident = resident_pair_grid(grouped_gemm_pair_kernel<PANEL>, kPairThreads, kPairSmemBytes);
  grid &= ~1;  // whole pairs only
  const int g = grid < resident ? grid : resident;
  g_pair_grid_used = g;
  if constexpr (PANEL) {
    p.unit_cols = weight_grad_unit_cols(groups * (p.m_tiles / 2), p.n_tiles, g / 2);
    p.row_units = (p.n_tiles + p.unit_cols - 1) / p.unit_cols;
  }
  launch_maybe_behind(behind, grouped_gemm_pair_kernel<PANEL>, g, kPairThreads, kPairSmemBytes, stream, p, map_a, map_b, map_c);
}

// Panels pay where most experts can have one and there are units enough to even them out: at up to 320 rows an expert on average and
// from 32 tiles a pair on (16 experts of 250 rows at D=2048, F=1024, 7 and 14 tiles a pair: the expert kernels 260 us without, 277 with;
// 32 of 750 with Zipf routing at D=7168 628 and 643 cycles per k-block, the walk along units costs a tile some 300).
void launch_weight_grad(const GemmParams& p, const CUtensorMap& map_a, const CUtensorMap& map_b, const CUtensorMap& map_c, int grid,
                        int64_t rows, cudaStream_t stream, bool behind) {
  const int groups = p.last_expert > 0 ? p.last_expert - p.first_expert : p.lay.L;
  const int64_t tiles = static_cast<int64_t>(groups) * (p.m_tiles / 2) * p.n_tiles;
  if (rows <= static_cast<int64_t>(kResidentBlocks * kBlockK) * p.lay.L && tiles >= 32 * (grid / 2))
    launch_pair<true>(p, map_a, map_b, map_c, grid, groups, stream, behind);
  else
    launch_pair<false>(p, map_a, map_b, map_c, grid, groups, stream, behind);
}

}  // namespace cem
