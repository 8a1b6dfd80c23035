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

namespace cem {

namespace {

constexpr int kPairStages = 6;
constexpr int kPairStageBytesA = kBlockM * kBlockK * 2;        // 16 KB: this CTA's 128 rows
constexpr int kPairStageBytesB = (kBlockN / 2) * kBlockK * 2;  // 16 KB: this CTA's 128 columns
constexpr int kPairStageBytes = kPairStageBytesA + kPairStageBytesB;
constexpr int kPairThreads = 192;
constexpr int kPairStagingBytes = 4 * 8192;  // two swizzled 4 KB blocks per epilogue warp
constexpr int kPairSmemBytes = kSmemAlignSlack + kPairStages * kPairStageBytes + kPairStagingBytes + kSmemTailBytes;
static_assert(kPairSmemBytes + 1024 + 1024 + 16 <= 233472, "no room for a second, small CTA on the SM");

// Tile as seen by CTA `rank` of the pair.
struct Tile {
  int g;      // local expert
  int row0;   // first slice row of the group
  int nrows;  // rows of the group
  int flags;  // kGroupFirst | kGroupFinal
  int m;      // row tile of the weight gradient (128 rows)
  int n;      // column tile (256 columns)
  int kblocks;
};

__device__ __forceinline__ Tile decode_pair_tile(const GemmParams& p, int t, int rank) {
  Tile tl;
  const int per_group = (p.m_tiles / 2) * p.n_tiles;
  const int gi = t / per_group, rem = t - gi * per_group;
  const int4 e = reinterpret_cast<const int4*>(p.plan + p.lay.off_gtiles + 4 * p.lay.max_gtiles * p.slice)[p.first_expert + gi];
  tl.g = e.x; tl.row0 = e.y; tl.nrows = e.z; tl.flags = e.w;
  const int mp = rem / p.n_tiles;
  tl.m = 2 * mp + rank; tl.n = rem - mp * p.n_tiles;
  tl.kblocks = (e.z + kBlockK - 1) / kBlockK;
  return tl;
}

// `bar` is the LEADER's full barrier (pair-aware loads credit the leader directly), except for `direct == false`
// (the peer's ragged last k-block): then it is this CTA's own full barrier and the loads are plain ones.
__device__ __forceinline__ void issue_pair_kblock(const Tile& tl, int kb, int rank, const CUtensorMap* map_a,
                                                  const CUtensorMap* map_b, uint32_t sa, uint32_t sb, uint32_t bar,
                                                  bool direct) {
  const int chunk0 = tl.n * (kBlockN / 64) + rank * (kBlockN / 128);  // this CTA's half of the 256-wide column tile
  // A and B are both two 64-column chunks
  if (direct) {
    tma_load_3d_pair(sa, map_a, bar, tl.row0 + kb * kBlockK, tl.m * (kBlockM / 64));
    tma_load_3d_pair(sb, map_b, bar, tl.row0 + kb * kBlockK, chunk0);
  } else {
    tma_load_3d(sa, map_a, bar, tl.row0 + kb * kBlockK, tl.m * (kBlockM / 64));
    tma_load_3d(sb, map_b, bar, tl.row0 + kb * kBlockK, chunk0);
  }
}

// Epilogue of this CTA's 128 x 256 accumulator. `tacc` is this warp's TMEM address (lane quarter q, accumulator buffer),
// `stage_gen` the warp's 8 KB staging buffer.
__device__ __forceinline__ void tgmm_epilogue(const GemmParams& p, const Tile& tl, uint32_t tacc, int q, int lane,
                                              uint8_t* stage_gen, const CUtensorMap* map_c) {
  const int row = q * 32 + lane;  // tile row owned by this thread
  uint32_t r[32];
  const size_t m_total = static_cast<size_t>(p.m_tiles) * kBlockM;
  const bool first = (tl.flags & kGroupFirst) != 0, final = (tl.flags & kGroupFinal) != 0;
  // The fp32 carry is private to this epilogue, so it is kept in the layout that suits it: tile by tile, and inside a
  // tile the 16-byte pieces (4 columns) of all 128 rows side by side. One warp load or store then covers 512
  // contiguous bytes (4 lines) instead of 32 rows 1 KB apart (32 requests at the SM's L2 port).
  const size_t tile_base = (static_cast<size_t>(tl.m) * p.n_tiles + tl.n) * (kBlockM * kBlockN);
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
        tma_store_2d(map_c, smem_u32(blk), tl.n * kBlockN + col, out_row0);
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

// 168 registers per thread: 192 threads x 168 leave half of the SM's register file to a copy CTA (the dispatch put, the
// fp8 expansion), which has to become resident BESIDE this kernel for the overlap to happen.
__global__ void __cluster_dims__(2, 1, 1) __maxnreg__(168)
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
  // barriers: full[6], empty[6], acc_full[2], acc_empty[2], drain; then tmem slot, abort flag, early flag
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kPairStages + s); };
  auto acc_full_bar = [&](int s) { return bar_base + 8u * (2 * kPairStages + s); };
  auto acc_empty_bar = [&](int s) { return bar_base + 8u * (2 * kPairStages + 2 + s); };
  const uint32_t drain_bar = bar_base + 8u * (2 * kPairStages + 4);
  constexpr int kSlotOff = 8 * (2 * kPairStages + 5);
  static_assert(kSlotOff + 12 <= kSmemTailBytes, "barrier area too small");
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
  const int num_tiles = groups * (p.m_tiles / 2) * p.n_tiles;
  const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;

  if (warp == 0) {
    // ================================ TMA producer (both CTAs) ==============================
    uint32_t it = 0;
    uint32_t own_used = 0, own_parity = 0;  // per stage: this CTA's own full barrier has been used / parity of its next use
    long long empty_wait = 0;
    {
      // The whole warp walks the k-blocks in step; one elected lane issues the copies.
      uint32_t ps = 0, pph = 0;
      bool dead = false;
      // The next tile is decoded one iteration ahead, so its plan-table load is in flight while this tile runs.
      Tile nxt = {};
      if (first_tile < num_tiles) nxt = decode_pair_tile(p, first_tile, rank);
      for (int t = first_tile; t < num_tiles && !dead && !*abort_flag; t += tile_step) {
        const Tile tl = nxt;
        if (t + tile_step < num_tiles) nxt = decode_pair_tile(p, t + tile_step, rank);
        for (int kb = 0; kb < tl.kblocks; ++kb) {
          const long long w0 = counting ? clock64() : 0;
          const bool ok = __all_sync(0xffffffffu, mbar_wait(empty_bar(ps), pph ^ 1u, p.mbar_limit, abort_flag));
          if (!ok) {
            if (lane == 0) {
              report_status(p.status, kStatusMbarTimeout, kKernelGemm, kModeTgmm, t, 1100 + ps, 0, 0);
              raise_abort();
            }
            dead = true;
            break;
          }
          if (counting) empty_wait += clock64() - w0;
          const bool own = !leader && kb == tl.kblocks - 1 && (tl.nrows % kBlockK) != 0;
          if (own) {
            own_used |= 1u << ps;
            own_parity ^= 1u << ps;
          }
          if (elect_one()) {
            const uint32_t sa = smem_base + ps * kPairStageBytes;
            const uint32_t fb = own ? full_bar(ps) : map_to_cta(full_bar(ps), 0);
            if (own) mbar_expect_tx(fb, kPairStageBytes); else mbar_expect_tx_cluster(fb, kPairStageBytes);
            issue_pair_kblock(tl, kb, rank, &map_a, &map_b, sa, sa + kPairStageBytesA, fb, !own);
          }
          ++it;
          if (++ps == kPairStages) { ps = 0; pph ^= 1u; }
        }
      }
      __syncwarp();
    }
    if (counting && lane == 0) prof_add(kProfEmptyWait, empty_wait);
    // Unwinding: no exit while a copy may still land in this CTA's shared memory. The leader's barriers see every
    // stage of both CTAs; the peer's own barriers only its ragged-tail loads (their last use has the parity before
    // the next one's).
    if (lane == 0 && *abort_flag) {
      for (int s = 0; s < kPairStages; ++s) {
        if (leader) {
          if (it > static_cast<uint32_t>(s)) {
            const uint32_t last = it - 1 - ((it - 1 - s) % kPairStages);
            mbar_wait(full_bar(s), (last / kPairStages) & 1u, p.mbar_limit);
          }
        } else if ((own_used >> s) & 1u) {
          mbar_wait(full_bar(s), ((own_parity >> s) & 1u) ^ 1u, p.mbar_limit);
        }
      }
    }
  } else if (warp == 1) {
    // ================================ MMA issuer (leader) / stage relay (peer) ==============
    // The whole warp walks the k-blocks in step and one elected lane issues.
    constexpr uint32_t idesc = make_instr_desc_bf16(2 * kBlockM, kBlockN, true, true);
    constexpr uint32_t kDescStep = 2048u;  // bytes per 16-row k step inside a stage
    const uint32_t peer = static_cast<uint32_t>(rank ^ 1);
    uint32_t it = 0, tcount = 0;
    uint32_t own_phase = 0;  // peer, weight-gradient mode: parity of the next use of its own full barrier, per stage
    long long full_wait = 0, acc_wait = 0;
    const long long loop_c0 = counting ? clock64() : 0;
    const uint64_t loop_n0 = counting ? global_timer_ns() : 0;
    {
      // The whole warp walks the k-blocks in step; one elected lane (always the same one) issues MMAs and commits.
      uint32_t cs = 0, cph = 0;
      bool dead = false;
      auto issue_stage = [&](uint32_t s, uint32_t tmem_d, int ksteps, bool first_kblock) {
        const uint32_t sa = smem_base + s * kPairStageBytes;
        const uint64_t da = make_smem_desc(sa, 8192, 1024), db = make_smem_desc(sa + kPairStageBytesA, 8192, 1024);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < kBlockK / kUmmaK; ++k) {
            if (k < ksteps)
              umma_bf16_pair(tmem_d, da + ((k * kDescStep) >> 4), db + ((k * kDescStep) >> 4), idesc,
                             (!first_kblock || k > 0) ? 1u : 0u);
          }
          umma_commit_pair_both(empty_bar(s));
        }
      };
      auto fail = [&](int t, int detail) {
        if (lane == 0) {
          report_status(p.status, kStatusMbarTimeout, kKernelGemm, kModeTgmm, t, detail, 0, 0);
          raise_abort();
        }
        dead = true;
      };
      auto advance = [&]() {
        ++it;
        if (++cs == kPairStages) { cs = 0; cph ^= 1u; }
      };
      // The next tile is decoded one iteration ahead, so its plan-table load is in flight while this tile runs.
      Tile nxt = {};
      if (first_tile < num_tiles) nxt = decode_pair_tile(p, first_tile, rank);
      for (int t = first_tile; t < num_tiles && !dead && !*abort_flag; t += tile_step, ++tcount) {
        const Tile tl = nxt;
        if (t + tile_step < num_tiles) nxt = decode_pair_tile(p, t + tile_step, rank);
        const int as = tcount & 1;
        const uint32_t aph = (tcount >> 1) & 1u;
        const uint32_t tmem_d = tmem_base + as * kBlockN;
        const bool ragged_tail = (tl.nrows % kBlockK) != 0;
        const int solo_kblocks = ragged_tail ? tl.kblocks - 1 : tl.kblocks;
        bool ok = true;
        if (leader) {
          const long long w0 = counting ? clock64() : 0;
          ok = __all_sync(0xffffffffu, mbar_wait(acc_empty_bar(as), aph ^ 1u, p.mbar_limit, abort_flag));
          if (counting) acc_wait += clock64() - w0;
          if (!ok) { fail(t, 1200 + as); break; }
          tcgen05_fence_after_sync();
        }
        for (int kb = 0; kb < solo_kblocks; ++kb) {
          if (leader) {
            const long long w1 = counting ? clock64() : 0;
            ok = __all_sync(0xffffffffu, mbar_wait(full_bar(cs), cph, p.mbar_limit, abort_flag));
            if (counting) full_wait += clock64() - w1;
            if (!ok) { fail(t, 1300 + cs); break; }
            tcgen05_fence_after_sync();
            issue_stage(cs, tmem_d, kBlockK / kUmmaK, kb == 0);
          }
          advance();  // the peer only keeps count of the stages: its loads credit the leader's barrier
        }
        if (dead) break;
        if (ragged_tail) {
          const int kb = tl.kblocks - 1;
          // Leader: both halves have landed and the peer has zero-filled its rows. Peer: its own loads have landed.
          const uint32_t parity = leader ? cph : ((own_phase >> cs) & 1u);
          own_phase ^= 1u << cs;
          ok = __all_sync(0xffffffffu, mbar_wait(full_bar(cs), parity, p.mbar_limit, abort_flag));
          if (!ok) { fail(t, 1300 + cs); break; }
          const int valid = tl.nrows - kb * kBlockK;
          const int ksteps = (valid + kUmmaK - 1) / kUmmaK;
          // Zero this CTA's rows [valid, ksteps*16) in its four 64-column chunks (2 of A, 2 of B): a k row is 32
          // 16-byte pieces here, lane i clears piece i.
          uint8_t* ga = smem_gen + cs * kPairStageBytes;
          const int zrows = ksteps * kUmmaK - valid;
          uint8_t* piece = ga + (lane >> 3) * 8192 + (lane & 7) * 16 + valid * 128;
          for (int r = 0; r < zrows; ++r, piece += 128) *reinterpret_cast<int4*>(piece) = make_int4(0, 0, 0, 0);
          fence_proxy_async_smem();
          __syncwarp();
          if (!leader) {
            // the arrival the peer's producer makes for every other k-block, after the rows are clean
            if (elect_one()) mbar_arrive_cluster(map_to_cta(full_bar(cs), peer));
          } else {
            tcgen05_fence_after_sync();
            issue_stage(cs, tmem_d, ksteps, kb == 0);
          }
          advance();
        }
        if (leader && elect_one()) {
          if (tl.kblocks > 0) {
            umma_commit_pair_both(acc_full_bar(as));
          } else {
            mbar_arrive(acc_full_bar(as));  // empty group: both epilogues write zeros
            mbar_arrive_cluster(map_to_cta(acc_full_bar(as), peer));
          }
        }
      }
      __syncwarp();
    }
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
    // The next tile is decoded one iteration ahead, so its plan-table load is in flight while this tile runs.
    Tile nxt = {};
    if (first_tile < num_tiles) nxt = decode_pair_tile(p, first_tile, rank);
    for (int t = first_tile; t < num_tiles && !*abort_flag; t += tile_step, ++tcount) {
      const Tile tl = nxt;
      if (t + tile_step < num_tiles) nxt = decode_pair_tile(p, t + tile_step, rank);
      const int as = tcount & 1;
      const uint32_t aph = (tcount >> 1) & 1u;
      bool ok = mbar_wait(acc_full_bar(as), aph, p.mbar_limit, abort_flag);
      if (!ok) {
        report_status(p.status, kStatusMbarTimeout, kKernelGemm, kModeTgmm, t, 1500 + as, 0, 0);
        raise_abort();
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tcgen05_fence_after_sync();
      const uint32_t tacc = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + as * kBlockN;
      tgmm_epilogue(p, tl, tacc, q, lane, stage_gen, &map_c);
      tcgen05_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(leader_acc_empty0 + 8u * as);
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

int g_pair_grid_used = 0;  // last pair grid size, for diagnostics

void launch_weight_grad(const GemmParams& p, const CUtensorMap& map_a, const CUtensorMap& map_b,
                        const CUtensorMap& map_c, int grid, cudaStream_t stream, bool behind) {
  static const int resident = resident_pair_grid(grouped_gemm_pair_kernel, kPairThreads, kPairSmemBytes);
  grid &= ~1;  // whole pairs only
  const int g = grid < resident ? grid : resident;
  g_pair_grid_used = g;
  launch_maybe_behind(behind, grouped_gemm_pair_kernel, g, kPairThreads, kPairSmemBytes, stream, p, map_a, map_b, map_c);
}

}  // namespace cem
