// Row-wise grouped GEMMs (SwiGLU up-projection, down-projection + combine, SwiGLU', dX + combine) on CTA pairs with the
// WEIGHTS' columns on the MMA's M side and the TOKENS on its N side.
//
// A pair of CTAs drives one 256 x N x 16 tcgen05.mma (cta_group::2): M = 256 weight columns (128 per CTA), N = a tile of
// up to 256 rows of ONE expert, in steps of 32. With tokens on the M side a tile is 128 or 256 rows whatever the expert
// has left; here an expert's rows are cut into equal tiles of a multiple of 32 (`plan_tile_begin`), so the padding is 16
// rows per expert on average. Each CTA stages its 128 weight columns and half of the tile's rows: 32 KB per k-block at
// N = 256 (the SM's L2 port carries one request per 128-byte line, see grouped_gemm_pair.cu), less for narrow tiles.
//
//   warp 0       TMA producer of the CTA's operands (every load credits the leader's full barrier)
//   warp 1       leader only: MMA issue; commits to both CTAs' barriers
//   warps 2-9    epilogue of the CTA's 128 columns x N rows. A warp may read 32 of the 128 TMEM lanes, so four warps form
//                a group; the two groups take the tile's 32-row chunks in turn (SwiGLU needs a few thousand cycles of one
//                warp per SM sub-partition for a tile: with 16 k-blocks per tile one group could not keep up).
//
// Measured against the token-major kernels this one replaced (128 x 256 tiles on single CTAs below 768 rows per expert, 256 x
// 256 on pairs above), same box: 496-540 cycles per k-block at D=7168, F=2048 by mode (the tensor pipe's floor for the
// mean width; 515-540 for the pairs, 610-700 for single CTAs), layer forward + backward with 256 rows per expert 7.86 -> 7.33
// ms, Zipf routing in slices of 2048 rows 10.7 -> 9.1 ms, decode of 64 tokens (16 rows per expert) 776 -> 563 us, 2048 rows
// per expert 21.4 -> 20.4 ms (there the 1000 W power cap sets the clock, so fewer padded rows are what counts).
//
// The accumulator is transposed (TMEM lane = weight column, TMEM column = row). `tcgen05.ld.16x256b` hands it out as
// 8 x 8 matrix fragments, and `stmatrix.trans` / `ldmatrix.trans` turn those around in the group's staging buffer, whose
// rows are token rows; global accesses then move whole 128- to 512-byte row pieces. 16-byte pieces of a staging row are
// XOR-ed with the row number (mod 8): fragment and row accesses are both free of bank conflicts.
#pragma once

#include "grouped_gemm.cuh"

#include "../common/pdl.cuh"
#include "../common/umma.cuh"
#include "gemm_common.cuh"

namespace cem {

namespace {

// Stages of the operand ring. SwiGLU' gives one up for two buffers of h for each epilogue warp.
template <int MODE>
constexpr int kRowStagesOf = MODE == kModeDswiglu ? 5 : 6;
constexpr int kRowStageBytesA = kBlockM * kBlockK * 2;  // this CTA's 128 weight columns
constexpr int kRowStageBytesB = (kTileTokens / 2) * kBlockK * 2;  // up to 128 rows
constexpr int kRowStageBytes = kRowStageBytesA + kRowStageBytesB;
constexpr int kRowBand = 4;                             // token tiles swept together over the weight columns, in short launches
constexpr int kRowBandMax = 12;                         // and of one expert in long ones
constexpr int kByExpert = 512;                          // 256 x 64 pieces of an expert's weights (32 KB) from which this pays: 16 MB
constexpr int kRowThreads = 64 + 8 * 32;
constexpr int kGroupStaging = 16384;                    // per epilogue group
constexpr int kRowSmemBytes = kSmemAlignSlack + 6 * kRowStageBytes + 2 * kGroupStaging + kSmemTailBytes;
static_assert(5 * kRowStageBytes + 8 * 8192 <= 6 * kRowStageBytes + 2 * kGroupStaging, "SwiGLU' has no room for its buffers");
static_assert(kRowSmemBytes + 1024 + 1024 + 16 <= 233472, "no room for a second, small CTA on the SM");

struct RowTile {
  int g;      // local expert
  int row0;   // first slice row
  int nrows;  // rows of the tile
  int ncols;  // nrows rounded up to a multiple of 32: the MMA's N
  int n;      // 256-column tile of the weights
};

// Where a GEMM's token rows come from: a matrix in expert order (tensor maps); `p.gather`, by a table of tokens; or the same for at
// most 32 expert ids, which every CTA sorts for itself.
enum RowSource : int { kRowsMapped, kRowsGathered, kRowsFew };

// What a CTA keeps of few ids, in shared memory behind the barriers.
struct FewRows {
  int4 tiles[32];     // as in the plan's tables: one tile per expert that has rows
  int tokens[32];     // by row
  float weights[32];
};

// `RANGED`: the tiles of a range of experts. A variant of its own, with the range's first entry in shared memory: as a register of every
// warp it made the SwiGLU' GEMM spill, and passes without ranges up to 1.4 % slower (620 rows of 107 experts at D=1792, F=512, forward
// 134.1 -> 135.2 us; the expert kernels on 6086 rows of 9 experts at D=256, F=1024 127.7 -> 129.5).
//
// The order of the tiles decides how often weights and rows come from DRAM or from the other die's L2, and under the power cap that is
// time: 32 experts x 2048 rows, D=7168, F=2048, the up-projection runs at 1177 TFLOP/s and, with every load from a few lines in the nearest
// L2, at 1413. So an expert's tiles go over its weight columns together, up to `kRowBandMax` at a time, and its weights are read once; by
// fours, wherever experts end, the bands of one expert find them gone (an expert's are 59 and 29 MB; a die's L2 holds 63, of both dies'
// lines). DRAM reads at 8 experts: up-projection 1289 -> 1075 MB, dX 893 -> 631, down-projection 307 -> 302. Forward + backward of
// 8192 x 8 rows of 32 experts 1.033 and 1.031 times as fast, 4096 x 8 rows (fp8 put) 1.02, Zipf routing of 2999 x 8 rows 1.02, 256 rows
// per expert 1.00 to 1.02. At most 8 or 6 at a time: 1.019 and 1.000. (Cache hints gave nothing, weights as evict-first took 5 %.)
// The way to a tile is two dependent loads longer: in launches of few or cheap tiles 1 us of 50, and what an expert's bands share is still
// in L2 there. So by fours below 16 MB of weights an expert (`kByExpert`: the launcher then takes the variant without ranges) and below
// four tiles a pair.
template <bool RANGED>
__device__ __forceinline__ RowTile decode_row_tile(const GemmParams& p, int t, volatile const int* first_entry, int num_entries,
                                                   const FewRows* few = nullptr) {
  RowTile tl;
  const int first = RANGED ? *first_entry : 0;
  const int4* tiles = reinterpret_cast<const int4*>(p.plan + p.lay.off_tiles + 4 * p.lay.max_tiles * p.slice) + first;
  int ti;
  if (RANGED && p.n_tiles * p.k_blocks >= kByExpert && num_entries * p.n_tiles >= 4 * static_cast<int>(gridDim.x >> 1)) {
    // (every expert's tiles take the places of its entries, times the weight columns)
    const int* start = p.plan + p.lay.off_tile_start + (p.lay.L + 1) * p.slice + tiles[t / p.n_tiles].x;
    const int begin = start[0] - first, count = start[1] - first - begin;
    const int bands = (count + kRowBandMax - 1) / kRowBandMax, most = (count + bands - 1) / bands;
    int rem = t - begin * p.n_tiles;
    const int in_band = rem / (most * p.n_tiles) * most;
    rem -= in_band * p.n_tiles;
    const int width = min(most, count - in_band);
    tl.n = rem / width;
    ti = begin + in_band + (rem - tl.n * width);
  } else {
    const int band_tiles = kRowBand * p.n_tiles;
    const int band = t / band_tiles, rem = t - band * band_tiles;
    int width = num_entries - band * kRowBand;
    width = width > kRowBand ? kRowBand : width;
    tl.n = rem / width;
    ti = band * kRowBand + (rem - tl.n * width);
  }
  const int4 e = few != nullptr ? few->tiles[ti] : tiles[ti];
  tl.g = e.x; tl.row0 = e.y; tl.nrows = e.z; tl.ncols = e.w;
  return tl;
}

template <int MODE>
struct RowTraits {
  static constexpr bool kAMn = (MODE == kModeSwiglu || MODE == kModeDownFwd);  // weights read with K along rows
  static constexpr bool kCombine = (MODE == kModeDownFwd || MODE == kModeDx);
};

template <int MODE, RowSource SRC>
__device__ __forceinline__ void issue_row_kblock(const GemmParams& p, const RowTile& tl, int kb, int rank,
                                                 const CUtensorMap* map_a, const CUtensorMap* map_b, uint32_t sa,
                                                 uint32_t bar) {
  if constexpr (RowTraits<MODE>::kAMn) {
    const int y = tl.g * p.b_group_rows + kb * kBlockK;
    if (MODE == kModeSwiglu && p.stripe == 128) {
      // Stripes of 128: this CTA's 64 gate columns and the 64 up columns that belong to them are 128 columns apart.
      tma_load_3d_pair(sa, map_a, bar, y, tl.n * 4 + rank);
      tma_load_3d_pair(sa + kRowStageBytesA / 2, map_a, bar, y, tl.n * 4 + 2 + rank);
    } else {
      tma_load_3d_pair(sa, map_a, bar, y, tl.n * 4 + 2 * rank);  // two 64-column chunks
    }
  } else {
    tma_load_2d_pair(sa, map_a, bar, kb * kBlockK, tl.g * p.b_group_rows + tl.n * kBlockN + rank * kBlockM);
  }
  if constexpr (SRC == kRowsMapped) tma_load_2d_pair(sa + kRowStageBytesA, map_b, bar, kb * kBlockK, tl.row0 + rank * (tl.ncols >> 1));
}

// ---------------------------------------------------------------------------------------------
// Gathered token rows (calls of few tokens on a rank on its own, `FusedRank::runs_brief`): no put, two more warps in each CTA bring the
// CTA's half of a tile's rows, 128 bytes a k-block, straight from x into the stage, in the layout that the tensor map's swizzle would
// give. A thread owns one 16-byte piece of up to sixteen rows (8 i + 4 * warp + lane / 8) and keeps their offsets for the tile.
// The copies count themselves off on the stage's `gathered` barrier (`cp.async.mbarrier.arrive`), nobody waits for them. What lands
// through the generic proxy is fenced for the tensor cores by who waits for it: the leader's MMA warp for its own CTA, the peer's
// warp 1, which passes the arrival on, for the peer.
//
// Bound by the warps' issue, some 300 cycles of barriers a stage and 33 a copy instruction: no more than a k-block takes up to 96 rows a
// tile, 850 cycles at 256. (So not for larger calls: with this instead of a put, and six warps, forward + backward of 2048 x 8 rows at
// D=7168 5.64 -> 5.92 ms; a copy through the load/store unit also costs more power than TMA's.)
// ---------------------------------------------------------------------------------------------
constexpr int kGatherWarps = 2;

template <int MODE, bool RANGED, typename RaiseAbort>
__device__ __forceinline__ void gather_rows(const GemmParams& p, int warp, int lane, int rank, uint32_t smem_base, uint32_t empty0,
                                            uint32_t gathered0, int first_tile, int tile_step, int num_tiles,
                                            volatile const int* first_entry, int num_entries, const FewRows* few,
                                            volatile int* abort_flag, RaiseAbort&& raise_abort) {
  constexpr int kRows = kTileTokens / 16;
  const int piece = lane & 7, row = 4 * warp + (lane >> 3);  // (row < 8)
  const uint32_t dst0 = smem_base + kRowStageBytesA + row * 128 + ((piece ^ row) << 4);
  const uint32_t pitch = static_cast<uint32_t>(p.k_blocks) * (kBlockK * 2);
  uint32_t ps = 0, pph = 0;
  bool dead = false;
  for (int t = first_tile; t < num_tiles && !dead && !*abort_flag; t += tile_step) {
    const RowTile tl = decode_row_tile<RANGED>(p, t, first_entry, num_entries, few);
    const int half = tl.ncols >> 1;
    uint32_t at[kRows];  // bytes from p.gather; ~0: past the tile
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int r = rank * half + 8 * i + row;
      at[i] = ~0u;
      if (8 * i < half && r < tl.nrows)
        at[i] = static_cast<uint32_t>(few != nullptr ? few->tokens[tl.row0 + r] : p.tokens[tl.row0 + r]) * pitch + piece * 16;
    }
    const uint8_t* src = reinterpret_cast<const uint8_t*>(p.gather);
    for (int kb = 0; kb < p.k_blocks; ++kb, src += kBlockK * 2) {
      if (!__all_sync(0xffffffffu, mbar_wait(empty0 + 8u * ps, pph ^ 1u, p.mbar_limit, abort_flag))) {
        if (lane == 0) {
          report_status(p.status, kStatusMbarTimeout, kKernelGemm, MODE, t, 1600 + ps, 0, 0);
          raise_abort();
        }
        dead = true;
        break;
      }
      const uint32_t dst = dst0 + ps * kRowStageBytes;
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        if (8 * i >= half) break;
        if (at[i] != ~0u) cp_async_16(dst + i * 1024, src + at[i]);
      }
      cp_async_arrive(gathered0 + 8u * ps);
      if (++ps == static_cast<uint32_t>(kRowStagesOf<MODE>)) { ps = 0; pph ^= 1u; }
    }
  }
  cp_async_wait_all();  // no exit while a copy may still land
}

// Few ids: one warp, a lane an id, sorts them stably by expert. Ids outside the experts have no row. Returns the number of tiles.
__device__ __forceinline__ int sort_few(const GemmParams& p, int lane, int* expert, int* row, int* first_row, int* count) {
  const int e = lane < p.num_ids ? p.ids[lane] : -1;
  const bool good = e >= 0 && e < p.lay.L;
  const unsigned peers = __match_any_sync(0xffffffffu, good ? e : -1);
  const bool first = good && __ffs(peers) - 1 == lane;
  const int key = good ? e : 0x7fffffff;
  int before = 0, tiles_before = 0;
#pragma unroll
  for (int l = 0; l < 32; ++l) {
    const int other = __shfl_sync(0xffffffffu, first ? key | static_cast<int>(0x80000000u) : key, l);
    if ((other & 0x7fffffff) < key) {
      ++before;
      tiles_before += other < 0 ? 1 : 0;
    }
  }
  *expert = good ? e : -1;
  *first_row = before;
  *row = before + __popc(peers & ((1u << lane) - 1u));
  *count = first ? __popc(peers) : 0;
  // (lanes of one expert agree on tiles_before; it is the first one's that counts)
  *count |= tiles_before << 8;
  return __popc(__ballot_sync(0xffffffffu, first));
}

// The same for everybody behind this kernel: the tables that the down-projection and the sum read, header and status for the host.
__device__ __forceinline__ void publish_few(const GemmParams& p, const FewPlan& out, int lane) {
  int e, row, first_row, count;
  const int tiles = sort_few(p, lane, &e, &row, &first_row, &count);
  const int rows = __popc(__ballot_sync(0xffffffffu, e >= 0));
  if (lane < p.num_ids && e < 0)
    report_status(p.status, kStatusBadIndex, kKernelPlan, 1, 0, lane, static_cast<uint32_t>(p.lay.L), static_cast<uint32_t>(p.ids[lane]));
  if (e >= 0) {
    out.order[row] = lane;
    out.inv_order[lane] = row;
    const int n = count & 0xff;
    if (n > 0) {
      reinterpret_cast<int4*>(out.plan + p.lay.off_tiles)[count >> 8] = make_int4(e, first_row, n, kTileUnit);
      out.plan[p.lay.off_tile_start + e] = count >> 8;
      out.plan[p.lay.off_tile_start + e + 1] = (count >> 8) + 1;  // (what the next expert writes, if it has a tile)
      out.plan[p.lay.off_in_start + e] = first_row;
      out.plan[p.lay.off_in_size + e] = n;
      out.plan[p.lay.off_src_send_start + e] = first_row;
    }
  }
  if (lane == 0) {
    out.plan[p.lay.off_num_tiles] = tiles;
    out.plan[p.lay.off_tile_start + p.lay.L] = tiles;
  }
  // header: slices, rows of the stream (mine, the fullest), rows for other ranks, too many slices, token copies
  int word = lane == 0 ? 1 : lane == 1 || lane == 2 || lane == 5 ? rows : 0;
  if (lane < kPlanHeaderInts) out.plan[lane] = word;
  __syncwarp();
  if (lane >= kPlanHeaderInts && lane < kPlanHeaderInts + 8)
    word = p.status != nullptr ? __ldcg(reinterpret_cast<const int*>(p.status) + lane - kPlanHeaderInts) : 0;
  if (lane < kPlanHeaderInts + 8) out.host_out[lane] = word;
  __syncwarp();
  if (lane == 0) {
    __threadfence_system();
    st_release_sys(reinterpret_cast<uint32_t*>(out.host_out) + kPlanHeaderInts + 8, out.host_seq);
  }
}

// ---------------------------------------------------------------------------------------------
// Epilogues. `tacc`: TMEM address of this warp's 32 lanes, accumulator buffer included. A group of four warps (128
// threads, `gt` = thread in the group) works on 32-row chunks h, h + 2, ... of the tile.
// Register index of a chunk fragment: half * 16 + j * 4 + rr * 2 + e holds weight column 16 half + 8 rr + lane / 4 (of the
// warp's 32) and row 8 j + 2 (lane & 3) + e (of the chunk's 32).
// ---------------------------------------------------------------------------------------------
// (Barrier numbers as immediates: with a register operand the compiler reserves all sixteen of the CTA's barriers.)
__device__ __forceinline__ void group_sync(int h) {
  if (h == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
  else asm volatile("bar.sync 2, 128;" ::: "memory");
}

// True if `ok` holds in every thread of the group.
__device__ __forceinline__ bool group_vote(int h, bool ok) {
  uint32_t r;
#define CEM_VOTE(BAR)                                                                                             \
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, " BAR ", 128, p;\n\t"         \
               "selp.u32 %0, 1, 0, q;\n\t}\n"                                                                     \
               : "=r"(r) : "r"(ok ? 1u : 0u) : "memory")
  if (h == 0) CEM_VOTE("1");
  else CEM_VOTE("2");
#undef CEM_VOTE
  return r != 0;
}

__device__ __forceinline__ void load_fragment(uint32_t taddr, uint32_t (&r)[32]) {
  tmem_ld_16x256_x4(taddr, r);
  tmem_ld_16x256_x4(taddr + (16u << 16), r + 16);
  tmem_ld_wait();
}

// Address of 16-byte piece `piece` of staging row `row`, rows of ROWB bytes.
template <int ROWB>
__device__ __forceinline__ uint32_t staged(uint32_t buf, int row, int piece) {
  return buf + row * ROWB + ((piece ^ (row & 7)) << 4);
}

// Copies staging rows (ROWB bytes = consecutive columns at `out + row * ld`) below `nvalid` to global memory.
template <int ROWB>
__device__ __forceinline__ void flush_rows(uint32_t buf, int gt, uint8_t* out, size_t ld_bytes, int nvalid) {
  constexpr int kPieces = ROWB / 16, kRows = 128 / kPieces;  // rows per sweep of the group
  const int piece = gt % kPieces;
#pragma unroll
  for (int i = 0; i < 32 / kRows; ++i) {
    const int row = gt / kPieces + i * kRows;
    const int4 v = ld_shared_v4(staged<ROWB>(buf, row, piece));
    if (row < nvalid) *reinterpret_cast<int4*>(out + row * ld_bytes + piece * 16) = v;
  }
}

struct GroupCtx {
  int h, q, lane, gt, rank;
  uint32_t staging;  // this group's staging buffer (SwiGLU': this warp's)
};

template <typename Release>
__device__ __forceinline__ void swiglu_epilogue(const GemmParams& p, const RowTile& tl, uint32_t tacc,
                                                const GroupCtx& c, const FewRows* few, Release&& release) {
  const int chunks = (tl.nrows + 31) >> 5;
  // Lanes 0-63 of the accumulator are gate columns and 64-127 the up columns that belong to them (stripes of 32: both
  // kinds alternate every 32 lanes), so a gate warp and its partner exchange half of a chunk through shared memory
  // (fp32, thread to thread) and each computes 32 activation columns of 16 rows.
  const bool narrow = p.stripe == 32;
  const bool is_gate = narrow ? !(c.q & 1) : c.q < 2;
  const int partner = narrow ? (c.q ^ 1) : (c.q ^ 2);
  const int act_piece = (narrow ? (c.q >> 1) : (c.q & 1)) * 4;  // first 16-byte piece of the 32 activation columns
  const bool with_h = p.out1 != nullptr;
  const uint32_t hbuf = c.staging, exch = c.staging + 8192;
  const uint32_t abuf = with_h ? exch : hbuf;  // activations go where the exchange was; without h its place is free
  const int act_col = tl.n * 128 + c.rank * 64;
  const int h_col0 = tl.n * kBlockN + c.rank * (p.stripe == 128 ? 64 : 128);
  const int h_col1 = h_col0 + (p.stripe == 128 ? 128 : 64);
  for (int ch = c.h; ch < chunks; ch += 2) {
    const int row0 = tl.row0 + ch * 32, nvalid = tl.nrows - ch * 32;
    // Router weights of this thread's four rows, asked for before anything else: they come from L2 (read past L1: the line
    // may also hold weights of rows that had not arrived when another tile read it).
    float w[4] = {1.0f, 1.0f, 1.0f, 1.0f};
    if (few != nullptr || p.row_w != nullptr) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = (is_gate ? 0 : 16) + 8 * (i >> 1) + 2 * (c.lane & 3) + (i & 1);
        if (t < nvalid) w[i] = few != nullptr ? few->weights[row0 + t] : __ldcg(p.row_w + row0 + t);
      }
    }
    uint32_t r[32];
    load_fragment(tacc + ch * 32, r);
    if (ch + 2 >= chunks) release();
    if (with_h) group_sync(c.h);  // the previous chunk's rows have left the buffers
    const uint32_t mine = exch + c.q * 2048 + c.lane * 16;
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // register quads (half, j) of the rows the partner works on
      const int half = i >> 1, jj = i & 1;
      uint32_t v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = is_gate ? r[half * 16 + (2 + jj) * 4 + k] : r[half * 16 + jj * 4 + k];
      st_shared_v4(mine + i * 512, v[0], v[1], v[2], v[3]);
    }
    if (with_h) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t o[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int b = (s >> 1) * 16 + j * 4 + (s & 1) * 2;
          o[s] = pack_bf16(__uint_as_float(r[b]), __uint_as_float(r[b + 1]));
        }
        stmatrix_x4_trans(staged<256>(hbuf, 8 * j + (c.lane & 7), c.q * 4 + (c.lane >> 3)), o);
      }
    }
    group_sync(c.h);
    uint32_t in[16];
    const uint32_t theirs = exch + partner * 2048 + c.lane * 16;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int4 v = ld_shared_v4(theirs + i * 512);
      in[4 * i] = v.x; in[4 * i + 1] = v.y; in[4 * i + 2] = v.z; in[4 * i + 3] = v.w;
    }
    if (with_h) group_sync(c.h);  // everybody has read the exchange: its place takes the activations
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      const int trow = (is_gate ? 0 : 16) + 8 * jj;
      uint32_t o[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int half = s >> 1, rr = s & 1;
        float a[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t own = is_gate ? r[half * 16 + jj * 4 + rr * 2 + e] : r[half * 16 + (2 + jj) * 4 + rr * 2 + e];
          const uint32_t other = in[(half * 2 + jj) * 4 + rr * 2 + e];
          const float gate = __uint_as_float(is_gate ? own : other), up = __uint_as_float(is_gate ? other : own);
          a[e] = silu_f(gate) * up;
        }
        o[s] = pack_bf16(a[0] * w[2 * jj], a[1] * w[2 * jj + 1]);
      }
      stmatrix_x4_trans(staged<128>(abuf, trow + (c.lane & 7), act_piece + (c.lane >> 3)), o);
    }
    group_sync(c.h);
    flush_rows<128>(abuf, c.gt, reinterpret_cast<uint8_t*>(p.out0 + static_cast<size_t>(row0) * p.ld0 + act_col),
                    static_cast<size_t>(p.ld0) * 2, nvalid);
    if (with_h) {
      // 256-byte staging rows: two 128-byte halves whose places in a row of h depend on the stripe
      const int piece = c.gt & 15;
      __nv_bfloat16* out = p.out1 + static_cast<size_t>(row0) * p.ld1 + (piece < 8 ? h_col0 : h_col1) + (piece & 7) * 8;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = (c.gt >> 4) + i * 8;
        const int4 v = ld_shared_v4(staged<256>(hbuf, row, piece));
        if (row < nvalid) *reinterpret_cast<int4*>(out + static_cast<size_t>(row) * p.ld1) = v;
      }
    }
  }
  if (c.h >= chunks) release();
}

// Down-projection / dX: every row's 128 columns go to the rank the row came from, at its send-order position.
// `dst` (shared memory, one entry per row of this group's chunks): source << 27 | position, or ~0 for rows past the tile.
template <typename Release>
__device__ __forceinline__ void combine_epilogue(const GemmParams& p, const RowTile& tl, uint32_t tacc,
                                                 const GroupCtx& c, const uint32_t* dst, Release&& release) {
  const int chunks = (tl.nrows + 31) >> 5;
  const int col = tl.n * kBlockN + c.rank * kBlockM;
  for (int ch = c.h; ch < chunks; ch += 2) {
    const int list0 = (ch >> 1) * 32;
    uint32_t r[32];
    load_fragment(tacc + ch * 32, r);
    if (ch + 2 >= chunks) release();
    uint32_t o[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int b = (s >> 1) * 16 + j * 4 + (s & 1) * 2;
        o[j][s] = pack_bf16(__uint_as_float(r[b]), __uint_as_float(r[b + 1]));
      }
    }
    const uint32_t buf = c.staging;
    group_sync(c.h);  // the previous chunk's rows have left the buffer
#pragma unroll
    for (int j = 0; j < 4; ++j)
      stmatrix_x4_trans(staged<256>(buf, 8 * j + (c.lane & 7), c.q * 4 + (c.lane >> 3)), o[j]);
    group_sync(c.h);
    const int piece = c.gt & 15;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = (c.gt >> 4) + i * 8;
      const int4 v = ld_shared_v4(staged<256>(buf, row, piece));
      const uint32_t d = dst[list0 + row];
      if (d != ~0u) {
        __nv_bfloat16* base = p.peer_rows != nullptr ? p.peer_rows[d >> 27] : p.out0;
        *reinterpret_cast<int4*>(base + static_cast<size_t>(d & ((1u << 27) - 1)) * p.ld0 + col + piece * 8) = v;
      }
    }
  }
  if (c.h >= chunks) release();
}

// SwiGLU': 128 columns of d_act and the 256 striped columns of h / dh that belong to them. A warp's 32 columns of d_act need 32 gate
// and 32 up columns of h and nothing of what the other warps have, so every warp brings its own two 64-byte pieces of a chunk's
// rows into its own staging, turns gate and up into gradients in place and writes them out as dh: no group barrier anywhere, and two
// elements an instruction (f32x2). With short contractions this epilogue is what bounds the GEMM: 1029 cycles per k-block at D=1024, F=512
// (16 k-blocks a tile), where the group moving whole 512-byte rows through six barriers a chunk, an element at a time, took 1363
// (75,000 instructions a scheduler and launch, now 44,000). Forward + backward, with the launches of one-range backwards: 8192 x 6
// rows there 698 -> 667 us, 1999 x 4 at D=2048 411 -> 393 us, the expert kernels on 4001 rows 250 -> 246.5 us.
//
// d_weight = <acc, act> is summed against the stored w * act and divided by w where the shares are added up
// (`weight_divides`): one rounding of act away from exact. Against the act that h gives, two rounded factors, it is 8 % further
// from 64 bits than a GEMM on the rounded act is (0.00253 against 0.00235 at D=7168, F=2048; this way 0.00167). A chunk of
// w * act passes through the buffer that the next chunk's h goes into.
//
// What a chunk needs is asked for a whole chunk earlier, across tiles: h by asynchronous copies into the one of the warp's two buffers that
// the chunk before is not in, w * act and the router weight into registers. (Asked for half a chunk ahead and the weight when
// needed, a chunk took 5000 cycles, most of them waiting for L2 in turn; now 3700.)
struct DswigluNext {
  int4 act[4];  // row 8 i + lane / 4: a 16-byte piece of the 64 bytes of w * act
  float w;      // router weight of row `lane`
};

// First of the warp's 32 gate columns among the CTA's 256 striped ones; the up columns are `stripe` further.
__device__ __forceinline__ int gate_column(const GemmParams& p, int q) { return 2 * p.stripe * (q * 32 / p.stripe) + q * 32 % p.stripe; }

// A chunk: its first row, how many of its 32 rows there are (none: no chunk) and its column tile.
struct Chunk {
  int row0, rows, n;
};

__device__ __forceinline__ Chunk chunk_of(const RowTile& tl, int ch) { return {tl.row0 + ch * 32, tl.nrows - ch * 32, tl.n}; }

// This lane's 16-byte piece of the warp's columns of h and dh.
__device__ __forceinline__ int dswiglu_column(const GemmParams& p, int n, const GroupCtx& c) {
  return 2 * (n * kBlockN + c.rank * kBlockM) + gate_column(p, c.q) + (c.lane & 4 ? p.stripe : 0) + (c.lane & 3) * 8;
}

// 16-byte piece `piece` of row `row` in the warp's staging: h (128 bytes a row) and w * act (64 bytes, two rows side by side).
__device__ __forceinline__ uint32_t staged_h(uint32_t buf, int row, int piece) { return buf + row * 128 + ((piece ^ (row & 7)) << 4); }
__device__ __forceinline__ uint32_t staged_act(uint32_t buf, int row, int piece) {
  return buf + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4);
}

// Router weight of row `lane` of a chunk (read past L1: the line may also hold weights of rows that had not arrived when another tile
// read it).
__device__ __forceinline__ float dswiglu_weight(const GemmParams& p, const GroupCtx& c, const Chunk& at) {
  return p.row_w != nullptr && c.lane < at.rows ? __ldcg(p.row_w + at.row0 + c.lane) : 1.0f;
}

// This lane's 16-byte piece of the chunk's row lane / 8.
__device__ __forceinline__ size_t dswiglu_offset(const GemmParams& p, const GroupCtx& c, const Chunk& at) {
  return static_cast<size_t>(at.row0 + (c.lane >> 3)) * p.ld0 + dswiglu_column(p, at.n, c);
}

// Asks for a chunk: its h, w * act and weights. Rows past the tile keep what is there: they are worked on and thrown away.
__device__ __forceinline__ void fetch_dswiglu(const GemmParams& p, const GroupCtx& c, const Chunk& at, uint32_t buf, bool weights,
                                              DswigluNext* v) {
  const __nv_bfloat16* h = p.in0 + dswiglu_offset(p, c, at);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if ((c.lane >> 3) + 4 * i < at.rows)
      cp_async_16(staged_h(buf, (c.lane >> 3) + 4 * i, c.lane & 7), h + static_cast<size_t>(4 * i) * p.ld0);
  if (p.dwp != nullptr) {
    const __nv_bfloat16* act =
        p.in1 + static_cast<size_t>(at.row0 + (c.lane >> 2)) * p.ld1 + at.n * kBlockN + c.rank * kBlockM + c.q * 32 + (c.lane & 3) * 8;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if ((c.lane >> 2) + 8 * i < at.rows) v->act[i] = *reinterpret_cast<const int4*>(act + static_cast<size_t>(8 * i) * p.ld1);
  }
  if (weights) v->w = dswiglu_weight(p, c, at);
}

// w * act of the chunk at hand from `v` into the accumulator's fragment layout (m[j][s]: columns 8 s + lane / 4, rows
// 8 j + 2 (lane & 3) + e), by way of a buffer that is free.
__device__ __forceinline__ void turn_act(const GroupCtx& c, uint32_t buf, const DswigluNext& v, uint32_t (&m)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    st_shared_v4(staged_act(buf, (c.lane >> 2) + 8 * i, c.lane & 3), v.act[i].x, v.act[i].y, v.act[i].z, v.act[i].w);
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 4; ++j) ldmatrix_x4_trans(staged_act(buf, 8 * j + (c.lane & 7), c.lane >> 3), m[j]);
  __syncwarp();  // every lane has read it: the next chunk's h goes over it
}

// A chunk's d_weight shares. `r`: the accumulator; `m`: w * act (in fragments); `odd`: rows whose weight is nothing to divide by, their
// sum is <acc, act> with act from h in `buf` (`h_landed` waits for it).
template <typename Landed>
__device__ __forceinline__ void dswiglu_shares(const GemmParams& p, const uint32_t (&r)[32], const GroupCtx& c, const Chunk& at,
                                               uint32_t buf, const uint32_t (&m)[4][4], uint32_t odd, Landed&& h_landed) {
  float part[8];  // <acc, w * act> over this thread's columns, rows 8 j + 2 (lane & 3) + e
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    f32x2 sum = make_f32x2(0.0f, 0.0f);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int b = (s >> 1) * 16 + j * 4 + (s & 1) * 2;
      sum = fma2(make_f32x2(__uint_as_float(r[b]), __uint_as_float(r[b + 1])), bf16x2_to_f32x2(m[j][s]), sum);
    }
    split_f32x2(sum, &part[2 * j], &part[2 * j + 1]);
  }
  if (odd != 0) {  // (rare)
    h_landed();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t g[4], u[4];
      ldmatrix_x4_trans(staged_h(buf, 8 * j + (c.lane & 7), c.lane >> 3), g);
      ldmatrix_x4_trans(staged_h(buf, 8 * j + (c.lane & 7), 4 + (c.lane >> 3)), u);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float sum = 0.0f;
#pragma unroll
        for (int s = 0; s < 4; ++s)
          sum += __uint_as_float(r[(s >> 1) * 16 + j * 4 + (s & 1) * 2 + e]) *
                 (silu_f(e ? bf16_hi(g[s]) : bf16_lo(g[s])) * (e ? bf16_hi(u[s]) : bf16_lo(u[s])));
        if ((odd >> (8 * j + 2 * (c.lane & 3) + e)) & 1u) part[2 * j + e] = sum;
      }
    }
    __syncwarp();
  }
  // Sum over the 8 lanes that hold the same rows, halving the rows a lane keeps at each step: then lane l has row
  // 8 (k / 2) + 2 (l & 3) + k % 2, k = l / 4, of one partial per (row, 32 columns).
#pragma unroll
  for (int step = 0; step < 3; ++step) {
    const int o = 4 << step;
    const bool upper = (c.lane & o) != 0;
#pragma unroll
    for (int k = 0; k < 8; k += 2 << step) {
      const float keep = upper ? part[k + (1 << step)] : part[k], give = upper ? part[k] : part[k + (1 << step)];
      part[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  const int k = c.lane >> 2, t = 8 * (k >> 1) + 2 * (c.lane & 3) + (k & 1);
  if (t < at.rows) p.dwp[static_cast<size_t>(at.row0 + t) * p.dwp_tiles + (at.n * 2 + c.rank) * 4 + c.q] = part[0];
}

// A chunk's dh. `buf`: its h, from here on dh; `wl`: the router weight of row `lane`. (Writing eight rows out and asking for eight of the
// next chunk's while the next eight are worked on is slower: 1107 against 1029 cycles per k-block at D=1024, F=512.)
__device__ __forceinline__ void dswiglu_chunk(const GemmParams& p, const uint32_t (&r)[32], const GroupCtx& c, const Chunk& at,
                                              uint32_t buf, float wl) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t ga = staged_h(buf, 8 * j + (c.lane & 7), c.lane >> 3);
    const uint32_t ua = staged_h(buf, 8 * j + (c.lane & 7), 4 + (c.lane >> 3));
    const f32x2 w = make_f32x2(__shfl_sync(0xffffffffu, wl, 8 * j + 2 * (c.lane & 3)),
                               __shfl_sync(0xffffffffu, wl, 8 * j + 2 * (c.lane & 3) + 1));
    uint32_t g[4], u[4];
    ldmatrix_x4_trans(ga, g);
    ldmatrix_x4_trans(ua, u);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int b = (s >> 1) * 16 + j * 4 + (s & 1) * 2;
      // d_act is rounded to bf16 first, as the unfused reference stores it.
      const f32x2 d = bf16x2_to_f32x2(pack_bf16(mul2(w, make_f32x2(__uint_as_float(r[b]), __uint_as_float(r[b + 1])))));
      const f32x2 gate = bf16x2_to_f32x2(g[s]), up = bf16x2_to_f32x2(u[s]);
      const f32x2 sig = sigmoid_f(gate), sl = mul2(gate, sig);
      const f32x2 rest = fma2(sig, make_f32x2(-1.0f, -1.0f), make_f32x2(1.0f, 1.0f));  // 1 - sig, rounded like the subtraction
      g[s] = pack_bf16(mul2(mul2(d, up), fma2(sl, rest, sig)));
      u[s] = pack_bf16(mul2(d, sl));
    }
    __syncwarp();  // all lanes' ldmatrix reads of these rows are done (they cross lanes) before the rows are overwritten
    stmatrix_x4_trans(ga, g);
    stmatrix_x4_trans(ua, u);
  }
  __syncwarp();
  __nv_bfloat16* out = p.out0 + dswiglu_offset(p, c, at);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int4 o = ld_shared_v4(staged_h(buf, (c.lane >> 3) + 4 * i, c.lane & 7));
    if ((c.lane >> 3) + 4 * i < at.rows) *reinterpret_cast<int4*>(out + static_cast<size_t>(4 * i) * p.ld0) = o;
  }
  __syncwarp();  // the chunk has left the buffer
}

// Zeroes an output's rows past the groups' last one, a row per CTA and turn, by the epilogue warps while the first tile is
// being made. (A fill of the whole output in front of the kernel took 6 us and a launch per output of 4096 x 4096.)
__device__ __forceinline__ void zero_tail(const GemmParams& p, int thread) {
  for (int i = 0; i < 2; ++i) {
    if (p.tail[i] == nullptr) continue;
    const int units = p.tail_cols[i] >> 3;
    for (int row = p.plan[1] + blockIdx.x; row < p.lay.S; row += gridDim.x) {
      int4* at = reinterpret_cast<int4*>(p.tail[i] + static_cast<size_t>(row) * p.tail_cols[i]);
      for (int u = thread; u < units; u += 8 * 32) at[u] = make_int4(0, 0, 0, 0);
    }
  }
}

// The kernels' common body (`maps_b`: null with gathered rows; `plan`: with few ids).
template <int MODE, bool RANGED, RowSource SRC>
__device__ __forceinline__ void row_gemm_body(const GemmParams& p, const CUtensorMap& map_a, const TokenMaps* maps_b,
                                              const FewPlan* plan = nullptr) {
  constexpr bool GATHER = SRC != kRowsMapped;
  using Traits = RowTraits<MODE>;
  constexpr int kRowStages = kRowStagesOf<MODE>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t staging_base = smem_base + kRowStages * kRowStageBytes;
  uint8_t* staging_gen = smem_gen + kRowStages * kRowStageBytes;
  constexpr int kBarriers = 6 * kRowStageBytes + 2 * kGroupStaging;  // offset, behind ring and staging
  const uint32_t bar_base = smem_base + kBarriers;
  // barriers: full[6], empty[6], acc_full[2], acc_empty[2], drain; then tmem slot, abort flag, early flag, first entry;
  // gathered[6] behind them
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kRowStages + s); };
  auto acc_full_bar = [&](int s) { return bar_base + 8u * (2 * kRowStages + s); };
  auto acc_empty_bar = [&](int s) { return bar_base + 8u * (2 * kRowStages + 2 + s); };
  const uint32_t drain_bar = bar_base + 8u * (2 * kRowStages + 4);
  constexpr int kSlotOff = 8 * (2 * kRowStages + 5);
  auto gathered_bar = [&](int s) { return bar_base + kSlotOff + 16u + 8u * s; };
  static_assert(kSlotOff % 8 == 0 && kSlotOff + 16 + 8 * kRowStages <= kSmemTailBytes, "barrier area too small");
  const uint32_t tmem_slot = bar_base + kSlotOff;
  uint8_t* tail_gen = smem_gen + kBarriers;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(tail_gen + kSlotOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail_gen + kSlotOff + 4);
  volatile int* early_flag = reinterpret_cast<volatile int*>(tail_gen + kSlotOff + 8);
  volatile int* first_entry = reinterpret_cast<volatile int*>(tail_gen + kSlotOff + 12);

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
    if (threadIdx.x == 0) report_status(p.status, kStatusBadIndex, kKernelGemm, MODE, -1, 1, kSmemAlignSlack,
                                        smem_base - smem_u32(smem_raw));
    return;
  }
  // (Few ids: the successor writes nothing before this kernel's own predecessor has ended.)
  if constexpr (SRC != kRowsFew) release_successor();
  cluster_sync_all();  // both CTAs run

  if (threadIdx.x == 0) {
    for (int s = 0; s < kRowStages; ++s) {
      mbar_init(full_bar(s), 2);  // leader: one arrival from each CTA's producer (the peer's own barrier is not used)
      mbar_init(empty_bar(s), 1);
      if constexpr (GATHER) mbar_init(gathered_bar(s), 32 * kGatherWarps + (leader ? 1 : 0));  // leader: and the peer's warp 1
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(acc_full_bar(s), 1);
      mbar_init(acc_empty_bar(s), 16);  // eight epilogue warps in each CTA of the pair
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    mbar_init_fence();
    tma_prefetch_desc(&map_a);
    if constexpr (!GATHER) {
      for (int i = 0; i < 8; ++i) tma_prefetch_desc(&maps_b->by_width[i]);
    }
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  // Launched behind its predecessor, the kernel has come this far in that one's tail; global memory from here on.
  wait_predecessor();
  FewRows* few = nullptr;
  if constexpr (SRC == kRowsFew) {
    static_assert(kSlotOff + 16 + 8 * kRowStages <= kSmemTailBytes && kSmemTailBytes % 16 == 0, "no place for the few rows");
    release_successor();
    few = reinterpret_cast<FewRows*>(tail_gen + kSmemTailBytes);
    if (warp == 0) {
      int e, row, first_row, count;
      const int tiles = sort_few(p, lane, &e, &row, &first_row, &count);
      if (e >= 0) {
        few->tokens[row] = lane / p.top_k;
        few->weights[row] = p.w_flat[lane];
        if ((count & 0xff) > 0) few->tiles[count >> 8] = make_int4(e, first_row, count & 0xff, kTileUnit);
      }
      if (lane == 0) *first_entry = tiles;  // (read back behind the barrier below)
    }
  }
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

  const bool gave_up = *early_flag != 0;
  int num_entries = 0;
  if (!gave_up) {
    if constexpr (RANGED) {
      const int* start = p.plan + p.lay.off_tile_start + (p.lay.L + 1) * p.slice;
      const int first = p.first_expert > 0 ? start[p.first_expert] : 0;  // (past the last slice only start[L] is written)
      num_entries = start[p.last_expert] - first;
      *first_entry = first;  // (the same from every thread; each reads back what it has written itself)
    } else if constexpr (SRC == kRowsFew) {
      num_entries = *first_entry;
    } else {
      num_entries = p.plan[p.lay.off_num_tiles + p.slice];
    }
  }
  const int num_tiles = num_entries * p.n_tiles;
  const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;

  if (warp == 0) {
    // ================================ TMA producer (both CTAs) ==============================
    // The whole warp walks the k-blocks in step (every lane waits on the stage's barrier, one elected lane issues the
    // copies), so stage index, phase and addresses stay warp-uniform values.
    uint32_t it = 0, ps = 0, pph = 0;
    int waited_expert = -1;
    long long empty_wait = 0;
    bool dead = false;
    // The next tile is decoded one iteration ahead, so its plan-table load is in flight while this tile runs.
    RowTile nxt = {};
    if (first_tile < num_tiles) nxt = decode_row_tile<RANGED>(p, first_tile, first_entry, num_entries, few);
    for (int t = first_tile; t < num_tiles && !dead && !*abort_flag; t += tile_step) {
      const RowTile tl = nxt;
      if (t + tile_step < num_tiles) nxt = decode_row_tile<RANGED>(p, t + tile_step, first_entry, num_entries, few);
      if constexpr (!GATHER && (MODE == kModeSwiglu || MODE == kModeDswiglu)) {  // whichever reads a slice's dispatched rows first
        if ((p.arrive != nullptr || p.ready != nullptr) && tl.g != waited_expert) {
          if (!wait_expert_rows(p, MODE, tl.g, lane, abort_flag)) {
            if (lane == 0) raise_abort();
            break;
          }
          waited_expert = tl.g;
        }
      }
      const CUtensorMap* map_b = GATHER ? nullptr : &maps_b->by_width[(tl.ncols >> 5) - 1];
      const uint32_t bytes = kRowStageBytesA + (GATHER ? 0u : static_cast<uint32_t>(tl.ncols >> 1) * (kBlockK * 2));
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        const long long w0 = counting ? clock64() : 0;
        const bool ok = __all_sync(0xffffffffu, mbar_wait(empty_bar(ps), pph ^ 1u, p.mbar_limit, abort_flag));
        if (!ok) {
          if (lane == 0) {
            report_status(p.status, kStatusMbarTimeout, kKernelGemm, MODE, t, 1100 + ps, 0, 0);
            raise_abort();
          }
          dead = true;
          break;
        }
        if (counting) empty_wait += clock64() - w0;
        if (elect_one()) {
          const uint32_t fb = map_to_cta(full_bar(ps), 0);
          mbar_expect_tx_cluster(fb, bytes);
          issue_row_kblock<MODE, SRC>(p, tl, kb, rank, &map_a, map_b, smem_base + ps * kRowStageBytes, fb);
        }
        ++it;
        if (++ps == kRowStages) { ps = 0; pph ^= 1u; }
      }
    }
    __syncwarp();
    if (counting && lane == 0) prof_add(kProfEmptyWait, empty_wait);
    // Unwinding: no exit while a copy may still land in this CTA's shared memory (the leader's barriers see every stage
    // of both CTAs; the peer leaves after the leader, at the cluster barrier below).
    if (lane == 0 && *abort_flag && leader) {
      for (int s = 0; s < kRowStages; ++s) {
        if (it > static_cast<uint32_t>(s)) {
          const uint32_t last = it - 1 - ((it - 1 - s) % kRowStages);
          mbar_wait(full_bar(s), (last / kRowStages) & 1u, p.mbar_limit);
        }
      }
    }
  } else if (warp == 1) {
    // ================================ MMA issuer (leader) ===================================
    constexpr uint32_t idesc0 = make_instr_desc_bf16(2 * kBlockM, 0, Traits::kAMn, false);
    constexpr uint32_t kDescStepA = Traits::kAMn ? 2048u : 32u;
    constexpr uint32_t kDescStepB = 32u;
    uint32_t it = 0, tcount = 0, cs = 0, cph = 0;
    long long full_wait = 0, acc_wait = 0;
    const long long loop_c0 = counting ? clock64() : 0;
    const uint64_t loop_n0 = counting ? global_timer_ns() : 0;
    bool dead = false;
    auto fail = [&](int t, int detail) {
      if (lane == 0) {
        report_status(p.status, kStatusMbarTimeout, kKernelGemm, MODE, t, detail, 0, 0);
        raise_abort();
      }
      dead = true;
    };
    RowTile nxt = {};
    if (leader && first_tile < num_tiles) nxt = decode_row_tile<RANGED>(p, first_tile, first_entry, num_entries, few);
    for (int t = first_tile; leader && t < num_tiles && !dead && !*abort_flag; t += tile_step, ++tcount) {
      const RowTile tl = nxt;
      if (t + tile_step < num_tiles) nxt = decode_row_tile<RANGED>(p, t + tile_step, first_entry, num_entries, few);
      const int as = tcount & 1;
      const uint32_t aph = (tcount >> 1) & 1u;
      const uint32_t tmem_d = tmem_base + as * kTileTokens;
      const uint32_t idesc = idesc0 | (static_cast<uint32_t>(tl.ncols >> 3) << 17);
      const long long w0 = counting ? clock64() : 0;
      bool ok = __all_sync(0xffffffffu, mbar_wait(acc_empty_bar(as), aph ^ 1u, p.mbar_limit, abort_flag));
      if (counting) acc_wait += clock64() - w0;
      if (!ok) { fail(t, 1200 + as); break; }
      tcgen05_fence_after_sync();
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        const long long w1 = counting ? clock64() : 0;
        ok = __all_sync(0xffffffffu, mbar_wait(full_bar(cs), cph, p.mbar_limit, abort_flag));
        if constexpr (GATHER) {
          if (ok) ok = __all_sync(0xffffffffu, mbar_wait(gathered_bar(cs), cph, p.mbar_limit, abort_flag));
          fence_proxy_async_smem();
        }
        if (counting) full_wait += clock64() - w1;
        if (!ok) { fail(t, 1300 + cs); break; }
        tcgen05_fence_after_sync();
        const uint32_t sa = smem_base + cs * kRowStageBytes;
        const uint64_t da = Traits::kAMn ? make_smem_desc(sa, 8192, 1024) : make_smem_desc(sa, 16, 1024);
        const uint64_t db = make_smem_desc(sa + kRowStageBytesA, 16, 1024);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < kBlockK / kUmmaK; ++k)
            umma_bf16_pair(tmem_d, da + ((k * kDescStepA) >> 4), db + ((k * kDescStepB) >> 4), idesc,
                           (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit_pair_both(empty_bar(cs));
        }
        ++it;
        if (++cs == kRowStages) { cs = 0; cph ^= 1u; }
      }
      if (dead) break;
      if (elect_one()) umma_commit_pair_both(acc_full_bar(as));
    }
    if constexpr (GATHER) {  // the peer's gathered stages
      for (int t = first_tile; !leader && t < num_tiles && !dead && !*abort_flag; t += tile_step) {
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!__all_sync(0xffffffffu, mbar_wait(gathered_bar(cs), cph, p.mbar_limit, abort_flag))) { fail(t, 1700 + cs); break; }
          fence_proxy_async_smem();
          if (elect_one()) mbar_arrive_cluster(map_to_cta(gathered_bar(cs), 0));
          if (++cs == kRowStages) { cs = 0; cph ^= 1u; }
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
  } else if (GATHER && warp >= kRowThreads / 32) {
    // ================================ gathered rows (both CTAs) =============================
    gather_rows<MODE, RANGED>(p, warp - kRowThreads / 32, lane, rank, smem_base, empty_bar(0), gathered_bar(0), first_tile, tile_step,
                              num_tiles, first_entry, num_entries, few, abort_flag, raise_abort);
  } else {
    // ================================ epilogue (both CTAs) ==================================
    GroupCtx c;
    c.h = (warp - 2) >> 2;
    c.q = warp & 3;  // TMEM lane quarter this warp may read
    c.lane = lane;
    c.gt = c.q * 32 + lane;
    c.rank = rank;
    c.staging = staging_base + c.h * kGroupStaging;
    if constexpr (MODE == kModeDswiglu) c.staging = staging_base + (c.h * 4 + c.q) * 8192;  // two buffers for each warp
    const uint32_t leader_acc_empty0 = map_to_cta(acc_empty_bar(0), 0);
    // Combine modes: the row table sits behind the 8 KB that a chunk is staged in.
    uint32_t* s_dst = reinterpret_cast<uint32_t*>(staging_gen + c.h * kGroupStaging + 8192);
    uint32_t turn = 0, returned = 0;  // turn: accumulator buffer in bit 0, its phase in bit 1
    if (!gave_up) zero_tail(p, (warp - 2) * 32 + lane);
    // (The last CTA is the last to get a tile. Also when an earlier kernel gave up: the host waits for it.)
    if constexpr (SRC == kRowsFew) {
      if (warp == 9 && blockIdx.x == gridDim.x - 1) publish_few(p, *plan, lane);
    }
    // SwiGLU': the next chunk, whether it has been asked for and the buffer it is in.
    DswigluNext ahead = {};
    bool fetched = false;
    uint32_t cur = 0;
    // Where this GEMM is the one that waits for a slice's rows, a tile's weights are there once its accumulator is.
    const bool arrives = p.arrive != nullptr || p.ready != nullptr;
    RowTile nxt = {};
    if (first_tile < num_tiles) nxt = decode_row_tile<RANGED>(p, first_tile, first_entry, num_entries, few);
    for (int t = first_tile; t < num_tiles; t += tile_step, turn = (turn + 1) & 3u) {
      const RowTile tl = nxt;
      if (t + tile_step < num_tiles) nxt = decode_row_tile<RANGED>(p, t + tile_step, first_entry, num_entries, few);
      const int as = turn & 1;
      const uint32_t aph = turn >> 1;
      if constexpr (Traits::kCombine) {
        // Where the rows of this group's chunks go (thread = row), worked out while the accumulator is being made.
        group_sync(c.h);  // the previous tile's table has been used up
        const int row = (c.gt >> 5) * 64 + c.h * 32 + lane;  // entry gt: row of chunk 2 (gt / 32) + h
        int src = -1, pos = 0;
        if (row < tl.nrows) resolve_source(p, tl.g, tl.row0 + row, &src, &pos);
        s_dst[c.gt] = src >= 0 ? (static_cast<uint32_t>(src) << 27) | static_cast<uint32_t>(pos) : ~0u;
        // Lane s keeps the count of row pieces this warp accounts for at source rank s (`flush_returned`).
        for (int s = 0; s < p.lay.P; ++s) {
          const uint32_t cnt = __popc(__ballot_sync(0xffffffffu, src == s));
          if (lane == s) returned += cnt;
        }
      }
      if constexpr (MODE == kModeDswiglu) {
        if (!fetched && c.h * 32 < tl.nrows) fetch_dswiglu(p, c, chunk_of(tl, c.h), c.staging + cur * 4096, !arrives, &ahead);
        fetched = false;
      }
      const long long w0 = counting ? clock64() : 0;
      const bool reached_acc = mbar_wait(acc_full_bar(as), aph, p.mbar_limit, abort_flag);
      if (counting && warp == 2 && lane == 0) prof_add(kProfEpiWait, clock64() - w0);
      if (!reached_acc && lane == 0) {
        report_status(p.status, kStatusMbarTimeout, kKernelGemm, MODE, t, 1500 + as, 0, 0);
        raise_abort();
      }
      // One decision for the whole group: nobody may be left alone at a group barrier. (SwiGLU' has none.)
      if (MODE == kModeDswiglu ? !__all_sync(0xffffffffu, reached_acc) : !group_vote(c.h, reached_acc)) break;
      tcgen05_fence_after_sync();
      const uint32_t tacc = tmem_base + (static_cast<uint32_t>(c.q * 32) << 16) + as * kTileTokens;
      auto release = [&]() {  // this warp has read its last accumulator value
        tcgen05_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(leader_acc_empty0 + 8u * as);
      };
      if constexpr (MODE == kModeSwiglu) swiglu_epilogue(p, tl, tacc, c, few, release);
      else if constexpr (MODE == kModeDswiglu) {
        const int chunks = (tl.nrows + 31) >> 5;
        for (int ch = c.h; ch < chunks; ch += 2) {
          const uint32_t buf = c.staging + cur * 4096, other = c.staging + (cur ^ 1) * 4096;
          const bool last = ch + 2 >= chunks;
          const Chunk at = chunk_of(tl, ch);
          auto h_landed = [&]() { cp_async_wait_all(); __syncwarp(); };
          const float wl = arrives && ch == c.h ? dswiglu_weight(p, c, at) : ahead.w;
          const uint32_t odd = __ballot_sync(0xffffffffu, !weight_divides(wl));
          uint32_t m[4][4], r[32];
          if (p.dwp != nullptr) turn_act(c, other, ahead, m);
          load_fragment(tacc + ch * 32, r);
          if (last) release();
          if (p.dwp != nullptr) dswiglu_shares(p, r, c, at, buf, m, odd, h_landed);
          // (Behind the last use of what the chunk before asked for: a load that shares its scoreboard would be waited for with it.)
          Chunk next = chunk_of(last ? nxt : tl, last ? c.h : ch + 2);
          if (last && t + tile_step >= num_tiles) next.rows = 0;
          fetched = next.rows > 0;
          h_landed();
          if (fetched) fetch_dswiglu(p, c, next, other, !last || !arrives, &ahead);
          dswiglu_chunk(p, r, c, at, buf, wl);
          cur ^= 1;
        }
        if (c.h >= chunks) release();
      }
      else combine_epilogue(p, tl, tacc, c, s_dst, release);
    }
    if constexpr (MODE == kModeDswiglu) cp_async_wait_all();  // (on the way out of an error: no exit while a copy may still land)
    if constexpr (Traits::kCombine) {
      // The group's stores are all issued before any of its warps releases its counts (also on the unwind path).
      group_sync(c.h);
      if (p.peer_count != nullptr && lane < p.lay.P && returned > 0) release_count(p.peer_count[lane], returned, p.lay.P);
    }
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
}  // namespace cem
