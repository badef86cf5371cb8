// EXL3 GEMM over a list of (expert, row tile) pairs, 3.0 and 4.0 bpw, decoded weights in TENSOR MEMORY (sm_100a).  Contract of the grouped form in
// exl3_gemm.cu: part[split][row][n] = partial sums of xs @ W_q[expert], rows sorted by expert, tile_tab[t] = {expert, first row, rows}; tiles of no
// rows, which the planner puts last, may stand anywhere.  Without a table the tiles are those of a plain GEMM.
//
// Bound by the trellis decode (two integer pipes, see exl3_decode.cuh).  Decode as in exl3_gemm_tm.cu: a thread owns one of the strip's 128 columns
// (one TMEM lane) and emits its k-values as packed fp16 pairs, the MMA reads A from tensor memory and the activations from shared memory.
// What is different is the schedule: the work items of a routed window are many and short (tile x 128-column strip x K split: 4 chunks of
// 128 k), so the CTAs are PERSISTENT and every ring runs on across items - the weights of the next item stream in while this one is decoded -
// and the accumulator is double buffered, its epilogue done by one decode group while the others go on.  One CTA per item in exl3_gemm.cu
// spent most of its life in its prologue and on shared-memory traffic of the decoded tile: 16 rows x 8 picks of 128 experts (2048 -> 1536 and
// 768 -> 2048, 3.0 bpw) took 235 us for both products,
// 141 us here; one row 83 and 26 us.  What is left is the decode's own: the integer pipe is 70 % busy.  (Fetching the next item's table entry
// ahead costs registers that the decode groups do not have: 5 % slower.)
//
// Tiles of up to 256 rows (TALL, for prompt slices): both accumulators hold rows of one item, a unit of 128 rows each, so that its weights are decoded once.
// The activations then come in boxes of 64 rows, no more of them than the tile has rows, and a unit is written out by two groups, half each: with one
// group a unit the next item waited for them (4.0 bpw, 128 experts, 16,800 pairs, 2048 -> 1536: 229 us by tiles of 128, 211 with one group a unit, 190 so).  What is left
// of it is the L2's: every strip reads the activations again, 6 TB/s at 65,536 pairs (3.0 bpw, 678 -> 510 us).
//
// Warp roles: 0 weight producer (one bulk copy per k-tile row), 1 TMEM owner + MMA issuer, 2 activation producer, then NG decode groups of 4 warps.
// Group e % NG writes out item e, after its first chunk of a later item: the accumulator of item e is needed again by item e + 2 only, whose
// first MMA waits for it.  No circle of waits: that chunk's A stage was last read by a chunk of item e or before.  Every wait is bounded.
#include <cuda.h>
#include "exl3_decode.cuh"
#include "exl3_gemm.cuh"

namespace rx {

constexpr int GR_KCH = 128, GR_HALF = 64, GR_STRIP = 128, GR_OP_STAGES = 3, GR_RAW_STAGES = 8;
constexpr int GR_A_COLS = GR_KCH / 2;             // TMEM columns of one A stage (two fp16 per column)
constexpr int GR_ROLE_WARPS = 3;
// A decode group waits for "the MMA that last read this stage": sound while no group can run two phases ahead, i.e. with as many stages as groups.
__host__ __device__ constexpr int gr_a_stages(int ng) { return ng; }
__host__ __device__ constexpr int gr_acc_cols(int brows) { return brows < 32 ? 32 : brows; }
constexpr int GR_TALL_ROWS = 256, GR_UNIT_ROWS = 128, GR_TALL_OPS = 5, GR_BOX_ROWS = 64;
__host__ __device__ inline int gr_smem_bytes(int brows, int twice) {
  return (brows > GR_UNIT_ROWS ? GR_TALL_OPS * GR_UNIT_ROWS : GR_OP_STAGES * brows) * 256 + GR_RAW_STAGES * 1024 * twice + 512;
}

// One k-tile (16 k) of a thread's column: 8 packed pairs, regs[m] = k (2m, 2m + 1), regs[4 + m] = k (8 + 2m, 9 + 2m).
// w[0] = the word before the thread's eighth of the tile, w[1..] = the eighth's words (see exl3_decode.cuh); b2: which of its two columns.
// shift: where the column's first window starts in its word pair (column_shift).
template <int TWICE>
__device__ __forceinline__ uint32_t column_shift(int b2) { return TWICE == 8 ? (b2 ? 32u : 16u) : (b2 ? 31u : 19u); }
template <int TWICE, int CB, bool ALIGN>
__device__ __forceinline__ void decode_column(const uint32_t (&w)[TWICE / 2 + 1], uint32_t shift, uint32_t* regs) {
  uint32_t y[4] = {};
  if constexpr (TWICE == 6 && ALIGN) {
#pragma unroll
    for (int i = 0; i < 3; ++i) y[i] = __funnelshift_l(w[i + 1], w[i], shift);
    y[3] = w[3] << shift;
  }
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    uint32_t s0, s1, s2, s3;
    if constexpr (TWICE == 8) {
      // b2 = 0: the 4 values that straddle the word boundary; b2 = 1: the word's own 4
      const uint32_t X = __funnelshift_lc(w[m + 1], w[m], shift);
      extract4<CB != CB_MUL1>(X, s0, s1, s2, s3);
    } else {
      // windows start at bit 19 + 24 m + 12 b2 + 3 i of w: 25 bits from the first one's start hold all four.  The word they start in does not
      // depend on b2 but for m = 3, and the funnel shift takes its amount modulo 32.
      static_assert(TWICE == 6, "widths of this kernel: 3.0 and 4.0 bpw");
      uint32_t X;
      if constexpr (ALIGN) {
        // the words once brought to the first window's start: no shift by a register behind it (2 % of a decode window; prompt tiles lose 1 %)
        X = m == 0 ? y[0] : m == 3 ? __funnelshift_l(y[3], y[2], 8) : __funnelshift_l(y[m], y[m - 1], m == 1 ? 24 : 16);
        s0 = __byte_perm(X, 0, 0x4432);
        s1 = __byte_perm(X << 3, 0, 0x4432);
      } else {
        if (m < 3) X = __funnelshift_l(w[m + 1], w[m], shift + 24 * m);
        else X = shift == 31u ? w[3] << 7 : __funnelshift_l(w[3], w[2], 27);
        s0 = X >> 16;
        s1 = (X >> 13) & 0xFFFFu;
      }
      const uint32_t x2 = X >> 10, x3 = X >> 7;
      s2 = CB != CB_MUL1 ? low16_mul(x2) : x2 & 0xFFFFu;        // (the multiply pipe has room for two of the masks)
      s3 = CB != CB_MUL1 ? low16_mul(x3) : x3 & 0xFFFFu;
    }
    regs[m] = pair_to_half2<CB>(s0, s1);
    regs[4 + m] = pair_to_half2<CB>(s2, s3);
  }
}

// HALVES: the last chunk of a split may be half a chunk (its checks cost the MMA issuer and the producers 1 % of a window of 80 rows).
template <int TWICE, int CB, int NG, bool HALVES, bool TALL>
__global__ void __launch_bounds__(GR_ROLE_WARPS * 32 + NG * 128, (NG <= 3 ? 2 : 1))
exl3_gemm_grouped_kernel(const __grid_constant__ CUtensorMap tmap_x, const uint32_t* __restrict__ trellis, size_t expert_words,
                         float* __restrict__ part, int rows, int K, int N, int splits, int cut, int brows, const int* tile_tab, int max_tiles,
                         int* status) {
  pdl_launch();
  constexpr int SA = gr_a_stages(NG), EW = TWICE / 2;            // EW: words of an eighth of a tile
  constexpr int OPS = TALL ? GR_TALL_OPS : GR_OP_STAGES;
  const int urows = TALL ? GR_UNIT_ROWS : brows;                 // rows of a unit: one accumulator, one B stage
  // Quarters of a chunk unrolled: short items keep to the instruction cache, long ones gain 5 % (86 experts 2048 -> 1536 in 4 splits 96.7 us with one, 93.2 with
  // two or four; 79 experts 768 -> 2048 in 3 splits 52.0, 52.0, 54.8).
  constexpr int QT = NG <= 3 ? 2 : 4;
  constexpr int TILE_WORDS = 4 * TWICE, ROW_BYTES = 8 * TILE_WORDS * 4, RAW_STAGE = 8 * ROW_BYTES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int b_half = urows * 128, b_stage = 2 * b_half;          // one [urows x 64] swizzled sub-tile
  uint8_t* b_base = smem;
  uint8_t* raw_base = smem + OPS * b_stage;
  uint64_t* a_full = (uint64_t*)(raw_base + GR_RAW_STAGES * RAW_STAGE);   // [SA] 4 decode warps
  uint64_t* a_empty = a_full + SA;                   // [SA] tcgen05.commit
  uint64_t* b_full = a_empty + SA;                   // [OP] activation producer expect_tx
  uint64_t* b_empty = b_full + OPS;         // [OP] tcgen05.commit
  uint64_t* raw_full = b_empty + OPS;       // [RAW] weight producer expect_tx
  uint64_t* raw_empty = raw_full + GR_RAW_STAGES;    // [RAW] 4 decode warps
  // A parity wait tells a phase from the next one only.  A group may ask for item e before item e - 2 is complete, but its own last write-out was
  // item e - NG, so e - 4 is: four barriers in turn for two accumulators.
  uint64_t* acc_full = raw_empty + GR_RAW_STAGES;    // [4] tcgen05.commit
  uint64_t* acc_empty = acc_full + 4;                // [2] 4 decode warps
  uint64_t* drained = acc_empty + 2;                 // every MMA of this CTA has completed
  uint32_t* tmem_slot = (uint32_t*)(drained + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  volatile int* last_flag = abort_flag + 1;          // of the wait before the tensor memory is freed, which an abort does not cut short

  volatile int* tile_end = last_flag + 1;             // the last live tile + 1, -1: not known yet
  volatile int* n_sent = tile_end + 1;                // [2] chunks that the producers have issued: weights, activations
  int* split_c0 = (int*)(n_sent + 2);                 // [splits + 1] where each split begins, in halves of a chunk
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int strips = N / GR_STRIP, per_tile = strips * splits, nt_total = N / 16;
  const int acc_cols = gr_acc_cols(urows);
  uint32_t ncols = 32;
  while ((int)ncols < 2 * acc_cols + SA * GR_A_COLS) ncols <<= 1;
  if (threadIdx.x == 0) {
    for (int i = 0; i < SA; ++i) { mbar_init(&a_full[i], 4); mbar_init(&a_empty[i], 1); }
    for (int i = 0; i < OPS; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
    for (int i = 0; i < GR_RAW_STAGES; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 4); }
    for (int i = 0; i < 4; ++i) mbar_init(&acc_full[i], 1);
    for (int i = 0; i < 2; ++i) mbar_init(&acc_empty[i], TALL ? 8 : 4);
    mbar_init(drained, 1);
    *abort_flag = *last_flag = 0;
    *tile_end = -1;
    fence_barrier_init();
    prefetch_tmap(&tmap_x);
  }
  // splits are cut at multiples of `cut` k (64 or 128), where the other kernels of the same form cut them
  if (warp == 2 && lane <= splits) split_c0[lane] = (int)((unsigned)(K / cut * lane) / (unsigned)splits) * (cut / GR_HALF);
  if (warp == 1) {
    tmem_alloc(tmem_slot, ncols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();                                        // the tile table and the rows come from the kernels before
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t a_tmem0 = tmem_base + 2 * acc_cols;

  // Items are taken tile by tile: a tile's splits, a split's strips.  A walker steps from item to item of this CTA by additions with carries.
  struct Walk { int tile, split, strip; };
  auto walk_of = [&](unsigned idx) {
    Walk w;
    w.tile = (int)(idx / (unsigned)per_tile);
    const unsigned rem = idx - (unsigned)w.tile * (unsigned)per_tile;
    w.split = (int)(rem / (unsigned)strips);
    w.strip = (int)(rem - (unsigned)w.split * (unsigned)strips);
    return w;
  };
  auto step = [&](Walk& w, const Walk& d) {
    w.strip += d.strip, w.split += d.split, w.tile += d.tile;
    if (w.strip >= strips) w.strip -= strips, ++w.split;
    if (w.split >= splits) w.split -= splits, ++w.tile;
  };
  struct Item { int expert, row0, nrows; };
  auto tile_of = [&](const Walk& w, Item& it) {        // false past the last item
    if (w.tile >= max_tiles) return false;
    if (tile_tab != nullptr) {
      it.expert = tile_tab[3 * w.tile], it.row0 = tile_tab[3 * w.tile + 1], it.nrows = tile_tab[3 * w.tile + 2];
    } else {
      it.expert = 0, it.row0 = w.tile * brows, it.nrows = min(brows, rows - it.row0);
    }
    if (it.nrows > 0) return true;
    // an idle tile: the end, or, before live ones, an item like the others whose rows are written nowhere
    it.expert = it.row0 = it.nrows = 0;
    int end = -1;
    for (int i = 0; i < (1 << 20) && (end = *tile_end) < 0; ++i) {}
    return w.tile < end;
  };
  auto units_of = [&](const Item& i) { return TALL && i.nrows > GR_UNIT_ROWS ? 2 : 1; };
  Item it;
  Walk at = walk_of(blockIdx.x);
  const Walk stride = walk_of(gridDim.x);

  if (warp == 0) {
    // ---- weight producer: a chunk is 8 k-tile rows of the strip, one copy each
    bool ok = true;
    int gc = 0;
    for (; ok && tile_of(at, it); step(at, stride)) {
      const int c0 = split_c0[at.split], halves = split_c0[at.split + 1] - c0, n = (halves + 1) >> 1;
      const uint32_t* src = trellis + (size_t)it.expert * expert_words + ((size_t)(c0 * 4 + (lane & 7)) * nt_total + (size_t)at.strip * 8) * TILE_WORDS;
      for (int c = 0; c < n && ok; ++c, ++gc) {
        const int s = gc % GR_RAW_STAGES;
        if (lane == 0) {
          if (gc >= GR_RAW_STAGES) ok = mbar_wait(&raw_empty[s], ((gc / GR_RAW_STAGES) - 1) & 1, abort_flag, status, 210, 500);
          if (ok) mbar_arrive_expect_tx(&raw_full[s], HALVES && 2 * c + 2 > halves ? RAW_STAGE / 2 : RAW_STAGE);
        }
        ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        if (ok && lane < (HALVES ? min(8, 4 * (halves - 2 * c)) : 8)) bulk_g2s(raw_base + s * RAW_STAGE + lane * ROW_BYTES, src + (size_t)c * 8 * nt_total * TILE_WORDS, ROW_BYTES, &raw_full[s]);
      }
    }
    if (lane == 0) n_sent[0] = ok ? gc : gc - 1;       // (the chunk whose wait gave up was counted)
  } else if (warp == 2) {
    // ---- activation producer: two [brows x 64] swizzled boxes per chunk
    if (elect_one()) {
      bool ok = true;
      int gc = 0;
      for (; ok && tile_of(at, it); step(at, stride)) {
        const int c0 = split_c0[at.split], halves = split_c0[at.split + 1] - c0, n = (halves + 1) >> 1;
        const int units = units_of(it);
        for (int c = 0; c < n && ok; ++c) {
          const int x = c0 * GR_HALF + c * GR_KCH;
          const bool half = HALVES && 2 * c + 2 > halves;
          for (int u = 0; u < units; ++u, ++gc) {
            const int s = gc % OPS;
            if (gc >= OPS && !mbar_wait(&b_empty[s], ((gc / OPS) - 1) & 1, abort_flag, status, 211, 250)) { ok = false; break; }
            uint8_t* dst = b_base + s * b_stage;
            if constexpr (TALL) {                      // only as many boxes as the unit has rows for: its other columns are neither multiplied nor written
              const int row0 = it.row0 + u * GR_UNIT_ROWS, boxes = min(it.nrows - u * GR_UNIT_ROWS, GR_UNIT_ROWS) > GR_BOX_ROWS ? 2 : 1;
              mbar_arrive_expect_tx(&b_full[s], (uint32_t)(boxes * GR_BOX_ROWS * 128 * (half ? 1 : 2)));
              for (int b = 0; b < boxes; ++b) {
                tma_load_2d(dst + b * GR_BOX_ROWS * 128, &tmap_x, x, row0 + b * GR_BOX_ROWS, &b_full[s]);
                if (!half) tma_load_2d(dst + b_half + b * GR_BOX_ROWS * 128, &tmap_x, x + GR_HALF, row0 + b * GR_BOX_ROWS, &b_full[s]);
              }
            } else {
              mbar_arrive_expect_tx(&b_full[s], (uint32_t)(half ? b_half : b_stage));
              tma_load_2d(dst, &tmap_x, x, it.row0, &b_full[s]);
              if (!half) tma_load_2d(dst + b_half, &tmap_x, x + GR_HALF, it.row0, &b_full[s]);
            }
          }
        }
      }
      n_sent[1] = gc;
    }
  } else if (warp == 1) {
    // ---- MMA issuer: A from tensor memory, B from shared memory; as many rows as the tile has, in sixteens
    {
      int last = -1;
      if (tile_tab != nullptr)
#pragma unroll 4
        for (int t = lane; t < max_tiles; t += 32)
          if (tile_tab[3 * t + 2] > 0) last = t;
      last = __reduce_max_sync(0xffffffffu, last);
      if (lane == 0) *tile_end = last + 1;
    }
    if (elect_one()) {
      const uint64_t desc0 = umma_desc_k_sw128(smem_u32(b_base));
      const uint32_t half_units = (uint32_t)b_half >> 4, stage_units = (uint32_t)b_stage >> 4;
      bool ok = true;
      int gc = 0, gb = 0;
      for (int e = 0, units = 0; ok && tile_of(at, it); e += units, step(at, stride)) {       // e: the item's first unit
        const int halves = split_c0[at.split + 1] - split_c0[at.split], n = (halves + 1) >> 1;
        units = units_of(it);
        for (int u = 0; u < units && ok; ++u)
          if (e + u >= 2) ok = mbar_wait(&acc_empty[(e + u) & 1], (((e + u) >> 1) - 1) & 1, abort_flag, status, 222);
        if (!ok) break;
        tc_fence_after();
        for (int c = 0; c < n && ok; ++c, ++gc) {
          const int sa = gc % SA;
          const uint32_t a_at = a_tmem0 + sa * GR_A_COLS;
          for (int u = 0; u < units; ++u, ++gb) {
            const int s = gb % OPS;
            if (!mbar_wait(&b_full[s], (gb / OPS) & 1, abort_flag, status, 220) ||
                (u == 0 && !mbar_wait(&a_full[sa], (gc / SA) & 1, abort_flag, status, 221, 100))) { ok = false; break; }
            tc_fence_after();
            const int nrows = TALL ? min(it.nrows - u * GR_UNIT_ROWS, GR_UNIT_ROWS) : it.nrows;
            const uint32_t idesc = umma_idesc_f16(GR_STRIP, max(16, (nrows + 15) & ~15), 0, 0);
            const uint32_t acc = tmem_base + ((e + u) & 1) * acc_cols;
            const uint64_t bd = desc0 + (uint64_t)(s * stage_units);
#pragma unroll
            for (int k = 0; k < GR_KCH / 16; ++k)
              if (!HALVES || k < GR_HALF / 16 || 2 * c + 2 <= halves) tc_mma_f16_ts(acc, a_at + k * 8, bd + (uint64_t)((k >> 2) * half_units + (k & 3) * 2), idesc, (c | k) != 0);
            tc_commit(&b_empty[s]);
          }
          if (ok) tc_commit(&a_empty[sa]);
        }
        for (int u = 0; u < units && ok; ++u) tc_commit(&acc_full[(e + u) & 3]);
      }
      tc_commit(drained);
    }
  } else {
    const int dw = warp - GR_ROLE_WARPS, grp = dw >> 2;
    const int q = warp & 3;                       // TMEM lane quarter this warp may touch
    const int n = q * 32 + lane;                  // output column of the strip owned by this thread
    const int nt = n >> 4, g = n & 7;
    const uint32_t shift = column_shift<TWICE>((n >> 3) & 1);
    const int prev_lane = (lane & ~7) | ((lane + 7) & 7);
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    const uint32_t my_words = (uint32_t)(nt * TILE_WORDS + g * EW) * 4u;     // byte offset of this thread's eighth inside a k-tile row
    bool ok = true;
    int next_out = grp;                           // the next unit (TALL: half of one) that this group writes out, and where it stands
    Walk out_at = walk_of(blockIdx.x + (TALL ? 0u : (unsigned)grp * gridDim.x));
    const Walk out_stride = walk_of((unsigned)NG * gridDim.x);
    int out_first = 0;                            // TALL: the first unit of the item at out_at
    auto write_out = [&](int job) {
      const int e = TALL ? job >> 1 : job, from = TALL ? (job & 1) * (GR_UNIT_ROWS / 2) : 0;
      Item o;
      tile_of(out_at, o);
      if constexpr (TALL) {
        for (int u; (u = units_of(o)) <= e - out_first;) {
          out_first += u;
          step(out_at, stride);
          tile_of(out_at, o);
        }
        o.row0 += (e - out_first) * GR_UNIT_ROWS;
        o.nrows = min(GR_UNIT_ROWS, o.nrows - (e - out_first) * GR_UNIT_ROWS);
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[e & 3], (e >> 2) & 1, abort_flag, status, 240))) return false;
      tc_fence_after();
      float* out = part + ((size_t)out_at.split * rows + o.row0) * N + out_at.strip * GR_STRIP + n;
      const int to = TALL ? min(o.nrows, from + GR_UNIT_ROWS / 2) : o.nrows;
      for (int cb = from; cb < to; cb += 16) {
        uint32_t r[16];
        tc_ld_32x32b_x16(tmem_base + (e & 1) * acc_cols + lane_addr + cb, r);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (cb + i < to) out[(size_t)(cb + i) * N] = __uint_as_float(r[i]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[e & 1]);
      if constexpr (!TALL) step(out_at, out_stride);
      return true;
    };
    int gc0 = 0, e = 0;                           // chunks up to the end of this item, units before it
    for (int gc = grp; ok && tile_of(at, it); e += units_of(it), step(at, stride)) {
      gc0 += (split_c0[at.split + 1] - split_c0[at.split] + 1) >> 1;
      for (; gc < gc0 && ok; gc += NG) {
        const int rs = gc % GR_RAW_STAGES, os = gc % SA;
        // (a wait that ran out is the whole warp's: lanes must not part before the next shuffle)
        ok = __all_sync(0xffffffffu, mbar_wait(&raw_full[rs], (gc / GR_RAW_STAGES) & 1, abort_flag, status, 230, 100));
        if (!ok) break;
        const uint32_t raw = smem_u32(raw_base + rs * RAW_STAGE) + my_words;
#pragma unroll QT
        for (int qt = 0; qt < 4; ++qt) {
          // two k-tiles at a time: the thread's eighth of each and, from the lane before it, the word those follow
          uint32_t w[2][EW + 1];
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            const uint32_t src = raw + (uint32_t)((qt * 2 + kk) * ROW_BYTES);
            if constexpr (TWICE == 8) {
              const uint4 v = lds128(src);
              w[kk][1] = v.x, w[kk][2] = v.y, w[kk][3] = v.z, w[kk][4] = v.w;
            } else {
#pragma unroll
              for (int i = 0; i < EW; ++i) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[kk][1 + i]) : "r"(src + 4u * i));
            }
          }
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) w[kk][0] = __shfl_sync(0xffffffffu, w[kk][EW], prev_lane);
          if (qt == 3) release_read_stage(&raw_empty[rs], lane);   // the stage's last read has landed in registers; proxy fence before the refill
          uint32_t regs[16];
          decode_column<TWICE, CB, NG <= 3>(w[0], shift, regs);
          decode_column<TWICE, CB, NG <= 3>(w[1], shift, regs + 8);
          if (qt == 0) {
            if (gc >= SA) ok = __all_sync(0xffffffffu, mbar_wait(&a_empty[os], ((gc / SA) - 1) & 1, abort_flag, status, 231));
            if (!ok) break;
            tc_fence_after();
          }
          tc_st_32x32b_x16(a_tmem0 + lane_addr + os * GR_A_COLS + qt * 16, regs);
        }
        if (!ok) break;
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[os]);
        for (; (TALL ? next_out >> 1 : next_out) < e && ok; next_out += NG) ok = write_out(next_out);
      }
    }
    for (; (TALL ? next_out >> 1 : next_out) < e && ok; next_out += NG) ok = write_out(next_out);
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0 && lane == 0) {                // consumers that gave up have not seen the last copies arrive
    if (warp == 0) ring_landed(raw_full, GR_RAW_STAGES, n_sent[0]);
    if (warp == 2) ring_landed(b_full, OPS, n_sent[1]);
  }
  if (warp == 1) {
    if (lane == 0) mbar_wait(drained, 0, last_flag, status, 241);      // nothing may still write the tensor memory that is freed
    __syncwarp();
    tmem_dealloc(tmem_base, ncols);
  }
}

int make_tmap_f16_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows);

template <int TWICE, int CB, int NG, bool HALVES, bool TALL>
static int launch_grouped(const CUtensorMap& tm, const uint32_t* trellis, size_t expert_words, float* part, int rows, int K, int N, int splits, int cut, int brows,
                          const int* tile_tab, int max_tiles, int* status, cudaStream_t st) {
  int smem = gr_smem_bytes(brows, TWICE) + 1024;
  if (NG <= 3 && smem < 80 * 1024) smem = 80 * 1024;   // at most two CTAs per SM: each allocates 256 TMEM columns
  auto kern = exl3_gemm_grouped_kernel<TWICE, CB, NG, HALVES, TALL>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const long long items = (long long)max_tiles * (N / GR_STRIP) * splits;
  if (items >= (1ll << 30)) return (int)cudaErrorInvalidValue;          // (item numbers are 32-bit)
  const long long slots = (NG <= 3 ? 2 : 1) * 148;
  rx::launch(kern, dim3((unsigned)(items < slots ? items : slots)), dim3(GR_ROLE_WARPS * 32 + NG * 128), smem, st, tm, trellis, expert_words, part, rows, K, N,
             splits, cut, brows, tile_tab, max_tiles, status);
  return (int)cudaGetLastError();
}

// Whether gemm_persistent takes the product: widths with a column decoder, tiles whose two accumulators fit beside the A stages, splits of a chunk
// and more and no more of them than its table of their bounds holds.
bool gemm_persistent_takes(int K, int twice, int splits, int brows) {
  return (twice == 6 || twice == 8) && (brows <= GR_UNIT_ROWS || (brows == GR_TALL_ROWS && splits == 1)) && splits <= K / GR_KCH && splits < 32;
}

int gemm_persistent(const void* xs, int rows, int K, const void* trellis, size_t expert_words, int N, int twice, int codebook, void* part, int splits, int cut,
                    const int* tile_tab, int max_tiles, int brows, int* status, cudaStream_t st) {
  CUtensorMap tm;
  int e = make_tmap_f16_2d(&tm, xs, (uint64_t)rows, (uint64_t)K, (uint32_t)(brows > GR_UNIT_ROWS ? GR_BOX_ROWS : brows));
  if (e != 0) return e;
  const uint32_t* tr = (const uint32_t*)trellis;
  const bool halves = cut == GR_HALF && (K / GR_KCH) % splits != 0;
#define RX_GR_L(T, CBV, NGV, H, TL) launch_grouped<T, CBV, NGV, H, TL>(tm, tr, expert_words, (float*)part, rows, K, N, splits, cut, brows, tile_tab, max_tiles, status, st)
#define RX_GR_H(T, CBV, H) (brows > GR_UNIT_ROWS ? RX_GR_L(T, CBV, 4, false, true) : brows > 32 ? RX_GR_L(T, CBV, 4, H, false) : RX_GR_L(T, CBV, 3, H, false))
#define RX_GR(T, CBV) (halves ? RX_GR_H(T, CBV, true) : RX_GR_H(T, CBV, false))
  switch (codebook) {
    case CB_3INST: return twice == 6 ? RX_GR(6, CB_3INST) : RX_GR(8, CB_3INST);
    case CB_MCG: return twice == 6 ? RX_GR(6, CB_MCG) : RX_GR(8, CB_MCG);
    case CB_MUL1: return twice == 6 ? RX_GR(6, CB_MUL1) : RX_GR(8, CB_MUL1);
    default: return (int)cudaErrorInvalidValue;
  }
#undef RX_GR
#undef RX_GR_H
#undef RX_GR_L
}

}  // namespace rx
