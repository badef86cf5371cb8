// EXL3 4.0 bpw GEMM of decode windows of up to 96 rows (sm_100a): one persistent CTA per SM, each with an equal share of the weights.
//
// Contract, decode and data path of exl3_gemm_tm.cu (weights decoded into tensor memory, part[split][row][n]), another schedule.  There a CTA has one (strip,
// split) and two CTAs share an SM: 272 items on 296 places leave an SM in six half idle, 224 one in two.  Here the strips' chunks of 128 k stand in a row that is cut
// into 148 equal shares.  A share begins and ends inside an item (a strip's split): the first k of an item are the end of a share, the last k the beginning of
// the next one.  A CTA takes its first-k piece first and hands its accumulator on through the item's place in `part`; it takes whole items next and its last-k
// piece, with the accumulator of the CTA before, at the end.  So an accumulator meets its k in the one order that a single CTA would, and the bits are those of
// exl3_gemm_tm.cu.  No circle of waits: a CTA waits for one that was numbered before it and was running when it began, and no piece is both taken and handed on.
// (That would be a share strictly inside an item, which is then two chunks longer at least.  But with no fewer items than CTAs a share has at least as many whole
// chunks as the mean item, and the longest item is at most one more.)
//
// What bounds it: the decode's integer work (18 of the 20 weights a clock that its loop reaches alone) and 9 us that no weight is decoded in: the start, the last
// MMAs, and CTAs that begin late because their SM's last one ended late; and, where shares are hardly longer than items, the accumulators that CTAs wait for.
//
// Up to 32 rows tensor memory holds two accumulators beside the six A stages.  More rows (TALL) have one, which 96 rows still leave room for: what its write-out
// costs is kept short by giving each 16 rows of it to another decode group, and up to six chunks are decoded meanwhile.
//
// Warp roles: 0 weight producer, 1 TMEM owner + MMA issuer, 2 activation producer, then six decode groups of four warps; group g takes every sixth chunk and
// writes out every sixth piece, after its first chunk of a later one.  Every wait is bounded.
#include <cuda.h>
#include "exl3_decode.cuh"
#include "exl3_gemm.cuh"

namespace rx {

constexpr int ST_CTAS = 148, ST_NG = 6, ST_ROLE_WARPS = 3, ST_THREADS = ST_ROLE_WARPS * 32 + ST_NG * 128;
constexpr int ST_KCH = 128, ST_A_COLS = ST_KCH / 2;
// Operand stages, A in tensor memory and B in shared memory.  Two chunks stand behind one pair of barriers: the MMA issuer's waits and commits, instructions that
// have to win their issue slots from 24 busy decode warps, come once in 256 k.
// (TALL has one chunk behind a barrier: its last chunk of a piece must not wait for a chunk of the next one, which may wait for the accumulator.)
constexpr int ST_STAGES = ST_NG;
__host__ __device__ constexpr int st_per(bool tall) { return tall ? 1 : 2; }
__host__ __device__ constexpr int st_raw(bool tall) { return tall ? 8 : 12; }
constexpr int ST_RAW_BYTES = 8 * 8 * 128;
constexpr int ST_ACC = 64;                         // columns of one of two accumulators; TALL: one of up to 96
constexpr int ST_FLAT_ROWS = 32, ST_TALL_ROWS = 96;
constexpr int ST_PIECES = 32;                      // of a share, at most
constexpr int ST_OUT = 8;                          // barriers of finished pieces (a group asks for piece f when piece f - 6 is complete)
static_assert(2 * ST_ACC + ST_STAGES * ST_A_COLS <= 512, "tensor memory");
__host__ __device__ inline int st_smem_bytes(int brows, bool tall) { return ST_STAGES * brows * 256 + st_raw(tall) * ST_RAW_BYTES + 512 + ST_PIECES * 16; }

struct StepArgs {
  float* part;
  // [0]: CTAs begun, modulo ST_CTAS; [32 + 4 share + quarter], TALL [32 + 32 share + 8 quarter + 16-row block]: accumulator handed on.  Zero between calls, those that
  // gave up among them: in every call the CTA that hands on sets a flag once and the one that takes clears it once, as its last act if it has given up.
  int* flags;
  int* status;
  int rows, K, N, splits, brows;
};

// A piece of a share: n chunks from chunk c0 of a strip, inside one split.
struct StepPiece { int strip, split, c0, n; bool hand, take; };

// The pieces of a share in the order in which they are done, one lane each: {strip, split | hand << 16 | take << 17, first chunk, chunks}.  Returns their number.
// (Walked by every role instead, with a division at each step, it cost every call 4 us.)
__device__ __forceinline__ int step_pieces(const StepArgs& a, int share, int lane, int4* table) {
  const unsigned nct = a.K / ST_KCH, splits = a.splits, u = (unsigned)(a.N / 128) * nct;
  const unsigned x0 = u * share / ST_CTAS, x1 = u * (share + 1) / ST_CTAS;
  auto item_of = [&](unsigned x) { const unsigned s = x / nct; return s * splits + ((x - s * nct + 1) * splits - 1) / nct; };
  const unsigned k0 = item_of(x0), k1 = item_of(x1 - 1);
  const int count = (int)(k1 - k0) + 1;
  auto begin = [&](unsigned k) { const unsigned s = k / splits; return s * nct + nct * (k - s * splits) / splits; };
  const bool take = begin(k0) < x0, hand = begin(k1 + 1) > x1;
  // first the piece that is handed on (the last in place), then whole items, then the piece that takes an accumulator (the first in place)
  int at = lane;
  if (count > 1) at = hand && lane == 0 ? count - 1 : take && lane == count - 1 ? 0 : lane - hand + take;
  if (lane < count) {
    const unsigned k = k0 + at, s = k / splits, j = k - s * splits, item = begin(k), b = max(item, x0), e = min(begin(k + 1), x1);
    table[lane] = make_int4((int)s, (int)(j | (hand && k == k1 ? 1u << 16 : 0u) | (b > item ? 1u << 17 : 0u)), (int)(b - s * nct), (int)(e - b));
  }
  return count;
}

// TALL: the block of piece f, of nb, that a group writes out; nb and more: none.  Over the pieces the blocks go round the groups.
__device__ __forceinline__ int step_block(int grp, int f, int nb) { return (int)((unsigned)(grp + ST_NG * ST_PIECES - f * nb) % (unsigned)ST_NG); }

template <int CB, bool TALL>
__global__ void __launch_bounds__(ST_THREADS, 1)
exl3_gemm_step_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ StepArgs a) {
  constexpr int PER = st_per(TALL), LOG = PER - 1, ST_BARS = ST_STAGES / PER, ST_RAW = st_raw(TALL);
  const int nb = a.brows / 16;                                     // TALL: blocks of 16 rows, each written out by another group
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int b_half = a.brows * 128, b_stage = 2 * b_half;          // one [brows x 64] swizzled sub-tile
  uint8_t* b_base = smem;
  uint8_t* raw_base = smem + ST_STAGES * b_stage;
  int4* table = (int4*)(raw_base + ST_RAW * ST_RAW_BYTES);
  uint64_t* full = (uint64_t*)(table + ST_PIECES);                 // [PER stages each] their decode warps and the copies of the activations
  uint64_t* empty = full + ST_BARS;                                // commit
  uint64_t* raw_full = empty + ST_BARS;                            // [RAW] weight producer
  uint64_t* raw_empty = raw_full + ST_RAW;                         // [RAW] four decode warps
  uint64_t* acc_full = raw_empty + ST_RAW;                         // [8] commit
  uint64_t* acc_empty = acc_full + ST_OUT;                         // [2] the decode warps that write out
  uint64_t* acc_taken = acc_empty + 2;                             // the decode warps that take in
  uint64_t* drained = acc_taken + 1;                               // every MMA of this CTA has completed
  uint32_t* tmem_slot = (uint32_t*)(drained + 1);
  volatile int* share_slot = (volatile int*)(tmem_slot + 1);       // [3]: share, pieces, chunks
  volatile int* abort_flag = share_slot + 3;
  volatile int* last_flag = abort_flag + 1;                        // of the wait before the tensor memory is freed, which an abort does not cut short
  volatile int* n_sent = last_flag + 1;                            // [2] chunks that the producers have issued: weights, activations
  volatile int* ended = n_sent + 2;                                // when the kernel before had ended
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < ST_BARS; ++i) { mbar_init(&full[i], 4 * PER + 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < ST_RAW; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 4); }
    for (int i = 0; i < ST_OUT; ++i) mbar_init(&acc_full[i], 1);
    for (int i = 0; i < 2; ++i) mbar_init(&acc_empty[i], TALL ? 4 * nb : 4);
    mbar_init(acc_taken, TALL ? 4 * nb : 4);
    mbar_init(drained, 1);
    *abort_flag = *last_flag = *ended = 0;
    n_sent[0] = n_sent[1] = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_x);
    prefetch_tmap(&tmap_w);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (warp == 2) {
    // CTAs are numbered in the order in which they begin
    const int share = __shfl_sync(0xffffffffu, lane == 0 ? (int)atomicInc((unsigned*)a.flags, ST_CTAS - 1) : 0, 0);
    const int count = step_pieces(a, share, lane, table);
    const unsigned u = (unsigned)(a.N / 128) * (a.K / ST_KCH);
    if (lane == 0) share_slot[0] = share, share_slot[1] = count, share_slot[2] = (int)(u * (share + 1) / ST_CTAS - u * share / ST_CTAS);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // The next kernel may begin: every CTA has its number and its tensor memory (which a CTA of that kernel, waiting for this one, must not have taken).
  pdl_launch();
  // The weights were not written by the kernel before, everything else may have been: the weights stream in and are decoded, up to the depth of the
  // operand ring, while it still runs.
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t a_tmem0 = tmem_base + 2 * ST_ACC;
  const int pieces = share_slot[1], total = share_slot[2];
  constexpr int FLAGS = TALL ? 32 : 4, QFLAGS = FLAGS / 4;         // of a share: a quarter's blocks of 16 rows, or all rows
  auto piece = [&](int f) {
    const int4 v = table[f];
    return StepPiece{v.x, v.y & 0xffff, v.z, v.w, (v.y >> 16 & 1) != 0, (v.y >> 17 & 1) != 0};
  };

  int gc_next = total + ST_NG;                      // decode warps: the first chunk of theirs that they have not announced
  int passed = 0;                                   // decode warps, bits: the kernel before has ended; this warp has handed on; it has taken

  if (warp == 0) {
    // ---- weight producer: ONE 2-D tiled copy per chunk (8 k-tile rows x 1 KB of the strip)
    if (elect_one()) {
      int gc = 0;
      bool ok = true;
      for (int f = 0; ok && f < pieces; ++f) {
        const StepPiece p = piece(f);
        for (int c = 0; c < p.n; ++c, ++gc) {
          const int s = gc % ST_RAW;
          if (gc >= ST_RAW && !(ok = mbar_wait_early(&raw_empty[s], ((gc / ST_RAW) - 1) & 1, abort_flag, ended, a.status, 170, 300))) break;
          mbar_arrive_expect_tx(&raw_full[s], ST_RAW_BYTES);
          tma_load_2d(raw_base + s * ST_RAW_BYTES, &tmap_w, p.strip * 256, (p.c0 + c) * 8, &raw_full[s]);
        }
      }
      n_sent[0] = gc;
    }
  } else if (warp == 2) {
    // ---- activation producer: two [brows x 64] swizzled boxes per chunk
    pdl_wait();
    if (elect_one()) {
      int gc = 0;
      bool ok = true;
      for (int f = 0; ok && f < pieces; ++f) {
        const StepPiece p = piece(f);
        for (int c = 0; c < p.n; ++c, ++gc) {
          const int s = gc % ST_STAGES, x = (p.c0 + c) * ST_KCH;
          uint64_t* bar = &full[s >> LOG];
          if ((gc & (PER - 1)) == 0) {
            if (gc >= ST_STAGES && !(ok = mbar_wait(&empty[s >> LOG], ((gc / ST_STAGES) - 1) & 1, abort_flag, a.status, 171, 100))) break;
            mbar_arrive_expect_tx(bar, (uint32_t)b_stage * (PER == 2 && gc + 1 < total ? 2 : 1));
          }
          tma_load_2d(b_base + s * b_stage, &tmap_x, x, 0, bar);
          tma_load_2d(b_base + s * b_stage + b_half, &tmap_x, x + 64, 0, bar);
          if (gc == 0) *ended = kernel_ended_at();
        }
      }
      n_sent[1] = gc;
    }
  } else if (warp == 1) {
    // ---- MMA issuer: A from tensor memory, B from shared memory
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_f16(128, a.brows, 0, 0);
      const uint64_t desc0 = umma_desc_k_sw128(smem_u32(b_base));
      const uint32_t half_units = (uint32_t)b_half >> 4, stage_units = (uint32_t)b_stage >> 4;
      int ps = 0, parity = 0, f = 0, c = 0;
      bool ok = true;
      StepPiece p = piece(0);
      uint32_t acc = 0, accumulate = 0;
      for (int gc = 0; gc < total; gc += PER) {
        if (!(ok = mbar_wait_early(&full[ps], parity, abort_flag, ended, a.status, 173))) break;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < PER; ++h) {
          if (PER == 2 && h == 1 && gc + 1 >= total) break;
          if (c == 0) {
            if (p.take) ok = mbar_wait(acc_taken, 0, abort_flag, a.status, 174);
            if (TALL && ok && f >= 1) ok = mbar_wait(&acc_empty[0], (f - 1) & 1, abort_flag, a.status, 172);
            if (!TALL && ok && f >= 2) ok = mbar_wait(&acc_empty[f & 1], ((f >> 1) - 1) & 1, abort_flag, a.status, 172);
            if (!ok) break;
            tc_fence_after();
            acc = tmem_base + (TALL ? 0 : (f & 1) * ST_ACC);
            accumulate = p.take;
          }
          const uint64_t bd = desc0 + (uint64_t)((PER * ps + h) * stage_units);
          const uint32_t at = a_tmem0 + (PER * ps + h) * ST_A_COLS;
#pragma unroll
          for (int k = 0; k < ST_KCH / 16; ++k)
            tc_mma_f16_ts(acc, at + k * 8, bd + (uint64_t)((k >> 2) * half_units + (k & 3) * 2), idesc, k == 0 ? accumulate : 1u);
          accumulate = 1;
          if (++c == p.n) {
            tc_commit(&acc_full[f % ST_OUT]);
            c = 0;
            if (++f < pieces) p = piece(f);
          }
        }
        if (!ok) break;
        tc_commit(&empty[ps]);
        if (++ps == ST_BARS) ps = 0, parity ^= 1;
      }
      tc_commit(drained);
    }
  } else {
    const int dw = warp - ST_ROLE_WARPS, grp = dw >> 2;
    const int q = warp & 3;                       // TMEM lane quarter this warp may touch
    const int n = q * 32 + lane;                  // output column of the strip owned by this thread
    const uint32_t sh = (n >> 3) & 1 ? 32u : 16u; // as in exl3_gemm_tm.cu: every other group of four values of eighth g
    const int prev_lane = (lane & ~7) | ((lane + 7) & 7);
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    const uint32_t my_words = (uint32_t)((n >> 4) * 8 + (n & 7)) * 16u;
    const int share = *share_slot;
    int* flag_out = a.flags + 32 + share * FLAGS + q * QFLAGS;
    bool ok = true;
    auto kernel_before = [&]() {                  // `part` and the flags may be in use until it has ended
      if (passed == 0) pdl_wait();
      passed |= 1;
    };
    auto place = [&](const StepPiece& o) { return a.part + ((size_t)o.split * a.rows) * a.N + o.strip * 128 + n; };
    // piece f has had its last MMA: its accumulator (TALL: block b of it) goes to its place
    auto write_out = [&](const StepPiece& o, int f, int b) {
      kernel_before();
      tc_fence_after();
      float* out = place(o);
      for (int cb = 16 * b; cb < (TALL ? 16 * b + 1 : a.rows); cb += 16) {
        uint32_t r[16];
        tc_ld_32x32b_x16(tmem_base + (TALL ? 0 : (f & 1) * ST_ACC) + lane_addr + cb, r);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (cb + i < a.rows) out[(size_t)(cb + i) * a.N] = __uint_as_float(r[i]);
      }
      tc_fence_before();
      if (o.hand) __threadfence();
      __syncwarp();
      if (lane == 0) {
        if (o.hand) atomicExch(flag_out + b, 1);
        mbar_arrive(&acc_empty[TALL ? 0 : f & 1]);
      }
      if (o.hand) passed |= 2;
    };
    // The accumulator of the last piece f, as the CTA before left it.  The group that writes out piece f - 2 (TALL: block b of piece f - 1), whose place it takes,
    // brings it in: a wait of another group could miss two phases of that buffer's barrier.
    auto take_in = [&](const StepPiece& o, int f, int b) {
      kernel_before();
      if (!__all_sync(0xffffffffu, wait_count(flag_out - FLAGS + b, 1, abort_flag, a.status, 178))) return false;
      const float* in = place(o);
      for (int cb = 16 * b; cb < (TALL ? 16 * b + 1 : a.rows); cb += 16) {
        uint32_t r[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = cb + i < a.rows ? __float_as_uint(__ldcg(in + (size_t)(cb + i) * a.N)) : 0u;
        tc_st_32x32b_x16(tmem_base + (TALL ? 0 : (f & 1) * ST_ACC) + lane_addr + cb, r);
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        atomicExch(flag_out - FLAGS + b, 0);
        mbar_arrive(acc_taken);
      }
      passed |= 4;
      return true;
    };
    int next_out = TALL ? 0 : grp, f = 0;         // the next piece that this group writes out (TALL: or looks at); the piece it is in
    // Writes out this group's pieces before piece `end`.  (Left for later when the last MMA is still to come, a group could wait for an operand stage whose MMA
    // waits for that very accumulator.)
    auto write_before = [&](int end) {
      for (; ok && next_out < end; next_out += TALL ? 1 : ST_NG) {
        const int b = TALL ? step_block(grp, next_out, nb) : 0;
        if (TALL && b >= nb) continue;
        ok = __all_sync(0xffffffffu, mbar_wait_early(&acc_full[next_out % ST_OUT], (next_out / ST_OUT) & 1, abort_flag, ended, a.status, 176));
        if (ok) write_out(piece(next_out), next_out, b);
        if (TALL && ok && next_out + 1 < pieces) {
          const StepPiece p = piece(next_out + 1);
          if (p.take) ok = take_in(p, next_out + 1, b);
        }
      }
    };
    int gc = grp, gc0 = 0;                        // chunks up to the end of piece f
    for (; ok && f < pieces; ++f) {
      const StepPiece p = piece(f);
      gc0 += p.n;
      // (not before: the CTA before may still be at it)
      if (TALL) {
        if (p.take && f == 0 && grp < nb) ok = take_in(p, 0, grp);
      } else if (p.take && grp == (f < 2 ? f : (f - 2) % ST_NG)) {
        write_before(f - 1);
        if (ok) ok = take_in(p, f, 0);
      }
      for (; gc < gc0 && ok; gc += ST_NG) {
        const int rs = gc % ST_RAW, os = gc % ST_STAGES;
        ok = __all_sync(0xffffffffu, mbar_wait_early(&raw_full[rs], (gc / ST_RAW) & 1, abort_flag, ended, a.status, 179, 100));
        if (!ok) break;
        const uint32_t raw4 = smem_u32(raw_base + rs * ST_RAW_BYTES) + my_words;
#pragma unroll
        for (int qt = 0; qt < 4; ++qt) {
          // two k-tiles at a time: the thread's eighth of each (4 words) and, from the lane before it, the word those follow
          uint4 cur[2];
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) cur[kk] = lds128(raw4 + (uint32_t)((qt * 2 + kk) * 1024));
          uint32_t prev[2];
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) prev[kk] = __shfl_sync(0xffffffffu, cur[kk].w, prev_lane);
          if (qt == 3) release_read_stage(&raw_empty[rs], lane);   // the stage's last read has landed in registers; proxy fence before the refill
          uint32_t regs[16];
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            const uint32_t w[5] = {prev[kk], cur[kk].x, cur[kk].y, cur[kk].z, cur[kk].w};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              const uint32_t X = __funnelshift_lc(w[m + 1], w[m], sh);
              uint32_t s0, s1, s2, s3;
              extract4<CB != CB_MUL1>(X, s0, s1, s2, s3);
              regs[8 * kk + m] = pair_to_half2<CB>(s0, s1);       // k = 16 kt + 2m, 2m+1
              regs[8 * kk + 4 + m] = pair_to_half2<CB>(s2, s3);   // k = 16 kt + 8 + 2m, +1
            }
          }
          if (qt == 0) {
            if (gc >= ST_STAGES) ok = __all_sync(0xffffffffu, mbar_wait_early(&empty[os >> LOG], ((gc / ST_STAGES) - 1) & 1, abort_flag, ended, a.status, 180));
            if (!ok) break;
            tc_fence_after();
          }
          tc_st_32x32b_x16(a_tmem0 + lane_addr + os * ST_A_COLS + qt * 16, regs);
        }
        if (!ok) break;
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[os >> LOG]);
        write_before(f);
      }
      if (PER == 2 && f == pieces - 1 && gc == total && (total & 1) != 0 && ok) {
        // the last pair has one chunk: the arrivals of the other
        const int os = gc % ST_STAGES;
        if (gc >= ST_STAGES) ok = __all_sync(0xffffffffu, mbar_wait_early(&empty[os >> LOG], ((gc / ST_STAGES) - 1) & 1, abort_flag, ended, a.status, 180));
        if (ok) {
          if (lane == 0) mbar_arrive(&full[os >> LOG]);
          gc += ST_NG;
        }
      }
    }
    gc_next = gc;
    write_before(f);
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0 && lane == 0) {
    // Consumers that gave up have not seen the last copies arrive.  A barrier of operands is complete with the arrivals of its decode warps, too: those that
    // are missing are made up for.
    const int begun = (n_sent[1] + PER - 1) / PER;
    if (warp >= ST_ROLE_WARPS)
      for (; gc_next < begun * PER; gc_next += ST_NG) mbar_arrive(&full[(gc_next % ST_STAGES) >> LOG]);
    if (warp == 0) ring_landed(raw_full, ST_RAW, n_sent[0]);
    if (warp == 2) ring_landed(full, ST_BARS, begun);
  }
  if (*abort_flag != 0 && warp >= ST_ROLE_WARPS && lane == 0) {
    // the next CTA gets its flags all the same, and those of the CTA before, which has begun and whose own waits are bounded, are cleared
    const int grp = (warp - ST_ROLE_WARPS) >> 2;
    int* flag = a.flags + 32 + *share_slot * FLAGS + (warp & 3) * QFLAGS;
    pdl_wait();
    for (int f = 0; f < share_slot[1]; ++f) {
      const StepPiece p = piece(f);
      const int b = TALL ? step_block(grp, f, nb) : 0;
      if (p.hand && (TALL ? b < nb : grp == f % ST_NG) && !(passed & 2)) atomicExch(flag + b, 1);
    }
    for (int f = 0; f < share_slot[1]; ++f) {
      const StepPiece p = piece(f);
      const int b = !TALL ? 0 : f == 0 ? grp : step_block(grp, f - 1, nb);
      if (p.take && (TALL ? b < nb : grp == (f < 2 ? f : (f - 2) % ST_NG)) && !(passed & 4))
        for (int i = 0; i < (1 << 22) && atomicExch(flag - FLAGS + b, 0) == 0; ++i) __nanosleep(100);
    }
  }
  __syncwarp();
  if (warp == 1) {
    if (lane == 0) mbar_wait(drained, 0, last_flag, a.status, 181);      // nothing may still write the tensor memory that is freed
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
}

int make_tmap_f16_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows);
int make_tmap_trellis(CUtensorMap* out, const void* base, uint64_t kt_rows, uint64_t row_words, uint32_t box_words, uint32_t box_rows);

template <int CB, bool TALL>
static int launch_step(const CUtensorMap& tx, const CUtensorMap& tw, const StepArgs& a, cudaStream_t st) {
  auto kern = exl3_gemm_step_kernel<CB, TALL>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  int smem = st_smem_bytes(a.brows, TALL) + 1024;
  if (smem < 120 * 1024) smem = 120 * 1024;        // one CTA per SM: it allocates all 512 TMEM columns
  return (int)rx::launch(kern, dim3(ST_CTAS), dim3(ST_THREADS), smem, st, tx, tw, a);
}

}  // namespace rx

using namespace rx;

RX_API int rx_exl3_tile_rows(int rows);

RX_API int rx_exl3_step_flags() { return 32 + ST_CTAS * 32; }

// At least one item for every CTA, no more pieces than the table holds.
static bool step_fits(int rows, int K, int N, int splits) {
  if (rows < 1 || rows > ST_TALL_ROWS || K % ST_KCH != 0 || N % 128 != 0 || splits < 1 || splits > K / ST_KCH) return false;
  const long long items = (long long)(N / 128) * splits, chunks = (long long)(N / 128) * (K / ST_KCH);
  return items >= ST_CTAS && items / ST_CTAS + 3 <= ST_PIECES && chunks < (1 << 24);
}

// Whether the call below is faster than exl3_gemm_tm.cu: that one takes 0.527 us a chunk on the SMs with two items and 3 us, this one 0.505 us a chunk of an equal
// share and 9.5 us (its start, and the spread of CTAs that wait for one another's accumulators), 11.5 from 17 rows on.  What an accumulator takes from one CTA to the next
// is hidden by the chunks that a share is longer than an item: with fewer than 4 of them, from 5 rows on 8 and from 17 rows on 10, the CTAs wait.  Layers of dense
// models, us by that one and this one, every other product the same: 4608 -> 24,576 (share 47, item 36) one row 93.6 and 85.5, 32 rows 102.2 and 100.9; 4096 ->
// 28,672 (48, 32) 88.1 and 84.9, 100.8 and 100.3; 4096 -> 22,016 (37, 32) 89.4 and 84.5, 113.0 and 118.9; 2560 -> 19,456 (20.5, 20) 60.0 and 66.0, 74.3 and 86.6;
// 5120 -> 34,816 (73.5, 40) 108.7 and 109.6, 124.3 and 124.9; 7168 -> 36,864 (109, 56) 149.9 and 151.9.  From 33 to 64 rows that one still has two CTAs to an SM
// and the gains are below 5 % (5120 -> 34,816 45.1 and 49.4; 4096 -> 28,672 36.3 and 34.8).
// Verify windows of 65 to 96 rows, one CTA per SM either way: the persistent kernel of whole items (exl3_gemm_grouped.cu) takes 0.78 us a chunk of the CTAs with
// most of them and 5 us, this one, with half as many decode warps more, 0.514 us a chunk of an equal share and 11.5 us.  80 rows, us: 5120 -> 34,816 65.0
// and 49.4; 4096 -> 28,672 50.8 and 36.0; 5120 -> 151,936 283 and 221; 17,408 -> 5120 34.0 and 30.5; 5120 -> 8192 in four splits 21.2 and 19.9; 6144 -> 5120 in
// seven 17.1 and 17.7; 5120 -> 5120 14.5 and 16.8.
RX_API int rx_exl3_step_takes(int rows, int K, int N, int splits) {
  if (!step_fits(rows, K, N, splits) || (rows > ST_FLAT_ROWS && rows <= 64)) return 0;
  const int item = (K / ST_KCH + splits - 1) / splits, items = (N / 128) * splits;
  const double share = (N / 128) * (K / ST_KCH) / (double)ST_CTAS;
  if (rows > 64) return (items + ST_CTAS - 1) / ST_CTAS * item * 0.78 + 5.0 > share * 0.514 + 11.5;
  if (items > 2 * ST_CTAS || share - item < (rows <= 4 ? 4 : rows <= 16 ? 8 : 10)) return 0;
  return 2 * item * 0.527 + 3.0 > share * 0.505 + (rows <= 16 ? 9.5 : 11.5);
}

// rx_exl3_gemm_b4 for decode windows; flags: int32 [rx_exl3_step_flags()], zero before the first call; calls that may overlap need one each.
RX_API int rx_exl3_gemm_step(const void* xr, int rows, int K, const void* trellis, int N, int codebook, void* part, int splits, void* flags, int* status,
                             void* stream) {
  if (!step_fits(rows, K, N, splits) || flags == nullptr) return (int)cudaErrorInvalidValue;
  if ((((uintptr_t)xr) & 15) != 0 || (((uintptr_t)trellis) & 15) != 0) return (int)cudaErrorMisalignedAddress;
  StepArgs a = {};
  a.part = (float*)part, a.flags = (int*)flags, a.status = status;
  a.rows = rows, a.K = K, a.N = N, a.splits = splits, a.brows = rows <= ST_FLAT_ROWS ? rx_exl3_tile_rows(rows) : (rows + 15) & ~15;
  CUtensorMap tx, tw;
  int e = make_tmap_f16_2d(&tx, xr, (uint64_t)rows, (uint64_t)K, (uint32_t)a.brows);
  if (e == 0) e = make_tmap_trellis(&tw, trellis, (uint64_t)(K / 16), (uint64_t)(N / 16) * 32, 256, 8);
  if (e != 0) return e;
#define RX_STEP(CBV) (rows <= ST_FLAT_ROWS ? launch_step<CBV, false>(tx, tw, a, (cudaStream_t)stream) : launch_step<CBV, true>(tx, tw, a, (cudaStream_t)stream))
  switch (codebook) {
    case CB_3INST: return RX_STEP(CB_3INST);
    case CB_MCG: return RX_STEP(CB_MCG);
    case CB_MUL1: return RX_STEP(CB_MUL1);
    default: return (int)cudaErrorInvalidValue;
  }
#undef RX_STEP
}
