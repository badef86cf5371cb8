// EXL3 4.0 bpw GEMM for prompt slices of many rows (sm_100a): every weight is decoded ONCE per call.
//
// The kernels of exl3_gemm_tm.cu decode a weight again for each tile of 256 rows, beside as many cycles of the tensor core.  Here the decode warps of all
// CTAs expand the matrix into a workspace of fp16 tiles, column tile by column tile and ahead of their use, while the tensor cores run an ordinary
// pipelined product over it: pairs of CTAs (cta_group::2), tiles of 256 rows x 256 columns, two accumulators in tensor memory, so that the write-out of
// one tile runs beside the products of the next.  Rows are the M side: a thread of the epilogue holds whole 128-column blocks of one row, and the
// 128-point transforms of a fused epilogue need no shuffle.  The sums meet k in the order of exl3_gemm_tm.cu (16 at a time, ascending, one
// accumulator), so a row's bits do not depend on which of the two kernels it went through.
//
// Nobody waits for a CTA that has not begun: pieces of the expansion are claimed one by one by warps that run, and the workspace holds the whole matrix.
//
// What bounds it: the power limit (1.3 GHz in a long loop) and the operands' way through shared memory (each SM copies 32 KB in and reads 32 KB per 512 tensor
// cycles, all that its 128 bytes a cycle carry: 620 to 650 cycles); beside it the expansion (178 M weights 98 us alone, its stores 3.6 TB/s).  Measured against
// exl3_gemm_tm.cu, four matrices after one another: 5120 -> 34,816 with its SwiGLU, 8192 rows 3.30 -> 2.07 ms (2.31 once the power limit holds the clock), 2048 rows 832 ->
// 649 us; 17,408 -> 5120, 2048 rows 405 -> 325 us; 5120 -> 5120, 1024 rows 66 -> 62 us.  Tried and slower: rows of W [N][K] instead of tiles (a copy of 128 rows then touches 128 DRAM pages; 17,408 ->
// 5120, 1024 rows 233 -> 188 us), f32 rows stored by their threads (150 -> 120 us at 2048 rows of 5120 x 5120), a last wave cut along the columns (narrow
// tiles are bound by their copies).
#include <cuda.h>
#include "exl3_decode.cuh"
#include "exl3_gemm.cuh"

namespace rx {

constexpr int WD_STAGES = 6;                       // stages of 64 k: 128 rows of xr and 128 columns of W per CTA
constexpr int WD_HALF = 128 * 128;                 // bytes of one operand tile [128][64] fp16
constexpr int WD_THREADS = 512;                    // warps 0 and 1: loads, MMA issue; 4-7 and, of the SwiGLU form, 8-11: epilogue; the others: expansion
constexpr int PIECE_KT = 16, WD_PIECE_K = 16 * PIECE_KT;   // k of one piece of the expansion (32 columns each)
constexpr int WD_SEG = 4;                          // pieces along k of a segment: what a tile waits for before it loads the segment's k
constexpr int WD_PAIRS = 74;                       // CTA pairs: one CTA per SM
// the workspace: counters (zero between calls), accumulators that one pair hands to the next, the decoded matrix
enum : int { WC_CLAIMED = 0, WC_FINISHED = 1, WC_SLOTS = 2, WC_HANDED = 16, WC_READY = WC_HANDED + WD_PAIRS * 8, WD_COUNTERS = 4096 };
constexpr long long WD_HAND = 256 * 256;           // floats of a pair's accumulator
constexpr long long WD_FRONT = WD_COUNTERS * 4ll + WD_PAIRS * WD_HAND * 4;
constexpr int WD_OUT = 2 * 32 * 128;               // bytes of an epilogue warp's staging: two boxes of 32 rows x 128 bytes, swizzled
constexpr int WD_SMEM = WD_STAGES * 2 * WD_HALF + 4 * WD_OUT + 256 + 1024;

enum : int { WD_PLAIN = 0, WD_SWIGLU = 1, WD_STORE = 2 };

struct WideArgs {
  const __half* svh;
  const float* bias;
  const __half* suh_next;
  const uint32_t* trellis;
  __half* act;               // SwiGLU: fp16 [rows][N / 2]
  __half* w;                 // workspace: the decoded matrix [N / 128][K / 64][128][64]
  float* hand;               // workspace: [pair][CTA][warp][256][32]
  int* count;                // workspace: [WD_COUNTERS]
  int* status;
  int rows, K, N;
  int row_tiles, col_tiles, band;    // column tiles of 256 (the last may be 128); tiles run through `band` row tiles, then to the next column
  int group;                         // column tiles that are expanded side by side: as many as the CTAs begin with
  int inter, region;                 // tiles that a pair takes one by one (every WD_PAIRS-th); tiles after those, shared out evenly
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void mbar_complete_tx(uint64_t* bar, uint32_t bytes) {      // as a copy of that many bytes does
  asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// mbar_wait for a barrier that threads of the other CTA arrive on
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, int site) {
  if (!mbar_wait(bar, parity, abort_flag, status, site)) return false;
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
  return true;
}
// 2-D tiled copy into this CTA's shared memory that reports to a barrier of the pair's first CTA
__device__ __forceinline__ void tma_load_2d_pair(void* dst_smem, const void* tmap, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst_smem)),
               "l"(tmap), "r"(bar), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tc_mma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair when the MMAs issued so far have completed
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tc_ld_32x32b_x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, "
      "%22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
        "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
        "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
// row `row` of a box of 128-byte rows in shared memory, 16-byte chunk j, in the copy engine's 128-byte swizzle (the box starts on 1024 bytes)
__device__ __forceinline__ void st_box(uint32_t box, int row, int j, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(box + row * 128 + ((j ^ (row & 7)) << 4)), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// 2-D tiled copy out of shared memory; rows past the tensor's end are not written
__device__ __forceinline__ void tma_store_2d(const void* tmap, uint32_t box, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(tmap), "r"(box), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void stg256(void* p, const uint32_t* r) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
               "r"(r[7])
               : "memory");
}
// Half of a 128-point transform that one thread holds: the additions of fwht128_warp but the last, in its order
__device__ __forceinline__ void fwht64_thread(uint32_t (&r)[64]) {
#pragma unroll
  for (int st = 1; st < 64; st <<= 1)
#pragma unroll
    for (int i = 0; i < 64; ++i)
      if (!(i & st)) {
        const float a = __uint_as_float(r[i]), b = __uint_as_float(r[i | st]);
        r[i] = __float_as_uint(a + b);
        r[i | st] = __float_as_uint(a - b);
      }
}
__device__ __forceinline__ void tc_ld_64(uint32_t taddr, uint32_t (&r)[64]) {
  tc_ld_32x32b_x32(taddr, r);
  tc_ld_32x32b_x32(taddr + 32, r + 32);
  tc_wait_ld();
}
__device__ __forceinline__ void tc_st_64(uint32_t taddr, uint32_t (&r)[64]) {
  tc_st_32x32b_x32(taddr, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
  tc_st_32x32b_x32(taddr + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
  tc_wait_st();
}
// v * 1/sqrt(128) * scale + bias for sixteen columns, with the roundings of finish_block
__device__ __forceinline__ void scale16(uint32_t (&v)[16], const float* scale, const float* bias) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float y = __fmul_rn(__fmul_rn(__uint_as_float(v[i]), 0.08838834764831845f), scale[i]);
    if (bias != nullptr) y += __ldg(bias + i);
    v[i] = __float_as_uint(y);
  }
}
// A 128-column block of the thread's row in tensor memory, transformed: `out` takes it sixteen columns at a time, columns c and 64 + c together.  One half is in
// registers at a time; both wait in tensor memory for the last addition (a thread that holds 128 values spills, with 512 threads per CTA).
template <typename Out>
__device__ __forceinline__ void transform_block(uint32_t taddr, Out out) {
#pragma unroll 1
  for (int h = 0; h < 128; h += 64) {
    uint32_t r[64];
    tc_ld_64(taddr + h, r);
    fwht64_thread(r);
    tc_st_64(taddr + h, r);
  }
#pragma unroll 1
  for (int c = 0; c < 64; c += 16) {
    uint32_t lo[16], hi[16];
    tc_ld_32x32b_x16(taddr + c, lo);
    tc_ld_32x32b_x16(taddr + 64 + c, hi);
    tc_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float a = __uint_as_float(lo[i]), b = __uint_as_float(hi[i]);
      lo[i] = __float_as_uint(a + b);
      hi[i] = __float_as_uint(a - b);
    }
    out(c, lo, hi);
  }
}

struct WideTile { int row, col, width, ct; };      // row tile, first column (plain), columns, column tile
__device__ __forceinline__ WideTile wide_tile(const WideArgs& a, int t) {
  const int b = t / (a.band * a.col_tiles), rb = min(a.band, a.row_tiles - b * a.band), u = t - b * a.band * a.col_tiles;
  WideTile w;
  w.row = b * a.band + u % rb;
  w.ct = u / rb;
  w.col = w.ct * 256;
  w.width = min(256, a.N - w.col);                 // the last column tile of an odd number of strips: 128 columns
  return w;
}

// What a pair does, in order.  Whole tiles first, every WD_PAIRS-th.  The last tiles, more than one and less than two for each pair, are cut into equal
// shares of their k: a share ends with the first k of a tile whose last k begin the next pair's share.  The first k come first in time and their
// accumulator is handed on through memory, the last k last: the sums are those of one pass over k, and the pair that waits has long got what it waits for.
struct WideItem { int tile, kb0, kb1; bool hand, take; };
struct WidePlan {
  int slot, inter, base, t0, k0, t1, k1, n;
  // boundary s of the shares, in k blocks of 64: within a tile a multiple of 8 that leaves 8 and more
  __device__ __forceinline__ static int bound(const WideArgs& a, int s, int kb_n) {
    const int x = (int)((long long)a.region * kb_n * s / WD_PAIRS), t = x / kb_n, k = (x - t * kb_n) & ~7;
    return k > 0 && kb_n - k < 8 ? (t + 1) * kb_n : t * kb_n + k;
  }
  __device__ __forceinline__ WidePlan(const WideArgs& a, int s) : slot(s), inter(a.inter), base(a.inter * WD_PAIRS), t0(0), k0(0), t1(0), k1(0) {
    const int kb_n = a.K / 64;
    if (a.region > 0) {
      const int x0 = bound(a, s, kb_n), x1 = bound(a, s + 1, kb_n);
      t0 = x0 / kb_n, k0 = x0 - t0 * kb_n, t1 = x1 / kb_n, k1 = x1 - t1 * kb_n;
    } else if (s >= a.row_tiles * a.col_tiles) {
      inter = 0;                                   // fewer tiles than pairs
    }
    n = inter + t1 - t0 + (k1 > 0);                // the tile that the share begins in is counted once, whole or its last k
  }
  __device__ __forceinline__ WideItem item(const WideArgs& a, int i) const {
    const int kb_n = a.K / 64;
    if (i < inter) return {slot + i * WD_PAIRS, 0, kb_n, false, false};
    i -= inter;
    if (k1 > 0 && i-- == 0) return {base + t1, 0, k1, true, false};
    // whole tiles, then the last k of the first tile
    if (k0 == 0) return {base + t0 + i, 0, kb_n, false, false};
    if (i < t1 - t0 - 1) return {base + t0 + 1 + i, 0, kb_n, false, false};
    return {base + t0, k0, kb_n, false, true};
  }
};

template <int CB, int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(WD_THREADS, 1)
exl3_gemm_wide_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_w64,
                      const __grid_constant__ CUtensorMap tmap_out, const __grid_constant__ WideArgs a) {
  pdl_launch();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + WD_STAGES * 2 * WD_HALF + 4 * WD_OUT);   // [stages] of the first CTA: both CTAs' copies
  uint64_t* empty = full + WD_STAGES;                             // [stages] commit
  uint64_t* acc_full = empty + WD_STAGES;                         // [2] commit
  uint64_t* acc_empty = acc_full + 2;                             // [2] of the first CTA: eight epilogue warps
  uint64_t* acc_taken = acc_empty + 2;                            // of the first CTA: eight epilogue warps have put the handed accumulator in place
  uint64_t* drained = acc_taken + 1;                              // every MMA of the pair has completed
  uint32_t* tmem_slot = (uint32_t*)(drained + 1);
  int* pair_slot = (int*)(tmem_slot + 1);
  volatile int* abort_flag = (volatile int*)(pair_slot + 1);
  int* n_sent = pair_slot + 2;                                    // stages that this CTA's copies were issued for
  int* sent = n_sent + 1;                                         // [stages] their bytes
  constexpr int GROUPS = MODE == WD_SWIGLU ? 2 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int kpieces = (a.K + WD_PIECE_K - 1) / WD_PIECE_K, segs = (kpieces + WD_SEG - 1) / WD_SEG, F = a.N / 2;
  int *claimed = a.count + WC_CLAIMED, *handed = a.count + WC_HANDED, *ready = a.count + WC_READY;

  if (threadIdx.x == 0) {
    for (int i = 0; i < WD_STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
    mbar_init(acc_taken, 8);
    mbar_init(drained, 1);
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_x);
    prefetch_tmap(&tmap_w);
    prefetch_tmap(&tmap_w64);
    prefetch_tmap(&tmap_out);
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  pdl_wait();   // the workspace may still be read by the product before, the rows still written
  const uint32_t tmem = *tmem_slot;
  // pairs are numbered in the order in which they begin: the one before, whose accumulator a pair may wait for, is running
  if (threadIdx.x == 0 && rank == 0) {
    const int slot = atomicAdd(a.count + WC_SLOTS, 1);
    *pair_slot = slot;
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(mapa_u32(smem_u32(pair_slot), 1)), "r"(slot) : "memory");
  }
  cluster_sync();
  const WidePlan plan(a, *pair_slot);

  if (warp == 0) {
    // ---- copies: this CTA's 128 rows of xr and its half of the tile's columns
    if (elect_one()) {
      int it = 0;
      bool ok = true;
      for (int i = 0; i < plan.n && ok; ++i) {
        const WideItem item = plan.item(a, i);
        const WideTile w = wide_tile(a, item.tile);
        const int half = w.width / 2, xrow = w.row * 256 + (int)rank * 128;
        // the decoded matrix: tiles of 128 columns x 64 k, each 16 KB in a row
        const int strip = MODE == WD_SWIGLU ? w.ct + (int)rank * (F / 128) : half == 128 ? 2 * w.ct + (int)rank : 2 * w.ct;
        const int wrow = strip * (a.K / 64) * 128 + (half == 128 ? 0 : (int)rank * 64);
        for (int kb = item.kb0; kb < item.kb1; ++kb, ++it) {
          const int s = it % WD_STAGES;
          if (kb == item.kb0 || kb % (WD_SEG * WD_PIECE_K / 64) == 0) {
            const int seg = kb / (WD_SEG * WD_PIECE_K / 64);
            ok = wait_count(ready + w.ct * segs + seg, 8 * min(WD_SEG, kpieces - seg * WD_SEG), abort_flag, a.status, 160);
            if (!ok) break;
            asm volatile("fence.proxy.async;" ::: "memory");   // written by ordinary stores, read by the copy engine
          }
          if (it >= WD_STAGES) ok = mbar_wait(&empty[s], ((it / WD_STAGES) - 1) & 1, abort_flag, a.status, 161, 20);
          if (!ok) break;
          uint8_t* st = smem + s * 2 * WD_HALF;
          const uint32_t bytes = WD_HALF + (uint32_t)half * 128u;
          sent[s] = (int)bytes;
          if (rank == 0) mbar_arrive_expect_tx(&full[s], 2u * bytes);
          const uint32_t bar = mapa_u32(smem_u32(&full[s]), 0);
          tma_load_2d_pair(st, &tmap_x, kb * 64, xrow, bar);
          tma_load_2d_pair(st + WD_HALF, half == 128 ? &tmap_w : &tmap_w64, 0, wrow + kb * 128, bar);
        }
      }
      *n_sent = it;
    }
  } else if (warp == 1) {
    // ---- MMA issuer of the pair
    if (rank == 0 && elect_one()) {
      int it = 0;
      const uint64_t desc0 = umma_desc_k_sw128(smem_u32(smem));
      bool ok = true;
      for (int n = 0; n < plan.n && ok; ++n) {
        const WideItem item = plan.item(a, n);
        const WideTile w = wide_tile(a, item.tile);
        const int acc = n & 1;
        if (item.take) ok = mbar_wait_cluster(acc_taken, 0, abort_flag, a.status, 166);
        if (ok && n >= 2) ok = mbar_wait_cluster(&acc_empty[acc], ((n >> 1) - 1) & 1, abort_flag, a.status, 162);
        if (!ok) break;
        tc_fence_after();
        const uint32_t idesc = umma_idesc_f16(256, w.width, 0, 0);
        for (int kb = item.kb0; kb < item.kb1; ++kb, ++it) {
          const int s = it % WD_STAGES;
          ok = mbar_wait(&full[s], (it / WD_STAGES) & 1, abort_flag, a.status, 163);
          if (!ok) break;
          tc_fence_after();
          const uint64_t ad = desc0 + (uint64_t)((s * 2 * WD_HALF) >> 4), bd = ad + (WD_HALF >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k) tc_mma_f16_pair(tmem + acc * 256, ad + k * 2, bd + k * 2, idesc, (kb | k) != 0);
          tc_commit_pair(&empty[s]);
        }
        if (ok) tc_commit_pair(&acc_full[acc]);
      }
      // nothing may still write the tensor memory that is freed, after a wait that gave up either
      asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(drained)) : "memory");
      ring_landed(drained, 1, 1);
    }
  } else if (warp >= 4 && warp < 4 + 4 * GROUPS) {
    // ---- epilogue: lane = row of this CTA's 128; with two groups of warps, each takes every other tile
    const int q = warp & 3, group = (warp >> 2) - 1;
    const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
    const uint32_t box0 = smem_u32(smem + WD_STAGES * 2 * WD_HALF + q * WD_OUT);
    float* scales = (float*)(smem + WD_STAGES * 2 * WD_HALF + (group * 4 + q) * 3 * 128 * 4);
    const size_t mine = (rank * 4 + q) * (size_t)(WD_HAND / 8) + lane;
    // the accumulator of item n, before its products: handed on by the pair before
    auto take = [&](int n) {
      const int from = plan.slot - 1;
      if (!__all_sync(0xffffffffu, wait_count(handed + from * 8 + rank * 4 + q, 1, abort_flag, a.status, 165))) return;
      const float* src = a.hand + from * WD_HAND + mine;
      for (int c = 0; c < 256; c += 16) {
        uint32_t r[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__ldcg(src + (c + i) * 32));
        tc_st_32x32b_x16(lane_base + (n & 1) * 256 + c, r);
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(acc_taken), 0));
    };
    const int last = plan.k0 > 0 ? plan.n - 1 : -1;   // the item that takes an accumulator
    if (last == group) take(last);
    for (int n = group; n < plan.n; n += GROUPS) {
      const WideItem item = plan.item(a, n);
      // one group: its buffer is free since item n - 1 was read.  Handed on first: a pair that waits must not keep the next one waiting.
      const bool before = GROUPS == 1 && n + 1 == last;
      if (before && !item.hand) take(last);
      const WideTile w = wide_tile(a, item.tile);
      const int acc = n & 1;
      if (MODE == WD_SWIGLU && !item.hand) {
        // the scales of the tile's gate and up columns and of the next product's input: a load beside its use would cost each of the blocks' chunks a round trip
        __syncwarp();
        for (int i = lane; i < 128; i += 32) {
          const int c = w.ct * 128 + i;
          scales[i] = __half2float(a.svh[c]), scales[128 + i] = __half2float(a.svh[F + c]), scales[256 + i] = __half2float(a.suh_next[c]);
        }
        __syncwarp();
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[acc], (n >> 1) & 1, abort_flag, a.status, 164, 100))) break;
      tc_fence_after();
      const int row0 = w.row * 256 + (int)rank * 128 + q * 32;
      const uint32_t src = lane_base + acc * 256;
      if (item.hand) {
        float* dst = a.hand + plan.slot * WD_HAND + mine;
        for (int c = 0; c < 256; c += 16) {
          uint32_t r[16];
          tc_ld_32x32b_x16(src + c, r);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) __stcg(dst + (c + i) * 32, __uint_as_float(r[i]));
        }
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicExch(handed + plan.slot * 8 + rank * 4 + q, 1);
        if (before) take(last);
      } else if constexpr (MODE == WD_PLAIN) {
        for (int c = 0; c < w.width; c += 32) {
          const uint32_t box = box0 + ((c >> 5) & 1) * (WD_OUT / 2);
          uint32_t r[32];
          tc_ld_32x32b_x32(src + c, r);
          tc_wait_ld();
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");      // the copy before the last has read this box
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j) st_box(box, lane, j, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            if (row0 < a.rows) tma_store_2d(&tmap_out, box, w.col + c, row0);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      } else if constexpr (MODE == WD_STORE) {
        if (row0 < a.rows)
#pragma unroll 1
          for (int b = 0; b < w.width; b += 128) {
            const int c0 = w.col + b;
            const float* bias = a.bias == nullptr ? nullptr : a.bias + c0;
            transform_block(src + b, [&](int c, uint32_t(&lo)[16], uint32_t(&hi)[16]) {
              float scale[2][16];
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const uint4* sv = reinterpret_cast<const uint4*>(a.svh + c0 + 64 * h + c);
                const uint4 v[2] = {__ldg(sv), __ldg(sv + 1)};
                const __half2* x = reinterpret_cast<const __half2*>(v);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  const float2 f = __half22float2(x[i]);
                  scale[h][2 * i] = f.x, scale[h][2 * i + 1] = f.y;
                }
              }
              scale16(lo, scale[0], bias == nullptr ? nullptr : bias + c);
              scale16(hi, scale[1], bias == nullptr ? nullptr : bias + 64 + c);
              if ((c & 16) == 0) {
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // the copies before have read the boxes
                __syncwarp();
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                st_box(box0, lane, (c & 16) / 4 + j, lo[4 * j], lo[4 * j + 1], lo[4 * j + 2], lo[4 * j + 3]);
                st_box(box0 + WD_OUT / 2, lane, (c & 16) / 4 + j, hi[4 * j], hi[4 * j + 1], hi[4 * j + 2], hi[4 * j + 3]);
              }
              if (c & 16) {
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                  tma_store_2d(&tmap_out, box0, c0 + c - 16, row0);
                  tma_store_2d(&tmap_out, box0 + WD_OUT / 2, c0 + 64 + c - 16, row0);
                  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
              }
            });
          }
      } else if (row0 < a.rows) {
        const int c0 = w.ct * 128;
        const bool live = row0 + lane < a.rows;    // the zeros of rows past the end would send the division down its slow path
        const float *bg = a.bias == nullptr ? nullptr : a.bias + c0, *bu = a.bias == nullptr ? nullptr : a.bias + F + c0;
        transform_block(src, [&](int c, uint32_t(&lo)[16], uint32_t(&hi)[16]) {
          scale16(lo, scales + c, bg == nullptr ? nullptr : bg + c);
          tc_st_32x32b_x16(src + c, lo);
          scale16(hi, scales + 64 + c, bg == nullptr ? nullptr : bg + 64 + c);
          tc_st_32x32b_x16(src + 64 + c, hi);
        });
        tc_wait_st();
        const uint32_t up = src + 128;
        auto act = [&](uint32_t(&v)[16], int c) {      // silu(gate) * up as bf16, times the next product's input scale
          scale16(v, scales + 128 + c, bu == nullptr ? nullptr : bu + c);
          uint32_t g[16];
          tc_ld_32x32b_x16(src + c, g);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float gv = live ? __uint_as_float(g[i]) : 1.f;
            const float x = gv / (1.f + __expf(-gv)) * __uint_as_float(v[i]);
            v[i] = __float_as_uint(__bfloat162float(__float2bfloat16_rn(x)) * scales[256 + c + i]);
          }
        };
        transform_block(up, [&](int c, uint32_t(&lo)[16], uint32_t(&hi)[16]) {
          act(lo, c);
          tc_st_32x32b_x16(up + c, lo);
          act(hi, 64 + c);
          tc_st_32x32b_x16(up + 64 + c, hi);
        });
        tc_wait_st();
        __half* out = a.act + (size_t)(row0 + lane) * F + c0;
        transform_block(up, [&](int c, uint32_t(&lo)[16], uint32_t(&hi)[16]) {
          uint32_t h[16];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const __half2 x = __floats2half2_rn(__uint_as_float(lo[2 * j]) * 0.08838834764831845f, __uint_as_float(lo[2 * j + 1]) * 0.08838834764831845f);
            const __half2 y = __floats2half2_rn(__uint_as_float(hi[2 * j]) * 0.08838834764831845f, __uint_as_float(hi[2 * j + 1]) * 0.08838834764831845f);
            h[j] = *reinterpret_cast<const uint32_t*>(&x);
            h[8 + j] = *reinterpret_cast<const uint32_t*>(&y);
          }
          if (live) {
            stg256(out + c, h);
            stg256(out + 64 + c, h + 8);
          }
        });
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[acc]), 0));
      if (GROUPS == 2 && n + 2 == last) take(last);
    }
    if (MODE != WD_SWIGLU && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  } else {
    // ---- expansion: a piece is 32 columns x 256 k, in the order in which the tiles need them.  The words of a piece are loaded as those of the piece
    // before are used up, and the piece after it is claimed meanwhile.
    const int strips = a.N / 128, per_ct = 8 * kpieces, pieces = a.col_tiles * per_ct;
    const uint4* tr = reinterpret_cast<const uint4*>(a.trellis);
    // A lane takes eighth g of the tiles of row j of four: columns g and g + 8, each every other group of four of its values (exl3_gemm_tm.cu).  The four
    // lanes of a column write 128 bytes of it side by side.
    const int g = lane & 7, j = lane >> 3, prev_lane = (lane & ~7) | ((lane + 7) & 7);
    const size_t kt_stride = (size_t)strips * 64;      // uint4 of one row of 16 k
    auto claim = [&]() { return lane == 0 ? atomicAdd(claimed, 1) : 0; };
    struct Piece { int strip, q, kt0, counter; bool live; };
    auto locate = [&](int p) {
      // a group of column tiles, segment by segment; in it column tile, 256 k, strip, 32 columns.  The last piece of an odd number of 128 k repeats half of
      // the piece before it (the same values).  Not live: past the end, or the second strip of a column tile that has one; the words of another are loaded.
      Piece r;
      r.live = p < pieces;
      p = min(p, pieces - 1);
      const int first = p / (a.group * per_ct) * a.group, tiles_g = min(a.group, a.col_tiles - first), u = p - first * per_ct;
      const int seg = min(u / (tiles_g * 8 * WD_SEG), segs - 1), v = u - seg * tiles_g * 8 * WD_SEG, n = 8 * min(WD_SEG, kpieces - seg * WD_SEG);
      const int ct = first + v / n, x = v % n, second = (x >> 2) & 1;
      r.q = x & 3;
      r.kt0 = min((seg * WD_SEG + (x >> 3)) * PIECE_KT, a.K / 16 - PIECE_KT);
      r.counter = ct * segs + seg;
      r.strip = MODE == WD_SWIGLU ? ct + second * (strips / 2) : 2 * ct + second;
      if (r.strip >= strips) r.strip = strips - 1, r.live = false;
      return r;
    };
    auto source = [&](const Piece& r) { return tr + (size_t)(r.kt0 + j) * kt_stride + r.strip * 64 + r.q * 16 + g; };
    constexpr int LOADS = PIECE_KT / 2;            // of a lane: two tiles of columns x four rows of k at a time
    int p = __shfl_sync(0xffffffffu, claim(), 0), ahead = claim();
    Piece now = locate(p);
    uint4 cur[LOADS];
    {
      const uint4* src = source(now);
#pragma unroll
      for (int i = 0; i < LOADS; ++i) cur[i] = __ldg(src + (i >> 1) * 4 * kt_stride + (i & 1) * 8);
    }
    while (p < pieces && __all_sync(0xffffffffu, *abort_flag == 0)) {
      const int pn = __shfl_sync(0xffffffffu, ahead, 0);
      const Piece nx = locate(pn);
      ahead = claim();
      const uint4* src = source(nx);
      __half* dst = a.w + ((size_t)(now.strip * (a.K / 64) + now.kt0 / 4) * 128 + now.q * 32 + g) * 64 + j * 16;
#pragma unroll
      for (int i = 0; i < LOADS; ++i) {
        const uint32_t w[5] = {__shfl_sync(0xffffffffu, cur[i].w, prev_lane), cur[i].x, cur[i].y, cur[i].z, cur[i].w};
        cur[i] = __ldg(src + (i >> 1) * 4 * kt_stride + (i & 1) * 8);
#pragma unroll
        for (int b2 = 0; b2 < 2; ++b2) {
          uint32_t h[8];
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            uint32_t s0, s1, s2, s3;
            extract4<CB != CB_MUL1>(b2 ? w[m + 1] : __funnelshift_l(w[m + 1], w[m], 16), s0, s1, s2, s3);
            h[m] = pair_to_half2<CB>(s0, s1);
            h[4 + m] = pair_to_half2<CB>(s2, s3);
          }
          if (now.live) stg256(dst + (i >> 1) * 128 * 64 + ((i & 1) * 16 + b2 * 8) * 64, h);
        }
      }
      __threadfence();
      __syncwarp();
      if (lane == 0) atomicAdd(ready + now.counter, 1);
      p = pn;
      now = nx;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0 && threadIdx.x == 0)
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(mapa_u32(smem_u32((const void*)abort_flag), rank ^ 1)), "r"(1) : "memory");
  __syncwarp();
  cluster_sync();
  if (*abort_flag != 0) {
    // Either CTA has given up, and the last copies may be under way.  A stage that only one CTA has issued its copies for gets the other's bytes here.
    if (rank == 0 && threadIdx.x == 0) {
      const int n0 = *n_sent, n1 = ld_cluster(n_sent, 1);
      for (int i = n1; i < n0; ++i) mbar_complete_tx(&full[i % WD_STAGES], (uint32_t)sent[i % WD_STAGES]);
      for (int i = n0; i < n1; ++i) mbar_arrive_expect_tx(&full[i % WD_STAGES], (uint32_t)ld_cluster(sent + i % WD_STAGES, 1));
      ring_landed(full, WD_STAGES, max(n0, n1));
    }
    __syncwarp();
    cluster_sync();
  }
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  if (warp == 0) {
    // the last CTA leaves the counters as it found them
    __threadfence();
    const int done = __shfl_sync(0xffffffffu, lane == 0 ? atomicAdd(a.count + WC_FINISHED, 1) : 0, 0);
    if (done == (int)gridDim.x - 1)
      for (int i = lane; i < WC_READY + a.col_tiles * segs; i += 32) a.count[i] = 0;
  }
}

int make_tmap_f16_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows);
int make_tmap_f32_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows);

template <int CB, int MODE>
static int launch_wide(const CUtensorMap& tx, const CUtensorMap& tw, const CUtensorMap& tw64, const CUtensorMap& to, const WideArgs& a, cudaStream_t st) {
  auto kern = exl3_gemm_wide_kernel<CB, MODE>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WD_SMEM);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return (int)rx::launch(kern, dim3(2 * WD_PAIRS), dim3(WD_THREADS), WD_SMEM, st, tx, tw, tw64, to, a);
}

static int wide_counters(int K, int N) { return WC_READY + (N + 255) / 256 * ((K + WD_SEG * WD_PIECE_K - 1) / (WD_SEG * WD_PIECE_K)); }

}  // namespace rx

using namespace rx;

// Whether the calls below are faster than exl3_gemm_tm.cu and, of the forms with one, the finish kernel after it; form: 0 plain, 1 SwiGLU, 2 store.  In units of that
// kernel's 8 per k and wave of 148 tiles: a share of 74 costs about as much per k here, the expansion and a longer start come on top, a wave's start and the finish
// kernel's rows fall away.  Fitted to 36 matrices (512 to 28,672 wide) at 19 row counts from 130 to 8192 each, both timed in turn: where it says yes the ratio of
// the times is 0.985 and more (plain 1.33 at the most, SwiGLU 1.54, store 1.74), where it says no below 1.06 (store 1.10 once).
RX_API int rx_exl3_wide_takes(int rows, int K, int N, int form) {
  if (K % 128 != 0 || K < WD_PIECE_K || N % 128 != 0 || wide_counters(K, N) > WD_COUNTERS || form < 0 || form > 2) return 0;
  static const struct { double wave, unit_k, unit, expand, start, finish; } F[3] = {
      {11770, 7.94, 30, 4.06e-4, 44750, 0}, {3760, 7.65, 40, 3.78e-4, 48900, 2.84e-3}, {11130, 7.97, 250, 5.98e-4, 46700, 2.97e-3}};
  const auto& f = F[form];
  const double rt = (rows + 255) / 256, tiles = rt * ((N + 255) / 256), units = tiles < WD_PAIRS ? 1.0 : tiles / WD_PAIRS;
  const double waves = (int)((rt * (N / 128) + 147) / 148);
  return waves * (K * 8.0 + f.wave) + f.finish * rows * (double)N > units * (K * f.unit_k + f.unit) + f.expand * (double)N * K + f.start;
}

// Bytes of workspace for a matrix; its first WD_COUNTERS * 4 bytes are zero before the first call.
RX_API long long rx_exl3_wide_bytes(int K, int N) { return WD_FRONT + 2ll * K * N; }

static int gemm_wide(WideArgs a, const void* xr, int codebook, int mode, void* out, void* work, long long work_bytes, cudaStream_t st) {
  if (a.rows <= 0 || a.K % 128 != 0 || a.K < WD_PIECE_K || a.N % (mode == WD_SWIGLU ? 256 : 128) != 0 || a.N <= 0) return (int)cudaErrorInvalidValue;
  if (work == nullptr || work_bytes < rx_exl3_wide_bytes(a.K, a.N) || wide_counters(a.K, a.N) > WD_COUNTERS) return (int)cudaErrorInvalidValue;
  if (mode == WD_STORE && ((((uintptr_t)a.svh) & 15) || (((uintptr_t)a.bias) & 15))) return (int)cudaErrorMisalignedAddress;
  if ((((uintptr_t)xr) & 15) || (((uintptr_t)out) & 31) || (((uintptr_t)a.trellis) & 15) || (((uintptr_t)work) & 127)) return (int)cudaErrorMisalignedAddress;
  a.count = (int*)work;
  a.hand = (float*)((char*)work + WD_COUNTERS * 4);
  a.w = (__half*)((char*)work + WD_FRONT);
  a.row_tiles = (a.rows + 255) / 256;
  a.col_tiles = (a.N + 255) / 256;
  const int bands = (a.row_tiles + 7) / 8;
  a.band = (a.row_tiles + bands - 1) / bands;
  const int total = a.row_tiles * a.col_tiles, rest = total % WD_PAIRS;
  a.inter = total < WD_PAIRS ? 1 : rest == 0 ? total / WD_PAIRS : total / WD_PAIRS - 1;
  a.region = total < WD_PAIRS ? 0 : total - a.inter * WD_PAIRS;
  a.group = a.inter == 0 ? a.col_tiles : (WD_PAIRS + a.band - 1) / a.band;
  CUtensorMap tx, tw, tw64, to;
  int e = make_tmap_f16_2d(&tx, xr, (uint64_t)a.rows, (uint64_t)a.K, 128);
  if (e == 0) e = make_tmap_f16_2d(&tw, a.w, (uint64_t)a.N * (a.K / 64), 64, 128);
  if (e == 0) e = make_tmap_f16_2d(&tw64, a.w, (uint64_t)a.N * (a.K / 64), 64, 64);
  to = tx;
  if (e == 0 && mode != WD_SWIGLU) e = make_tmap_f32_2d(&to, out, (uint64_t)a.rows, (uint64_t)a.N, 32);
  if (e != 0) return e;
#define RX_WD(CBV) (mode == WD_SWIGLU ? launch_wide<CBV, WD_SWIGLU>(tx, tw, tw64, to, a, st) \
                    : mode == WD_STORE ? launch_wide<CBV, WD_STORE>(tx, tw, tw64, to, a, st) : launch_wide<CBV, WD_PLAIN>(tx, tw, tw64, to, a, st))
  switch (codebook) {
    case CB_3INST: return RX_WD(CB_3INST);
    case CB_MCG: return RX_WD(CB_MCG);
    case CB_MUL1: return RX_WD(CB_MUL1);
    default: return (int)cudaErrorInvalidValue;
  }
#undef RX_WD
}

// 4.0 bpw: part[row][n] = rx_exl3_gemm_b4 in one split, the same bits.
RX_API int rx_exl3_gemm_wide(const void* xr, int rows, int K, const void* trellis, int N, int codebook, void* part, void* work, long long work_bytes, int* status,
                             void* stream) {
  WideArgs a = {};
  a.trellis = (const uint32_t*)trellis, a.status = status;
  a.rows = rows, a.K = K, a.N = N;
  return gemm_wide(a, xr, codebook, WD_PLAIN, part, work, work_bytes, (cudaStream_t)stream);
}

// The same with rx_finish_swiglu_rot in its epilogue: a tile is 128 gate columns and the 128 up columns beside them.
RX_API int rx_exl3_gemm_wide_swiglu(const void* xr, int rows, int K, const void* trellis, int F, int codebook, const void* svh, const void* bias,
                                    const void* suh_down, void* act, void* work, long long work_bytes, int* status, void* stream) {
  WideArgs a = {};
  a.act = (__half*)act, a.svh = (const __half*)svh, a.bias = (const float*)bias, a.suh_next = (const __half*)suh_down;
  a.trellis = (const uint32_t*)trellis, a.status = status;
  a.rows = rows, a.K = K, a.N = 2 * F;
  return gemm_wide(a, xr, codebook, WD_SWIGLU, act, work, work_bytes, (cudaStream_t)stream);
}

// The same with rx_finish_store of fp32 rows in its epilogue.
RX_API int rx_exl3_gemm_wide_store(const void* xr, int rows, int K, const void* trellis, int N, int codebook, const void* svh, const void* bias, void* out,
                                   void* work, long long work_bytes, int* status, void* stream) {
  WideArgs a = {};
  a.svh = (const __half*)svh, a.bias = (const float*)bias;
  a.trellis = (const uint32_t*)trellis, a.status = status;
  a.rows = rows, a.K = K, a.N = N;
  return gemm_wide(a, xr, codebook, WD_STORE, out, work, work_bytes, (cudaStream_t)stream);
}
