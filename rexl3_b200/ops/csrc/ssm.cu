// Mamba2 (SSD) token mixer for hybrid decoders: causal depthwise conv over x | B | C, discretization, fp32 state recurrence,
// grouped gated RMSNorm.  Semantics matched: reference crates/cuda/csrc/nemotron_ssm.cu:1-45 (conv k=4 with a 3-row history,
// dt = softplus(dt + bias), decay exp(dt * A), y = C . S + D * x, gated norm over d_inner / groups channels) and
// crates/model/src/families/nemotron_h_omni/ssm_ref.rs.
//
// This engine's own layout and schedule:
//   proj      f32 [M][ldp]: the in_proj output row, columns z (d_inner) | x (d_inner) | B (G*N) | C (G*N) | dt (H) | padding
//   conv pool f32 [slots][3][C]      C = d_inner + 2 G N; the last three pre-conv x|B|C rows of the sequence, oldest first
//   ssm pool  f32 [slots][H][P][N]   P = 64 (head dim), N = 128 (state); n contiguous
// Rows of one sequence are consecutive and in position order (a "segment"); a sequence appears in at most one segment of a
// launch.  A row at position 0 starts from a zero state whatever the pools hold, so a slot needs no reset when it is reused.
// Record / commit split (reference crates/cuda/csrc/gdn.cu:253-322: a verify window reads the pools, a later commit replays the accepted
// prefix): the recurrence kernels take a mode.  SCAN_OUT alone = a window whose rows may still be rejected: the pools are read, outputs are
// written, nothing is stored back; the caller keeps that launch's `proj` and `xbc` rows (per layer) as the record.  SCAN_STATE alone = the
// commit: the same kernel walks the first `keep` recorded rows of each sequence again (the same arithmetic on the same inputs, so the state
// equals what a serial decode of those rows leaves, bit for bit) and stores the state and the conv history; outputs are not written.
// SCAN_OUT | SCAN_STATE = rows that are final when fed (prefill, windows without drafts).
//
// The conv is parallel over rows (each row reads its three predecessors from the launch's own rows or from the pool); the
// recurrence is sequential over the rows of a segment with the state of one head in the registers of a 256-thread CTA
// (thread = one p, 32 of the 128 n), so a decode step moves each state once: 2 x 32 KB per (sequence, head).
#include <type_traits>
#include "common.cuh"

namespace rx {

constexpr int SSM_P = 64, SSM_N = 128, SSM_HIST = 3;
constexpr int SCAN_OUT = 1, SCAN_STATE = 2;

// asynchronous copies into shared memory: the inputs of the next tokens arrive while the current ones are computed
__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ float ssm_silu(float v) { return v / (1.f + __expf(-v)); }
__device__ __forceinline__ float ssm_bf(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }

// the pre-conv value of channel c at `back` positions before row r (back 1..3), or of row r itself (back 0)
__device__ __forceinline__ float ssm_conv_in(const float* __restrict__ proj, int ldp, int xoff, const float* pool, int C,
                                             const int* __restrict__ row_seq, const int* __restrict__ positions, int r, int back, int c) {
  const int pos = positions[r];
  if (pos - back < 0) return 0.f;
  const int seq = row_seq[r];
  if (r - back >= 0 && row_seq[r - back] == seq) return proj[(size_t)(r - back) * ldp + xoff + c];
  // not in this launch: the pool holds positions (first - 3, first - 2, first - 1) of the segment's first row
  int o = 0;                                   // rows of the segment before r (only 0..2 can get here)
  while (o < back && r - o - 1 >= 0 && row_seq[r - o - 1] == seq) ++o;
  return pool[((size_t)seq * SSM_HIST + (SSM_HIST - back + o)) * C + c];
}

// the segment's last three pre-conv rows become the sequence's conv history.  Every CTA of the segment (one per head) commits its own
// share of the channels after its recurrence: left to one CTA, this loop of dependent loads was most of a decode step's kernel time.
__device__ __forceinline__ void ssm_conv_commit(const float* __restrict__ proj, int ldp, int xoff, float* conv_pool, int C,
                                                const int* __restrict__ row_seq, const int* __restrict__ positions, int last, int seq, int part,
                                                int nparts) {
  const int chunk = (C + nparts - 1) / nparts, c0 = part * chunk, c1 = min(C, c0 + chunk);
  for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
    float v[SSM_HIST];
#pragma unroll
    for (int k = 0; k < SSM_HIST; ++k) v[k] = ssm_conv_in(proj, ldp, xoff, conv_pool, C, row_seq, positions, last, SSM_HIST - 1 - k, c);
#pragma unroll
    for (int k = 0; k < SSM_HIST; ++k) conv_pool[((size_t)seq * SSM_HIST + k) * C + c] = v[k];
  }
}

// xbc[r][c] = silu(b[c] + sum_j w[c][j] * in(pos - 3 + j)).  One channel of one row per thread: the form for the few rows of a decode window,
// where it is latency that counts.  grid (M, ceil(C / 256))
__global__ void __launch_bounds__(256) ssm_conv_kernel(const float* __restrict__ proj, int ldp, int xoff, int C, const int* __restrict__ row_seq,
                                                      const int* __restrict__ positions, const uint16_t* __restrict__ conv_w,
                                                      const uint16_t* __restrict__ conv_b, const float* __restrict__ pool, float* __restrict__ xbc) {
  pdl_launch();
  pdl_wait();
  const int r = blockIdx.x, c = blockIdx.y * 256 + threadIdx.x;
  if (c >= C) return;
  float acc = ssm_bf(conv_b[c]);
#pragma unroll
  for (int j = 0; j < 4; ++j) acc += ssm_bf(conv_w[c * 4 + j]) * ssm_conv_in(proj, ldp, xoff, pool, C, row_seq, positions, r, 3 - j, c);
  xbc[(size_t)r * C + c] = ssm_silu(acc);
}

// The same for many rows, bound by memory (one read of the rows, one write): a thread takes two neighbouring channels and walks CONV_RB rows, all
// loaded before the first is used, with the three rows before them in registers.  The form above reads every input four times through the
// caches: 137 us for 2048 rows x 10240 channels against 46 us here; the two passes need 26.  grid (ceil(M / CONV_RB), ceil(C / 512)), 256 threads.
constexpr int CONV_RB = 8;
__global__ void __launch_bounds__(256) ssm_conv_rows_kernel(const float* __restrict__ proj, int ldp, int xoff, int C, const int* __restrict__ row_seq,
                                                           const int* __restrict__ positions, const uint16_t* __restrict__ conv_w,
                                                           const uint16_t* __restrict__ conv_b, const float* __restrict__ pool,
                                                           float* __restrict__ xbc, int M) {
  pdl_launch();
  pdl_wait();
  const int rb = blockIdx.x * CONV_RB, c = (blockIdx.y * 256 + threadIdx.x) * 2;
  if (c >= C) return;
  float2 x[CONV_RB + 3];                            // rows rb - 3 .. rb + CONV_RB - 1
  int seq[CONV_RB + 3];
#pragma unroll
  for (int i = 0; i < CONV_RB + 3; ++i) {
    const int r = max(0, min(rb + i - 3, M - 1));
    seq[i] = rb + i < 3 ? -1 : row_seq[r];
    x[i] = *reinterpret_cast<const float2*>(proj + (size_t)r * ldp + xoff + c);
  }
  float w[2][4], bias[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    bias[e] = ssm_bf(conv_b[c + e]);
#pragma unroll
    for (int j = 0; j < 4; ++j) w[e][j] = ssm_bf(conv_w[(c + e) * 4 + j]);
  }
  auto put = [&](int i, float2 a, float2 b, float2 d) {
    const float in[2][4] = {{a.x, b.x, d.x, x[i + 3].x}, {a.y, b.y, d.y, x[i + 3].y}};
    float o[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float acc = bias[e];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc += w[e][j] * in[e][j];
      o[e] = ssm_silu(acc);
    }
    if (rb + i < M) *reinterpret_cast<float2*>(xbc + (size_t)(rb + i) * C + c) = make_float2(o[0], o[1]);
  };
  bool whole = true;                                // every row's three predecessors are its sequence's
#pragma unroll
  for (int i = 0; i < CONV_RB; ++i) whole = whole && seq[i] == seq[i + 3];
  if (whole) {
#pragma unroll
    for (int i = 0; i < CONV_RB; ++i) put(i, x[i], x[i + 1], x[i + 2]);
    return;
  }
  // Short segments: what a row's own segment does not have in this launch comes from the pool (positions first - 3 .. first - 1 of the segment) or
  // is zero.  All rows' values are on their way before the first is used (layer of the delta net, 16 x 5 rows 62.5 us row after row, 56.3 so).
  float2 p[CONV_RB][3];
  int own = 0;
#pragma unroll
  for (int i = 0; i < CONV_RB; ++i) {
    if (i == 0) own = seq[2] != seq[3] ? 0 : seq[1] != seq[3] ? 1 : seq[0] != seq[3] ? 2 : 3;
    else own = seq[i + 3] == seq[i + 2] ? min(own + 1, 3) : 0;
    const int pos = own < 3 ? positions[min(rb + i, M - 1)] : 0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {                   // 3 - j positions back
      p[i][j] = x[i + j];
      if (3 - j > own) {
        p[i][j] = make_float2(0.f, 0.f);
        if (pos >= 3 - j) p[i][j] = *reinterpret_cast<const float2*>(pool + ((size_t)seq[i + 3] * SSM_HIST + j + own) * C + c);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < CONV_RB; ++i) put(i, p[i][0], p[i][1], p[i][2]);
}

// Recurrence.  grid (segments or rows, H).  With a segment table (seg_start != nullptr) block x is segment x; without one block x is
// row x and returns unless that row opens a segment.  Each block also writes its share of the segment's last three pre-conv rows to the conv pool.
__global__ void __launch_bounds__(256) ssm_scan_kernel(const float* __restrict__ xbc, int C, const float* __restrict__ proj, int ldp, int xoff,
                                                      int dtoff, int M, int H, int G, const int* __restrict__ row_seq,
                                                      const int* __restrict__ positions, const int* __restrict__ seg_start,
                                                      const int* __restrict__ seg_len, const float* __restrict__ dt_bias,
                                                      const float* __restrict__ a_neg, const float* __restrict__ d_skip,
                                                      float* __restrict__ ssm_pool, float* conv_pool, float* __restrict__ y, int mode) {
  pdl_launch();
  pdl_wait();
  __shared__ __align__(16) float sB[SSM_N], sC[SSM_N], sx[SSM_P];
  int r0, len;
  if (seg_start != nullptr) {
    r0 = seg_start[blockIdx.x];
    len = seg_len[blockIdx.x];
  } else {
    r0 = blockIdx.x;
    if (r0 > 0 && row_seq[r0 - 1] == row_seq[r0]) return;
    len = 1;
    while (r0 + len < M && row_seq[r0 + len] == row_seq[r0]) ++len;
  }
  if (len <= 0) return;
  const int h = blockIdx.y, tid = threadIdx.x, p = tid >> 2, nq = tid & 3;
  const int seq = row_seq[r0], g = h / (H / G), DI = H * SSM_P;
  float st[32];
  float* sp = ssm_pool + (((size_t)seq * H + h) * SSM_P + p) * SSM_N + nq * 32;
  if (positions[r0] == 0) {
#pragma unroll
    for (int i = 0; i < 32; ++i) st[i] = 0.f;
  } else {
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      const float4 v = *reinterpret_cast<const float4*>(sp + i);
      st[i] = v.x, st[i + 1] = v.y, st[i + 2] = v.z, st[i + 3] = v.w;
    }
  }
  const float A = a_neg[h], Dh = d_skip[h], dtb = dt_bias[h];
  // this thread's share of a token's inputs (one B or C value, one x value for the first 64 threads, the head's dt); the next token's are
  // fetched while the current one is computed, so a long segment is not a chain of dependent global loads
  const int bc_off = tid < SSM_N ? DI + g * SSM_N + tid : DI + G * SSM_N + g * SSM_N + (tid - SSM_N);
  float n_bc = xbc[(size_t)r0 * C + bc_off], n_x = tid < SSM_P ? xbc[(size_t)r0 * C + h * SSM_P + tid] : 0.f, n_dt = proj[(size_t)r0 * ldp + dtoff + h];
  for (int t = 0; t < len; ++t) {
    const int r = r0 + t;
    const float c_bc = n_bc, c_x = n_x, c_dt = n_dt;
    if (t + 1 < len) {
      const float* xn = xbc + (size_t)(r + 1) * C;
      n_bc = xn[bc_off];
      if (tid < SSM_P) n_x = xn[h * SSM_P + tid];
      n_dt = proj[(size_t)(r + 1) * ldp + dtoff + h];
    }
    __syncthreads();
    if (tid < SSM_N) sB[tid] = c_bc;
    else sC[tid - SSM_N] = c_bc;
    if (tid < SSM_P) sx[tid] = c_x;
    __syncthreads();
    float dt = c_dt + dtb;
    dt = dt > 20.f ? dt : log1pf(__expf(dt));            // softplus
    const float dA = __expf(dt * A), xdt = sx[p] * dt;
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;     // four partial sums: dependent chains of 8 instead of 32
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      const float4 bb = *reinterpret_cast<const float4*>(sB + nq * 32 + i), cc = *reinterpret_cast<const float4*>(sC + nq * 32 + i);
      // (the roundings are spelled out: the split kernel below repeats them, so that a commit leaves the bits of a direct run)
      st[i] = __fmaf_rn(xdt, bb.x, __fmul_rn(st[i], dA)); st[i + 1] = __fmaf_rn(xdt, bb.y, __fmul_rn(st[i + 1], dA));
      st[i + 2] = __fmaf_rn(xdt, bb.z, __fmul_rn(st[i + 2], dA)); st[i + 3] = __fmaf_rn(xdt, bb.w, __fmul_rn(st[i + 3], dA));
      a0 = __fmaf_rn(st[i], cc.x, a0); a1 = __fmaf_rn(st[i + 1], cc.y, a1); a2 = __fmaf_rn(st[i + 2], cc.z, a2); a3 = __fmaf_rn(st[i + 3], cc.w, a3);
    }
    float acc = (a0 + a1) + (a2 + a3);
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    if (nq == 0 && (mode & SCAN_OUT)) y[(size_t)r * DI + h * SSM_P + p] = __fmaf_rn(Dh, sx[p], acc);
  }
  if (!(mode & SCAN_STATE)) return;
#pragma unroll
  for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(sp + i) = make_float4(st[i], st[i + 1], st[i + 2], st[i + 3]);
  ssm_conv_commit(proj, ldp, xoff, conv_pool, C, row_seq, positions, r0 + len - 1, seq, h, (int)gridDim.y);
}

// Prefill / commit form of the recurrence, bound by the multiply pipe and by issue: three fp32 operations per state value and token.  A head's 64
// state rows p are split over two CTAs of four warps; a thread holds four rows of every fourth n of a quarter (n = 32 nq + 4 m + k, m = 0 .. 7), so
// that B and C cost a token four vector loads from shared memory for 96 operations (a 1 x 32 tile needs sixteen) and a thread's share of an
// output is one of the sixteen chains that ssm_scan_kernel adds up.  Every rounding and every order of a sum is that kernel's: states and outputs
// are the same bits.  (Packed pairs along n took 436 us, 463 us this way: what they save in issue slots is small, two of the three operations
// read three registers, which the packed form issues every third cycle; a 4 x 4 tile on twice the warps is bound by the loads again: 506 us.)
// The inputs of TC tokens at a time come by cp.async into two buffers, x dt and the decays are made from them by the CTA: two block barriers per
// TC tokens, no global load on the per-token path.  The dependents are released only when the recurrence is done: released at the start, their
// waiting CTAs (thousands) took the SMs' slots and slowed it by half.
// One sequence of 2047 tokens, 128 heads: 463 us; 2159 us before (1 x 32 tiles, one warp per CTA, register ring; 3220 us with early release).
// The states come and go through shared memory, whole rows in 16-byte pieces: a thread's own values, every fourth of a row, are half sectors, and a commit
// is little else than its states (8 x 1 rows 57.5 us with them, 32 us in the one-warp form, 20 us now).
// grid (segments, H, SSM_PS), 128 threads; TC tokens to a chunk.
constexpr int SSM_PS = 2, SSM_CP = SSM_P / SSM_PS;
template <int TC> struct SsmChunk { float B[TC][SSM_N], C[TC][SSM_N], x[TC][SSM_CP], dt[TC]; };
// where n stands in a token's B and C: the eight values of a thread (nq, k) as two vectors, sixteen threads' vectors side by side
__device__ __forceinline__ int ssm_place(int n) { return ((n >> 4) & 1) * 64 + ((n >> 5) * 4 + (n & 3)) * 4 + ((n >> 2) & 3); }
// where value n of a state row stands on its way through shared memory: the lanes of a warp, at any m, then meet different banks
constexpr int SSM_SROW = SSM_N + 4;
__device__ __forceinline__ int ssm_stage(int n) { return n ^ ((n >> 5) << 2); }
template <int TC>
__global__ void __launch_bounds__(128) ssm_scan_split_kernel(const float* __restrict__ xbc, int C, const float* __restrict__ proj, int ldp, int xoff,
                                                            int dtoff, int M, int H, int G, const int* __restrict__ row_seq,
                                                            const int* __restrict__ positions, const int* __restrict__ seg_start,
                                                            const int* __restrict__ seg_len, const float* __restrict__ dt_bias,
                                                            const float* __restrict__ a_neg, const float* __restrict__ d_skip,
                                                            float* __restrict__ ssm_pool, float* conv_pool, float* __restrict__ y, int mode) {
  pdl_wait();
  // two chunks; the states' way in and out takes the second one's place
  constexpr int STAGE = SSM_CP * SSM_SROW * 4, CHUNK = (int)sizeof(SsmChunk<TC>);
  __shared__ __align__(16) uint8_t raw[CHUNK + (CHUNK > STAGE ? CHUNK : STAGE)];
  SsmChunk<TC>* buf = reinterpret_cast<SsmChunk<TC>*>(raw);
  float* stage = reinterpret_cast<float*>(raw + CHUNK);
  __shared__ float xdt[TC][SSM_CP], dec[TC];                         // x dt and the decay of the current chunk
  const int r0 = seg_start[blockIdx.x], len = seg_len[blockIdx.x];
  if (len <= 0) return;
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ln = lane & 15, lp = lane >> 4;
  const int seq = row_seq[r0], g = h / (H / G), DI = H * SSM_P, p0 = blockIdx.z * SSM_CP;
  // Slot i of a thread is state row pl + (i ^ sel) with sel from lane bits 0 and 1: what a lane passes on in the output sums' tree is then always its
  // upper slots, without selects.
  const int pl = warp * 8 + lp * 4, sel = (ln & 1 ? 2 : 0) | (ln & 2 ? 1 : 0);
  float st[4][8];
  float* sp = ssm_pool + (((size_t)seq * H + h) * SSM_P + p0) * SSM_N;
  const bool fresh = positions[r0] == 0;
  if (!fresh)
#pragma unroll
    for (int i = 0; i < SSM_CP / 4; ++i) cp16(&stage[(4 * i + warp) * SSM_SROW + ssm_stage(4 * lane)], sp + (4 * i + warp) * SSM_N + 4 * lane);
  const int place = ssm_place(tid);
  auto issue = [&](int c) {                         // tokens c * TC ..; past the end the last row again (never used)
    SsmChunk<TC>& d = buf[c & 1];
    const float* src = xbc + DI + g * SSM_N + tid;
#pragma unroll
    for (int t = 0; t < TC; ++t) {
      const float* xr = src + (size_t)(r0 + min(c * TC + t, len - 1)) * C;
      cp4(&d.B[t][place], xr);
      cp4(&d.C[t][place], xr + G * SSM_N);
    }
    const int t = tid >> 3;
    if (t < TC) cp16(&d.x[t][4 * (tid & 7)], xbc + (size_t)(r0 + min(c * TC + t, len - 1)) * C + h * SSM_P + p0 + 4 * (tid & 7));
    if (tid < TC) cp4(&d.dt[tid], proj + (size_t)(r0 + min(c * TC + tid, len - 1)) * ldp + dtoff + h);
    cp_commit();
  };
  const float A = a_neg[h], Dh = d_skip[h], dtb = dt_bias[h];
  const bool b2 = (ln & 4) != 0, b3 = (ln & 8) != 0;
  float* yp = y + h * SSM_P + p0 + pl + sel;        // slot 0's row: the one whose sums end in this lane
  // NT tokens (4, or 1 at the end): the states in turn, then all NT x 4 output sums over the 16 lanes together, each step halving what a lane
  // carries on.  A sum's tree over the lanes (distances 1, 2, 4, 8) does not depend on NT.
  auto tokens = [&](const SsmChunk<TC>& d, auto n, int t0, int r) {
    constexpr int NT = decltype(n)::value;
    float k[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int t = t0 + i;
      const float4 B0 = *reinterpret_cast<const float4*>(&d.B[t][4 * ln]), B1 = *reinterpret_cast<const float4*>(&d.B[t][64 + 4 * ln]);
      const float4 C0 = *reinterpret_cast<const float4*>(&d.C[t][4 * ln]), C1 = *reinterpret_cast<const float4*>(&d.C[t][64 + 4 * ln]);
      const float b[8] = {B0.x, B0.y, B0.z, B0.w, B1.x, B1.y, B1.z, B1.w}, c[8] = {C0.x, C0.y, C0.z, C0.w, C1.x, C1.y, C1.z, C1.w};
      const float dA = dec[t];
      float xd[4], o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int p = 0; p < 4; ++p) xd[p] = xdt[t][pl + (p ^ sel)];
#pragma unroll
      for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          st[p][m] = __fmaf_rn(xd[p], b[m], __fmul_rn(st[p][m], dA));
          o[p] = __fmaf_rn(st[p][m], c[m], o[p]);
        }
      const float k0 = o[0] + __shfl_xor_sync(0xffffffffu, o[2], 1), k1 = o[1] + __shfl_xor_sync(0xffffffffu, o[3], 1);
      k[i] = k0 + __shfl_xor_sync(0xffffffffu, k1, 2);
    }
    if (!(mode & SCAN_OUT)) return;
    if constexpr (NT == 4) {                        // lane bits 2 and 3 pick the token
      const float m0 = (b2 ? k[2] : k[0]) + __shfl_xor_sync(0xffffffffu, b2 ? k[0] : k[2], 4);
      const float m1 = (b2 ? k[3] : k[1]) + __shfl_xor_sync(0xffffffffu, b2 ? k[1] : k[3], 4);
      const float m = (b3 ? m1 : m0) + __shfl_xor_sync(0xffffffffu, b3 ? m0 : m1, 8);
      const int t = (b2 ? 2 : 0) + (b3 ? 1 : 0);
      yp[(size_t)(r + t) * DI] = __fmaf_rn(Dh, d.x[t0 + t][pl + sel], m);
    } else {
      float m = k[0];
      m += __shfl_xor_sync(0xffffffffu, m, 4);
      m += __shfl_xor_sync(0xffffffffu, m, 8);
      if (!b2 && !b3) yp[(size_t)r * DI] = __fmaf_rn(Dh, d.x[t0][pl + sel], m);
    }
  };
  issue(0);
  const int own = (ln >> 2) * 32 + (ln & 3);
  cp_wait_all();
  __syncthreads();
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int m = 0; m < 8; ++m) st[p][m] = fresh ? 0.f : stage[(pl + (p ^ sel)) * SSM_SROW + ssm_stage(own + 4 * m)];
  const int nc = (len + TC - 1) / TC;
  for (int c = 0; c < nc; ++c) {
    cp_wait_all();
    __syncthreads();                                // chunk c has landed, everybody is done with chunk c - 1
    if (c + 1 < nc) issue(c + 1);
    const SsmChunk<TC>& d = buf[c & 1];
    if (TC == 16 || tid < 8 * TC) {
      const int t = tid >> 3, p = 4 * (tid & 7);    // eight threads per token
      float dt = d.dt[t] + dtb;
      dt = dt > 20.f ? dt : log1pf(__expf(dt));     // softplus
      const float4 x = *reinterpret_cast<const float4*>(&d.x[t][p]);
      xdt[t][p] = x.x * dt, xdt[t][p + 1] = x.y * dt, xdt[t][p + 2] = x.z * dt, xdt[t][p + 3] = x.w * dt;
      if (p == 0) dec[t] = __expf(dt * A);
    }
    __syncthreads();
    const int nt = min(TC, len - c * TC);
    int t = 0;
    for (; t + 4 <= nt; t += 4) tokens(d, std::integral_constant<int, 4>(), t, r0 + c * TC + t);
    for (; t < nt; ++t) tokens(d, std::integral_constant<int, 1>(), t, r0 + c * TC + t);
  }
  pdl_launch();
  if (!(mode & SCAN_STATE)) return;
  __syncthreads();                                  // (the last tokens have been read)
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int m = 0; m < 8; ++m) stage[(pl + (p ^ sel)) * SSM_SROW + ssm_stage(own + 4 * m)] = st[p][m];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < SSM_CP / 4; ++i)
    *reinterpret_cast<float4*>(sp + (4 * i + warp) * SSM_N + 4 * lane) = *reinterpret_cast<const float4*>(&stage[(4 * i + warp) * SSM_SROW + ssm_stage(4 * lane)]);
  ssm_conv_commit(proj, ldp, xoff, conv_pool, C, row_seq, positions, r0 + len - 1, seq, h * SSM_PS + blockIdx.z, (int)(gridDim.y * SSM_PS));
}

// The next projection's input rotation of a 128-block of bf16 values, a warp: x[4 lane ..] * suh, transformed, to fp16.  The values are those that would have been
// stored and read again (norm_rot_in_kernel without a norm), so the bits are the same.
__device__ __forceinline__ void ssm_rotate(const uint16_t (&b)[4], const __half* suh, __half* xr) {
  const int lane = threadIdx.x & 31;
  const uint2 u = *reinterpret_cast<const uint2*>(suh + 4 * lane);
  const float2 s0 = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), s1 = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
  float v[4] = {ssm_bf(b[0]) * s0.x, ssm_bf(b[1]) * s0.y, ssm_bf(b[2]) * s1.x, ssm_bf(b[3]) * s1.y};
  fwht128_warp(v);
  const __half2 a = __floats2half2_rn(v[0], v[1]), c = __floats2half2_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(xr + 4 * lane) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&c));
}

// out[r][c] = bf16( rmsnorm_group( y * silu(z) )[c] * w[c] ), grid (M, G); the group is d_inner / G channels wide.  Bound by memory: a thread's
// first GN_KEEP channels stay in registers between the sum and the scaling (loaded together; read and gated twice, one after the other, it took
// 68 us for 2047 rows of 8 x 1024 channels, 46 us now); a wider group is gated again beyond that.
// With `suh` the rows leave rotated (xr, fp16) by way of shared memory (W * 2 bytes): a launch less, 2.7 us in a step and 22 us in that prompt slice.
constexpr int GN_KEEP = 4;
__global__ void __launch_bounds__(256) ssm_gate_norm_kernel(const float* __restrict__ y, const float* __restrict__ proj, int ldp, int DI, int G,
                                                           const uint16_t* __restrict__ norm_w, float eps, uint16_t* __restrict__ out,
                                                           const __half* __restrict__ suh, __half* __restrict__ xr) {
  pdl_launch();
  pdl_wait();
  __shared__ float red[8];
  extern __shared__ __align__(8) uint16_t gn_row[];
  const int r = blockIdx.x, g = blockIdx.y, W = DI / G, c0 = g * W;
  const float* yr = y + (size_t)r * DI + c0;
  const float* zr = proj + (size_t)r * ldp + c0;
  float keep[GN_KEEP], z[GN_KEEP], ss = 0.f;
#pragma unroll
  for (int i = 0; i < GN_KEEP; ++i) {
    const int c = threadIdx.x + 256 * i;
    keep[i] = c < W ? yr[c] : 0.f;
    z[i] = c < W ? zr[c] : 0.f;
  }
#pragma unroll
  for (int i = 0; i < GN_KEEP; ++i) {
    keep[i] = __fmul_rn(keep[i], ssm_silu(z[i]));
    ss = __fmaf_rn(keep[i], keep[i], ss);
  }
  for (int c = threadIdx.x + 256 * GN_KEEP; c < W; c += 256) {
    const float v = __fmul_rn(yr[c], ssm_silu(zr[c]));
    ss = __fmaf_rn(v, v, ss);
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += red[i];
  const float rinv = rsqrtf(tot / (float)W + eps);
  auto put = [&](int c, float v) {
    __nv_bfloat16 b = __float2bfloat16_rn(v * rinv * ssm_bf(norm_w[c0 + c]));
    if (suh != nullptr) gn_row[c] = *reinterpret_cast<uint16_t*>(&b);
    else out[(size_t)r * DI + c0 + c] = *reinterpret_cast<uint16_t*>(&b);
  };
#pragma unroll
  for (int i = 0; i < GN_KEEP; ++i)
    if (threadIdx.x + 256 * i < W) put(threadIdx.x + 256 * i, keep[i]);
  for (int c = threadIdx.x + 256 * GN_KEEP; c < W; c += 256) put(c, yr[c] * ssm_silu(zr[c]));
  if (suh == nullptr) return;
  __syncthreads();
  for (int b = (threadIdx.x >> 5) * 128; b < W; b += 8 * 128) {
    const uint2 u = *reinterpret_cast<const uint2*>(gn_row + b + 4 * (threadIdx.x & 31));
    const uint16_t v[4] = {(uint16_t)u.x, (uint16_t)(u.x >> 16), (uint16_t)u.y, (uint16_t)(u.y >> 16)};
    ssm_rotate(v, suh + c0 + b, xr + (size_t)r * DI + c0 + b);
  }
}

// ------------------------------------------------------------------------------------------------ gated delta net
// Gated DeltaNet linear attention (reference crates/cuda/csrc/gdn.cu:1-25: 16 key heads x 128, 32/48/64 value heads x 128, conv
// width 4 over q | k | v, l2-normalised q and k, q scaled by 1/sqrt(128), decay exp(g) with g = A * softplus(a + dt_bias), A < 0,
// beta = sigmoid(b); delta rule S = S e^g; S += k (x) (beta (v - S^T k)); o = S^T q; per-head RMSNorm(o) * w * silu(z)).
//   proj     f32 [M][ldp]: z (Hv*128) | q (Hk*128) | k (Hk*128) | v (Hv*128) | b (Hv) | a (Hv) | padding
//   S pool   f32 [slots][Hv][64 KB], one head's state S[value j][key i] stored in the order the kernel reads it: thread (j, half) owns
//            i = 64 half + 4 s + e (s = 0..15 load steps, e = 0..3), and the float4 of step s sits at ((warp * 16 + s) * 32 + lane) * 4 with
//            warp = j / 16, lane = 2 (j % 16) + half: every load and store instruction of a warp covers one contiguous 512-byte run
//            (the obvious [j][i] layout made each instruction touch 32 different 128-byte lines; measured in the profile note).
//            conv pool as above with C = (2 Hk + Hv) * 128
// One CTA per (segment, value head), 256 threads: thread = value column j and one half of the 128 keys (64 state values in registers);
// the two halves meet in one shuffle.  The gated norm runs in the same kernel (the CTA holds the head's whole output row).
//
// KDA = true: Kimi delta attention (reference crates/cuda/csrc/kda.cu: per-key-channel decay).  The decay is a vector over the key
// channels, exp(A * softplus(a_i + dt_bias_i)) with a_i taken from 128 columns per head (proj: ... | b (Hv) | a (Hv*128)), and the
// output gate is a sigmoid instead of SiLU.  Everything else is the same code.
constexpr int GDN_D = 128;

// the write of a token: beta (v - S.k / |k|), with the key's 1 / |k| once more (k enters the update normalised as well)
__device__ __forceinline__ float gdn_delta(float v, float kv, float beta, float kinv) { return __fmaf_rn(-kv, kinv, v) * beta * kinv; }
// One token of the delta rule for the 64 state values of a thread (value column j, one half of the keys): decay, S.k (both halves meet in one
// shuffle), the rank-one write, S.q.  Four partial sums per dot product, key i in sum i % 4, keep the dependent chains at 16 instead of 64; a thread of
// gdn_scan_split_kernel holds one such chain, so that both kernels leave the same bits.
// sk / sq / sd: this half's 64 keys, queries and (KDA) decays in shared memory, 16-byte aligned.  o is returned before the 1 / |q| factor.
template <bool KDA>
__device__ __forceinline__ void gdn_token_update(float (&st)[64], const float* sk, const float* sq, const float* sd, float decay, float v, float beta,
                                                 float kinv, float& o_out) {
  float k0 = 0.f, k1 = 0.f, k2 = 0.f, k3 = 0.f;
#pragma unroll
  for (int i = 0; i < 64; i += 4) {
    const float4 kk = *reinterpret_cast<const float4*>(sk + i);
    if (KDA) {
      const float4 dd = *reinterpret_cast<const float4*>(sd + i);
      st[i] *= dd.x; st[i + 1] *= dd.y; st[i + 2] *= dd.z; st[i + 3] *= dd.w;
    } else {
      st[i] *= decay; st[i + 1] *= decay; st[i + 2] *= decay; st[i + 3] *= decay;
    }
    k0 = __fmaf_rn(st[i], kk.x, k0); k1 = __fmaf_rn(st[i + 1], kk.y, k1); k2 = __fmaf_rn(st[i + 2], kk.z, k2); k3 = __fmaf_rn(st[i + 3], kk.w, k3);
  }
  float kv = (k0 + k1) + (k2 + k3);
  kv = kv + __shfl_xor_sync(0xffffffffu, kv, 1);
  const float delta = gdn_delta(v, kv, beta, kinv);
  float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
  for (int i = 0; i < 64; i += 4) {
    const float4 kk = *reinterpret_cast<const float4*>(sk + i);
    const float4 qq = *reinterpret_cast<const float4*>(sq + i);
    st[i] = __fmaf_rn(kk.x, delta, st[i]); st[i + 1] = __fmaf_rn(kk.y, delta, st[i + 1]);
    st[i + 2] = __fmaf_rn(kk.z, delta, st[i + 2]); st[i + 3] = __fmaf_rn(kk.w, delta, st[i + 3]);
    o0 = __fmaf_rn(st[i], qq.x, o0); o1 = __fmaf_rn(st[i + 1], qq.y, o1); o2 = __fmaf_rn(st[i + 2], qq.z, o2); o3 = __fmaf_rn(st[i + 3], qq.w, o3);
  }
  float o = (o0 + o1) + (o2 + o3);
  o = o + __shfl_xor_sync(0xffffffffu, o, 1);
  o_out = o;
}

// Two CTAs per SM (128 registers, a few dozen bytes of spill): a decode step is a chain of dependent loads per CTA, and a second resident
// CTA hides it; measured 54 us -> see the profile note for 16 streams x 48 heads.
template <bool KDA>
__global__ void __launch_bounds__(256, 2) gdn_scan_kernel(const float* __restrict__ xbc, int C, const float* __restrict__ proj, int ldp, int xoff,
                                                      int goff, int M, int Hk, int Hv, const int* __restrict__ row_seq,
                                                      const int* __restrict__ positions, const int* __restrict__ seg_start,
                                                      const int* __restrict__ seg_len, const float* __restrict__ dt_bias,
                                                      const float* __restrict__ a_neg, const uint16_t* __restrict__ norm_w, float eps,
                                                      float* __restrict__ s_pool, float* conv_pool, uint16_t* __restrict__ out, int mode,
                                                      const __half* __restrict__ suh, __half* __restrict__ xr_out) {
  pdl_launch();
  pdl_wait();
  __shared__ __align__(16) float sqk[2 * GDN_D], sdec[KDA ? GDN_D : 4];
  __shared__ float red[8], red2[8];
  int r0, len;
  if (seg_start != nullptr) {
    r0 = seg_start[blockIdx.x];
    len = seg_len[blockIdx.x];
  } else {
    r0 = blockIdx.x;
    if (r0 > 0 && row_seq[r0 - 1] == row_seq[r0]) return;
    len = 1;
    while (r0 + len < M && row_seq[r0 + len] == row_seq[r0]) ++len;
  }
  if (len <= 0) return;
  __shared__ __align__(8) uint16_t srow[GDN_D];
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, j = tid >> 1, half = tid & 1;
  const int seq = row_seq[r0], hk = h / (Hv / Hk), DI = Hv * GDN_D;
  float st[64];
  float* sp = s_pool + ((size_t)seq * Hv + h) * (GDN_D * GDN_D) + (size_t)warp * (16 * 128) + lane * 4;   // step s adds 128 floats
  if (positions[r0] == 0) {
#pragma unroll
    for (int i = 0; i < 64; ++i) st[i] = 0.f;
  } else {
#pragma unroll
    for (int i = 0; i < 64; i += 4) {
      const float4 v = *reinterpret_cast<const float4*>(sp + (i >> 2) * 128);
      st[i] = v.x, st[i + 1] = v.y, st[i + 2] = v.z, st[i + 3] = v.w;
    }
  }
  const float A = a_neg[h], dtb = KDA ? 0.f : dt_bias[h], wj = ssm_bf(norm_w[j]);
  const float* sq = sqk + half * 64;
  const float* sk = sqk + GDN_D + half * 64;
  for (int t = 0; t < len; ++t) {
    const int r = r0 + t;
    const float* xr = xbc + (size_t)r * C;
    __syncthreads();
    const float val = tid < GDN_D ? xr[hk * GDN_D + tid] : xr[(Hk + hk) * GDN_D + (tid - GDN_D)];
    sqk[tid] = val;
    const float ss = warp_sum(__fmul_rn(val, val));
    if (lane == 0) red[warp] = ss;
    if (KDA && tid < GDN_D) {
      float ai = proj[(size_t)r * ldp + goff + Hv + h * GDN_D + tid] + dt_bias[h * GDN_D + tid];
      ai = ai > 20.f ? ai : log1pf(__expf(ai));
      sdec[tid] = __expf(A * ai);
    }
    __syncthreads();
    const float qinv = rsqrtf(red[0] + red[1] + red[2] + red[3] + 1e-6f) * 0.08838834764831845f;
    const float kinv = rsqrtf(red[4] + red[5] + red[6] + red[7] + 1e-6f);
    const float v = xr[2 * Hk * GDN_D + h * GDN_D + j];
    float decay = 1.f;
    if (!KDA) {
      float a = proj[(size_t)r * ldp + goff + Hv + h] + dtb;
      a = a > 20.f ? a : log1pf(__expf(a));
      decay = __expf(A * a);
    }
    const float beta = 1.f / (1.f + __expf(-proj[(size_t)r * ldp + goff + h]));
    float o;
    gdn_token_update<KDA>(st, sk, sq, sdec + (KDA ? half * 64 : 0), decay, v, beta, kinv, o);
    o *= qinv;
    const float ss2 = warp_sum(half == 0 ? __fmul_rn(o, o) : 0.f);
    if (lane == 0) red2[warp] = ss2;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) tot += red2[i];
    if (half == 0 && (mode & SCAN_OUT)) {
      const float z = proj[(size_t)r * ldp + h * GDN_D + j];
      const float gate = KDA ? 1.f / (1.f + __expf(-z)) : ssm_silu(z);
      __nv_bfloat16 b = __float2bfloat16_rn(o * rsqrtf(tot / (float)GDN_D + eps) * wj * gate);
      if (suh != nullptr) srow[j] = *reinterpret_cast<uint16_t*>(&b);
      else out[(size_t)r * DI + h * GDN_D + j] = *reinterpret_cast<uint16_t*>(&b);
    }
    if (suh != nullptr && (mode & SCAN_OUT)) {         // the head's row leaves rotated
      __syncthreads();
      if (warp == 0) {
        const uint2 u = *reinterpret_cast<const uint2*>(srow + 4 * lane);
        const uint16_t v4[4] = {(uint16_t)u.x, (uint16_t)(u.x >> 16), (uint16_t)u.y, (uint16_t)(u.y >> 16)};
        ssm_rotate(v4, suh + h * GDN_D, xr_out + (size_t)r * DI + h * GDN_D);
      }
    }
  }
  if (!(mode & SCAN_STATE)) return;
#pragma unroll
  for (int i = 0; i < 64; i += 4) *reinterpret_cast<float4*>(sp + (i >> 2) * 128) = make_float4(st[i], st[i + 1], st[i + 2], st[i + 3]);
  ssm_conv_commit(proj, ldp, xoff, conv_pool, C, row_seq, positions, r0 + len - 1, seq, h, (int)gridDim.y);
}

// ---- prefill / commit form of the delta-rule scan.  A head's 128 value columns evolve independently (S_j only meets q and k): they are split over
// GDN_JS CTAs of four warps.  A thread holds two columns x one of the partial sums of gdn_token_update, 16 keys (4 i + sub of a half): what bounds the
// kernel is the way of k and q out of shared memory (a vector load costs four cycles of the SM however many lanes read the same word), and two columns
// share what is loaded; k, q and the decays are laid out by thread, so that its 16 keys are four vectors.  A token's critical path is
// a 16-key dot product, three shuffles and the rank-one write; the output sums of four tokens go over the lanes together, off that path.  What a
// token needs besides (1 / |q|, 1 / |k|, decay, write strength) is computed for TC tokens at a time by the CTA from the inputs that cp.async
// brought into two buffers (norm sums per token and warp: 40 shuffles, 0.96 us per token).  With convolution and norm, 1024
// tokens of one sequence, 48 heads, take 462 us (1090 with one warp per 16 columns; 422 with dot products in eighths of the keys, which are other sums).  Every rounding and every order of a sum
// is gdn_scan_kernel's, so states and outputs are the same bits; the per-head gated norm, which needs all 128 outputs, runs afterwards in
// gdn_norm_kernel.  The dependents are released at the end (see ssm_scan_split_kernel).  grid (segments, Hv, GDN_JS), 128 threads.
constexpr int GDN_JS = 4, GDN_PAD = GDN_D + 32;                       // 16 keys every 20 floats: eight lanes' vectors in different banks
template <bool KDA, int TC> struct GdnChunk {
  float q[TC][GDN_PAD], k[TC][GDN_PAD], d[KDA ? TC : 1][GDN_PAD], v[TC][GDN_D / GDN_JS], a[TC], b[TC];
};
__device__ __forceinline__ int gdn_place(int i) { return (((i >> 4) & 4) + (i & 3)) * 20 + ((i >> 2) & 15); }     // key i: thread group, place in its 16
template <bool KDA, int TC>
__global__ void __launch_bounds__(128) gdn_scan_split_kernel(const float* __restrict__ xbc, int C, const float* __restrict__ proj, int ldp, int xoff,
                                                            int goff, int M, int Hk, int Hv, const int* __restrict__ row_seq,
                                                            const int* __restrict__ positions, const int* __restrict__ seg_start,
                                                            const int* __restrict__ seg_len, const float* __restrict__ dt_bias,
                                                            const float* __restrict__ a_neg, float* __restrict__ s_pool, float* conv_pool,
                                                            float* __restrict__ y32, int mode) {
  constexpr int JC = GDN_D / GDN_JS;
  pdl_wait();
  __shared__ __align__(16) GdnChunk<KDA, TC> buf[2];
  __shared__ __align__(16) float4 gate[TC];                            // decay, beta, 1 / |k|, 1 / |q| of a token
  const int r0 = seg_start[blockIdx.x], len = seg_len[blockIdx.x];
  if (len <= 0) return;
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int sub = lane & 3, half = (lane >> 2) & 1, jl = warp * 8 + (lane >> 3), j = blockIdx.z * JC + jl;     // columns j and j + 4
  const bool odd = (lane & 1) != 0;       // an odd lane holds them the other way round: of a pair, a lane passes its slot 1 on in a sum's tree
  const int seq = row_seq[r0], hk = h / (Hv / Hk), DI = Hv * GDN_D;
  float st[2][16];                                                     // keys 64 half + 4 (0 .. 15) + sub of the two columns
  float* sp = s_pool + ((size_t)seq * Hv + h) * (GDN_D * GDN_D) + (size_t)(j >> 4) * (16 * 128) + (2 * (j & 15) + half) * 4 + sub;
  const bool fresh = positions[r0] == 0;
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const float a = fresh ? 0.f : sp[m * 128], b = fresh ? 0.f : sp[m * 128 + 32];
    st[0][m] = odd ? b : a, st[1][m] = odd ? a : b;
  }
  const float A = a_neg[h], dtb = KDA ? dt_bias[h * GDN_D + tid] : dt_bias[h];
  const int place = gdn_place(tid);
  auto issue = [&](int c) {                                            // past the end the last row again (never used)
    GdnChunk<KDA, TC>& d = buf[c & 1];
#pragma unroll
    for (int t = 0; t < TC; ++t) {
      const float* xr = xbc + (size_t)(r0 + min(c * TC + t, len - 1)) * C + hk * GDN_D + tid;
      cp4(&d.q[t][place], xr);
      cp4(&d.k[t][place], xr + Hk * GDN_D);
    }
    if (tid < TC * 8) {
      const int t = tid >> 3, kv = tid & 7;
      cp16(&d.v[t][4 * kv], xbc + (size_t)(r0 + min(c * TC + t, len - 1)) * C + (2 * Hk + h) * GDN_D + blockIdx.z * JC + 4 * kv);
    }
    if (KDA) {
#pragma unroll
      for (int t = 0; t < TC; ++t)
        cp4(&d.d[t][place], proj + (size_t)(r0 + min(c * TC + t, len - 1)) * ldp + goff + Hv + h * GDN_D + tid);
    }
    if (tid < TC) {
      const float* pr = proj + (size_t)(r0 + min(c * TC + tid, len - 1)) * ldp + goff;
      cp4(&d.b[tid], pr + h);
      if (!KDA) cp4(&d.a[tid], pr + Hv + h);
    }
    cp_commit();
  };
  const int kb = (4 * half + sub) * 20, j0 = jl + (odd ? 4 : 0);       // j0: the column of slot 0
  // NT tokens (4, or 1 at the end): the states in turn, then the NT x 2 output sums over the eight lanes of a column pair together
  auto tokens = [&](const GdnChunk<KDA, TC>& d, auto n, int t0, int r) {
    constexpr int NT = decltype(n)::value;
    float o[NT][2];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int t = t0 + i;
      const float4 gt = gate[t];
      float kk[16], a[2] = {0.f, 0.f};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 v = *reinterpret_cast<const float4*>(&d.k[t][kb + 4 * u]);
        kk[4 * u] = v.x, kk[4 * u + 1] = v.y, kk[4 * u + 2] = v.z, kk[4 * u + 3] = v.w;
        float4 dd = make_float4(gt.x, gt.x, gt.x, gt.x);
        if (KDA) dd = *reinterpret_cast<const float4*>(&d.d[t][kb + 4 * u]);
        const float de[4] = {dd.x, dd.y, dd.z, dd.w};
#pragma unroll
        for (int m = 4 * u; m < 4 * u + 4; ++m)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            st[c][m] *= de[m & 3];
            a[c] = __fmaf_rn(st[c][m], kk[m], a[c]);
          }
      }
      float kv = a[0] + __shfl_xor_sync(0xffffffffu, a[1], 1);         // the four partial sums of a half, then the halves
      kv += __shfl_xor_sync(0xffffffffu, kv, 2);
      kv += __shfl_xor_sync(0xffffffffu, kv, 4);
      const float delta = gdn_delta(d.v[t][j0], kv, gt.y, gt.z), dl[2] = {delta, __shfl_xor_sync(0xffffffffu, delta, 1)};
      a[0] = a[1] = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 v = *reinterpret_cast<const float4*>(&d.q[t][kb + 4 * u]);
        const float qq[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int m = 4 * u; m < 4 * u + 4; ++m)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            st[c][m] = __fmaf_rn(kk[m], dl[c], st[c][m]);
            a[c] = __fmaf_rn(st[c][m], qq[m & 3], a[c]);
          }
      }
      o[i][0] = a[0], o[i][1] = a[1];
    }
    if (!(mode & SCAN_OUT)) return;
    const bool b1 = (lane & 2) != 0, b2 = (lane & 4) != 0;
    float m[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) m[i] = o[i][0] + __shfl_xor_sync(0xffffffffu, o[i][1], 1);
    float* yp = y32 + (size_t)r * DI + h * GDN_D + blockIdx.z * JC + j0;
    if constexpr (NT == 4) {                                           // bits 1 and 2 pick the token
      const float n0 = (b1 ? m[2] : m[0]) + __shfl_xor_sync(0xffffffffu, b1 ? m[0] : m[2], 2);
      const float n1 = (b1 ? m[3] : m[1]) + __shfl_xor_sync(0xffffffffu, b1 ? m[1] : m[3], 2);
      const float s = (b2 ? n1 : n0) + __shfl_xor_sync(0xffffffffu, b2 ? n0 : n1, 4);
      const int i = (b1 ? 2 : 0) + (b2 ? 1 : 0);
      yp[(size_t)i * DI] = s * gate[t0 + i].w;
    } else {
      float s = m[0] + __shfl_xor_sync(0xffffffffu, m[0], 2);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      if (!b1 && !b2) yp[0] = s * gate[t0].w;
    }
  };
  issue(0);
  const int nc = (len + TC - 1) / TC;
  for (int c = 0; c < nc; ++c) {
    cp_wait_all();
    __syncthreads();                                                   // chunk c has landed, everybody is done with chunk c - 1
    if (c + 1 < nc) issue(c + 1);
    GdnChunk<KDA, TC>& d = buf[c & 1];
    // norms: gdn_scan_kernel's warp sums over 32 values (tree over lane distances 16, 8, 4, 2, 1), eight lanes with four values each
    float rs[TC / 4][2];
#pragma unroll
    for (int i = 0; i < TC / 4; ++i)
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        // values n, n + 8, n + 16 and n + 24 of a 32 stand two places apart each
        const float* x = (w ? d.k[warp + 4 * i] : d.q[warp + 4 * i]) + gdn_place(32 * (lane >> 3) + (lane & 7));
        rs[i][w] = (__fmul_rn(x[0], x[0]) + __fmul_rn(x[4], x[4])) + (__fmul_rn(x[2], x[2]) + __fmul_rn(x[6], x[6]));
      }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < TC / 4; ++i)
#pragma unroll
        for (int w = 0; w < 2; ++w) rs[i][w] += __shfl_xor_sync(0xffffffffu, rs[i][w], o);
#pragma unroll
    for (int i = 0; i < TC / 4; ++i) {
      float tot[2];
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        tot[w] = __shfl_sync(0xffffffffu, rs[i][w], 0);
#pragma unroll
        for (int k = 1; k < 4; ++k) tot[w] += __shfl_sync(0xffffffffu, rs[i][w], 8 * k);
      }
      const int t = warp + 4 * i;
      if (lane == i) {
        float decay = 1.f;
        if (!KDA) {
          float al = d.a[t] + dtb;
          al = al > 20.f ? al : log1pf(__expf(al));
          decay = __expf(A * al);
        }
        gate[t] = make_float4(decay, 1.f / (1.f + __expf(-d.b[t])), rsqrtf(tot[1] + 1e-6f), rsqrtf(tot[0] + 1e-6f) * 0.08838834764831845f);
      }
    }
    if (KDA) {
#pragma unroll
      for (int t = 0; t < TC; ++t) {
        float ai = d.d[t][place] + dtb;
        ai = ai > 20.f ? ai : log1pf(__expf(ai));
        d.d[t][place] = __expf(A * ai);
      }
    }
    __syncthreads();
    const int nt = min(TC, len - c * TC);
    int t = 0;
    for (; t + 4 <= nt; t += 4) tokens(d, std::integral_constant<int, 4>(), t, r0 + c * TC + t);
    for (; t < nt; ++t) tokens(d, std::integral_constant<int, 1>(), t, r0 + c * TC + t);
  }
  pdl_launch();
  if (!(mode & SCAN_STATE)) return;
#pragma unroll
  for (int m = 0; m < 16; ++m) sp[m * 128] = odd ? st[1][m] : st[0][m], sp[m * 128 + 32] = odd ? st[0][m] : st[1][m];
  ssm_conv_commit(proj, ldp, xoff, conv_pool, C, row_seq, positions, r0 + len - 1, seq, h * GDN_JS + blockIdx.z, (int)(gridDim.y * GDN_JS));
}

// out[r][h][j] = bf16( o * rsqrt(mean_j o^2 + eps) * w[j] * gate(z) ), bound by memory: one warp per (row, head), four columns per lane.  The sum of
// squares is taken in gdn_scan_kernel's order: trees over 16 columns (distances 8, 4, 2, 1), the eight sums added in sequence.
// grid (M, ceil(Hv / 8)), 256 threads.
template <bool KDA>
__global__ void __launch_bounds__(256) gdn_norm_kernel(const float* __restrict__ y32, const float* __restrict__ proj, int ldp, int Hv,
                                                      const uint16_t* __restrict__ norm_w, float eps, uint16_t* __restrict__ out,
                                                      const __half* __restrict__ suh, __half* __restrict__ xr) {
  pdl_launch();
  pdl_wait();
  const int r = blockIdx.x, lane = threadIdx.x & 31, h = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (h >= Hv) return;
  const size_t at = ((size_t)r * Hv + h) * GDN_D + 4 * lane;
  const float* zp = proj + (size_t)r * ldp + h * GDN_D + 4 * lane;
  const float4 o = *reinterpret_cast<const float4*>(y32 + at);
  const float z[4] = {zp[0], zp[1], zp[2], zp[3]}, v[4] = {o.x, o.y, o.z, o.w};
  float s[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) s[e] = __fmul_rn(v[e], v[e]);
#pragma unroll
  for (int e = 0; e < 4; ++e) s[e] += __shfl_xor_sync(0xffffffffu, s[e], 2);
#pragma unroll
  for (int e = 0; e < 4; ++e) s[e] += __shfl_xor_sync(0xffffffffu, s[e], 1);
  const float s16 = (s[0] + s[2]) + (s[1] + s[3]);
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += __shfl_sync(0xffffffffu, s16, 4 * i);
  const float rinv = rsqrtf(tot / (float)GDN_D + eps);
  uint16_t b[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float gt = KDA ? 1.f / (1.f + __expf(-z[e])) : ssm_silu(z[e]);
    __nv_bfloat16 t = __float2bfloat16_rn(v[e] * rinv * ssm_bf(norm_w[4 * lane + e]) * gt);
    b[e] = *reinterpret_cast<uint16_t*>(&t);
  }
  if (suh != nullptr) {                                // the row leaves rotated: 17 us less for 2048 rows of 6144
    ssm_rotate(b, suh + h * GDN_D, xr + ((size_t)r * Hv + h) * GDN_D);
    return;
  }
  uint16_t* op = out + at;
  if ((((uintptr_t)out) & 7) == 0) *reinterpret_cast<uint2*>(op) = make_uint2(b[0] | ((uint32_t)b[1] << 16), b[2] | ((uint32_t)b[3] << 16));
  else op[0] = b[0], op[1] = b[1], op[2] = b[2], op[3] = b[3];
}

// The walking form needs pairs of channels (even widths, 8-byte alignment), enough rows to fill the chip with eighths of them (64 of 10240 channels), and
// rows that follow one another: prompt slices and verify windows.  A plain decode window has one row of each sequence and keeps the other form
// (layer of the delta net, 64 x 1 rows 104.6 us and 108.1, 256 x 1 388 and 397; 16 x 5 rows 59.2 and 56.3, 32 x 8 167 and 158).
static void launch_conv(const void* proj, int ldp, int xoff, int C, const void* row_seq, const void* positions, const void* conv_w, const void* conv_b,
                        const void* conv_pool, void* xbc, int M, bool follow, cudaStream_t st) {
  const bool pairs = C % 2 == 0 && ldp % 2 == 0 && xoff % 2 == 0 && ((((uintptr_t)proj) | ((uintptr_t)xbc) | ((uintptr_t)conv_pool)) & 7) == 0;
  const int cg = (C + 511) / 512;
  if (follow && pairs && (long long)(M / CONV_RB) * cg >= 148)
    launch(ssm_conv_rows_kernel, dim3((M + CONV_RB - 1) / CONV_RB, cg), dim3(256), 0, st, (const float*)proj, ldp, xoff, C, (const int*)row_seq,
           (const int*)positions, (const uint16_t*)conv_w, (const uint16_t*)conv_b, (const float*)conv_pool, (float*)xbc, M);
  else
    launch(ssm_conv_kernel, dim3(M, (C + 255) / 256), dim3(256), 0, st, (const float*)proj, ldp, xoff, C, (const int*)row_seq, (const int*)positions,
           (const uint16_t*)conv_w, (const uint16_t*)conv_b, (const float*)conv_pool, (float*)xbc);
}

}  // namespace rx

// One Mamba2 mixer between its two projections: conv, recurrence (pools updated), gated norm.  seg_start / seg_len (device, nseg
// entries) describe the segments when the host knows them (prefill, commit); pass nullptr and nseg = 0 to have the kernel find them.
// mode: 3 = rows are final (outputs and pools written), 1 = window record (outputs only; keep proj and xbc for the commit),
// 2 = commit (the recurrence over the recorded proj / xbc rows of the given segments, pools written; conv and norm are not launched).
// suh not null: the rows leave with the next projection's input rotation, fp16 to xr, and out_bf16 is not written (groups of whole 128-blocks).
RX_API int rx_ssm_mixer(const void* proj, int ldp, int M, int H, int P, int G, int N, const void* row_seq, const void* positions,
                        const void* seg_start, const void* seg_len, int nseg, const void* conv_w, const void* conv_b, const void* dt_bias,
                        const void* a_neg, const void* d_skip, const void* norm_w, float eps, void* conv_pool, void* ssm_pool, void* xbc,
                        void* y, void* out_bf16, void* stream, int mode, const void* suh, void* xr) {
  using namespace rx;
  if (mode < 1 || mode > 3) return (int)cudaErrorInvalidValue;
  if (P != SSM_P || N != SSM_N || G <= 0 || H % G || M <= 0) return (int)cudaErrorInvalidValue;
  const int DI = H * P, C = DI + 2 * G * N, xoff = DI, dtoff = DI + C;
  if (ldp < dtoff + H) return (int)cudaErrorInvalidValue;
  if (suh != nullptr && ((DI / G) % 128 != 0 || DI / G > 16384)) return (int)cudaErrorInvalidValue;
  if ((((uintptr_t)ssm_pool) & 15) != 0) return (int)cudaErrorMisalignedAddress;       // every form moves the states in 16-byte pieces
  cudaStream_t st = (cudaStream_t)stream;
  if (mode & SCAN_OUT)
    launch_conv(proj, ldp, xoff, C, row_seq, positions, conv_w, conv_b, conv_pool, xbc, M, seg_start != nullptr || mode == SCAN_OUT, st);
  // Commits begin early (the layers' follow one another: one row 7.4 us alone, 5.7 so for the delta net), and short ones take chunks of four tokens: a quarter
  // of the shared memory and of the gates' work (8 x 1 rows of the delta net 21.3 -> 15.8 us, of Mamba2 57.5 -> 20.1 together with the states' way).
  const bool short_commit = mode == SCAN_STATE && M <= 4 * nseg;
  if (seg_start != nullptr && (((uintptr_t)xbc) & 15) == 0)     // segments known on the host (prefill, commit); its copies take 16 bytes
    launch_pdl(mode == SCAN_STATE, short_commit ? ssm_scan_split_kernel<4> : ssm_scan_split_kernel<16>, dim3(nseg, H, SSM_PS), dim3(128), 0, st, (const float*)xbc, C, (const float*)proj, ldp, xoff, dtoff, M, H, G,
           (const int*)row_seq, (const int*)positions, (const int*)seg_start, (const int*)seg_len, (const float*)dt_bias, (const float*)a_neg,
           (const float*)d_skip, (float*)ssm_pool, (float*)conv_pool, (float*)y, mode);
  else
  launch(ssm_scan_kernel, dim3(seg_start ? nseg : M, H), dim3(256), 0, st, (const float*)xbc, C, (const float*)proj, ldp, xoff, dtoff, M, H, G,
         (const int*)row_seq, (const int*)positions, (const int*)seg_start, (const int*)seg_len, (const float*)dt_bias, (const float*)a_neg,
         (const float*)d_skip, (float*)ssm_pool, (float*)conv_pool, (float*)y, mode);
  if (mode & SCAN_OUT)
    launch(ssm_gate_norm_kernel, dim3(M, G), dim3(256), suh != nullptr ? DI / G * 2 : 0, st, (const float*)y, (const float*)proj, ldp, DI, G,
           (const uint16_t*)norm_w, eps, (uint16_t*)out_bf16, (const __half*)suh, (__half*)xr);
  return (int)cudaGetLastError();
}

// One gated-delta-net (kda = 0) or Kimi-delta-attention (kda = 1; dt_bias then has Hv*128 entries) mixer between its two projections:
// conv, then recurrence + gated norm (pools updated).  Two launches; with a host segment table and y32 (f32 [M][Hv*128] scratch) the
// recurrence runs column-split with the norm as a third launch (prefill and commit).
RX_API int rx_gdn_mixer(const void* proj, int ldp, int M, int Hk, int Hv, int D, const void* row_seq, const void* positions, const void* seg_start,
                        const void* seg_len, int nseg, const void* conv_w, const void* conv_b, const void* dt_bias, const void* a_neg,
                        const void* norm_w, float eps, void* conv_pool, void* s_pool, void* xbc, void* out_bf16, void* stream, int kda, int mode,
                        void* y32, const void* suh, void* xr) {
  using namespace rx;
  if (mode < 1 || mode > 3) return (int)cudaErrorInvalidValue;
  if (D != GDN_D || Hk <= 0 || Hv % Hk || M <= 0) return (int)cudaErrorInvalidValue;
  const int DI = Hv * D, C = (2 * Hk + Hv) * D, xoff = DI, goff = DI + C;
  if (ldp < goff + Hv + (kda ? Hv * D : Hv)) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)stream;
  if (mode & SCAN_OUT)
    launch_conv(proj, ldp, xoff, C, row_seq, positions, conv_w, conv_b, conv_pool, xbc, M, seg_start != nullptr || mode == SCAN_OUT, st);
  if (seg_start != nullptr && y32 != nullptr && ((((uintptr_t)xbc) | ((uintptr_t)y32)) & 15) == 0) {
    // segments known on the host (prefill, commit): the column-split scan with prefetched inputs, then the norm (same bits as the fused kernel).  Commits
    // begin early and short ones take chunks of four tokens (see rx_ssm_mixer).
    const bool short_commit = mode == SCAN_STATE && M <= 4 * nseg;
    auto gdn_scan = kda ? gdn_scan_split_kernel<true, 8> : gdn_scan_split_kernel<false, 16>;
    if (short_commit) gdn_scan = kda ? gdn_scan_split_kernel<true, 4> : gdn_scan_split_kernel<false, 4>;
    launch_pdl(mode == SCAN_STATE, gdn_scan, dim3(nseg, Hv, GDN_JS), dim3(128), 0, st, (const float*)xbc, C,
           (const float*)proj, ldp, xoff, goff, M, Hk, Hv, (const int*)row_seq, (const int*)positions, (const int*)seg_start, (const int*)seg_len,
           (const float*)dt_bias, (const float*)a_neg, (float*)s_pool, (float*)conv_pool, (float*)y32, mode);
    if (mode & SCAN_OUT)
      launch(kda ? gdn_norm_kernel<true> : gdn_norm_kernel<false>, dim3(M, (Hv + 7) / 8), dim3(256), 0, st, (const float*)y32, (const float*)proj, ldp, Hv,
             (const uint16_t*)norm_w, eps, (uint16_t*)out_bf16, (const __half*)suh, (__half*)xr);
    return (int)cudaGetLastError();
  }
  launch(kda ? gdn_scan_kernel<true> : gdn_scan_kernel<false>, dim3(seg_start ? nseg : M, Hv), dim3(256), 0, st, (const float*)xbc, C, (const float*)proj, ldp, xoff, goff, M, Hk, Hv,
         (const int*)row_seq, (const int*)positions, (const int*)seg_start, (const int*)seg_len, (const float*)dt_bias, (const float*)a_neg,
         (const uint16_t*)norm_w, eps, (float*)s_pool, (float*)conv_pool, (uint16_t*)out_bf16, mode,
         (const __half*)suh, (__half*)xr);
  return (int)cudaGetLastError();
}
