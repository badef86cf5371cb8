// Everything around the EXL3 GEMM: input rotation (x * suh -> Hadamard -> fp16) fused with RMSNorm, and the finish
// kernels that sum the GEMM's K-split partials in split order, apply the output Hadamard, svh and bias, and fuse what
// follows (residual add + RMSNorm + the next layer's input rotation, or SwiGLU + the down projection's rotation).
// Also: trellis -> dense W_q unpack (test oracle / weight reconstruction) and embedding gather.
//
// What these match in the reference: crates/cuda/csrc/exl3_linear.cu:136-208 (rot_in / rot_out), glue.cu:99 (add_rmsnorm),
// :139 (swiglu), ling_kda_proj_fused.cu:1432,1595,2088 (the fused forms).  One warp owns one 128-wide Hadamard block;
// lane L holds elements 4L..4L+3.  All reductions have a fixed order, so results never depend on the row count.
#include "exl3_decode.cuh"

namespace rx {

__device__ __forceinline__ float bf16_to_f(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }
__device__ __forceinline__ uint16_t f_to_bf16(float f) {
  __nv_bfloat16 b = __float2bfloat16_rn(f);
  return *reinterpret_cast<uint16_t*>(&b);
}

__device__ __forceinline__ void load4_bf16(const uint16_t* p, float (&v)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  v[0] = __uint_as_float(u.x << 16); v[1] = __uint_as_float(u.x & 0xFFFF0000u);
  v[2] = __uint_as_float(u.y << 16); v[3] = __uint_as_float(u.y & 0xFFFF0000u);
}
__device__ __forceinline__ void store4_bf16(uint16_t* p, const float (&v)[4]) {
  uint2 u;
  u.x = (uint32_t)f_to_bf16(v[0]) | ((uint32_t)f_to_bf16(v[1]) << 16);
  u.y = (uint32_t)f_to_bf16(v[2]) | ((uint32_t)f_to_bf16(v[3]) << 16);
  *reinterpret_cast<uint2*>(p) = u;
}
__device__ __forceinline__ void load4_f16(const __half* p, float (&v)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void store4_f16(__half* p, const float (&v)[4]) {
  const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
  uint2 u;
  u.x = *reinterpret_cast<const uint32_t*>(&a); u.y = *reinterpret_cast<const uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = u;
}

// Block-wide sum with a fixed order: warp shuffles, then warp 0 adds the per-warp values in warp order.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = 0.f;
  for (int i = 0; i < nw; ++i) t += red[i];
  return t;
}

// ------------------------------------------------------------------------------------------------ unpack
template <int TWICE, int CB>
__global__ void unpack_kernel(const uint32_t* __restrict__ trellis, __half* __restrict__ w, int kt, int nt) {
  pdl_launch();
  pdl_wait();
  const int tile = blockIdx.x * (blockDim.x / 4) + threadIdx.x / 4;
  if (tile >= kt * nt) return;
  const int h = threadIdx.x & 3;
  uint32_t h2[32];
  decode_span<TWICE, CB, 64>(trellis + (size_t)tile * 4 * TWICE, h * TWICE, h2);
  const int tk = tile / nt, tn = tile % nt, N = nt * 16;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int q = 2 * i, lanep = (64 * h + q) / 8, j = q % 8;
    const int r = 2 * (lanep % 4) + (j & 1) + 8 * ((j >> 1) & 1), c = lanep / 4 + 8 * (j >> 2);
    const __half2 v = *reinterpret_cast<const __half2*>(&h2[i]);
    w[(size_t)(tk * 16 + r) * N + tn * 16 + c] = __low2half(v);
    w[(size_t)(tk * 16 + r + 1) * N + tn * 16 + c] = __high2half(v);
  }
}

// ------------------------------------------------------------------------------------------------ embed
__global__ void embed_kernel(const int* __restrict__ ids, const uint16_t* __restrict__ table, uint16_t* __restrict__ h, int d, int vocab) {
  pdl_launch();
  pdl_wait();
  const int row = blockIdx.x;
  int id = ids[row];
  if (id < 0 || id >= vocab) id = 0;
  const uint4* src = reinterpret_cast<const uint4*>(table + (size_t)id * d);
  uint4* dst = reinterpret_cast<uint4*>(h + (size_t)row * d);
  for (int i = threadIdx.x; i < d / 8; i += blockDim.x) dst[i] = src[i];
}

// ------------------------------------------------------------------------------------------------ norm + rot_in
// xr[row] = fp16( H( rmsnorm(x[row]) * w * suh ) ), one block per row.  norm_w == nullptr: no norm (plain rotation).
__global__ void __launch_bounds__(1024) norm_rot_in_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ norm_w, float eps,
                                   const __half* __restrict__ suh, __half* __restrict__ xr, int K) {
  pdl_launch();
  pdl_wait();
  __shared__ float blk_ss[512];   // one partial per 128-block (K <= 65536), added in block order: independent of the block size
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint16_t* xrow = x + (size_t)row * K;
  float rinv = 1.f;
  if (norm_w != nullptr) {
    for (int b = warp; b < K / 128; b += nw) {
      float v[4];
      load4_bf16(xrow + b * 128 + lane * 4, v);
      const float ss = warp_sum(v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3]);
      if (lane == 0) blk_ss[b] = ss;
    }
    __syncthreads();
    float tot = 0.f;
    for (int b = 0; b < K / 128; ++b) tot += blk_ss[b];
    rinv = rsqrtf(tot / (float)K + eps);
  }
  for (int b = warp; b < K / 128; b += nw) {
    const int i = b * 128 + lane * 4;
    float v[4], s[4];
    load4_bf16(xrow + i, v);
    load4_f16(suh + i, s);
    if (norm_w != nullptr) {
      float w[4];
      load4_bf16(norm_w + i, w);
#pragma unroll
      for (int r = 0; r < 4; ++r) v[r] = bf16_to_f(f_to_bf16(v[r] * rinv)) * w[r];
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] *= s[r];
    fwht128_warp(v);
    store4_f16(xr + (size_t)row * K + i, v);
  }
}

// The plain rotation of many rows: eight lanes to a 128-block.  x and xr of [rows * nb] blocks, suh of nb.
__global__ void __launch_bounds__(256) rot_in_rows_kernel(const uint16_t* x, const __half* __restrict__ suh, __half* __restrict__ xr, long long blocks,
                                                          int nb) {
  pdl_launch();
  pdl_wait();
  const long long at = ((long long)blockIdx.x * 256 + threadIdx.x) >> 3, item = min(at, blocks - 1);
  const int l4 = (threadIdx.x & 7) * 4, n0 = (int)(item % nb) * 128 + l4;
  float v[4][4], s[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    load4_bf16(x + item * 128 + l4 + 32 * j, v[j]);
    load4_f16(suh + n0 + 32 * j, s[j]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) v[j][e] *= s[j][e];        // exact: 8 and 11 bits
  fwht128_oct(v);
  if (at >= blocks) return;
#pragma unroll
  for (int j = 0; j < 4; ++j) store4_f16(xr + item * 128 + l4 + 32 * j, v[j]);
}

// ------------------------------------------------------------------------------------------------ finish kernels
// y[row][n] = H_N( sum_s part[s][row][:] )[n] * svh[n] + bias[n] for one 128-block, lane holds 4 consecutive n.
// ONE: a single plane, known at compile time.  The loop over planes keeps eight loads in registers; a kernel that carries it for nothing holds a
// third as many warps per SM (100 registers against 32-48), which for the many rows of a prompt is what bounded these kernels.
template <bool ONE = false>
__device__ __forceinline__ void sum_planes(const float* __restrict__ part, int S, size_t split_stride, size_t off, float (&y)[4]) {
  // loads are issued eight at a time (independent, so their latencies overlap) and added in split order
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (ONE || S == 1) acc = __ldg(reinterpret_cast<const float4*>(part + off));
  else
  for (int s0 = 0; s0 < S; s0 += 8) {
    float4 p[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (s0 + j < S) p[j] = __ldg(reinterpret_cast<const float4*>(part + (size_t)(s0 + j) * split_stride + off));
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (s0 + j < S) {
        if (s0 + j == 0) acc = p[j];
        else { acc.x += p[j].x; acc.y += p[j].y; acc.z += p[j].z; acc.w += p[j].w; }
      }
  }
  y[0] = acc.x; y[1] = acc.y; y[2] = acc.z; y[3] = acc.w;
}
template <bool ONE = false>
__device__ __forceinline__ void finish_block(const float* __restrict__ part, int S, size_t split_stride, size_t off, const __half* svh,
                                             const float* bias, int n0, float (&y)[4]) {
  sum_planes<ONE>(part, S, split_stride, off, y);
  fwht128_warp(y);
  float sv[4];
  load4_f16(svh + n0, sv);
#pragma unroll
  for (int r = 0; r < 4; ++r) y[r] = __fmul_rn(y[r], sv[r]);     // (never contracted into what follows: the variants of a kernel give the same bits)
  if (bias != nullptr) {
    const float4 b = *reinterpret_cast<const float4*>(bias + n0);
    y[0] += b.x; y[1] += b.y; y[2] += b.z; y[3] += b.w;
  }
}

// mode 0: out bf16 [M, N];  mode 1: out f32 [M, N]
template <bool ONE>
__global__ void __launch_bounds__(256) finish_store_kernel(const float* __restrict__ part, int S, int M, int N, const __half* __restrict__ svh,
                                    const float* __restrict__ bias, void* __restrict__ out, int f32_out) {
  pdl_launch();
  pdl_wait();
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int b = blockIdx.y * nw + warp; b < N / 128; b += gridDim.y * nw) {
    const int n0 = b * 128 + lane * 4;
    float y[4];
    finish_block<ONE>(part, S, (size_t)M * N, (size_t)row * N + n0, svh, bias, n0, y);
    if (f32_out) *reinterpret_cast<float4*>((float*)out + (size_t)row * N + n0) = make_float4(y[0], y[1], y[2], y[3]);
    else store4_bf16((uint16_t*)out + (size_t)row * N + n0, y);
  }
}

// h[row] += y (bf16 residual stream, updated in place); then xr = fp16(H(rmsnorm(h) * w * suh_next)).
// norm_w == nullptr skips the norm, suh_next == nullptr skips the rotation output entirely (residual update only).
// The products with suh_next stay plain: they are fused into the rotation's first additions, here and in norm_rot_in_kernel alike (a norm weight times
// a scale that is not +-1 has more bits than fp32 holds).
__global__ void __launch_bounds__(1024) finish_add_norm_rot_kernel(const float* __restrict__ part, int S, int M, int N, const __half* __restrict__ svh,
                                           const float* __restrict__ bias, uint16_t* __restrict__ h, const uint16_t* __restrict__ norm_w,
                                           float eps, const __half* __restrict__ suh_next, __half* __restrict__ xr,
                                           uint16_t* __restrict__ xn_out) {
  pdl_launch();
  pdl_wait();
  extern __shared__ float rowbuf[];  // N floats: the updated residual row (as stored, bf16-rounded)
  __shared__ float blk_ss[512];      // per-128-block sums of squares, added in block order (independent of the block size)
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int b = warp; b < N / 128; b += nw) {
    float ss = 0.f;
    const int n0 = b * 128 + lane * 4;
    float y[4], r[4];
    finish_block(part, S, (size_t)M * N, (size_t)row * N + n0, svh, bias, n0, y);
    load4_bf16(h + (size_t)row * N + n0, r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      r[i] = bf16_to_f(f_to_bf16(r[i] + y[i]));
      ss = __fmaf_rn(r[i], r[i], ss);
      rowbuf[n0 + i] = r[i];
    }
    store4_bf16(h + (size_t)row * N + n0, r);
    ss = warp_sum(ss);
    if (lane == 0) blk_ss[b] = ss;
  }
  if (suh_next == nullptr && xn_out == nullptr) return;
  float rinv = 1.f;
  __syncthreads();  // orders the rowbuf / blk_ss writes before the reads below
  if (norm_w != nullptr) {
    float tot = 0.f;
    for (int b = 0; b < N / 128; ++b) tot += blk_ss[b];
    rinv = rsqrtf(tot / (float)N + eps);
  }
  for (int b = warp; b < N / 128; b += nw) {
    const int n0 = b * 128 + lane * 4;
    float v[4], s[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = rowbuf[n0 + i];
    if (suh_next != nullptr) load4_f16(suh_next + n0, s);
    if (norm_w != nullptr) {
      float w[4];
      load4_bf16(norm_w + n0, w);
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = __fmul_rn(bf16_to_f(f_to_bf16(v[i] * rinv)), w[i]);
    }
    if (xn_out != nullptr) store4_bf16(xn_out + (size_t)row * N + n0, v);   // the normalised row itself (router input, per-expert rotations)
    if (suh_next == nullptr) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] *= s[i];
    fwht128_warp(v);
    store4_f16(xr + (size_t)row * N + n0, v);
  }
}

// The same for the rows of a decode window, bound by latency: one SM is slow to fetch the planes of a row (7 x 5120 floats), and 32 warps need two passes
// over its 40 blocks.  So a cluster of four CTAs takes a row, a warp one 128-block of it, kept in registers; the blocks' sums of squares reach every
// CTA through the cluster's shared memory and are added there in block order.  The weights are loaded before the wait for the predecessor.
// One row of 5120 in 7 planes 3.2 us, 5.8 by one CTA; 64 rows 4.0 and 6.0 (launch included); clusters of eight 3.0 and 4.7.
constexpr int FEW_CTAS = 4, FEW_WARPS = 16;
__global__ void __cluster_dims__(FEW_CTAS, 1, 1) __launch_bounds__(FEW_WARPS * 32) finish_add_norm_rot_few_kernel(
    const float* __restrict__ part, int S, int M, int N, const __half* __restrict__ svh, const float* __restrict__ bias, uint16_t* __restrict__ h,
    const uint16_t* __restrict__ norm_w, float eps, const __half* __restrict__ suh_next, __half* __restrict__ xr, uint16_t* __restrict__ xn_out) {
  pdl_launch();
  __shared__ float blk_ss[FEW_CTAS * FEW_WARPS];
  const int row = blockIdx.x / FEW_CTAS, rank = blockIdx.x % FEW_CTAS, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = N / 128;
  const int b = rank * (blockDim.x >> 5) + warp, n0 = b * 128 + lane * 4;
  const bool live = b < nb, out = suh_next != nullptr || xn_out != nullptr, sums = out && norm_w != nullptr;
  if (sums) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // every CTA of the cluster has begun: its shared memory may be written
  alignas(16) float bi[4] = {};
  float sv[4] = {}, w[4] = {}, s[4] = {};
  if (live) {
    load4_f16(svh + n0, sv);
    if (bias != nullptr) *reinterpret_cast<float4*>(bi) = *reinterpret_cast<const float4*>(bias + n0);
    if (sums) load4_bf16(norm_w + n0, w);
    if (suh_next != nullptr) load4_f16(suh_next + n0, s);
  }
  pdl_wait();
  float r[4] = {};
  if (live) {
    float y[4];
    load4_bf16(h + (size_t)row * N + n0, r);
    sum_planes(part, S, (size_t)M * N, (size_t)row * N + n0, y);
    fwht128_warp(y);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      y[i] = __fmul_rn(y[i], sv[i]);
      if (bias != nullptr) y[i] += bi[i];
      r[i] = bf16_to_f(f_to_bf16(r[i] + y[i]));
    }
    store4_bf16(h + (size_t)row * N + n0, r);
  }
  if (!out) return;
  float rinv = 1.f;
  if (sums) {
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) ss = __fmaf_rn(r[i], r[i], ss);
    ss = warp_sum(ss);
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (live && lane < FEW_CTAS)
      asm volatile("{.reg .b32 a; mapa.shared::cluster.u32 a, %0, %1; st.shared::cluster.f32 [a], %2;}" ::"r"(smem_u32(&blk_ss[b])), "r"(lane), "f"(ss) : "memory");
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    float tot = 0.f;
    for (int i = 0; i < nb; ++i) tot += blk_ss[i];
    rinv = rsqrtf(tot / (float)N + eps);
  }
  if (!live) return;
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = sums ? __fmul_rn(bf16_to_f(f_to_bf16(r[i] * rinv)), w[i]) : r[i];
  if (xn_out != nullptr) store4_bf16(xn_out + (size_t)row * N + n0, v);
  if (suh_next == nullptr) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] *= s[i];
  fwht128_warp(v);
  store4_f16(xr + (size_t)row * N + n0, v);
}

// The same for the many rows of a prompt slice (one plane, rows of up to ROWS_MAX elements): a CTA per row, eight lanes to a 128-block and ROWS_NB blocks to a
// lane, which stay in registers between the sum of squares and the scaling, all of them loaded before the first is used.  By warps, a block each, it was
// bound by the shuffles of its two transforms: 8192 rows of 5120 122 us, 96 now; 900 rows of 4096 24.6 -> 16.4.
constexpr int ROWS_NB = 2, ROWS_MAX = 5120;
__global__ void __launch_bounds__(ROWS_MAX / 16 / ROWS_NB) finish_add_norm_rot_rows_kernel(const float* part, int N, const __half* __restrict__ svh,
                                                                      const float* __restrict__ bias, uint16_t* h,
                                                                      const uint16_t* __restrict__ norm_w, float eps, const __half* __restrict__ suh_next,
                                                                      __half* __restrict__ xr, uint16_t* __restrict__ xn_out) {
  pdl_launch();
  pdl_wait();
  __shared__ float blk_ss[ROWS_MAX / 128];
  const int row = blockIdx.x, nb = N / 128, groups = blockDim.x / 8, grp = threadIdx.x >> 3, l4 = (threadIdx.x & 7) * 4;
  const size_t base = (size_t)row * N + l4;
  float v[ROWS_NB][4][4], r[ROWS_NB][4][4];
#pragma unroll
  for (int i = 0; i < ROWS_NB; ++i) {
    const int b = min(grp + groups * i, nb - 1);          // (past the end the last block again: nothing of it is stored)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 p = *reinterpret_cast<const float4*>(part + base + b * 128 + 32 * j);
      v[i][j][0] = p.x, v[i][j][1] = p.y, v[i][j][2] = p.z, v[i][j][3] = p.w;
      load4_bf16(h + base + b * 128 + 32 * j, r[i][j]);
    }
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < ROWS_NB; ++i) {
    const int b = grp + groups * i, n0 = min(b, nb - 1) * 128 + l4;
    fwht128_oct(v[i]);
    float ss[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float sv[4];
      load4_f16(svh + n0 + 32 * j, sv);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[i][j][e] = __fmul_rn(v[i][j][e], sv[e]);
      if (bias != nullptr) {
        const float4 bb = *reinterpret_cast<const float4*>(bias + n0 + 32 * j);
        v[i][j][0] += bb.x, v[i][j][1] += bb.y, v[i][j][2] += bb.z, v[i][j][3] += bb.w;
      }
      ss[j] = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[i][j][e] = bf16_to_f(f_to_bf16(r[i][j][e] + v[i][j][e]));
        ss[j] = __fmaf_rn(v[i][j][e], v[i][j][e], ss[j]);
      }
      if (b < nb) store4_bf16(h + base + b * 128 + 32 * j, v[i][j]);
    }
    float sum = (ss[0] + ss[2]) + (ss[1] + ss[3]);         // warp_sum's order over the 32 fours of a block
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (l4 == 0 && b < nb) blk_ss[b] = sum;
  }
  if (suh_next == nullptr && xn_out == nullptr) return;
  float rinv = 1.f;
  __syncthreads();
  if (norm_w != nullptr) {
    float tot = 0.f;
    for (int b = 0; b < nb; ++b) tot += blk_ss[b];
    rinv = rsqrtf(tot / (float)N + eps);
  }
#pragma unroll
  for (int i = 0; i < ROWS_NB; ++i) {
    const int b = grp + groups * i, n0 = min(b, nb - 1) * 128 + l4;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (norm_w != nullptr) {
        float w[4];
        load4_bf16(norm_w + n0 + 32 * j, w);
#pragma unroll
        for (int e = 0; e < 4; ++e) v[i][j][e] = __fmul_rn(bf16_to_f(f_to_bf16(v[i][j][e] * rinv)), w[e]);
      }
      if (xn_out != nullptr && b < nb) store4_bf16(xn_out + base + b * 128 + 32 * j, v[i][j]);
    }
    if (suh_next == nullptr) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float s[4];
      load4_f16(suh_next + n0 + 32 * j, s);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[i][j][e] *= s[e];
    }
    fwht128_oct(v[i]);
    if (b < nb)
#pragma unroll
      for (int j = 0; j < 4; ++j) store4_f16(xr + base + b * 128 + 32 * j, v[i][j]);
  }
}

// part [S, M, 2F] = gate | up.  act = silu(gate) * up (bf16-rounded like an unfused pipeline would store it), then
// xr[row][F] = fp16(H(act * suh_down)).
template <bool ONE>
__global__ void __launch_bounds__(256) finish_swiglu_rot_kernel(const float* __restrict__ part, int S, int M, int F, const __half* __restrict__ svh,
                                         const float* __restrict__ bias, const __half* __restrict__ suh_down, __half* __restrict__ xr) {
  pdl_launch();
  pdl_wait();
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int N = 2 * F;
  for (int b = blockIdx.y * nw + warp; b < F / 128; b += gridDim.y * nw) {
    const int n0 = b * 128 + lane * 4;
    float g[4], u[4], s[4];
    finish_block<ONE>(part, S, (size_t)M * N, (size_t)row * N + n0, svh, bias, n0, g);
    finish_block<ONE>(part, S, (size_t)M * N, (size_t)row * N + F + n0, svh, bias, F + n0, u);
    load4_f16(suh_down + n0, s);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float a = g[i] / (1.f + __expf(-g[i])) * u[i];
      g[i] = bf16_to_f(f_to_bf16(a)) * s[i];
    }
    fwht128_warp(g);
    store4_f16(xr + (size_t)row * F + n0, g);
  }
}

}  // namespace rx

using namespace rx;

RX_API int rx_exl3_unpack(const void* trellis, int K, int N, int twice, int codebook, void* w_f16, void* stream) {
  if (K % 16 || N % 16) return (int)cudaErrorInvalidValue;
  const int kt = K / 16, nt = N / 16, tiles = kt * nt;
  cudaStream_t st = (cudaStream_t)stream;
  const dim3 grid((tiles + 31) / 32), block(128);
#define RX_GO(CBV) RX_DISPATCH_TWICE(twice, rx::launch(unpack_kernel<T_, CBV>, dim3(grid), dim3(block), 0, st, (const uint32_t*)trellis, (__half*)w_f16, kt, nt))
  switch (codebook) {
    case CB_3INST: RX_GO(CB_3INST); break;
    case CB_MCG: RX_GO(CB_MCG); break;
    case CB_MUL1: RX_GO(CB_MUL1); break;
    default: return (int)cudaErrorInvalidValue;
  }
#undef RX_GO
  return (int)cudaGetLastError();
}

RX_API int rx_embed(const void* ids, const void* table, void* h, int rows, int d, int vocab, void* stream) {
  if (d % 8) return (int)cudaErrorInvalidValue;
  rx::launch(embed_kernel, dim3(rows), dim3(128), 0, (cudaStream_t)stream, (const int*)ids, (const uint16_t*)table, (uint16_t*)h, d, vocab);
  return (int)cudaGetLastError();
}

// Eight lanes a block from 8192 blocks on (8192 rows of 4096 32.9 -> 27.3 us, 512 rows of 8192 7.0 -> 5.3), of rows of up to 1024 from 16,384 (1500 of 1024 level, 1024
// 3.1 us by a warp a block and 3.3).  Not from 149 to 296 rows of up to 8192, which the form below has in one wave of two CTAs per SM (256 of 4096 2.5 and 3.4 us).
RX_API int rx_rot_in_by_lanes(int rows, int K) {
  return (long long)rows * (K / 128) >= (K <= 1024 ? 16384 : 8192) && (rows <= 148 || rows > 296 || K > 8192);
}

RX_API int rx_norm_rot_in(const void* x_bf16, const void* norm_w_bf16, float eps, const void* suh, void* xr, int rows, int K, void* stream) {
  if (K % 128 || K / 128 > 512) return (int)cudaErrorInvalidValue;
  const long long blocks = (long long)rows * (K / 128);
  if (norm_w_bf16 == nullptr && rx_rot_in_by_lanes(rows, K)) {
    rx::launch(rot_in_rows_kernel, dim3((unsigned)((blocks + 31) / 32)), dim3(256), 0, (cudaStream_t)stream, (const uint16_t*)x_bf16, (const __half*)suh, (__half*)xr,
               blocks, K / 128);
    return (int)cudaGetLastError();
  }
  rx::launch(norm_rot_in_kernel, dim3(rows), dim3(rows >= 512 ? 256 : 1024), 0, (cudaStream_t)stream, (const uint16_t*)x_bf16, (const uint16_t*)norm_w_bf16, eps, (const __half*)suh,
                                                            (__half*)xr, K);
  return (int)cudaGetLastError();
}

static int blocks_y(int rows, int nblocks128) {
  // one warp per 128-block (8 warps per CTA): the kernels without a row-wide reduction get their memory-level parallelism
  // from many resident warps with one or two loads each.  For a few rows that means one CTA per 8 blocks; for a prefill
  // chunk of thousands of rows the CTAs take several blocks each instead (a grid of 10^5 very short CTAs is bound by the
  // rate at which CTAs can be launched, not by memory).
  int per_row = (nblocks128 + 7) / 8;
  if (per_row < 1) per_row = 1;
  int cap = 16384 / (rows < 1 ? 1 : rows);
  if (cap < 1) cap = 1;
  return per_row < cap ? per_row : cap;
}

RX_API int rx_finish_store(const void* part, int S, int M, int N, const void* svh, const void* bias, void* out, int f32_out, void* stream) {
  if (N % 128) return (int)cudaErrorInvalidValue;
  dim3 grid(M, blocks_y(M, N / 128));
  rx::launch(S == 1 ? finish_store_kernel<true> : finish_store_kernel<false>, dim3(grid), dim3(256), 0, (cudaStream_t)stream, (const float*)part, S, M, N, (const __half*)svh, (const float*)bias, out, f32_out);
  return (int)cudaGetLastError();
}

// Whether a prompt slice of one plane goes by the row form.  The general form below has up to 296 rows in one wave of two CTAs of 1024 threads per SM, and from 512 on,
// where its CTAs are smaller, up to 592 in one wave again; rows wider than 4096 take it a second pass.  us, general and row form: 149 rows of 4224 9.5 and 6.9, 296 of
// 2048 6.0 and 6.4, 297 8.1 and 7.0, 511 10.3 and 7.2, 592 6.4 and 7.6, 593 8.5 and 7.6; 296 of 4096 7.1 and 8.2, 297 9.9 and 7.6, 592 10.3 and 8.5.
RX_API int rx_add_norm_rot_by_rows(int M, int N) {
  if (N <= 1024 || N > ROWS_MAX) return 0;
  return N > 4096 ? M > 148 : M > 296 && (N > 2048 || M < 512 || M > 592);
}

RX_API int rx_finish_add_norm_rot(const void* part, int S, int M, int N, const void* svh, const void* bias, void* h_bf16, const void* norm_w,
                                  float eps, const void* suh_next, void* xr, void* stream, void* xn_out) {
  if (N % 128 || N * 4 > 200 * 1024 || N / 128 > 512) return (int)cudaErrorInvalidValue;
  if (S == 1 && rx_add_norm_rot_by_rows(M, N)) {
    rx::launch(finish_add_norm_rot_rows_kernel, dim3(M), dim3((N / 128 + 4 * ROWS_NB - 1) / (4 * ROWS_NB) * 32), 0, (cudaStream_t)stream, (const float*)part, N, (const __half*)svh, (const float*)bias,
               (uint16_t*)h_bf16, (const uint16_t*)norm_w, eps, (const __half*)suh_next, (__half*)xr, (uint16_t*)xn_out);
    return (int)cudaGetLastError();
  }
  // Up to 64 rows (256 CTAs) the clusters are the faster form of rows of 4096 and more, up to 16 rows also of shorter ones, which one CTA has in one
  // pass: 37 rows of 2048 in 18 planes take 4.65 us by clusters, 4.40 otherwise; 37 rows of 4096 in 9 planes 4.75 and 5.10; 74 of 5120 6.5 and 6.1.
  if ((N >= 4096 ? M <= 64 : M <= 16) && N <= FEW_CTAS * FEW_WARPS * 128) {
    const int warps = (N / 128 + FEW_CTAS - 1) / FEW_CTAS;
    rx::launch(finish_add_norm_rot_few_kernel, dim3(M * FEW_CTAS), dim3(warps * 32), 0, (cudaStream_t)stream, (const float*)part, S, M, N, (const __half*)svh,
               (const float*)bias, (uint16_t*)h_bf16, (const uint16_t*)norm_w, eps, (const __half*)suh_next, (__half*)xr, (uint16_t*)xn_out);
    return (int)cudaGetLastError();
  }
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(finish_add_norm_rot_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  // a window of a few rows wants every row finished fast (1024 threads per row); a prefill chunk wants many rows in flight per SM
  const int threads = M >= 512 ? 256 : 1024;
  rx::launch(finish_add_norm_rot_kernel, dim3(M), dim3(threads), (size_t)N * 4, (cudaStream_t)stream, (const float*)part, S, M, N, (const __half*)svh, (const float*)bias,
                                                                     (uint16_t*)h_bf16, (const uint16_t*)norm_w, eps, (const __half*)suh_next,
                                                                     (__half*)xr, (uint16_t*)xn_out);
  return (int)cudaGetLastError();
}

RX_API int rx_finish_swiglu_rot(const void* part, int S, int M, int F, const void* svh, const void* bias, const void* suh_down, void* xr,
                                void* stream) {
  if (F % 128) return (int)cudaErrorInvalidValue;
  dim3 grid(M, blocks_y(M, F / 128));
  rx::launch(S == 1 ? finish_swiglu_rot_kernel<true> : finish_swiglu_rot_kernel<false>, dim3(grid), dim3(256), 0, (cudaStream_t)stream, (const float*)part, S, M, F, (const __half*)svh, (const float*)bias,
                                                                  (const __half*)suh_down, (__half*)xr);
  return (int)cudaGetLastError();
}

// Turn programmatic dependent launch on (1, default) or off (0) for every later launch of this library.
RX_API int rx_set_pdl(int on) {
  rx::pdl_enabled() = on ? 1 : 0;
  return 0;
}
