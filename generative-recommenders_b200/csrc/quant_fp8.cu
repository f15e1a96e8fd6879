// Block quantiser for the FP8 forward: x [total_L, H, d] (bf16 / f16 / f32) -> e4m3 with one fp32
// scale = absmax / 448 per (128-token block counted from the start of each sequence, head).
// One CTA per (block, head).
//
// 16-bit inputs of head dimension 64 / 128 on the 16-byte grid (what the FP8 forward is fed) run
// quantize_e4m3_vec_kernel: HBM-bound, (2 + 1) bytes per element.  A block is 128 rows of at most
// sixteen 16-byte vectors, so 256 threads hold all of it in eight vectors each: one read, the
// maximum on packed 16-bit values, conversion from registers.  Anything else runs the element-wise
// kernel, which reads the block twice (the second time from L1/L2).
#include <cuda_fp8.h>

#include "common.cuh"

namespace b200hstu {
namespace {

constexpr int QBLOCK = 128;

template <typename E> struct Pair16;
template <> struct Pair16<__nv_bfloat16> { using type = __nv_bfloat162; };
template <> struct Pair16<__half> { using type = __half2; };

__device__ __forceinline__ uint32_t pack_e4m3(float lo, float hi) {
  return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3);
}

template <typename E>
__global__ void __launch_bounds__(256) quantize_e4m3_block_kernel(const E *__restrict__ x, int64_t rs, int64_t hs,
                                                                  uint8_t *__restrict__ x8, float *__restrict__ scale,
                                                                  const int32_t *__restrict__ seq_offsets,
                                                                  const int32_t *__restrict__ block_offsets, int B,
                                                                  int H, int d, int max_seq_len) {
  __shared__ float red[8];
  __shared__ float s_scale;
  const int h = blockIdx.y;
  const int total_blocks = block_offsets[B];
  for (int blk = blockIdx.x; blk < total_blocks; blk += gridDim.x) {
    // sequence that owns this block: last b with block_offsets[b] <= blk
    int lo = 0, hi = B - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (block_offsets[mid] <= blk) lo = mid; else hi = mid - 1;
    }
    const int b = lo;
    const int start = seq_offsets[b], len = seq_offsets[b + 1] - start;
    const int r0 = (blk - block_offsets[b]) * QBLOCK;
    const int nrows = min(QBLOCK, len - r0);
    const int n = nrows * d;
    float amax = 0.f;
    for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
      int r = idx / d, c = idx - r * d;
      amax = fmaxf(amax, fabsf(to_f32(x[(int64_t)(start + r0 + r) * rs + (int64_t)h * hs + c])));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    if (threadIdx.x == 0) {
      float m = red[0];
      for (int w = 1; w < 8; ++w) m = fmaxf(m, red[w]);
      float sc = fmaxf(m, 1e-12f) / 448.f;
      s_scale = sc;
      scale[(int64_t)blk * H + h] = sc;
    }
    __syncthreads();
    const float sc = s_scale;  // true division below: bit-identical to x / scale on the host
    for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
      int r = idx / d, c = idx - r * d;
      float v = to_f32(x[(int64_t)(start + r0 + r) * rs + (int64_t)h * hs + c]) / sc;
      x8[((int64_t)(start + r0 + r) * H + h) * d + c] = (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
    }
    __syncthreads();
  }
}

// Rows are taken by the sequence's own length (a block at the end of a sequence is short); heads of
// one block are neighbours in the grid, so that the CTAs in flight together read whole rows.
// Measured on 977 k tokens x 4 heads x 128 (1.5 GB): 265 us = 5.7 TB/s, against 1904 us element-wise; with
// a division per element 440 us (bound by the XU pipe), with more but spilling warps (48 registers) 320 us.
constexpr int QTHREADS = 256;
template <typename E, int D>
__global__ void __launch_bounds__(QTHREADS, 4) quantize_e4m3_vec_kernel(const E *__restrict__ x, int64_t rs, int64_t hs,
                                                                uint8_t *__restrict__ x8, float *__restrict__ scale,
                                                                const int32_t *__restrict__ seq_offsets,
                                                                const int32_t *__restrict__ block_offsets, int B,
                                                                int H) {
  constexpr int VPR = D / 8;                 // vectors per row
  constexpr int NV = QBLOCK * VPR / QTHREADS;     // vectors per thread
  using E2 = typename Pair16<E>::type;
  __shared__ float red[QTHREADS / 32];
  __shared__ int seg[3];                     // first row of the block in x, its rows, (-1: no such block)
  const int blk = blockIdx.x / H, h = blockIdx.x - blk * H;
  if (threadIdx.x < 32) {
    // the sequence that owns the block: the last b with block_offsets[b] <= blk, found by a 32-way
    // search (two dependent loads for up to 1024 sequences, where halving takes ten)
    int lo = 0, n = B;                       // the answer lies in [lo, lo + n)
    while (n > 1) {
      const int step = (n + 31) / 32;
      const int at = threadIdx.x * step;
      const bool le = at < n && block_offsets[lo + at] <= blk;
      const int last = 31 - __clz(__ballot_sync(0xffffffffu, le) | 1u);
      lo += last * step;
      n = min(step, n - last * step);
    }
    if (threadIdx.x == 0) {
      const int start = seq_offsets[lo], r0 = (blk - block_offsets[lo]) * QBLOCK;
      seg[0] = start + r0;
      seg[1] = blk < block_offsets[B] ? min(QBLOCK, seq_offsets[lo + 1] - start - r0) : -1;
    }
  }
  __syncthreads();
  const int nrows = seg[1];
  if (nrows < 0) return;                     // (rows of `scale` beyond the last block stay as they are)
  const int64_t row0 = seg[0];
  const int c = threadIdx.x % VPR, r = threadIdx.x / VPR;
  constexpr int RSTEP = QTHREADS / VPR;
  const E *src = x + row0 * rs + (int64_t)h * hs + c * 8;
  uint4 v[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int row = r + i * RSTEP;
    v[i] = row < nrows ? __ldcs(reinterpret_cast<const uint4 *>(src + (int64_t)row * rs)) : make_uint4(0, 0, 0, 0);
  }
  E2 m = *reinterpret_cast<const E2 *>(&v[0].x);
  m = __habs2(m);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const E2 *e = reinterpret_cast<const E2 *>(&v[i]);
#pragma unroll
    for (int j = 0; j < 4; ++j) m = __hmax2(m, __habs2(e[j]));
  }
  float amax = fmaxf(to_f32(m.x), to_f32(m.y));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int w = 1; w < QTHREADS / 32; ++w) amax = fmaxf(amax, red[w]);
  const float sc = fmaxf(amax, 1e-12f) / 448.f;
  if (threadIdx.x == 0) scale[(int64_t)blk * H + h] = sc;
  // The result is defined by the true quotient f / sc, rounded to fp32 and then to e4m3.  With the
  // reciprocal rounded to nearest, one residual step gives the same fp32 value as the division
  // (Markstein, IBM J. Res. Dev. 34, 1990) in three instructions: q = f y, q' = q + (q sc - f)(-y).  The
  // residual is taken with that sign so that -0 stays -0: where it vanishes it is +0, its product with -y
  // is -0, and q - 0 = q (with f - q sc the sum -0 + 0 gave +0).  Only results far below e4m3's smallest
  // step can see an underflow in it, and those round to zero either way: the bytes are the division's for
  // every pair of a 16-bit f and a 16-bit maximum.  A block with an infinity has sc = inf and takes the
  // division.
  const float inv = 1.f / sc;
  uint8_t *dst = x8 + (row0 * H + h) * D + c * 8;
  if (!(sc < INFINITY)) {   // (its own loop over memory: inside the one below the compiler divides always)
    for (int row = r; row < nrows; row += RSTEP)
#pragma unroll 1
      for (int j = 0; j < 8; ++j)
        dst[(int64_t)row * H * D + j] =
            (uint8_t)__nv_cvt_float_to_fp8(to_f32(src[(int64_t)row * rs + j]) / sc, __NV_SATFINITE, __NV_E4M3);
    return;
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int row = r + i * RSTEP;
    const E2 *e = reinterpret_cast<const E2 *>(&v[i]);
    float q[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float f = to_f32(j & 1 ? e[j / 2].y : e[j / 2].x);
      const float t = f * inv;
      q[j] = fmaf(fmaf(t, sc, -f), -inv, t);
    }
    uint2 o;
    o.x = pack_e4m3(q[0], q[1]) | pack_e4m3(q[2], q[3]) << 16;
    o.y = pack_e4m3(q[4], q[5]) | pack_e4m3(q[6], q[7]) << 16;
    if (row < nrows) *reinterpret_cast<uint2 *>(dst + (int64_t)row * H * D) = o;
  }
}

template <typename E>
bool launch_vec(const E *x, int64_t rs, int64_t hs, uint8_t *x8, float *scale, const int32_t *seq_offsets,
                const int32_t *block_offsets, int B, int H, int d, int64_t max_blocks, cudaStream_t st) {
  if ((d != 64 && d != 128) || rs % 8 != 0 || hs % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0 ||
      (reinterpret_cast<uintptr_t>(x8) & 7) != 0 || max_blocks * H > 0x7fffffffll)
    return false;
  const unsigned grid = (unsigned)(max_blocks * H);
  if (d == 128)
    quantize_e4m3_vec_kernel<E, 128><<<grid, QTHREADS, 0, st>>>(x, rs, hs, x8, scale, seq_offsets, block_offsets, B, H);
  else
    quantize_e4m3_vec_kernel<E, 64><<<grid, QTHREADS, 0, st>>>(x, rs, hs, x8, scale, seq_offsets, block_offsets, B, H);
  return true;
}

}  // namespace

int quantize_e4m3_block(const void *x, int dtype, int64_t row_stride, int64_t head_stride, void *x8, float *scale,
                        const int32_t *seq_offsets, const int32_t *block_offsets, int B, int H, int d, int64_t total_L,
                        int max_seq_len, cudaStream_t st) {
  int64_t max_blocks = total_L / QBLOCK + B;
  int gx = (int)(max_blocks < 65535 ? max_blocks : 65535);
  if (gx < 1) gx = 1;
  dim3 grid((unsigned)gx, (unsigned)H);
  ProfileScope prof(PROF_QUANT, st);
  switch (dtype) {
    case B200_HSTU_F32:
      quantize_e4m3_block_kernel<float><<<grid, 256, 0, st>>>((const float *)x, row_stride, head_stride, (uint8_t *)x8,
                                                              scale, seq_offsets, block_offsets, B, H, d, max_seq_len);
      break;
    case B200_HSTU_BF16:
      if (launch_vec((const __nv_bfloat16 *)x, row_stride, head_stride, (uint8_t *)x8, scale, seq_offsets,
                     block_offsets, B, H, d, max_blocks, st))
        break;
      quantize_e4m3_block_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16 *)x, row_stride, head_stride,
                                                                      (uint8_t *)x8, scale, seq_offsets, block_offsets,
                                                                      B, H, d, max_seq_len);
      break;
    case B200_HSTU_F16:
      if (launch_vec((const __half *)x, row_stride, head_stride, (uint8_t *)x8, scale, seq_offsets, block_offsets, B,
                     H, d, max_blocks, st))
        break;
      quantize_e4m3_block_kernel<__half><<<grid, 256, 0, st>>>((const __half *)x, row_stride, head_stride,
                                                               (uint8_t *)x8, scale, seq_offsets, block_offsets, B, H,
                                                               d, max_seq_len);
      break;
    default:
      return fail(B200_HSTU_EINVAL, "unknown dtype %d", dtype);
  }
  count_launch();
  B200_CHECK_LAUNCH("e4m3 block quantiser");
  return 0;
}

}  // namespace b200hstu
