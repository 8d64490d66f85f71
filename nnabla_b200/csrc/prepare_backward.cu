// Operand preparation for the convolution backward passes. Both passes run on
// the implicit-GEMM contraction kernel of the forward; these kernels only
// bring the gradients and activations into the layouts that kernel reads.
//
//   input gradient:  dx = conv(dy stuffed with the forward stride, flipped
//                    and transposed weights)          -> dy_to_nhwc_stuffed,
//                                                        flip_transpose_weights
//   weight gradient: dW[o, c, ky, kx] = sum over (n, oy, ox) = a convolution of
//                    x^T (batch as the channel axis) with dy^T as the filter,
//                    stride and dilation exchanged     -> batch_to_inner
//   bias gradient:   sums of dy over batch and pixels  -> channel_sums
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "pdl.cuh"
#include "prepare.cuh"

namespace nb200 {
namespace {

__device__ __forceinline__ void split3(float v, __nv_bfloat16 &h, __nv_bfloat16 &m, __nv_bfloat16 &l) {
  h = __float2bfloat16_rn(v);
  const float r1 = __fsub_rn(v, __bfloat162float(h));
  m = __float2bfloat16_rn(r1);
  const float r2 = __fsub_rn(r1, __bfloat162float(m));
  l = __float2bfloat16_rn(r2);
}

// dy [N][Ko][Ho][Wo] fp32 -> three bf16 planes [N][Hs][Ws][ctot]: map o of group g
// lands at slot g * k_pad_g + (o - g * Kog), pixel (oy, ox) at (oy * sh, ox * sw);
// every other position of the (pre-zeroed) output stays zero. chan_scale (per
// map, may be NULL) is multiplied in first with one rounding: dy * alpha.
__global__ void __launch_bounds__(256) dy_to_nhwc_stuffed_kernel(const float *__restrict__ dy, int Ko, int Ho, int Wo,
                                                                 int groups, int Kog, int k_pad_g, int ctot, int Hs,
                                                                 int Ws, int sh, int sw,
                                                                 const float *__restrict__ chan_scale,
                                                                 __nv_bfloat16 *__restrict__ out,
                                                                 int64_t plane_stride) {
  pdl_wait();
  pdl_trigger();
  __shared__ float tile[32][33];
  const int n = blockIdx.z;
  const int HW = Ho * Wo;
  const int p0 = blockIdx.x * 32, d0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int dd = ty; dd < 32; dd += 8) {
    const int d = d0 + dd, p = p0 + tx;
    const int g = d / k_pad_g, oo = d - g * k_pad_g;
    float v = 0.0f;
    if (d < ctot && g < groups && oo < Kog && p < HW) {
      const int o = g * Kog + oo;
      v = dy[((int64_t)n * Ko + o) * HW + p];
      if (chan_scale)
        v = __fmul_rn(v, chan_scale[o]);
    }
    tile[dd][tx] = v;
  }
  __syncthreads();
  for (int pp = ty; pp < 32; pp += 8) {
    const int p = p0 + pp, d = d0 + tx;
    if (p < HW && d < ctot) {
      const int oy = p / Wo, ox = p - oy * Wo;
      const int64_t dst = (((int64_t)n * Hs + (int64_t)oy * sh) * Ws + (int64_t)ox * sw) * ctot + d;
      __nv_bfloat16 h, m, l;
      split3(tile[tx][pp], h, m, l);
      out[dst] = h;
      out[plane_stride + dst] = m;
      out[2 * plane_stride + dst] = l;
    }
  }
}

// parts[n][gridDim.x]: the bits of the largest magnitude of image n's shares (non-negative floats order like their bits; a
// NaN ends above infinity). HBM-bound, four loads in flight per thread.
__global__ void __launch_bounds__(256) image_absmax_kernel(const float *__restrict__ x, int64_t per_image,
                                                           uint32_t *__restrict__ parts) {
  pdl_wait();
  pdl_trigger();
  const float *xs = x + (int64_t)blockIdx.y * per_image;
  const int64_t begin = per_image / 4 * blockIdx.x / gridDim.x * 4;
  const int64_t end = blockIdx.x + 1 == gridDim.x ? per_image : per_image / 4 * (blockIdx.x + 1) / gridDim.x * 4;
  uint32_t m = 0;
  if (((reinterpret_cast<uintptr_t>(x) & 15) | (per_image & 3)) == 0) {
#pragma unroll 4
    for (int64_t i = begin + 4 * threadIdx.x; i < end; i += 1024) {
      const float4 v = __ldg(reinterpret_cast<const float4 *>(xs + i));
      m = max(max(m, __float_as_uint(fabsf(v.x))), max(__float_as_uint(fabsf(v.y)), __float_as_uint(fabsf(v.z))));
      m = max(m, __float_as_uint(fabsf(v.w)));
    }
  } else {
#pragma unroll 8
    for (int64_t i = begin + threadIdx.x; i < end; i += 256)
      m = max(m, __float_as_uint(fabsf(__ldg(xs + i))));
  }
  m = __reduce_max_sync(0xffffffffu, m);
  __shared__ uint32_t warps[8];
  if ((threadIdx.x & 31) == 0)
    warps[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = __reduce_max_sync(0xffffffffu, threadIdx.x < 8 ? warps[threadIdx.x] : 0u);
    if (threadIdx.x == 0)
      parts[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = m;
  }
}

// src [N][C][HW] fp32 -> channel-last bf16 planes [planes][N][HW][ctot]: the pieces (hi, mid, lo) of every value, channel
// c of group g at slot g * c_pad_g + c - g * Cg, all other slots zero. `scaled` receives the pieces of
// src * chan_scale[c] (one rounding: dy * alpha), `plain` those of src itself; either may be NULL, so that dy is read
// once for both gradients. HBM-bound: 4 B read and 2 B per piece written per value. Blocks of 64 pixels x 64 slots, a
// thread converts four slots of four pixels; a pixel's row of 64 slots is transposed through shared memory in 16-byte
// chunks (XORed with the pixel quad, at most two lanes to a bank) and leaves as 128 bytes.
// kHalf: two fp16 pieces of src * 2^-e with e from the image's largest magnitude, the maximum of image_parts[n][parts],
// left in image_max[n]. The images go last to first, against the order that the maxima were taken in, so that most of
// them still come from L2: [128, 256, 28, 28] 50 us for the two passes (82 us with the maximum of the whole tensor and
// 4-byte stores).
struct NhwcPieces {
  const float *src;
  int N, C, HW, groups, Cg, c_pad_g, ctot;
  const float *chan_scale;
  uint16_t *scaled, *plain;
  const uint32_t *image_parts; // kHalf
  int parts;
  uint32_t *image_max;
  float *sums; // not kHalf: the channels' sums over each tile's pixels, [N * tiles_x][C], or NULL
  __host__ __device__ int tiles_x() const { return (HW + 63) / 64; }
  __host__ __device__ int tiles_y() const { return (ctot + 63) / 64; }
  __host__ __device__ int64_t blocks() const { return (int64_t)tiles_x() * tiles_y() * N; }
  bool vec() const { return HW % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0; }
};

template <bool kVec, int PLANES, bool kHalf>
__device__ __forceinline__ void nhwc_pieces_tile(const NhwcPieces &P, int block, uint4 (*tile)[64][8]) {
  const float *__restrict__ src = P.src;
  const float *__restrict__ chan_scale = P.chan_scale;
  const uint32_t *__restrict__ image_parts = P.image_parts;
  uint16_t *__restrict__ scaled = P.scaled, *__restrict__ plain = P.plain;
  const int C = P.C, HW = P.HW, groups = P.groups, Cg = P.Cg, c_pad_g = P.c_pad_g, ctot = P.ctot, parts = P.parts;
  const int64_t plane_stride = (int64_t)P.N * HW * ctot;
  const int tx = P.tiles_x(), ty = P.tiles_y();
  const int bx = block % tx, by = block / tx % ty, bz = block / (tx * ty);
  const int n = kHalf ? P.N - 1 - bz : bz, p0 = bx * 64, d0 = by * 64;
  const int px4 = threadIdx.x & 15, chq = threadIdx.x >> 4;
  const int p = p0 + 4 * px4, dq = d0 + 4 * chq;
  const int g = dq / c_pad_g, cc0 = dq - g * c_pad_g; // c_pad_g is a multiple of 16: one group for the four slots
  const bool ok = dq < ctot && g < groups;
  const float *base = src + ((int64_t)n * C + (g * Cg + cc0)) * HW + p;
  float down = 1.0f;
  if (kHalf) {
    uint32_t m = 0;
    for (int i = threadIdx.x & 31; i < parts; i += 32)
      m = max(m, __ldg(image_parts + (int64_t)n * parts + i));
    m = __reduce_max_sync(0xffffffffu, m);
    down = __int_as_float((127 - half_pair_exponent(m)) << 23);
    if (bx == 0 && by == 0 && threadIdx.x == 0)
      P.image_max[n] = m;
  }
  float v[4][4], f[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const bool live = ok && cc0 + r < Cg;
    f[r] = kHalf ? down : live && scaled && chan_scale ? __ldg(chan_scale + g * Cg + cc0 + r) : 1.0f;
    if (kVec) {
      const float4 q = live && p < HW ? __ldcs(reinterpret_cast<const float4 *>(base + (int64_t)r * HW))
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
      v[r][0] = q.x, v[r][1] = q.y, v[r][2] = q.z, v[r][3] = q.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        v[r][k] = live && p + k < HW ? __ldcs(base + (int64_t)r * HW + k) : 0.0f;
    }
  }
  if (!kHalf && P.sums) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float s = (v[r][0] + v[r][1]) + (v[r][2] + v[r][3]);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o);
      if (px4 == 0 && ok && cc0 + r < Cg)
        P.sums[((int64_t)n * tx + bx) * C + g * Cg + cc0 + r] = s;
    }
  }
#pragma unroll
  for (int pass = 0; pass < (kHalf ? 1 : 2); ++pass) {
    uint16_t *out = pass == 0 ? scaled : plain;
    if (!out)
      continue;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint16_t piece[3][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float a = kHalf || (pass == 0 && chan_scale) ? __fmul_rn(v[r][k], f[r]) : v[r][k];
        if (kHalf) {
          const __half h = __float2half_rn(a);
          piece[0][r] = __half_as_ushort(h);
          piece[1][r] = __half_as_ushort(__float2half_rn(__fsub_rn(a, __half2float(h))));
        } else {
          __nv_bfloat16 h, m, l;
          split3(a, h, m, l);
          piece[0][r] = __bfloat16_as_ushort(h);
          piece[1][r] = __bfloat16_as_ushort(m);
          piece[2][r] = __bfloat16_as_ushort(l);
        }
      }
      const int chunk = (chq >> 1) ^ (px4 & 7);
#pragma unroll
      for (int pl = 0; pl < PLANES; ++pl)
        reinterpret_cast<uint2 *>(&tile[pl][4 * px4 + k][chunk])[chq & 1] =
            make_uint2(piece[pl][0] | (uint32_t)piece[pl][1] << 16, piece[pl][2] | (uint32_t)piece[pl][3] << 16);
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int i = threadIdx.x + 256 * it, pp = i >> 3, c = i & 7;
      const int pix = p0 + pp, d = d0 + 8 * c;
      if (pix < HW && d < ctot) {
        const int64_t dst = ((int64_t)n * HW + pix) * ctot + d;
#pragma unroll
        for (int pl = 0; pl < PLANES; ++pl)
          *reinterpret_cast<uint4 *>(out + pl * plane_stride + dst) = tile[pl][pp][c ^ ((pp >> 2) & 7)];
      }
    }
    __syncthreads();
  }
}

template <bool kVec, int PLANES, bool kHalf>
__global__ void __launch_bounds__(256) nhwc_pieces_kernel(const __grid_constant__ NhwcPieces P) {
  __shared__ uint4 tile[PLANES][64][8];
  pdl_wait();
  pdl_trigger();
  nhwc_pieces_tile<kVec, PLANES, kHalf>(P, blockIdx.x, tile);
}

// wb [Ko][Cg][kh][kw] of +-1 (exact in bf16) -> side [C][kh * kw][k_slots] bf16, row g * Cg + c, maps of the group
// innermost, zero past them: the weights of the input gradient, one block per row.
struct TransposedWeights {
  const float *wb;
  int rows, Cg, taps, Kog, k_slots;
  __nv_bfloat16 *side;
};

__device__ __forceinline__ void transpose_binary_weights_row(const TransposedWeights &W, int row) {
  const int g = row / W.Cg, c = row - g * W.Cg, taps = W.taps;
  const float *src = W.wb + ((int64_t)g * W.Kog * W.Cg + c) * taps;
  __nv_bfloat16 *dst = W.side + (int64_t)row * taps * W.k_slots;
#pragma unroll 4
  for (int i = threadIdx.x; i < taps * W.k_slots; i += 256) {
    const int t = i / W.k_slots, o = i - t * W.k_slots;
    dst[i] = o < W.Kog ? __float2bfloat16_rn(__ldg(src + (int64_t)o * W.Cg * taps + t)) : __float2bfloat16_rn(0.0f);
  }
}

// Everything that the two gradients of a convolution read, in one launch: the weights' rows first (short blocks of
// scattered loads), then the pieces of dy and of x. Three launches took 17 to 19 us at 256 maps of 14 x 14 where this takes
// 9.
template <bool kVecDy, bool kVecX, int XP>
__global__ void __launch_bounds__(256) conv_backward_operands_kernel(const __grid_constant__ TransposedWeights W,
                                                                     const __grid_constant__ NhwcPieces dy,
                                                                     const __grid_constant__ NhwcPieces x) {
  __shared__ uint4 tile[3][64][8];
  pdl_wait();
  pdl_trigger();
  int block = blockIdx.x;
  if (block < W.rows)
    return transpose_binary_weights_row(W, block);
  block -= W.rows;
  const int dy_blocks = (int)dy.blocks();
  if (block < dy_blocks)
    nhwc_pieces_tile<kVecDy, 3, false>(dy, block, tile);
  else
    nhwc_pieces_tile<kVecX, XP, false>(x, block - dy_blocks, tile);
}

// wb [Ko][Cg][kh][kw] fp32 -> side [planes][C][kh * kw][k_slots] bf16:
// side[g * Cg + c][ky * kw + kx][o] = wb[g * Kog + o][c][kh - 1 - ky][kw - 1 - kx]; one plane for values
// exact in bf16 (binary weights), three (hi, mid, lo) for full-precision weights.
template <int PLANES>
__global__ void flip_transpose_weights_kernel(const float *__restrict__ wb, int Ko, int Cg, int kh, int kw, int Kog,
                                              int k_slots, __nv_bfloat16 *__restrict__ side, int64_t plane_stride) {
  pdl_wait();
  pdl_trigger();
  const int taps = kh * kw;
  const int64_t total = (int64_t)Ko * Cg * taps;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int t = (int)(i % taps);
    const int c = (int)((i / taps) % Cg);
    const int o = (int)(i / ((int64_t)taps * Cg));
    const int g = o / Kog, oo = o - g * Kog;
    const int ky = t / kw, kx = t - ky * kw;
    const int tf = (kh - 1 - ky) * kw + (kw - 1 - kx);
    const int64_t dst = ((int64_t)(g * Cg + c) * taps + tf) * k_slots + oo;
    if (PLANES == 1) {
      side[dst] = __float2bfloat16_rn(wb[i]);
    } else {
      __nv_bfloat16 h, m, l;
      split3(wb[i], h, m, l);
      side[dst] = h;
      side[dst + plane_stride] = m;
      side[dst + 2 * plane_stride] = l;
    }
  }
}

// src: N rows of R values, rows src_row_stride apart -> out [planes][R][Np] bf16
// (the batch index becomes the innermost axis; positions n >= N stay zero in
// the pre-zeroed output). Tile transpose through shared memory.
template <int PLANES>
__global__ void __launch_bounds__(256) batch_to_inner_kernel(const float *__restrict__ src, int N, int64_t R,
                                                             int64_t src_row_stride, int Np,
                                                             __nv_bfloat16 *__restrict__ out, int64_t plane_stride) {
  pdl_wait();
  pdl_trigger();
  __shared__ float tile[32][33];
  const int64_t r0 = (int64_t)blockIdx.x * 32;
  const int n0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int nn = ty; nn < 32; nn += 8) {
    const int n = n0 + nn;
    const int64_t r = r0 + tx;
    tile[nn][tx] = (n < N && r < R) ? src[(int64_t)n * src_row_stride + r] : 0.0f;
  }
  __syncthreads();
  for (int rr = ty; rr < 32; rr += 8) {
    const int64_t r = r0 + rr;
    const int n = n0 + tx;
    if (r < R && n < N) {
      const int64_t dst = r * Np + n;
      __nv_bfloat16 h, m, l;
      split3(tile[tx][rr], h, m, l);
      out[dst] = h;
      if (PLANES > 1)
        out[plane_stride + dst] = m;
      if (PLANES > 2)
        out[2 * plane_stride + dst] = l;
    }
  }
}

// Sums of dy [N][Ko][HW] over n and the pixels, per map (bias gradient,
// convolution.cpp:281-290): block (o, s) adds the images n = s, s + splits, ...;
// a second kernel adds the partials of each map in order.
__global__ void __launch_bounds__(256) channel_partial_sums_kernel(const float *__restrict__ dy, int N, int Ko, int HW,
                                                                   float *__restrict__ partial) {
  pdl_wait();
  pdl_trigger();
  const int o = blockIdx.x, s = blockIdx.y, splits = gridDim.y;
  float acc = 0.0f;
  for (int n = s; n < N; n += splits) {
    const float *p = dy + ((int64_t)n * Ko + o) * HW;
    for (int i = threadIdx.x; i < HW; i += 256)
      acc += p[i];
  }
  __shared__ float red[256];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int d = 128; d > 0; d >>= 1) {
    if ((int)threadIdx.x < d)
      red[threadIdx.x] += red[threadIdx.x + d];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    partial[(int64_t)s * Ko + o] = red[0];
}

__global__ void channel_finish_kernel(const float *__restrict__ partial, int Ko, int splits, float *__restrict__ out,
                                      int accumulate) {
  pdl_wait();
  pdl_trigger();
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= Ko)
    return;
  float s = 0.0f;
  for (int k = 0; k < splits; ++k)
    s += partial[(int64_t)k * Ko + o];
  out[o] = accumulate ? __fadd_rn(out[o], s) : s;
}

// The same where the pass that converts dy has left its sums, `rows` of them per map: 32 rows by 8 maps per block.
__global__ void __launch_bounds__(256) channel_rows_finish_kernel(const float *__restrict__ partial, int Ko, int rows,
                                                                  float *__restrict__ out, int accumulate) {
  pdl_wait();
  pdl_trigger();
  __shared__ float warps[8][8];
  const int o = blockIdx.x * 8 + (threadIdx.x & 7);
  float s = 0.0f;
  if (o < Ko) {
#pragma unroll 8
    for (int r = threadIdx.x >> 3; r < rows; r += 32)
      s += __ldg(partial + (int64_t)r * Ko + o);
  }
  s += __shfl_xor_sync(0xffffffffu, s, 8);
  s += __shfl_xor_sync(0xffffffffu, s, 16);
  if ((threadIdx.x & 31) < 8)
    warps[threadIdx.x >> 5][threadIdx.x & 7] = s;
  __syncthreads();
  if (threadIdx.x < 8 && o < Ko) {
    s = 0.0f;
    for (int w = 0; w < 8; ++w)
      s += warps[w][threadIdx.x];
    out[o] = accumulate ? __fadd_rn(out[o], s) : s;
  }
}

// staged [splits][Cg][Kog][taps] (the contraction's NCHW-shaped output with the
// input channel as the image axis, one partial result per K split) ->
// dW[o][c][taps]: the splits are added in order, then dW is overwritten or added to.
__global__ void permute_weight_grad_kernel(const float *__restrict__ staged, int splits, int Cg, int Kog, int taps,
                                           float *__restrict__ dw, int accumulate) {
  pdl_wait();
  pdl_trigger();
  const int64_t total = (int64_t)Cg * Kog * taps;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int t = (int)(i % taps);
    const int c = (int)((i / taps) % Cg);
    const int o = (int)(i / ((int64_t)taps * Cg));
    float v = 0.0f;
    for (int k = 0; k < splits; ++k)
      v = __fadd_rn(v, staged[k * total + ((int64_t)c * Kog + o) * taps + t]);
    dw[i] = accumulate ? __fadd_rn(dw[i], v) : v;
  }
}

inline unsigned capped(int64_t work, int threads) {
  int64_t b = (work + threads - 1) / threads;
  const int64_t cap = (int64_t)sm_count() * 32;
  b = b > cap ? cap : b;
  return (unsigned)(b < 1 ? 1 : b);
}

} // namespace

int dy_to_nhwc_stuffed(const float *dy, int N, int Ko, int Ho, int Wo, int groups, int Kog, int k_pad_g, int ctot,
                       int Hs, int Ws, int sh, int sw, const float *chan_scale, void *out, cudaStream_t st) {
  NB_CHECK(N <= 65535, NB200_ENOTIMPL, "batch larger than 65535");
  const dim3 grid((Ho * Wo + 31) / 32, (ctot + 31) / 32, N);
  NB_CUDA(launch_dependent(dy_to_nhwc_stuffed_kernel, grid, dim3(256), 0, st, dy, Ko, Ho, Wo, groups, Kog, k_pad_g,
                           ctot, Hs, Ws, sh, sw, chan_scale, reinterpret_cast<__nv_bfloat16 *>(out), (int64_t)N * Hs *
                           Ws * ctot));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

int nchw_to_nhwc_half_pair_images(const float *x, int N, int C, int HW, int groups, int Cg, int c_pad_g, int ctot,
                                  void *out, uint32_t *image_max, cudaStream_t st) {
  NB_CHECK(N <= 65535, NB200_ENOTIMPL, "batch larger than 65535");
  const int64_t per_image = (int64_t)C * HW;
  // shares of at least 4096 values, not many more than fill the chip twice (a block's start and end cost two microseconds)
  const int64_t most = std::min<int64_t>(kHalfPairParts, 16ll * sm_count() / N);
  const int parts = (int)std::max<int64_t>(1, std::min(per_image / 4096, most));
  NB_CUDA(launch_dependent(image_absmax_kernel, dim3(parts, N), dim3(256), 0, st, x, per_image, image_max + N));
  const NhwcPieces P{x,       N,       C, HW, groups, Cg, c_pad_g, ctot, nullptr, static_cast<uint16_t *>(out),
                     nullptr, image_max + N, parts, image_max, nullptr};
  NB_CHECK(P.blocks() < (1ll << 31), NB200_ENOTIMPL, "tensor too large");
  NB_CUDA(launch_dependent(P.vec() ? nhwc_pieces_kernel<true, 2, true> : nhwc_pieces_kernel<false, 2, true>,
                           dim3((unsigned)P.blocks()), dim3(256), 0, st, P));
  return NB200_OK;
}

int conv_backward_operands(const ConvBackwardOperands &o, cudaStream_t st) {
  const TransposedWeights W{o.wb, o.side ? o.groups * o.Cg : 0, o.Cg, o.taps, o.Kog, o.k_slots,
                            static_cast<__nv_bfloat16 *>(o.side)};
  const NhwcPieces dy{o.dy, o.N, o.groups * o.Kog, o.dy_pixels, o.groups, o.Kog, o.k_pad_g, o.k_total, o.alpha,
                      static_cast<uint16_t *>(o.dy_scaled), static_cast<uint16_t *>(o.dy_plain), nullptr, 0, nullptr, o.dy_sums};
  const NhwcPieces x{o.x, o.x_pieces ? o.N : 0, o.groups * o.Cg, o.x_pixels, o.groups, o.Cg, o.c_pad_g, o.c_total, nullptr,
                     nullptr, static_cast<uint16_t *>(o.x_pieces), nullptr, 0, nullptr, nullptr};
  const int64_t blocks = W.rows + dy.blocks() + x.blocks();
  NB_CHECK(blocks < (1ll << 31), NB200_ENOTIMPL, "tensor too large");
  const bool vd = dy.vec(), vx = x.vec();
  auto kernel = o.x_planes == 3 ? (vd ? (vx ? conv_backward_operands_kernel<true, true, 3> : conv_backward_operands_kernel<true, false, 3>)
                                      : (vx ? conv_backward_operands_kernel<false, true, 3> : conv_backward_operands_kernel<false, false, 3>))
                                : (vd ? (vx ? conv_backward_operands_kernel<true, true, 1> : conv_backward_operands_kernel<true, false, 1>)
                                      : (vx ? conv_backward_operands_kernel<false, true, 1> : conv_backward_operands_kernel<false, false, 1>));
  NB_CUDA(launch_dependent(kernel, dim3((unsigned)blocks), dim3(256), 0, st, W, dy, x));
  return NB200_OK;
}

int flip_transpose_weights(const float *wb, int Ko, int Cg, int kh, int kw, int groups, int k_slots, void *side,
                           cudaStream_t st, int planes) {
  const int64_t plane_stride = (int64_t)groups * Cg * kh * kw * k_slots;
  if (planes == 3)
    NB_CUDA(launch_dependent(flip_transpose_weights_kernel<3>, dim3(capped((int64_t)Ko * Cg * kh * kw, 256)), dim3(256),
                             0, st, wb, Ko, Cg, kh, kw, Ko / groups, k_slots, reinterpret_cast<__nv_bfloat16 *>(side),
                             plane_stride));
  else
    NB_CUDA(launch_dependent(flip_transpose_weights_kernel<1>, dim3(capped((int64_t)Ko * Cg * kh * kw, 256)), dim3(256),
                             0, st, wb, Ko, Cg, kh, kw, Ko / groups, k_slots, reinterpret_cast<__nv_bfloat16 *>(side),
                             plane_stride));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

int batch_to_inner(const float *src, int N, int64_t R, int64_t src_row_stride, int Np, int planes, void *out,
                   cudaStream_t st) {
  NB_CHECK((R + 31) / 32 < (1ll << 31) && (N + 31) / 32 <= 65535, NB200_ENOTIMPL, "tensor too large for the batch transpose");
  const dim3 grid((unsigned)((R + 31) / 32), (unsigned)((N + 31) / 32));
  __nv_bfloat16 *o = reinterpret_cast<__nv_bfloat16 *>(out);
  if (planes == 3)
    NB_CUDA(launch_dependent(batch_to_inner_kernel<3>, grid, dim3(256), 0, st, src, N, R, src_row_stride, Np, o, R *
                             Np));
  else
    NB_CUDA(launch_dependent(batch_to_inner_kernel<1>, grid, dim3(256), 0, st, src, N, R, src_row_stride, Np, o, R *
                             Np));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

int channel_sums(const float *dy, int N, int Ko, int HW, float *out, int accumulate, float *partial, int splits,
                 cudaStream_t st) {
  NB_CHECK(splits >= 1 && splits <= 65535, NB200_EVALUE, "bad split count");
  NB_CUDA(launch_dependent(channel_partial_sums_kernel, dim3(Ko, splits), dim3(256), 0, st, dy, N, Ko, HW, partial));
  NB_LAUNCH_CHECK();
  NB_CUDA(launch_dependent(channel_finish_kernel, dim3((Ko + 255) / 256), dim3(256), 0, st, partial, Ko, splits, out,
                           accumulate));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

int channel_rows_finish(const float *partial, int Ko, int rows, float *out, int accumulate, cudaStream_t st) {
  NB_CUDA(launch_dependent(channel_rows_finish_kernel, dim3((Ko + 7) / 8), dim3(256), 0, st, partial, Ko, rows, out,
                           accumulate));
  return NB200_OK;
}

int permute_weight_grad(const float *staged, int splits, int Cg, int Kog, int taps, float *dw, int accumulate,
                        cudaStream_t st) {
  NB_CUDA(launch_dependent(permute_weight_grad_kernel, dim3(capped((int64_t)Cg * Kog * taps, 256)), dim3(256), 0, st,
                           staged, splits, Cg, Kog, taps, dw, accumulate));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

} // namespace nb200
