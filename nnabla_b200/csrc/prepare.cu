// Operand preparation for the tensor-core contractions (all HBM-bound passes):
//  * weight binarisation fused with the per-output alpha = mean|W| reduction
//    and with the emission of the K-major +-1 side-band the MMA reads,
//  * fp32 -> three bf16 planes (hi, mid, lo with hi + mid + lo == x exactly
//    for normal-range values), optionally with NCHW -> NHWC re-layout,
//  * int8 code transposition.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "prepare.cuh"
#include "pdl.cuh"

namespace nb200 {
namespace {

__device__ __forceinline__ float sign_of(float w, float zero_to) {
  // include/nbla/function/sign.hpp:48-50 (+0, -0 and NaN take zero_to)
  return (w > 0.0f) ? 1.0f : ((w < 0.0f) ? -1.0f : zero_to);
}

// ---------------------------------------------------------------------------
// BinaryWeightAffine / BinaryConnectAffine weights: W is [R, C] row-major, one
// alpha per COLUMN (binary_weight_affine.cpp:83-107). Grid (C/64, R/64);
// each block handles a 64 x 64 tile: reads W coalesced along c, writes Wb
// coalesced, transposes the signs through shared memory and writes the
// side-band [C][Kp] (K = R contiguous) coalesced along r, and stores the
// tile's column sums of |W| to partial[row_block][c]. A second tiny kernel
// sums the partials in a fixed order (deterministic) and scales by 1/R.
// ---------------------------------------------------------------------------
constexpr int kBT = 64;

template <bool kInt8>
__global__ void __launch_bounds__(256) binarize_columns_kernel(const float *__restrict__ w, int R, int C,
                                                               float zero_to, float *__restrict__ wb,
                                                               void *__restrict__ side, int64_t side_pitch,
                                                               float *__restrict__ partial) {
  pdl_wait();
  pdl_trigger();
  __shared__ float s_sign[kBT][kBT + 1];
  __shared__ float s_sum[4][kBT];
  const int c0 = blockIdx.x * kBT, r0 = blockIdx.y * kBT;
  const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6; // 64 x 4
  const int c = c0 + tx;
  float acc = 0.0f;
  for (int rr = ty; rr < kBT; rr += 4) {
    const int r = r0 + rr;
    float s = 0.0f;
    if (r < R && c < C) {
      const float v = w[(int64_t)r * C + c];
      s = sign_of(v, zero_to);
      wb[(int64_t)r * C + c] = s;
      acc += fabsf(v);
    }
    s_sign[rr][tx] = s;
  }
  s_sum[ty][tx] = acc;
  __syncthreads();
  if (partial != nullptr && ty == 0 && c < C)
    partial[(int64_t)blockIdx.y * C + c] = (s_sum[0][tx] + s_sum[1][tx]) + (s_sum[2][tx] + s_sum[3][tx]);
  // side-band: row = output column c, contiguous index = input row r
  for (int cc = ty; cc < kBT; cc += 4) {
    const int oc = c0 + cc, r = r0 + tx;
    if (oc < C && r < R) {
      const float s = s_sign[tx][cc];
      if (kInt8)
        reinterpret_cast<int8_t *>(side)[(int64_t)oc * side_pitch + r] = (int8_t)(int)s;
      else
        reinterpret_cast<__nv_bfloat16 *>(side)[(int64_t)oc * side_pitch + r] = __float2bfloat16_rn(s);
    }
  }
}

// The same with 128-bit accesses (C a multiple of 4, 16-byte aligned W / Wb, side-band rows
// aligned to 8 bytes): a thread handles four columns of a row, and four rows of a side-band row.
template <bool kInt8>
__device__ __forceinline__ void binarize_columns_vec_tile(int bx, int by, const float *__restrict__ w, int R, int C,
                                                          float zero_to, float *__restrict__ wb, void *__restrict__ side,
                                                          int64_t side_pitch, float *__restrict__ partial) {
  __shared__ float s_sign[kBT][kBT + 1];
  __shared__ float s_sum[16][kBT];
  const int c0 = bx * kBT, r0 = by * kBT;
  const int tx4 = threadIdx.x & 15, ty = threadIdx.x >> 4; // 16 column quads x 16 rows
  const int c = c0 + 4 * tx4;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int rr = ty + 16 * it, r = r0 + rr;
    float4 sg = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < R && c < C) { // C % 4 == 0: the quad is inside or outside as a whole
      const float4 v = __ldg(reinterpret_cast<const float4 *>(w + (int64_t)r * C + c));
      sg = make_float4(sign_of(v.x, zero_to), sign_of(v.y, zero_to), sign_of(v.z, zero_to), sign_of(v.w, zero_to));
      *reinterpret_cast<float4 *>(wb + (int64_t)r * C + c) = sg;
      acc[0] += fabsf(v.x), acc[1] += fabsf(v.y), acc[2] += fabsf(v.z), acc[3] += fabsf(v.w);
    }
    s_sign[rr][4 * tx4 + 0] = sg.x;
    s_sign[rr][4 * tx4 + 1] = sg.y;
    s_sign[rr][4 * tx4 + 2] = sg.z;
    s_sign[rr][4 * tx4 + 3] = sg.w;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    s_sum[ty][4 * tx4 + i] = acc[i];
  __syncthreads();
  if (partial != nullptr && threadIdx.x < kBT && c0 + threadIdx.x < C) {
    float t = 0.0f; // fixed order: deterministic
#pragma unroll
    for (int k = 0; k < 16; ++k)
      t += s_sum[k][threadIdx.x];
    partial[(int64_t)by * C + c0 + threadIdx.x] = t;
  }
  // side-band: row = output column, contiguous index = input row; four input rows per thread
  const int r = r0 + 4 * tx4;
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int cc = ty + 16 * it, oc = c0 + cc;
    if (oc >= C || r >= R)
      continue;
    float sv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      sv[i] = (r + i < R) ? s_sign[4 * tx4 + i][cc] : 0.0f;
    if (kInt8) {
      const uint32_t packed = ((uint32_t)(uint8_t)(int8_t)(int)sv[0]) | ((uint32_t)(uint8_t)(int8_t)(int)sv[1] << 8) |
                              ((uint32_t)(uint8_t)(int8_t)(int)sv[2] << 16) | ((uint32_t)(uint8_t)(int8_t)(int)sv[3] << 24);
      *reinterpret_cast<uint32_t *>(reinterpret_cast<int8_t *>(side) + (int64_t)oc * side_pitch + r) = packed;
    } else {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(sv[0], sv[1]), hi = __floats2bfloat162_rn(sv[2], sv[3]);
      uint2 out;
      out.x = *reinterpret_cast<const uint32_t *>(&lo);
      out.y = *reinterpret_cast<const uint32_t *>(&hi);
      *reinterpret_cast<uint2 *>(reinterpret_cast<__nv_bfloat16 *>(side) + (int64_t)oc * side_pitch + r) = out;
    }
  }
}

template <bool kInt8>
__global__ void __launch_bounds__(256) binarize_columns_vec_kernel(const float *__restrict__ w, int R, int C,
                                                                   float zero_to, float *__restrict__ wb,
                                                                   void *__restrict__ side, int64_t side_pitch,
                                                                   float *__restrict__ partial) {
  pdl_wait();
  pdl_trigger();
  binarize_columns_vec_tile<kInt8>(blockIdx.x, blockIdx.y, w, R, C, zero_to, wb, side, side_pitch, partial);
}

__global__ void finalize_alpha_kernel(const float *__restrict__ partial, int blocks, int C, float inv,
                                      float *__restrict__ alpha) {
  pdl_wait();
  pdl_trigger();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C)
    return;
  float s = 0.0f;
  for (int b = 0; b < blocks; ++b)
    s += partial[(int64_t)b * C + c];
  alpha[c] = __fmul_rn(s, inv);
}

// ---------------------------------------------------------------------------
// BinaryWeightConvolution / BinaryConnectConvolution weights: W is
// [Ko, Cg, kh, kw]; one alpha per output map = mean over its Cg*kh*kw taps
// (binary_weight_convolution.cpp:81-102). One block per output map; the
// side-band is [Ko][Kp] with K ordered (ky, kx, c) so that one 128-byte K
// block is one filter tap over consecutive channels, matching the NHWC
// activation planes.
// ---------------------------------------------------------------------------
// Zeros in the channel slots [Cg, c_pad) of every tap of one row of weights (a memset of all weights in front cost 4 us: a
// launch that the ones around it do not overlap).
__device__ __forceinline__ void zero_slots(uint8_t *row, int taps, int Cg, int c_pad, int bytes) {
  const int pad = (c_pad - Cg) * bytes;
  for (int i = threadIdx.x; i < taps * pad; i += 256) {
    const int t = i / pad;
    row[(t * c_pad + Cg) * bytes + (i - t * pad)] = 0;
  }
}

// kMode: 0 = bf16 signs, 1 = int8 signs, 2 = fp16 signs.
template <int kMode>
__device__ __forceinline__ void binarize_row(int o, const float *__restrict__ w, int Cg, int kh, int kw,
                                             float zero_to, float inv, float *__restrict__ wb,
                                             float *__restrict__ alpha, void *__restrict__ side, int64_t side_pitch,
                                             int c_pad) {
  const int taps = kh * kw, Kd = Cg * taps;
  const float *wr = w + (int64_t)o * Kd;
  zero_slots(reinterpret_cast<uint8_t *>(side) + (int64_t)o * side_pitch * (kMode == 1 ? 1 : 2), taps, Cg, c_pad,
             kMode == 1 ? 1 : 2);
  float acc = 0.0f;
  for (int k0 = threadIdx.x; k0 < Kd; k0 += 8 * 256) { // eight loads in flight
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      v[u] = k0 + 256 * u < Kd ? __ldg(wr + k0 + 256 * u) : 0.0f;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + 256 * u;
      if (k >= Kd)
        break;
      const float s = sign_of(v[u], zero_to);
      wb[(int64_t)o * Kd + k] = s;
      acc += fabsf(v[u]);
      const int c = k / taps, t = k - c * taps;
      const int64_t dst = (int64_t)o * side_pitch + (int64_t)t * c_pad + c;
      if (kMode == 1) {
        reinterpret_cast<int8_t *>(side)[dst] = (int8_t)(int)s;
      } else if (kMode == 2) {
        reinterpret_cast<__half *>(side)[dst] = __float2half_rn(s);
      } else {
        reinterpret_cast<__nv_bfloat16 *>(side)[dst] = __float2bfloat16_rn(s);
      }
    }
  }
  if (alpha == nullptr)
    return;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1)
    acc += __shfl_xor_sync(0xffffffffu, acc, d);
  __shared__ float s_part[8];
  if ((threadIdx.x & 31) == 0)
    s_part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.0f;
    for (int i = 0; i < 8; ++i)
      s += s_part[i];
    alpha[o] = __fmul_rn(s, inv);
  }
}

template <int kMode>
__global__ void __launch_bounds__(256) binarize_rows_kernel(const float *__restrict__ w, int Cg, int kh, int kw,
                                                            float zero_to, float inv, float *__restrict__ wb,
                                                            float *__restrict__ alpha, void *__restrict__ side,
                                                            int64_t side_pitch, int c_pad) {
  pdl_wait();
  pdl_trigger();
  binarize_row<kMode>(blockIdx.x, w, Cg, kh, kw, zero_to, inv, wb, alpha, side, side_pitch, c_pad);
}

// Fixed-point convolution weights: wq [Ko, Cg, kh, kw] holds multiples of delta
// (|code| <= 127); the int8 codes go to the same tap-major side-band layout.
__global__ void __launch_bounds__(256) codes_conv_weights_kernel(const float *__restrict__ wq, int Cg, int kh, int kw,
                                                                 float inv_delta, int8_t *__restrict__ side,
                                                                 int64_t side_pitch, int c_pad) {
  pdl_wait();
  pdl_trigger();
  const int o = blockIdx.x;
  const int taps = kh * kw, Kd = Cg * taps;
  const float *wr = wq + (int64_t)o * Kd;
  zero_slots(reinterpret_cast<uint8_t *>(side) + (int64_t)o * side_pitch, taps, Cg, c_pad, 1);
  for (int k = threadIdx.x; k < Kd; k += 256) {
    const int c = k / taps, t = k - c * taps;
    side[(int64_t)o * side_pitch + (int64_t)t * c_pad + c] = (int8_t)__float2int_rn(__fmul_rn(wr[k], inv_delta));
  }
}

// ---------------------------------------------------------------------------
// fp32 [rows, K] -> bf16 planes [3][rows][Kp]: hi = bf16(x), mid = bf16(x - hi),
// lo = bf16(x - hi - mid); the two subtractions are exact in fp32.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void split3(float x, __nv_bfloat16 &h, __nv_bfloat16 &m, __nv_bfloat16 &l) {
  h = __float2bfloat16_rn(x);
  const float r1 = __fsub_rn(x, __bfloat162float(h));
  m = __float2bfloat16_rn(r1);
  const float r2 = __fsub_rn(r1, __bfloat162float(m));
  l = __float2bfloat16_rn(r2);
}

// Four neighbouring values of a row of `extent` floats from column k on, zero past its end; kVec: one 128-bit load
// (the row starts on 16 bytes and extent is a multiple of 4).
template <bool kVec> __device__ __forceinline__ float4 load_quad(const float *__restrict__ row, int k, int extent) {
  if (kVec)
    return k < extent ? __ldcs(reinterpret_cast<const float4 *>(row + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
  return make_float4(k < extent ? row[k] : 0.f, k + 1 < extent ? row[k + 1] : 0.f, k + 2 < extent ? row[k + 2] : 0.f,
                     k + 3 < extent ? row[k + 3] : 0.f);
}

// Up to two operands with rows of Kp values in one launch. A thread takes eight values of a row (Kp is a multiple of 64): two
// 128-bit loads (kVec: K % 4 == 0, 16-byte aligned x) and a 128-bit store per plane. Bound by HBM; with a value per
// thread and a launch per operand the input gradient of a [16, 4096] . [4096, 4096] layer took 104 us, now 27, of
// [256, 1024] . [1024, 4096] 40, now 19.
template <bool kVec>
__global__ void __launch_bounds__(256) split_rows_kernel(const SplitRows A, const SplitRows B, unsigned a_blocks, int64_t Kp) {
  pdl_wait();
  pdl_trigger();
  const SplitRows &P = blockIdx.x < a_blocks ? A : B;
  const unsigned groups = (unsigned)(Kp / 8);
  const int64_t i = (int64_t)(blockIdx.x - (blockIdx.x < a_blocks ? 0u : a_blocks)) * 256 + threadIdx.x;
  const int64_t r = i / groups;
  const int k = 8 * (int)(i - r * groups);
  if (r >= P.rows)
    return;
  const float *src = P.x + r * P.K + k;
  float v[8];
#pragma unroll
  for (int q = 0; q < 8; q += 4) {
    if (kVec) {
      const float4 t = k + q < P.K ? ld_stream(reinterpret_cast<const float4 *>(src + q)) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[q] = t.x, v[q + 1] = t.y, v[q + 2] = t.z, v[q + 3] = t.w;
    } else {
#pragma unroll
      for (int j = q; j < q + 4; ++j)
        v[j] = k + j < P.K ? __ldcs(src + j) : 0.0f;
    }
  }
  if (P.col_scale != nullptr)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      v[j] = __fmul_rn(v[j], k + j < P.K ? __ldg(P.col_scale + k + j) : 1.0f);
  __align__(16) __nv_bfloat16 piece[3][8];
#pragma unroll
  for (int j = 0; j < 8; ++j)
    split3(v[j], piece[0][j], piece[1][j], piece[2][j]);
  __nv_bfloat16 *dst = static_cast<__nv_bfloat16 *>(P.out) + r * Kp + k;
#pragma unroll
  for (int pl = 0; pl < 3; ++pl)
    if (pl < P.planes)
      *reinterpret_cast<uint4 *>(dst + pl * P.rows * Kp) = *reinterpret_cast<const uint4 *>(piece[pl]);
}

// The same for operands along whose rows the product does not contract (x and dy of a weight gradient, plain weights):
// source [rows][cols] -> [planes][cols][Rp], rows padded with zeros to Rp, a multiple of 64. 64 x 64 tiles through shared
// memory, eight rows of a column per thread, 128 bytes of a plane per eight lanes. sums (may be NULL): receives the column
// sums of each tile, [tile row][cols]. With an fp32 transpose first and the split behind it, and dy read again for its
// sums, the weight gradient of [256, 1024] . [1024, 4096] took 43 us, now 24.5; of [1024, 2048] . [2048, 700] 56, now 36.
template <bool kVec>
__global__ void __launch_bounds__(256) split_columns_kernel(const SplitColumns A, const SplitColumns B, unsigned a_blocks,
                                                            int64_t Rp) {
  pdl_wait();
  pdl_trigger();
  __shared__ float tile[64][65];
  const bool first = blockIdx.x < a_blocks;
  const SplitColumns &P = first ? A : B;
  const unsigned b = blockIdx.x - (first ? 0u : a_blocks), row_tiles = (unsigned)(Rp / 64);
  const unsigned rt = b % row_tiles;
  const int r0 = 64 * (int)rt, c0 = 64 * (int)(b / row_tiles);
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int r = (threadIdx.x >> 4) + 16 * it, c = 4 * (threadIdx.x & 15);
    const float *row = P.x + (int64_t)(r0 + r) * P.cols;
    const float4 v = r0 + r < P.rows ? load_quad<kVec>(row, c0 + c, P.cols) : make_float4(0.f, 0.f, 0.f, 0.f);
    tile[r][c] = v.x, tile[r][c + 1] = v.y, tile[r][c + 2] = v.z, tile[r][c + 3] = v.w;
  }
  __syncthreads();
  const int g = threadIdx.x & 7;
  __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(P.out);
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int c = (threadIdx.x >> 3) + 32 * it;
    __align__(16) __nv_bfloat16 piece[3][8];
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float v = tile[8 * g + j][c];
      sum += v;
      split3(v, piece[0][j], piece[1][j], piece[2][j]);
    }
    if (P.sums) {
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (g == 0 && c0 + c < P.cols)
        P.sums[(int64_t)rt * P.cols + c0 + c] = sum;
    }
    if (c0 + c < P.cols)
#pragma unroll
      for (int pl = 0; pl < 3; ++pl)
        if (pl < P.planes)
          *reinterpret_cast<uint4 *>(out + ((int64_t)pl * P.cols + c0 + c) * Rp + r0 + 8 * g) =
              *reinterpret_cast<const uint4 *>(piece[pl]);
  }
}

// Both operands of a binary-weight affine layer in one launch: the weights' 64 x 64 tiles first, then four values of x per
// thread into three bf16 pieces [3][rows][Kp] (Kp a multiple of 64, zero padded; K a multiple of 4, 16-byte aligned).
__global__ void __launch_bounds__(256) binary_affine_operands_kernel(const float *__restrict__ w, int R, int C, float zero_to,
                                                                     float *__restrict__ wb, void *__restrict__ side,
                                                                     int64_t side_pitch, float *__restrict__ partial, int gx,
                                                                     int w_blocks, const float *__restrict__ x, int64_t rows,
                                                                     __nv_bfloat16 *__restrict__ pieces) {
  pdl_wait();
  pdl_trigger();
  if ((int)blockIdx.x < w_blocks) {
    binarize_columns_vec_tile<false>((int)blockIdx.x % gx, (int)blockIdx.x / gx, w, R, C, zero_to, wb, side, side_pitch,
                                     partial);
    return;
  }
  const unsigned quads = (unsigned)(side_pitch / 4); // x's rows are padded like the side-band's
  const int64_t i = (int64_t)(blockIdx.x - w_blocks) * 256 + threadIdx.x;
  const int64_t r = i / quads;
  const int k = 4 * (int)(i - r * quads);
  if (r >= rows)
    return;
  const float4 v = k < R ? __ldcs(reinterpret_cast<const float4 *>(x + r * R + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float e[4] = {v.x, v.y, v.z, v.w};
  __align__(8) __nv_bfloat16 p[3][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    split3(e[j], p[0][j], p[1][j], p[2][j]);
#pragma unroll
  for (int pl = 0; pl < 3; ++pl)
    *reinterpret_cast<uint2 *>(pieces + (pl * rows + r) * side_pitch + k) = *reinterpret_cast<const uint2 *>(p[pl]);
}

// Column sums of a row-major [rows, C] matrix (bias gradient, affine.cpp:130-137):
// block (cx, s) adds its share of the rows for 256 columns (coalesced along the
// columns), a second kernel adds the `splits` partials of each column in order.
__global__ void __launch_bounds__(256) column_partial_sums_kernel(const float *__restrict__ a, int64_t rows, int C,
                                                                  float *__restrict__ partial) {
  pdl_wait();
  pdl_trigger();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= C)
    return;
  const int64_t per = (rows + gridDim.y - 1) / gridDim.y;
  const int64_t r0 = blockIdx.y * per, r1 = (r0 + per < rows) ? r0 + per : rows;
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  int64_t r = r0;
  for (; r + 3 < r1; r += 4) {
    s0 += a[r * C + c];
    s1 += a[(r + 1) * C + c];
    s2 += a[(r + 2) * C + c];
    s3 += a[(r + 3) * C + c];
  }
  for (; r < r1; ++r)
    s0 += a[r * C + c];
  partial[(int64_t)blockIdx.y * C + c] = (s0 + s1) + (s2 + s3);
}

__global__ void __launch_bounds__(256) column_finish_kernel(const float *__restrict__ partial, int C, int splits,
                                                            float *__restrict__ out, int accumulate) {
  pdl_wait();
  pdl_trigger();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= C)
    return;
  float s = 0.f;
  for (int k = 0; k < splits; ++k)
    s += partial[(int64_t)k * C + c];
  out[c] = accumulate ? __fadd_rn(out[c], s) : s;
}

// fp32 NCHW -> planes of NHWC: out[plane][n][hw][ctot], where channel c of
// group g lands at g * c_pad_g + (c - g * Cg) and every other slot is zero.
// Tile transpose through shared memory: reads coalesced along hw, writes
// coalesced along the channel slots. OutT = bf16 (PLANES pieces) or int8
// (codes of values that are multiples of delta).
template <typename OutT, int PLANES>
__global__ void __launch_bounds__(256) nchw_to_nhwc_kernel(const float *__restrict__ x, int C, int HW, int groups,
                                                           int Cg, int c_pad_g, int ctot, OutT *__restrict__ out,
                                                           int64_t plane_stride, float inv_delta) {
  pdl_wait();
  pdl_trigger();
  __shared__ float tile[32][33];
  const int n = blockIdx.z;
  const int p0 = blockIdx.x * 32, d0 = blockIdx.y * 32; // d = destination channel slot
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5; // 32 x 8
  for (int dd = ty; dd < 32; dd += 8) {
    const int d = d0 + dd, p = p0 + tx;
    const int g = d / c_pad_g, cc = d - g * c_pad_g;
    const bool live = d < ctot && g < groups && cc < Cg && p < HW;
    tile[dd][tx] = live ? x[((int64_t)n * C + (g * Cg + cc)) * HW + p] : 0.0f;
  }
  __syncthreads();
  for (int pp = ty; pp < 32; pp += 8) {
    const int p = p0 + pp, d = d0 + tx;
    if (p < HW && d < ctot) {
      const float v = tile[tx][pp];
      const int64_t dst = ((int64_t)n * HW + p) * ctot + d;
      if constexpr (sizeof(OutT) == 1) {
        out[dst] = (OutT)__float2int_rn(__fmul_rn(v, inv_delta)); // v is k * delta
      } else {
        __nv_bfloat16 h, m, l;
        split3(v, h, m, l);
        out[dst] = h;
        if (PLANES > 1)
          out[plane_stride + dst] = m;
        if (PLANES > 2)
          out[2 * plane_stride + dst] = l;
      }
    }
  }
}

// Codes of four multiples of delta as one word: round(v / delta) on the add pipe, where for |t| < 2^22 the low
// byte of 1.5 * 2^23 + t is the two's complement code.
__device__ __forceinline__ uint32_t pack_codes(float a, float b, float c, float d, float inv_delta) {
  const uint32_t i = __float_as_uint(__fadd_rn(__fmul_rn(a, inv_delta), 12582912.0f));
  const uint32_t j = __float_as_uint(__fadd_rn(__fmul_rn(b, inv_delta), 12582912.0f));
  const uint32_t k = __float_as_uint(__fadd_rn(__fmul_rn(c, inv_delta), 12582912.0f));
  const uint32_t l = __float_as_uint(__fadd_rn(__fmul_rn(d, inv_delta), 12582912.0f));
  return __byte_perm(__byte_perm(i, j, 0x0040), __byte_perm(k, l, 0x0040), 0x5410);
}

// fp32 NCHW (multiples of delta) -> int8 NHWC codes, 64 pixels x 64 channel slots per block. A thread converts four
// neighbouring slots of four pixels 16 apart, sixteen loads in flight; the four codes of a pixel go to shared memory as
// one word and leave in 64-byte runs per pixel. For planes that 128-bit loads cannot read (the loop over single values
// with one load in flight took 27 us for [256, 512, 7, 7]).
__device__ __forceinline__ void nchw_to_nhwc_i8_tile(int bx, int by, int n, const float *__restrict__ x, int C, int HW,
                                                     int groups, int Cg, int c_pad_g, int ctot,
                                                     int8_t *__restrict__ out, float inv_delta) {
  __shared__ uint32_t tile[64][17]; // [pixel][16 words of 4 codes + 1 pad]
  const int p0 = bx * 64, d0 = by * 64;
  const int px = threadIdx.x & 15, chq = threadIdx.x >> 4;
  const int dq = d0 + 4 * chq;
  const int g = dq / c_pad_g, cc0 = dq - g * c_pad_g; // c_pad_g is a multiple of 16: one group for the four slots
  const bool ok = dq < ctot && g < groups;
  const float *base = x + ((int64_t)n * C + (g * Cg + cc0)) * HW;
  float v[4][4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int p = p0 + px + 16 * k;
      v[k][r] = ok && cc0 + r < Cg && p < HW ? __ldcs(base + (int64_t)r * HW + p) : 0.0f;
    }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    tile[px + 16 * k][chq] = pack_codes(v[k][0], v[k][1], v[k][2], v[k][3], inv_delta);
  __syncthreads();
  const int word = threadIdx.x & 15, prow = threadIdx.x >> 4; // 16 pixels per pass
#pragma unroll
  for (int pp = prow; pp < 64; pp += 16) {
    const int pix = p0 + pp, d = d0 + 4 * word;
    if (pix < HW && d < ctot)
      *reinterpret_cast<uint32_t *>(out + ((int64_t)n * HW + pix) * ctot + d) = tile[pp][word];
  }
}

__global__ void __launch_bounds__(256) nchw_to_nhwc_i8_kernel(const float *__restrict__ x, int C, int HW, int groups,
                                                              int Cg, int c_pad_g, int ctot,
                                                              int8_t *__restrict__ out, float inv_delta) {
  pdl_wait();
  pdl_trigger();
  nchw_to_nhwc_i8_tile(blockIdx.x, blockIdx.y, blockIdx.z, x, C, HW, groups, Cg, c_pad_g, ctot, out, inv_delta);
}

// Same conversion with 128-bit loads (HW a multiple of 4): every thread has
// four independent float4 loads in flight (4 pixels x 4 channel rows).
__device__ __forceinline__ void nchw_to_nhwc_i8_vec_tile(int bx, int by, int n, const float *__restrict__ x, int C,
                                                         int HW, int groups, int Cg, int c_pad_g, int ctot,
                                                         int8_t *__restrict__ out, float inv_delta) {
  __shared__ uint32_t tile[64][17];
  const int p0 = bx * 64, d0 = by * 64;
  // 16 pixel quads x 16 channel quads: a thread converts four neighbouring channel slots of four pixels, so
  // that the four codes of a pixel leave as one word
  const int px4 = threadIdx.x & 15, chq = threadIdx.x >> 4;
  const int p = p0 + 4 * px4;
  const int dq = d0 + 4 * chq;
  const int g = dq / c_pad_g, cc0 = dq - g * c_pad_g; // c_pad_g is a multiple of 16: one group for the four slots
  const bool ok = dq < ctot && g < groups && p < HW;
  const float *base = x + ((int64_t)n * C + (g * Cg + cc0)) * HW + p;
  // round(v / delta) on the add pipe: for |t| < 2^22 the low mantissa bits of 1.5 * 2^23 + t, rounded to
  // nearest even by the addition itself, are the two's complement integer (its low byte is the code)
  uint32_t f[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ok && cc0 + r < Cg)
      v = __ldcs(reinterpret_cast<const float4 *>(base + (int64_t)r * HW));
    f[r][0] = __float_as_uint(__fadd_rn(__fmul_rn(v.x, inv_delta), 12582912.0f));
    f[r][1] = __float_as_uint(__fadd_rn(__fmul_rn(v.y, inv_delta), 12582912.0f));
    f[r][2] = __float_as_uint(__fadd_rn(__fmul_rn(v.z, inv_delta), 12582912.0f));
    f[r][3] = __float_as_uint(__fadd_rn(__fmul_rn(v.w, inv_delta), 12582912.0f));
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    tile[4 * px4 + k][chq] = __byte_perm(__byte_perm(f[0][k], f[1][k], 0x0040), __byte_perm(f[2][k], f[3][k], 0x0040),
                                         0x5410);
  __syncthreads();
  const int word = threadIdx.x & 15, prow = threadIdx.x >> 4;
#pragma unroll
  for (int pp = prow; pp < 64; pp += 16) {
    const int pix = p0 + pp, d = d0 + 4 * word;
    if (pix < HW && d < ctot)
      *reinterpret_cast<uint32_t *>(out + ((int64_t)n * HW + pix) * ctot + d) = tile[pp][word];
  }
}

__global__ void __launch_bounds__(256) nchw_to_nhwc_i8_vec_kernel(const float *__restrict__ x, int C, int HW,
                                                                  int groups, int Cg, int c_pad_g, int ctot,
                                                                  int8_t *__restrict__ out, float inv_delta) {
  pdl_wait();
  pdl_trigger();
  nchw_to_nhwc_i8_vec_tile(blockIdx.x, blockIdx.y, blockIdx.z, x, C, HW, groups, Cg, c_pad_g, ctot, out, inv_delta);
}

// Both operands of a binary-weight convolution over fixed-point activations in one launch: blocks
// [0, Ko) binarise one filter each (sign, scale, int8 side-band), the others convert one 64 x 64 tile of
// the activations to channel-last codes. The two jobs are independent, and at a few dozen images the
// weights' pass costs as much as the activations': side by side it disappears behind them.
template <bool kVec>
__global__ void __launch_bounds__(256)
    binary_conv_operands_i8_kernel(const float *__restrict__ w, int Ko, int Cg_w, int kh, int kw, float zero_to, float inv,
                                   float *__restrict__ wb, float *__restrict__ alpha, void *__restrict__ side,
                                   int64_t side_pitch, int c_pad, const float *__restrict__ x, int C, int HW,
                                   int groups, int Cg, int c_pad_g, int ctot, int8_t *__restrict__ out,
                                   float inv_delta, int gx, int gy) {
  pdl_wait();
  pdl_trigger();
  if ((int)blockIdx.x < Ko) {
    binarize_row<1>(blockIdx.x, w, Cg_w, kh, kw, zero_to, inv, wb, alpha, side, side_pitch, c_pad);
    return;
  }
  const int lin = (int)blockIdx.x - Ko;
  const int bx = lin % gx, r = lin / gx;
  if (kVec)
    nchw_to_nhwc_i8_vec_tile(bx, r % gy, r / gy, x, C, HW, groups, Cg, c_pad_g, ctot, out, inv_delta);
  else
    nchw_to_nhwc_i8_tile(bx, r % gy, r / gy, x, C, HW, groups, Cg, c_pad_g, ctot, out, inv_delta);
}

// int8 [R, C] -> [C][pitch] (transpose), tile 64 x 64 through shared memory.
__global__ void __launch_bounds__(256) transpose_i8_kernel(const int8_t *__restrict__ src, int R, int C,
                                                           int8_t *__restrict__ dst, int64_t pitch) {
  pdl_wait();
  pdl_trigger();
  __shared__ int8_t tile[64][65];
  const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64;
  const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;
  for (int rr = ty; rr < 64; rr += 4) {
    const int r = r0 + rr, c = c0 + tx;
    tile[rr][tx] = (r < R && c < C) ? src[(int64_t)r * C + c] : (int8_t)0;
  }
  __syncthreads();
  for (int cc = ty; cc < 64; cc += 4) {
    const int c = c0 + cc, r = r0 + tx;
    if (c < C && r < R)
      dst[(int64_t)c * pitch + r] = tile[tx][cc];
  }
}

// Both operands of the 8-bit fixed-point affine in one launch: x [M, K] -> codes [M][Kp] and w [K, N] -> transposed
// codes [N][Kp] (Kp = K rounded up to 128, zero padded). HBM-bound: 5 bytes per value. The last x_blocks blocks: a warp
// converts four runs of 128 values, each one 512-byte load and one 128-byte store. The blocks before them, since w is what
// was quantized last and begins in L2: a tile of 128 k
// x 64 n; a thread converts 4 x 4 values, the word of four k of one n goes through shared memory (16-byte chunks
// XORed with the n quad, so that the transposed stores meet at most two to a bank) and leaves in 128-byte rows.
// 8192 x 4096 and 4096 x 8192: 54 us, 6.2 TB/s; one pass to codes per operand (one value per thread and store) and
// a separate byte transpose took 237 us.
template <bool kVecX, bool kVecW>
__global__ void __launch_bounds__(256) fxp8_operands_kernel(const float *__restrict__ x, int64_t M, int K, int64_t Kp,
                                                            float inv_dx, int8_t *__restrict__ xc,
                                                            const float *__restrict__ w, int N, float inv_dw,
                                                            int8_t *__restrict__ wt, unsigned w_blocks, int k_tiles) {
  __shared__ uint4 tile[64][8];
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.x >= w_blocks) {
    const int64_t runs_row = Kp / 128, runs = M * runs_row;
    const int64_t s0 = ((int64_t)(blockIdx.x - w_blocks) * 8 + warp) * 4;
    float4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t s = s0 + j, r = s / runs_row;
      const int k = (int)(s - r * runs_row) * 128 + 4 * lane;
      v[j] = s < runs ? load_quad<kVecX>(x + r * K, k, K) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (s0 + j < runs)
        reinterpret_cast<uint32_t *>(xc)[(s0 + j) * 32 + lane] = pack_codes(v[j].x, v[j].y, v[j].z, v[j].w, inv_dx);
    return;
  }
  const unsigned t = blockIdx.x;
  const int k0 = (int)(t % k_tiles) * 128, n0 = (int)(t / k_tiles) * 64;
  const int nq = threadIdx.x & 15, kr = threadIdx.x >> 4; // n quad, first k quad
  float4 v[2][4];
#pragma unroll
  for (int it = 0; it < 2; ++it)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + 4 * (kr + 16 * it) + j;
      v[it][j] = k < K ? load_quad<kVecW>(w + (int64_t)k * N, n0 + 4 * nq, N) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  uint32_t *words = reinterpret_cast<uint32_t *>(&tile[0][0]);
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int kq = kr + 16 * it, col = (((kq >> 2) ^ (nq & 7)) << 2) | (kq & 3);
    const float4 *q = v[it];
    words[(4 * nq + 0) * 32 + col] = pack_codes(q[0].x, q[1].x, q[2].x, q[3].x, inv_dw);
    words[(4 * nq + 1) * 32 + col] = pack_codes(q[0].y, q[1].y, q[2].y, q[3].y, inv_dw);
    words[(4 * nq + 2) * 32 + col] = pack_codes(q[0].z, q[1].z, q[2].z, q[3].z, inv_dw);
    words[(4 * nq + 3) * 32 + col] = pack_codes(q[0].w, q[1].w, q[2].w, q[3].w, inv_dw);
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int i = threadIdx.x + 256 * it, n = i >> 3, c = i & 7;
    if (n0 + n < N)
      *reinterpret_cast<uint4 *>(wt + (int64_t)(n0 + n) * Kp + k0 + 16 * c) = tile[n][c ^ ((n >> 2) & 7)];
  }
}

} // namespace

int binarize_columns(const float *w, int R, int C, float zero_to, float *wb, float *alpha, void *side,
                     int64_t side_pitch, bool int8, float *partial_scratch, cudaStream_t st) {
  const dim3 grid((C + kBT - 1) / kBT, (R + kBT - 1) / kBT);
  float *partial = alpha ? partial_scratch : nullptr;
  // the side-band rows hold K padded to a multiple of 64 values: four rows past R stay inside a row
  const bool vec = C % 4 == 0 && side_pitch % 4 == 0 && side_pitch >= (int64_t)(R + 3) / 4 * 4 &&
                   ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(wb)) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(side) & 7) == 0;
  if (vec && int8)
    NB_CUDA(launch_dependent(binarize_columns_vec_kernel<true>, grid, dim3(256), 0, st, w, R, C, zero_to, wb, side,
                             side_pitch, partial));
  else if (vec)
    NB_CUDA(launch_dependent(binarize_columns_vec_kernel<false>, grid, dim3(256), 0, st, w, R, C, zero_to, wb, side,
                             side_pitch, partial));
  else if (int8)
    NB_CUDA(launch_dependent(binarize_columns_kernel<true>, grid, dim3(256), 0, st, w, R, C, zero_to, wb, side,
                             side_pitch, partial));
  else
    NB_CUDA(launch_dependent(binarize_columns_kernel<false>, grid, dim3(256), 0, st, w, R, C, zero_to, wb, side,
                             side_pitch, partial));
  NB_LAUNCH_CHECK();
  if (alpha) {
    const float inv = (float)1 / R; // binary_weight_affine.cpp:68
    NB_CUDA(launch_dependent(finalize_alpha_kernel, dim3((C + 255) / 256), dim3(256), 0, st, partial, (int)grid.y, C,
                             inv, alpha));
    NB_LAUNCH_CHECK();
  }
  return NB200_OK;
}

int binary_affine_operands(const float *x, int64_t rows, const float *w, int R, int C, float zero_to, float *wb, float *alpha,
                           void *side, int64_t pitch, float *partial_scratch, void *pieces, cudaStream_t st, bool *leave_sums) {
  const int gx = (C + kBT - 1) / kBT, gy = (R + kBT - 1) / kBT;
  const int64_t w_blocks = (int64_t)gx * gy, x_blocks = (rows * (pitch / 4) + 255) / 256;
  const bool vec = C % 4 == 0 && R % 4 == 0 && w_blocks + x_blocks < (1ll << 31) &&
                   ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(wb) | reinterpret_cast<uintptr_t>(x)) & 15) == 0;
  if (!vec) {
    *leave_sums = false;
    NB_TRY(binarize_columns(w, R, C, zero_to, wb, alpha, side, pitch, false, partial_scratch, st));
    return split_rows_bf16(SplitRows{x, nullptr, pieces, rows, R, 3}, SplitRows{}, pitch, st);
  }
  NB_CUDA(launch_dependent(binary_affine_operands_kernel, dim3((unsigned)(w_blocks + x_blocks)), dim3(256), 0, st, w, R, C,
                           zero_to, wb, side, pitch, alpha ? partial_scratch : nullptr, gx, (int)w_blocks, x, rows,
                           static_cast<__nv_bfloat16 *>(pieces)));
  if (alpha && !*leave_sums)
    NB_CUDA(launch_dependent(finalize_alpha_kernel, dim3((C + 255) / 256), dim3(256), 0, st, partial_scratch, gy, C,
                             (float)1 / R, alpha)); // binary_weight_affine.cpp:68
  return NB200_OK;
}

int binarize_rows(const float *w, int Ko, int Cg, int kh, int kw, float zero_to, float *wb, float *alpha, void *side,
                  int64_t side_pitch, int c_pad, bool int8, cudaStream_t st, bool half) {
  const float inv = (float)1 / (Cg * kh * kw); // binary_weight_convolution.cpp:66
  if (int8)
    NB_CUDA(launch_dependent(binarize_rows_kernel<1>, dim3(Ko), dim3(256), 0, st, w, Cg, kh, kw, zero_to, inv, wb,
                             alpha,
                             side, side_pitch, c_pad));
  else if (half)
    NB_CUDA(launch_dependent(binarize_rows_kernel<2>, dim3(Ko), dim3(256), 0, st, w, Cg, kh, kw, zero_to, inv, wb,
                             alpha, side, side_pitch, c_pad));
  else
    NB_CUDA(launch_dependent(binarize_rows_kernel<0>, dim3(Ko), dim3(256), 0, st, w, Cg, kh, kw, zero_to, inv, wb,
                             alpha, side, side_pitch, c_pad));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

bool binary_conv_operands_i8_applies(const float *x, int N, int HW, int ctot, int Ko) {
  const int64_t blocks = (int64_t)Ko + (int64_t)((HW + 63) / 64) * ((ctot + 63) / 64) * N;
  return x != nullptr && blocks < (1ll << 31);
}

int binary_conv_operands_i8(const float *w, int Ko, int Cg, int kh, int kw, float zero_to, float *wb, float *alpha,
                            void *side, int64_t side_pitch, int c_pad, const float *x, int N, int C, int HW, int groups,
                            int c_pad_g, int ctot, float delta, void *out, cudaStream_t st) {
  const float inv = (float)1 / (Cg * kh * kw); // binary_weight_convolution.cpp:66
  const int gx = (HW + 63) / 64, gy = (ctot + 63) / 64;
  const int64_t blocks = (int64_t)Ko + (int64_t)gx * gy * N;
  NB_CHECK(binary_conv_operands_i8_applies(x, N, HW, ctot, Ko), NB200_EVALUE, "operand preparation does not apply");
  // 128-bit loads when the planes allow it (nchw_to_nhwc_planes has the same rule)
  if (HW % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0)
    NB_CUDA(launch_dependent(binary_conv_operands_i8_kernel<true>, dim3((unsigned)blocks), dim3(256), 0, st, w, Ko, Cg,
                             kh, kw, zero_to, inv, wb, alpha, side, side_pitch, c_pad, x, C, HW, groups, Cg, c_pad_g,
                             ctot, reinterpret_cast<int8_t *>(out), 1.0f / delta, gx, gy));
  else
    NB_CUDA(launch_dependent(binary_conv_operands_i8_kernel<false>, dim3((unsigned)blocks), dim3(256), 0, st, w, Ko, Cg,
                             kh, kw, zero_to, inv, wb, alpha, side, side_pitch, c_pad, x, C, HW, groups, Cg, c_pad_g,
                             ctot, reinterpret_cast<int8_t *>(out), 1.0f / delta, gx, gy));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

int codes_conv_weights(const float *wq, int Ko, int Cg, int kh, int kw, float delta, void *side, int64_t side_pitch,
                       int c_pad, cudaStream_t st) {
  NB_CUDA(launch_dependent(codes_conv_weights_kernel, dim3(Ko), dim3(256), 0, st, wq, Cg, kh, kw, 1.0f / delta,
                           reinterpret_cast<int8_t *>(side), side_pitch, c_pad));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

int split_rows_bf16(const SplitRows &a, const SplitRows &b, int64_t Kp, cudaStream_t st) {
  NB_CHECK(Kp % 64 == 0 && Kp / 64 < (1ll << 31), NB200_EVALUE, "the padded K extent must be a multiple of 64");
  auto blocks = [&](const SplitRows &p) { return (p.rows * (Kp / 8) + 255) / 256; };
  auto vec = [](const SplitRows &p) {
    return p.rows == 0 || (p.K % 4 == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0);
  };
  NB_CHECK(blocks(a) + blocks(b) < (1ll << 31), NB200_ENOTIMPL, "operand too large");
  NB_CUDA(launch_dependent(vec(a) && vec(b) ? split_rows_kernel<true> : split_rows_kernel<false>,
                           dim3((unsigned)(blocks(a) + blocks(b))), dim3(256), 0, st, a, b, (unsigned)blocks(a), Kp));
  return NB200_OK;
}

int split_columns_bf16(const SplitColumns &a, const SplitColumns &b, int64_t Rp, cudaStream_t st) {
  NB_CHECK(Rp % 64 == 0, NB200_EVALUE, "the padded row count must be a multiple of 64");
  auto blocks = [&](const SplitColumns &p) { return (Rp / 64) * ((p.cols + 63) / 64); };
  auto vec = [](const SplitColumns &p) {
    return p.cols == 0 || (p.cols % 4 == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0);
  };
  NB_CHECK(blocks(a) + blocks(b) < (1ll << 31), NB200_ENOTIMPL, "operand too large");
  NB_CUDA(launch_dependent(vec(a) && vec(b) ? split_columns_kernel<true> : split_columns_kernel<false>,
                           dim3((unsigned)(blocks(a) + blocks(b))), dim3(256), 0, st, a, b, (unsigned)blocks(a), Rp));
  return NB200_OK;
}

// ---------------------------------------------------------------------------
// Two fp16 pieces of an fp32 tensor: with s = 2^-e chosen from the tensor's largest magnitude so that
// max |x| * s lies in [2^14, 2^15), x * s = p0 + p1 with p0 = fp16(x * s), p1 = fp16(x * s - p0): 22
// significant bits for every element within 2^-18 of the maximum, an absolute error of at most 2^-40
// of the maximum below that (p1 is then subnormal), which no fp32 sum over a filter window resolves.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) absmax_bits_kernel(const float *__restrict__ x, size_t n,
                                                          uint32_t *__restrict__ maxbits) {
  pdl_wait();
  pdl_trigger();
  uint32_t m = 0;
  const size_t stride = (size_t)gridDim.x * 256;
  const size_t n4 = ((reinterpret_cast<uintptr_t>(x) & 15) == 0) ? n / 4 : 0;
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n4; i += stride) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(x) + i);
    m = max(max(m, __float_as_uint(fabsf(v.x))), max(__float_as_uint(fabsf(v.y)), __float_as_uint(fabsf(v.z))));
    m = max(m, __float_as_uint(fabsf(v.w)));
  }
  for (size_t i = n4 * 4 + (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += stride)
    m = max(m, __float_as_uint(fabsf(__ldg(x + i))));
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && m != 0)
    atomicMax(maxbits, m);
}

// out[i] = (in ? in[i] : 1) * 2^e: the per-row factor that undoes the activation scaling
__global__ void half_pair_row_scale_kernel(const float *__restrict__ in, int n, const uint32_t *__restrict__ maxbits,
                                           float *__restrict__ out) {
  pdl_wait();
  pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const float up = __int_as_float((127 + half_pair_exponent(*maxbits)) << 23);
    out[i] = in ? __fmul_rn(in[i], up) : up;
  }
}

// nchw_to_nhwc_kernel for the two fp16 pieces; plane 1 lies plane_stride elements behind plane 0.
// Tiles of 32 pixels x 64 channel slots: loads run along the pixels, every thread stores two
// neighbouring slots of a pixel as one 32-bit word per plane (ctot is even: slots come in sixteens).
__global__ void __launch_bounds__(256) nchw_to_nhwc_half_pair_kernel(const float *__restrict__ x, int C, int HW,
                                                                     int groups, int Cg, int c_pad_g, int ctot,
                                                                     const uint32_t *__restrict__ maxbits,
                                                                     __half *__restrict__ out, int64_t plane_stride) {
  pdl_wait();
  pdl_trigger();
  __shared__ float tile[64][33];
  const float down = __int_as_float((127 - half_pair_exponent(*maxbits)) << 23);
  const int n = blockIdx.z;
  const int p0 = blockIdx.x * 32, d0 = blockIdx.y * 64;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int dd = ty; dd < 64; dd += 8) {
    const int d = d0 + dd, p = p0 + tx;
    const int g = d / c_pad_g, cc = d - g * c_pad_g;
    const bool live = d < ctot && g < groups && cc < Cg && p < HW;
    tile[dd][tx] = live ? __ldcs(x + ((int64_t)n * C + (g * Cg + cc)) * HW + p) : 0.0f;
  }
  __syncthreads();
#pragma unroll
  for (int pp = ty; pp < 32; pp += 8) {
    const int p = p0 + pp, d = d0 + 2 * tx;
    if (p < HW && d < ctot) {
      const float v0 = __fmul_rn(tile[2 * tx][pp], down), v1 = __fmul_rn(tile[2 * tx + 1][pp], down);
      const __half a0 = __float2half_rn(v0), a1 = __float2half_rn(v1);
      const __half b0 = __float2half_rn(__fsub_rn(v0, __half2float(a0)));
      const __half b1 = __float2half_rn(__fsub_rn(v1, __half2float(a1)));
      const int64_t dst = ((int64_t)n * HW + p) * ctot + d;
      *reinterpret_cast<__half2 *>(out + dst) = __halves2half2(a0, a1);
      *reinterpret_cast<__half2 *>(out + plane_stride + dst) = __halves2half2(b0, b1);
    }
  }
}

int nchw_to_nhwc_half_pair(const float *x, int N, int C, int HW, int groups, int Cg, int c_pad_g, int ctot, void *out,
                           uint32_t *maxbits, const float *row_scale_in, int rows, float *row_scale_out,
                           cudaStream_t st) {
  NB_CHECK(N <= 65535, NB200_ENOTIMPL, "batch larger than 65535");
  NB_CUDA(cudaMemsetAsync(maxbits, 0, 4, st));
  const size_t n = (size_t)N * C * HW;
  size_t blocks = (n / 4 + 255) / 256;
  const size_t cap = (size_t)sm_count() * 16;
  blocks = blocks < 1 ? 1 : (blocks > cap ? cap : blocks);
  NB_CUDA(launch_dependent(absmax_bits_kernel, dim3((unsigned)blocks), dim3(256), 0, st, x, n, maxbits));
  NB_LAUNCH_CHECK();
  NB_CUDA(launch_dependent(half_pair_row_scale_kernel, dim3((rows + 255) / 256), dim3(256), 0, st, row_scale_in, rows,
                           maxbits, row_scale_out));
  NB_LAUNCH_CHECK();
  NB_CHECK(ctot % 2 == 0, NB200_EVALUE, "channel slots must come in pairs");
  const dim3 grid((HW + 31) / 32, (ctot + 63) / 64, N);
  NB_CUDA(launch_dependent(nchw_to_nhwc_half_pair_kernel, grid, dim3(256), 0, st, x, C, HW, groups, Cg, c_pad_g, ctot,
                           maxbits, reinterpret_cast<__half *>(out), (int64_t)N * HW * ctot));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

int nchw_to_nhwc_planes(const float *x, int N, int C, int HW, int groups, int Cg, int c_pad_g, int ctot, int planes,
                        float delta, void *out, cudaStream_t st) {
  const dim3 grid((HW + 31) / 32, (ctot + 31) / 32, N);
  NB_CHECK(N <= 65535, NB200_ENOTIMPL, "batch larger than 65535");
  const int64_t ps = (int64_t)N * HW * ctot;
  if (planes == 0) {
    // ctot is a multiple of 16 (channel slots are padded to 16 per group), so word stores are aligned.
    const dim3 grid8((HW + 63) / 64, (ctot + 63) / 64, N);
    if (HW % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0)
      NB_CUDA(launch_dependent(nchw_to_nhwc_i8_vec_kernel, grid8, dim3(256), 0, st, x, C, HW, groups, Cg, c_pad_g, ctot,
                               reinterpret_cast<int8_t *>(out), 1.0f / delta));
    else
      NB_CUDA(launch_dependent(nchw_to_nhwc_i8_kernel, grid8, dim3(256), 0, st, x, C, HW, groups, Cg, c_pad_g, ctot,
                               reinterpret_cast<int8_t *>(out), 1.0f / delta));
  } else if (planes == 3) {
    NB_CUDA(launch_dependent(nchw_to_nhwc_kernel<__nv_bfloat16, 3>, grid, dim3(256), 0, st, x, C, HW, groups, Cg,
                             c_pad_g, ctot, reinterpret_cast<__nv_bfloat16 *>(out), ps, 0.f));
  } else {
    NB_CUDA(launch_dependent(nchw_to_nhwc_kernel<__nv_bfloat16, 1>, grid, dim3(256), 0, st, x, C, HW, groups, Cg,
                             c_pad_g, ctot, reinterpret_cast<__nv_bfloat16 *>(out), ps, 0.f));
  }
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

int column_sums(const float *a, int64_t rows, int C, float *out, int accumulate, float *partial, int splits,
                cudaStream_t st) {
  const dim3 grid((C + 255) / 256, splits);
  NB_CUDA(launch_dependent(column_partial_sums_kernel, grid, dim3(256), 0, st, a, rows, C, partial));
  return column_sums_finish(partial, C, splits, out, accumulate, st);
}

int column_sums_finish(const float *partial, int C, int splits, float *out, int accumulate, cudaStream_t st) {
  NB_CUDA(launch_dependent(column_finish_kernel, dim3((C + 255) / 256), dim3(256), 0, st, partial, C, splits, out,
                           accumulate));
  return NB200_OK;
}

int transpose_i8(const int8_t *src, int R, int C, int8_t *dst, int64_t pitch, cudaStream_t st) {
  const dim3 grid((C + 63) / 64, (R + 63) / 64);
  NB_CUDA(launch_dependent(transpose_i8_kernel, grid, dim3(256), 0, st, src, R, C, dst, pitch));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

int fxp8_operands(const float *x, int64_t M, int K, int64_t Kp, float delta_x, int8_t *xc, const float *w, int N,
                  float delta_w, int8_t *wt, cudaStream_t st) {
  const int64_t x_blocks = (M * (Kp / 128) + 31) / 32, k_tiles = Kp / 128, w_blocks = k_tiles * ((N + 63) / 64);
  NB_CHECK(x_blocks + w_blocks < (1ll << 31), NB200_ENOTIMPL, "operands too large for one launch");
  const bool vx = K % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const bool vw = N % 4 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
  auto kernel = vx ? (vw ? fxp8_operands_kernel<true, true> : fxp8_operands_kernel<true, false>)
                   : (vw ? fxp8_operands_kernel<false, true> : fxp8_operands_kernel<false, false>);
  NB_CUDA(launch_dependent(kernel, dim3((unsigned)(x_blocks + w_blocks)), dim3(256), 0, st, x, M, K, Kp, 1.0f / delta_x,
                           xc, w, N, 1.0f / delta_w, wt, (unsigned)w_blocks, (int)k_tiles));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

} // namespace nb200
