// Small fp32 products on the FMA pipes, in one launch and without operand passes: y[M][N] (+)= op(A) . op(B) of operands
// as the layers hold them. The tensor-core route needs the operands split into bf16 pieces (and transposed) first: four
// to seven launches of 2 to 10 us for products that take the FMA pipes 1 us.
//
// A block makes a TM x 32 tile of y over the whole contraction, in chunks of 128 values through a ring of shared-memory
// stages (cp.async, zero-filled past the edges). Warp w takes values [16 w, 16 w + 16) of every chunk, all outputs of the
// tile in registers; the eight partial tiles are added in warp order at the end. Bound by the latency of a chunk (issue,
// wait, barrier) and by the FMA rate of the few SMs that a small tile grid reaches, so 16-row tiles are taken where
// 32-row tiles do not fill the chip.
//
// On the way through shared memory the B operand can be binarized (kBinarize: sign(w), which is also written to wb, and
// alpha from the column sums of |w|) or have its columns summed (kColumnSums: db), and A can be multiplied by a factor
// per contraction index (dy * alpha, one rounding): every thread changes the values that it fetched itself, before the
// chunk's only barrier. wb leaves chunk by chunk from all blocks of a column (from the first rows' alone, those were the
// last to end: [100, 784] . [784, 500] 10.6 us, now 9.5); the partial tiles go to shared memory in rows of 36 floats as
// 16-byte writes (one value at a time, eight rows to a bank, x^T . dy of the same layer took 9.6 us, now 7.8).
#pragma once
#include <algorithm>

#include "common.cuh"
#include "pdl.cuh"
#include "prepare.cuh"
#include "ptx.cuh"

namespace nb200 {

constexpr int kSmallK = 128;             // contraction values per stage
constexpr int kSmallPitch = kSmallK + 4; // rows along the contraction: 16-byte reads of eight rows hit 32 banks
constexpr int kSmallMaxK = 2048;         // the longest contraction with a factor per index (held in shared memory)

constexpr int kSmallPart = 36;           // row pitch of a warp's partial tile: 16-byte writes of eight rows hit 32 banks

// 25 KB (TM = 16) or 34 KB per stage: two blocks per SM
constexpr int small_stages(int rows) { return rows == 16 ? 4 : 3; }

enum class SmallB { kPlain, kBinarize, kColumnSums };

struct SmallGemm {
  const float *a, *b;
  float *y;
  int M, N, K;
  const float *a_scale;   // per contraction index, may be NULL
  const float *col_scale; // per column of y, may be NULL
  const float *col_bias;  // may be NULL
  int accumulate;
  float zero_to, inv;  // kBinarize
  float *wb, *alpha;   // kBinarize: wb is written by all blocks of a column, a chunk in turn; alpha (may be NULL) by the
                       // blocks of the first rows
  float *sums;         // kColumnSums: written (or accumulated into) by the blocks of the first rows
  int accumulate_sums;
};

// include/nbla/function/sign.hpp:48-50 (+0, -0 and NaN take zero_to)
__device__ __forceinline__ float small_sign(float v, float zero_to) { return v > 0.0f ? 1.0f : v < 0.0f ? -1.0f : zero_to; }

// One thread's share of a stage of R rows (rows of y or columns of y) x kSmallK contraction values: kQuads groups of four
// consecutive values of the source. kAlongK: the source is [rows][K], else [K][rows].
template <int R, bool kAlongK>
struct SmallShare {
  static constexpr int kPitch = kAlongK ? kSmallPitch : R, kFloats = kAlongK ? R * kSmallPitch : kSmallK * R;
  static constexpr int kQuads = R * kSmallK / 4 / 256;
  static constexpr int kPerRow = (kAlongK ? kSmallK : R) / 4; // quads in a row of the stage
  const float *src; // this thread's first quad in the first chunk
  int64_t step;     // from one of its quads to the next
  int64_t advance;  // from chunk to chunk
  int line, col;    // its first quad's row and column in the stage
  int row_left, col_left;
  bool vec;
  __device__ __forceinline__ SmallShare(const float *base, int r0, int rows, int K) {
    line = threadIdx.x / kPerRow, col = threadIdx.x % kPerRow * 4;
    const int ld = kAlongK ? K : rows;
    src = base + (kAlongK ? (int64_t)(r0 + line) * ld + col : (int64_t)line * ld + r0 + col);
    step = (int64_t)(256 / kPerRow) * ld;
    advance = kAlongK ? kSmallK : (int64_t)kSmallK * ld;
    row_left = kAlongK ? rows - r0 - line : K - line; // rows of the source from this thread's first one on
    col_left = kAlongK ? K - col : rows - r0 - col;
    vec = ((ld & 3) | (int)(reinterpret_cast<uintptr_t>(base) & 15)) == 0;
  }
  __device__ __forceinline__ float *quad(float *stage, int j) const {
    return stage + (line + 256 / kPerRow * j) * kPitch + col;
  }
  // contraction index of quad j in chunk 0 (its first value's when kAlongK)
  __device__ __forceinline__ int k_of(int j) const { return kAlongK ? col : line + 256 / kPerRow * j; }
  __device__ __forceinline__ void fetch(float *stage, int chunk) const {
    const float *p = src + chunk * advance;
    const int rows_left = row_left - (kAlongK ? 0 : chunk * kSmallK), cols_left = col_left - (kAlongK ? chunk * kSmallK : 0);
#pragma unroll
    for (int j = 0; j < kQuads; ++j) {
      const bool row_in = rows_left > 256 / kPerRow * j;
      const uint32_t dst = ptx::smem_u32(quad(stage, j));
      const float *q = p + j * step;
      if (vec) {
        const bool in = row_in && cols_left > 0; // a multiple of four values is left
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(in ? q : src), "r"(in ? 16 : 0)
                     : "memory");
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool in = row_in && cols_left > e;
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * e), "l"(in ? q + e : src),
                       "r"(in ? 4 : 0)
                       : "memory");
        }
      }
    }
  }
};

// The tile (bx, by) of a product, gy tiles along its rows, by one block. kAT: A is stored [K][M], else [M][K]; kBT: B is
// stored [N][K], else [K][N].
template <int TM, bool kAT, bool kBT, SmallB kMode>
__device__ __forceinline__ void small_gemm_tile(const SmallGemm &P, float *ring, float *s_scale, unsigned bx, unsigned by,
                                                unsigned gy) {
  static_assert(TM == 16 || TM == 32, "tile rows");
  static_assert(kMode == SmallB::kPlain || !kBT, "columns are summed along the rows of B");
  constexpr int TN = 32, kNJ = TM == 32 ? 8 : 4, kMI = TM / 4; // a lane's outputs: 4 rows x kNJ columns
  constexpr int kStages = small_stages(TM);
  using ShareA = SmallShare<TM, !kAT>;
  using ShareB = SmallShare<TN, kBT>;
  constexpr int kStage = ShareA::kFloats + ShareB::kFloats;
  const int m0 = by * TM, n0 = bx * TN, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, mi = lane % kMI, ni = lane / kMI;
  const int chunks = (P.K + kSmallK - 1) / kSmallK;
  const ShareA share_a(P.a, m0, P.M, P.K);
  const ShareB share_b(P.b, n0, P.N, P.K);
  auto fetch_chunk = [&](int chunk) {
    if (chunk < chunks) {
      float *stage = ring + chunk % kStages * kStage;
      share_a.fetch(stage, chunk);
      share_b.fetch(stage + ShareA::kFloats, chunk);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int c = 0; c < kStages - 1; ++c)
    fetch_chunk(c);
  const bool scale_a = !kAT && P.a_scale != nullptr;
  if (scale_a) {
    for (int k = tid; k < chunks * kSmallK; k += 256)
      s_scale[k] = k < P.K ? __ldg(P.a_scale + k) : 0.0f;
    __syncthreads();
  }

  float acc[4][kNJ];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int j = 0; j < kNJ; ++j)
      acc[r][j] = 0.0f;
  float col[4] = {0.0f, 0.0f, 0.0f, 0.0f}; // this thread's share of the sums of its four columns of B

  for (int chunk = 0; chunk < chunks; ++chunk) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    float *as = ring + chunk % kStages * kStage, *bs = as + ShareA::kFloats;
    const int k0 = chunk * kSmallK;
    if (scale_a) {
      const float4 f = *reinterpret_cast<const float4 *>(s_scale + (kAT ? 0 : k0 + share_a.col));
#pragma unroll
      for (int j = 0; j < ShareA::kQuads; ++j) {
        float4 *q = reinterpret_cast<float4 *>(share_a.quad(as, j));
        const float4 v = *q;
        *q = make_float4(__fmul_rn(v.x, f.x), __fmul_rn(v.y, f.y), __fmul_rn(v.z, f.z), __fmul_rn(v.w, f.w));
      }
    }
    if (kMode != SmallB::kPlain) {
#pragma unroll
      for (int j = 0; j < ShareB::kQuads; ++j) {
        float4 *q = reinterpret_cast<float4 *>(share_b.quad(bs, j));
        float4 v = *q;
        if (kMode == SmallB::kBinarize) {
          col[0] += fabsf(v.x), col[1] += fabsf(v.y), col[2] += fabsf(v.z), col[3] += fabsf(v.w);
          v = make_float4(small_sign(v.x, P.zero_to), small_sign(v.y, P.zero_to), small_sign(v.z, P.zero_to),
                          small_sign(v.w, P.zero_to));
          *q = v;
          const int k = k0 + share_b.k_of(j), n = n0 + share_b.col;
          if (chunk % gy == by && k < P.K) {
            float *w = P.wb + (int64_t)k * P.N + n;
            if (n + 3 < P.N && (reinterpret_cast<uintptr_t>(w) & 15) == 0) {
              *reinterpret_cast<float4 *>(w) = v;
            } else {
              const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (n + i < P.N)
                  w[i] = e[i];
            }
          }
        } else {
          col[0] += v.x, col[1] += v.y, col[2] += v.z, col[3] += v.w;
        }
      }
    }
    __syncthreads(); // the chunk is here and ready, and the stage that the next fetch overwrites has been read
    fetch_chunk(chunk + kStages - 1);
    if (k0 + warp * (kSmallK / 8) >= P.K) // this warp's share of the last chunk is padding
      break;
#pragma unroll
    for (int q = 0; q < kSmallK / 32; ++q) { // four contraction values at a time
      const int k = warp * (kSmallK / 8) + q * 4;
      float av[4][4], bv[4][kNJ]; // [k][row], [k][column]
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float4 t = kAT ? *reinterpret_cast<const float4 *>(as + (k + r) * TM + mi * 4)
                             : *reinterpret_cast<const float4 *>(as + (mi + kMI * r) * kSmallPitch + k);
        const float e[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (kAT)
            av[r][u] = e[u];
          else
            av[u][r] = e[u];
      }
      if (kBT) {
#pragma unroll
        for (int j = 0; j < kNJ; ++j) {
          const float4 t = *reinterpret_cast<const float4 *>(bs + (ni + TN / kNJ * j) * kSmallPitch + k);
          bv[0][j] = t.x, bv[1][j] = t.y, bv[2][j] = t.z, bv[3][j] = t.w;
        }
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int h = 0; h < kNJ / 4; ++h) {
            const float4 t = *reinterpret_cast<const float4 *>(bs + (k + u) * TN + 16 * h + ni * 4);
            bv[u][4 * h] = t.x, bv[u][4 * h + 1] = t.y, bv[u][4 * h + 2] = t.z, bv[u][4 * h + 3] = t.w;
          }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int j = 0; j < kNJ; ++j)
            acc[r][j] = __fmaf_rn(av[u][r], bv[u][j], acc[r][j]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // partial tiles of the warps, and the column sums, over the ring
  float *part = ring, *colsum = ring + 8 * TM * kSmallPart; // [warp][TM][kSmallPart], [32][TN]
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    float *row = part + (warp * TM + (kAT ? mi * 4 + r : mi + kMI * r)) * kSmallPart;
    if (kBT) {
#pragma unroll
      for (int j = 0; j < kNJ; ++j)
        row[ni + TN / kNJ * j] = acc[r][j];
    } else {
#pragma unroll
      for (int h = 0; h < kNJ / 4; ++h)
        *reinterpret_cast<float4 *>(row + 16 * h + ni * 4) =
            make_float4(acc[r][4 * h], acc[r][4 * h + 1], acc[r][4 * h + 2], acc[r][4 * h + 3]);
    }
  }
  if (kMode != SmallB::kPlain) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      colsum[(tid / 8) * TN + tid % 8 * 4 + j] = col[j];
  }
  __syncthreads();
  const int n = n0 + lane;
  float factor = 1.0f;
  bool scaled = P.col_scale != nullptr;
  if (scaled && n < P.N)
    factor = __ldg(P.col_scale + n);
  if (kMode != SmallB::kPlain) {
    float s = 0.0f;
#pragma unroll 8
    for (int i = 0; i < 32; ++i)
      s += colsum[i * TN + lane];
    if (kMode == SmallB::kBinarize && P.alpha) {
      factor = __fmul_rn(s, P.inv);
      scaled = true;
    }
    if (by == 0 && warp == 0 && n < P.N) {
      if (kMode == SmallB::kBinarize) {
        if (P.alpha)
          P.alpha[n] = factor;
      } else {
        P.sums[n] = P.accumulate_sums ? __fadd_rn(P.sums[n], s) : s;
      }
    }
  }
  const float bias = P.col_bias && n < P.N ? __ldg(P.col_bias + n) : 0.0f;
#pragma unroll
  for (int i = 0; i < TM / 8; ++i) {
    const int m = warp + 8 * i;
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w)
      v += part[(w * TM + m) * kSmallPart + lane];
    if (m0 + m < P.M && n < P.N) {
      if (scaled)
        v = __fmul_rn(v, factor);
      if (P.col_bias)
        v = __fadd_rn(v, bias);
      float *dst = P.y + (int64_t)(m0 + m) * P.N + n;
      *dst = P.accumulate ? __fadd_rn(*dst, v) : v;
    }
  }
}

template <int TM, bool kAT, bool kBT, SmallB kMode>
__global__ void __launch_bounds__(256, 2) small_gemm_kernel(const __grid_constant__ SmallGemm P) {
  extern __shared__ __align__(16) float ring[];
  __shared__ float s_scale[kAT ? 1 : kSmallMaxK];
  pdl_wait();
  pdl_trigger();
  small_gemm_tile<TM, kAT, kBT, kMode>(P, ring, s_scale, blockIdx.x, blockIdx.y, gridDim.y);
}

// Two products that do not depend on one another, the gradients of an affine layer, in one launch: dx = A . B^T by the
// first n_dx blocks, dW = A^T . B by the others. Each alone leaves SMs idle or starts a second round of blocks that the
// other's could fill: the gradients of [100, 784] . [784, 500] 16.5 us in two launches, 12.6 in one; [32, 2048] . [2048, 512]
// 24.4 and 17.5.
template <int TMX, int TMW, SmallB kSums>
__global__ void __launch_bounds__(256, 2) small_gemm_gradients_kernel(const __grid_constant__ SmallGemm X,
                                                                      const __grid_constant__ SmallGemm W, unsigned n_dx) {
  extern __shared__ __align__(16) float ring[];
  __shared__ float s_scale[kSmallMaxK];
  pdl_wait();
  pdl_trigger();
  if (blockIdx.x < n_dx) {
    const unsigned gx = (unsigned)(X.N + 31) / 32;
    small_gemm_tile<TMX, false, true, SmallB::kPlain>(X, ring, s_scale, blockIdx.x % gx, blockIdx.x / gx, n_dx / gx);
  } else {
    const unsigned gx = (unsigned)(W.N + 31) / 32, b = blockIdx.x - n_dx;
    small_gemm_tile<TMW, true, false, kSums>(W, ring, s_scale, b % gx, b / gx, (gridDim.x - n_dx) / gx);
  }
}

// Time of the launch in units of 10 ns: waves of 32 x 32 tiles, each with a fixed part worth 128 contraction values.
// Measured: [64, 512] . [512, 1000] 5.1 us, [256, 1024] . [1024, 1024] 21.7 us, [2048, 128] . [128, 512] 21.5 us.
inline int64_t small_gemm_tiles(int64_t M, int64_t N, int rows) { return ((M + rows - 1) / rows) * ((N + 31) / 32); }
inline int64_t small_gemm_cost(int64_t M, int64_t N, int64_t K) {
  const int64_t waves = (small_gemm_tiles(M, N, 32) + sm_count() - 1) / sm_count();
  return M > 65535 * 16 ? INT64_MAX : waves * (128 + (K + kSmallK - 1) / kSmallK * kSmallK);
}
// Lines to the tensor-core route, from both routes' times on 200 shapes of 1 to 4096 rows and 16 to 8192 columns: that
// route's launches are a constant and a part that grows with K, and its passes over B with N * K ([1, 4096] . [4096, 4096]
// 27 us here, 69 there, binarized 41 and 49). Where the first line of each allows more, the tensor-core route is up to a
// third the faster one by now, but seven times as far from 64-bit sums (1.4e-6 of the result against 2e-7).
inline bool small_gemm_binarized(int64_t M, int64_t N, int64_t K) {
  return small_gemm_cost(M, N, K) <= std::max(1024 + K / 4, 768 + K * 3 / 8 + N * K / 8192);
}
inline bool small_gemm_scaled(int64_t M, int64_t N, int64_t K) { // (the factors' place)
  return K <= kSmallMaxK && small_gemm_cost(M, N, K) <= std::max(1024 + K * 5 / 8, 768 + K * 3 / 8 + N * K / 8192);
}
inline bool small_gemm_plain(int64_t M, int64_t N, int64_t K) {
  return small_gemm_cost(M, N, K) <= std::max(1024 + K * 3 / 2, 1536 + K * 3 / 8 + N * K / 4096);
}
inline bool small_gemm_transposed(int64_t M, int64_t N, int64_t K) {
  return small_gemm_cost(M, N, K) <= std::max(2048 + K * 3, 1024 + K / 4 + N * K / 4096);
}

template <int TM, bool kAT, bool kBT> constexpr size_t small_gemm_smem() {
  constexpr size_t smem =
      small_stages(TM) * (SmallShare<TM, !kAT>::kFloats + SmallShare<32, kBT>::kFloats) * sizeof(float);
  static_assert(smem >= (8 * TM * kSmallPart + 32 * 32) * sizeof(float), "the partial tiles reuse the ring");
  return smem;
}

template <typename Kernel> int allow_small_gemm_smem(Kernel kernel, size_t smem, std::atomic<bool> (&configured)[64]) {
  int dev = 0;
  NB_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    NB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[dev & 63] = true;
  }
  return NB200_OK;
}

template <int TM, bool kAT, bool kBT, SmallB kMode>
int launch_small_gemm_tile(const SmallGemm &P, cudaStream_t st) {
  constexpr size_t smem = small_gemm_smem<TM, kAT, kBT>();
  auto kernel = small_gemm_kernel<TM, kAT, kBT, kMode>;
  static std::atomic<bool> configured[64]{};
  NB_TRY(allow_small_gemm_smem(kernel, smem, configured));
  const dim3 grid((unsigned)((P.N + 31) / 32), (unsigned)((P.M + TM - 1) / TM));
  NB_CUDA(launch_dependent(kernel, grid, dim3(256), smem, st, P));
  return NB200_OK;
}

template <int TMX, int TMW, SmallB kSums>
int launch_small_gradients_tile(const SmallGemm &X, const SmallGemm &W, cudaStream_t st) {
  constexpr size_t sx = small_gemm_smem<TMX, false, true>(), sw = small_gemm_smem<TMW, true, false>();
  constexpr size_t smem = sx > sw ? sx : sw;
  auto kernel = small_gemm_gradients_kernel<TMX, TMW, kSums>;
  static std::atomic<bool> configured[64]{};
  NB_TRY(allow_small_gemm_smem(kernel, smem, configured));
  const unsigned n_dx = (unsigned)small_gemm_tiles(X.M, X.N, TMX);
  NB_CUDA(launch_dependent(kernel, dim3(n_dx + (unsigned)small_gemm_tiles(W.M, W.N, TMW)), dim3(256), smem, st, X, W,
                           n_dx));
  return NB200_OK;
}

template <bool kAT, bool kBT, SmallB kMode>
int launch_small_gemm(const SmallGemm &P, cudaStream_t st) {
  return small_gemm_tiles(P.M, P.N, 32) < sm_count() ? launch_small_gemm_tile<16, kAT, kBT, kMode>(P, st)
                                                     : launch_small_gemm_tile<32, kAT, kBT, kMode>(P, st);
}

// Both gradients in one launch; each product's tiles as it would have them alone.
template <SmallB kSums> int launch_small_gradients_t(const SmallGemm &X, const SmallGemm &W, cudaStream_t st) {
  const bool fx = small_gemm_tiles(X.M, X.N, 32) < sm_count(), fw = small_gemm_tiles(W.M, W.N, 32) < sm_count();
  return fx ? (fw ? launch_small_gradients_tile<16, 16, kSums>(X, W, st) : launch_small_gradients_tile<16, 32, kSums>(X, W, st))
            : (fw ? launch_small_gradients_tile<32, 16, kSums>(X, W, st) : launch_small_gradients_tile<32, 32, kSums>(X, W, st));
}
inline int launch_small_gradients(const SmallGemm &X, const SmallGemm &W, cudaStream_t st) {
  return W.sums ? launch_small_gradients_t<SmallB::kColumnSums>(X, W, st) : launch_small_gradients_t<SmallB::kPlain>(X, W, st);
}

} // namespace nb200
