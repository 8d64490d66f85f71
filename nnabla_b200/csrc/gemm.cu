// Host side of the tcgen05 contractions: tensor-map encoding, kernel
// selection, and the C-ABI entry points for the affine layers.
#include <cstring>
#include <mutex>

#include <cstdlib>

#include "gemm.cuh"
#include "gemm2.cuh"
#include "small_gemm.cuh"
#include "prepare.cuh"

namespace nb200 {

// ---- driver entry point for tensor-map encoding (no link against libcuda) --
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int get_encode_fn(EncodeTiledFn *out) {
  static std::mutex m;
  static EncodeTiledFn fn = nullptr;
  std::lock_guard<std::mutex> lock(m);
  if (fn == nullptr) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    NB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    NB_CHECK(q == cudaDriverEntryPointSuccess && p != nullptr, NB200_ECUDA,
             "cuTensorMapEncodeTiled is not available from this driver");
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  *out = fn;
  return NB200_OK;
}

static CUtensorMapL2promotion l2_promotion() {
#ifdef NB200_CC_TRACE
  const char *e = std::getenv("NB_PROMO"); // timing experiments only
  if (e)
    return e[0] == '0' ? CU_TENSOR_MAP_L2_PROMOTION_NONE
                       : (e[0] == '1' ? CU_TENSOR_MAP_L2_PROMOTION_L2_64B
                                      : (e[0] == '2' ? CU_TENSOR_MAP_L2_PROMOTION_L2_128B : CU_TENSOR_MAP_L2_PROMOTION_L2_256B));
#endif
  return CU_TENSOR_MAP_L2_PROMOTION_L2_256B;
}

// dtype_code: 0 = bf16, 1 = uint8/int8 bytes, 2 = float32
int encode_tiled(CUtensorMap *map, int dtype_code, int rank, const void *base, const uint64_t *dims,
                 const uint64_t *strides_bytes, const uint32_t *box, const uint32_t *elem_strides,
                 int swizzle_bytes) {
  EncodeTiledFn fn;
  NB_TRY(get_encode_fn(&fn));
  NB_CHECK((reinterpret_cast<uintptr_t>(base) & 15) == 0, NB200_EVALUE, "tensor-map base must be 16-byte aligned");
  for (int i = 0; i < rank - 1; ++i)
    NB_CHECK(strides_bytes[i] % 16 == 0, NB200_EVALUE, "tensor-map stride %d (%llu bytes) is not a multiple of 16", i,
             (unsigned long long)strides_bytes[i]);
  cuuint64_t d[5], s[5];
  cuuint32_t b[5], e[5];
  for (int i = 0; i < rank; ++i) {
    d[i] = dims[i];
    b[i] = box[i];
    e[i] = elem_strides ? elem_strides[i] : 1;
    if (i < rank - 1)
      s[i] = strides_bytes[i];
  }
  const CUtensorMapDataType dt = dtype_code == 0   ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                 : dtype_code == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                                   : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  const CUresult r = fn(map, dt,
                        (cuuint32_t)rank, const_cast<void *>(base), d, s, b, e, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        swizzle_bytes == 0    ? CU_TENSOR_MAP_SWIZZLE_NONE
                        : swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                              : CU_TENSOR_MAP_SWIZZLE_128B,
                        l2_promotion(),
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  NB_CHECK(r == CUDA_SUCCESS, NB200_ECUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return NB200_OK;
}

int make_operand_map(CUtensorMap *map, const void *base, bool int8, int64_t k_extent, int64_t pitch_elems,
                     int64_t rows, int planes, int box_rows, int row_bytes) {
  const uint64_t es = int8 ? 1 : 2;
  const uint64_t dims[3] = {(uint64_t)k_extent, (uint64_t)rows, (uint64_t)planes};
  const uint64_t strides[2] = {(uint64_t)pitch_elems * es, (uint64_t)pitch_elems * es * (uint64_t)rows};
  const uint32_t box[3] = {(uint32_t)(row_bytes / es), (uint32_t)box_rows, 1};
  return encode_tiled(map, int8 ? 1 : 0, 3, base, dims, strides, box, nullptr, row_bytes);
}

// ---- per-device status word written by kernels whose bounded waits gave up --
int device_status_word(int **status) {
  static std::mutex m;
  static int *words[64];
  int dev = 0;
  NB_CUDA(cudaGetDevice(&dev));
  NB_CHECK(dev >= 0 && dev < 64, NB200_EVALUE, "device index %d out of range", dev);
  std::lock_guard<std::mutex> lock(m);
  if (words[dev] == nullptr) {
    NB_CUDA(cudaMalloc(&words[dev], sizeof(int)));
    NB_CUDA(cudaMemset(words[dev], 0, sizeof(int)));
  }
  *status = words[dev];
  return NB200_OK;
}

// ---- split K ----------------------------------------------------------------
// y (+)= (sum over the splits of parts[split][M][N], in order) * (scale * col_scale) + col_bias, each operation rounded as
// in the contraction's own epilogue. Four columns of a row per thread (kVec: N % 4 == 0, 16-byte aligned y rows).
template <bool kVec>
__global__ void __launch_bounds__(256) split_sums_kernel(const float *__restrict__ parts, int splits, int M, int N,
                                                         GemmEpilogue ep, int64_t ldy) {
  pdl_wait();
  pdl_trigger();
  const int quads = (N + 3) / 4;
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= (int64_t)M * quads)
    return;
  const int m = (int)(i / quads), n = 4 * (int)(i - (int64_t)m * quads);
  const float *p = parts + (int64_t)m * N + n;
  float *y = ep.y + m * ldy + n;
  float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 8
  for (int k = 0; k < splits; ++k, p += (int64_t)M * N) {
    if (kVec) {
      const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
      s[0] += v.x, s[1] += v.y, s[2] += v.z, s[3] += v.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        s[j] += n + j < N ? __ldg(p + j) : 0.0f;
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (n + j < N) {
      s[j] = __fmul_rn(s[j], ep.col_scale ? __fmul_rn(ep.scale, __ldg(ep.col_scale + n + j)) : ep.scale);
      if (ep.col_bias)
        s[j] = __fadd_rn(s[j], __ldg(ep.col_bias + n + j));
      if (ep.accumulate)
        s[j] = __fadd_rn(y[j], s[j]);
    }
  if (kVec) {
    *reinterpret_cast<float4 *>(y) = make_float4(s[0], s[1], s[2], s[3]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < N)
        y[j] = s[j];
  }
}

static int launch_split_sums(const float *parts, int splits, int M, int N, const GemmEpilogue &ep, int64_t ldy,
                             cudaStream_t st) {
  const bool vec = N % 4 == 0 && ldy % 4 == 0 && (reinterpret_cast<uintptr_t>(ep.y) & 15) == 0;
  const int64_t threads = (int64_t)M * ((N + 3) / 4);
  NB_CUDA(launch_dependent(vec ? split_sums_kernel<true> : split_sums_kernel<false>,
                           dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, st, parts, splits, M, N, ep, ldy));
  return NB200_OK;
}

// Into how many parts the K blocks of a floating-point product go whose tiles do not fill the chip. A tile's time is about
// 3 us and then its blocks', bound by L2 to shared memory (10 ns a KB); parts cost 5 us, a second launch that adds up what
// they stored. Whole layers, in one part and in parts: [60, 8192] . [8192, 1000] 64 and 29 us, [128, 8000] . [8000, 2000] 83
// and 60, input gradient of [16, 1024] . [1024, 4096] 48 and 30; [512, 1024] . [1024, 1024] 13.3 and, in two, 15.7.
static int k_splits_for(int64_t tiles, int k_blocks, int block_kb) {
  const double block_us = 0.01 * block_kb;
  int best = 1;
  double best_us = 0.0;
  for (int s = 1; s <= 16 && (s == 1 || k_blocks >= 4 * s); ++s) {
    const int64_t rounds = (tiles * s + sm_count() - 1) / sm_count();
    const double us = rounds * (3.0 + (k_blocks + s - 1) / s * block_us) + (s > 1 ? 5.0 : 0.0);
    if (s == 1 || us < best_us)
      best = s, best_us = us;
  }
  const int per = (k_blocks + best - 1) / best;
  return (k_blocks + per - 1) / per; // no empty part
}

// ---- launch -----------------------------------------------------------------
static void fill_problem(GemmProblem &prob, int M, int N, int k_blocks, int bn, int chunk_blocks, int64_t ldy) {
  prob.M = M;
  prob.N = N;
  prob.kblocks = k_blocks;
  prob.m_tiles = (M + kTileM - 1) / kTileM;
  prob.n_tiles = (N + bn - 1) / bn;
  prob.bn = bn;
  prob.row_bytes = kRowBytes;
  prob.chunk_blocks = chunk_blocks;
  prob.k_splits = 1;
  prob.split_blocks = k_blocks;
  prob.split_stride = 0;
  prob.ldy = ldy;
}

// Runs `launch(problem, epilogue)` whole or, for few tiles, in parts of K that split_sums_kernel adds up. y is M x N.
template <typename Problem, typename Launch>
static int run_in_parts(Problem &prob, int block_kb, int M, int N, const GemmEpilogue &ep, int64_t ldy, cudaStream_t st,
                        Launch launch) {
  const int splits = ep.n_peers == 0 && !ep.row_scale && !ep.row_bias && !ep.alpha_partial
                         ? k_splits_for((int64_t)prob.m_tiles * prob.n_tiles, prob.kblocks, block_kb)
                         : 1;
  if (splits == 1)
    return launch(prob, ep);
  AsyncScratch scratch(st);
  NB_TRY(scratch.alloc((size_t)splits * M * N * sizeof(float)));
  prob.k_splits = splits;
  prob.split_blocks = (prob.kblocks + splits - 1) / splits;
  prob.split_stride = (int64_t)M * N;
  prob.ldy = N;
  GemmEpilogue part{};
  part.y = static_cast<float *>(scratch.p);
  part.scale = 1.0f;
  NB_TRY(launch(prob, part));
  return launch_split_sums(part.y, splits, M, N, ep, ldy, st);
}

template <bool kInt8, int PA, int PB, int BN, int STAGES, bool kSkip>
static int launch_gemm(const CUtensorMap &ma, const CUtensorMap &mb, int M, int N, int k_blocks,
                       const GemmEpilogue &ep, int64_t ldy, cudaStream_t st) {
  GemmProblem prob;
  fill_problem(prob, M, N, k_blocks, BN, kInt8 ? 0 : k_chunk_blocks((kSkip ? 6 : PA * PB) * 4), ldy);
  auto launch = [&](const GemmProblem &p, const GemmEpilogue &e) {
    return launch_contraction<kInt8, PA, PB, BN, STAGES, kSkip, GemmProblem>(ma, mb, p, p.k_splits * p.m_tiles * p.n_tiles,
                                                                             e, st);
  };
  // (int32 sums are exact in one piece only)
  return kInt8 ? launch(prob, ep)
               : run_in_parts(prob, (PA * kTileM + PB * BN) * kRowBytes / 1024, M, N, ep, ldy, st, launch);
}
// Whether y = pieces of x (three) . weights (one plane) runs as GemmTransposedProblem: where 128 x 128 tiles would leave
// SMs idle, and its rounds of 128 x 64 tiles at 40 KB a K block cost less than those of 64 columns by 128 rows of x at 56.
// Whole layers, alpha made in the product's epilogue instead of a launch of its own, operands in L2 and, in brackets, read
// from HBM: [256, 1024] . [1024, 4096] 19.3 -> 16.1 us (23.5 -> 19.3), [512, 1024] . [1024, 1024] 16.3 -> 13.3 (19.0 ->
// 15.5), [64, 2048] . [2048, 8192] 53.6 -> 48.7 (55.7 -> 50.5), [128, 8000] . [8000, 2000], in parts, 63.8 -> 59.5 (65.4 ->
// 61.5).
static bool gemm_transposes(int64_t M, int64_t N) {
  const int64_t sms = sm_count();
  auto rounds = [&](int64_t rows, int64_t cols) {
    return (((M + rows - 1) / rows) * ((N + cols - 1) / cols) + sms - 1) / sms;
  };
  return ((M + 127) / 128) * ((N + 127) / 128) < sms && rounds(64, 128) * 40 <= rounds(128, 64) * 56;
}

// Which kernel a product takes: the one answer that run_gemm launches by and binary_affine prepares alpha by. `ep` as
// run_gemm gets it, but for col_scale and alpha's fields.
enum class GemmRoute { kPair, kTransposed, kSingle };
static GemmRoute gemm_route(bool int8, int planes_a, int planes_b, int M, int N, int k_blocks, const GemmEpilogue &ep,
                            int64_t ldy) {
  // Large problems: two-SM tiles (256 x 256 per CTA pair) halve the B traffic per SM.
  // NNABLA_B200_GEMM_PAIR=0 forces the single-CTA kernel (debugging aid).
  static const bool pair_enabled = []() {
    const char *e = std::getenv("NNABLA_B200_GEMM_PAIR");
    return !(e && e[0] == '0');
  }();
  const int64_t pair_tiles = (int64_t)((M + kPairTileM - 1) / kPairTileM) * ((N + kPairTileN - 1) / kPairTileN);
  // (the bulk stores of its epilogue need a 16-byte aligned y with a row pitch that is a multiple of 16 bytes)
  const bool y_tma_ok = (reinterpret_cast<uintptr_t>(ep.y) & 15) == 0 && (ldy % 4) == 0;
  // (peer copies of y and accumulation into y need the plain stores of the single-CTA kernel's epilogue)
  // (the two-SM kernel accumulates a whole tile in tensor memory; long floating-point K loops go to the
  // single-CTA kernel, whose chunked accumulation bounds the truncation error)
  if (pair_enabled && y_tma_ok && ep.n_peers == 0 && !ep.accumulate && planes_b == 1 && pair_tiles >= sm_count() / 2 &&
      (int8 || (planes_a == 3 && k_blocks * 12 <= 384)))
    return GemmRoute::kPair;
  return !int8 && planes_a == 3 && planes_b == 1 && ep.n_peers == 0 && !ep.row_scale && !ep.row_bias && gemm_transposes(M, N)
             ? GemmRoute::kTransposed
             : GemmRoute::kSingle;
}
// The transposed product's tiles (128 of y's columns by 64 rows) and the KB that a K block of one takes.
constexpr int kTransposedRows = 64, kTransposedBlockKb = 40;
static int64_t transposed_tiles(int M, int N) {
  return (int64_t)((N + kTileM - 1) / kTileM) * ((M + kTransposedRows - 1) / kTransposedRows);
}

// A: [planes_a][M][pitch_a], B: [planes_b][N][pitch_b], both K-major.
int run_gemm(bool int8, int planes_a, int planes_b, const void *A, int64_t pitch_a, const void *B, int64_t pitch_b,
             int M, int N, int K, const GemmEpilogue &ep, int64_t ldy, cudaStream_t st) {
  NB_CHECK(M > 0 && N > 0 && K > 0, NB200_EVALUE, "empty contraction (M=%d N=%d K=%d)", M, N, K);
  const int epb = int8 ? 128 : 64;
  const int k_blocks = (K + epb - 1) / epb;
  const int m_tiles = (M + kTileM - 1) / kTileM;
  // Narrower N tiles when wide ones would leave most SMs idle.
  const bool narrow = (int64_t)m_tiles * ((N + 127) / 128) < sm_count();
  CUtensorMap ma, mb;
  NB_TRY(make_operand_map(&ma, A, int8, K, pitch_a, M, planes_a, kTileM));
  const GemmRoute route = gemm_route(int8, planes_a, planes_b, M, N, k_blocks, ep, ldy);
  NB_CHECK(!ep.alpha_partial || route == GemmRoute::kTransposed, NB200_EVALUE, "this route does not make alpha");
  if (route == GemmRoute::kPair) {
    NB_TRY(make_operand_map(&mb, B, int8, K, pitch_b, N, 1, kPairTileN / 2));
    return int8 ? launch_pair_gemm<true, 1, 6>(ma, mb, M, N, k_blocks, ep, ldy, st)
                : launch_pair_gemm<false, 3, 3>(ma, mb, M, N, k_blocks, ep, ldy, st);
  }
  if (int8) {
    NB_CHECK(planes_a == 1 && planes_b == 1, NB200_EVALUE, "int8 operands have one plane");
    const bool wide = (int64_t)m_tiles * ((N + 255) / 256) >= sm_count();
    if (wide) {
      NB_TRY(make_operand_map(&mb, B, true, K, pitch_b, N, 1, 256));
      return launch_gemm<true, 1, 1, 256, 4, false>(ma, mb, M, N, k_blocks, ep, ldy, st);
    }
    if (!narrow) {
      NB_TRY(make_operand_map(&mb, B, true, K, pitch_b, N, 1, 128));
      return launch_gemm<true, 1, 1, 128, 6, false>(ma, mb, M, N, k_blocks, ep, ldy, st);
    }
    NB_TRY(make_operand_map(&mb, B, true, K, pitch_b, N, 1, 64));
    return launch_gemm<true, 1, 1, 64, 8, false>(ma, mb, M, N, k_blocks, ep, ldy, st);
  }
  if (planes_a == 3 && planes_b == 1) {
    if (route == GemmRoute::kTransposed) {
      GemmTransposedProblem prob;
      fill_problem(prob, N, M, k_blocks, kTransposedRows, k_chunk_blocks(3 * 4), ldy);
      NB_TRY(make_operand_map(&ma, B, false, K, pitch_b, N, 1, kTileM));
      NB_TRY(make_operand_map(&mb, A, false, K, pitch_a, M, 3, kTransposedRows));
      auto launch = [&](const GemmTransposedProblem &p, const GemmEpilogue &e) {
        GemmEpilogue t = e;
        t.row_scale = e.col_scale, t.row_bias = e.col_bias;
        t.col_scale = t.col_bias = nullptr;
        return launch_contraction<false, 1, 3, kTransposedRows, 4, 0, GemmTransposedProblem>(
            ma, mb, p, p.k_splits * p.m_tiles * p.n_tiles, t, st);
      };
      return run_in_parts(prob, kTransposedBlockKb, M, N, ep, ldy, st, launch);
    }
    if (!narrow) {
      NB_TRY(make_operand_map(&mb, B, false, K, pitch_b, N, 1, 128));
      return launch_gemm<false, 3, 1, 128, 3, false>(ma, mb, M, N, k_blocks, ep, ldy, st);
    }
    NB_TRY(make_operand_map(&mb, B, false, K, pitch_b, N, 1, 64));
    return launch_gemm<false, 3, 1, 64, 3, false>(ma, mb, M, N, k_blocks, ep, ldy, st);
  }
  if (planes_a == 3 && planes_b == 3) {
    NB_TRY(make_operand_map(&mb, B, false, K, pitch_b, N, 3, 64));
    return launch_gemm<false, 3, 3, 64, 2, true>(ma, mb, M, N, k_blocks, ep, ldy, st);
  }
  return fail(NB200_ENOTIMPL, "no kernel for %d x %d operand planes", planes_a, planes_b);
}

static inline int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

static bool bf16_exact(float v) {
  uint32_t b;
  std::memcpy(&b, &v, 4);
  return (b & 0xffffu) == 0;
}

// Shared body of BinaryWeightAffine / BinaryConnectAffine forward.
static int binary_affine(const float *x, const float *w, float *wb, float *alpha, const float *bias, float *y,
                         int64_t M, int64_t K, int64_t N, float zero_to, cudaStream_t st) {
  NB_CHECK(M > 0 && K > 0 && N > 0, NB200_EVALUE, "empty operand (M=%lld K=%lld N=%lld)", (long long)M, (long long)K,
           (long long)N);
  NB_CHECK(M < (1ll << 31) && K < (1ll << 31) && N < (1ll << 31), NB200_EVALUE, "extent exceeds 2^31");
  NB_CHECK(x && w && wb && y, NB200_EVALUE, "null data pointer");
  NB_CHECK(bf16_exact(zero_to), NB200_ENOTIMPL,
           "quantize_zero_to = %g is not representable in bf16; the exact tensor-core path needs it to be", zero_to);
  if (small_gemm_binarized(M, N, K)) {
    SmallGemm P{};
    P.a = x, P.b = w, P.y = y;
    P.M = (int)M, P.N = (int)N, P.K = (int)K;
    P.col_bias = bias;
    P.zero_to = zero_to, P.inv = (float)1 / K; // binary_weight_affine.cpp:68
    P.wb = wb, P.alpha = alpha;
    return launch_small_gemm<false, false, SmallB::kBinarize>(P, st);
  }
  const int64_t Kp = round_up(K, 64);
  const size_t planes_bytes = (size_t)3 * M * Kp * 2;
  const size_t side_bytes = (size_t)N * Kp * 2;
  const size_t partial_bytes = alpha ? (size_t)((K + 63) / 64) * N * 4 : 0;
  AsyncScratch scratch(st);
  NB_TRY(scratch.alloc(round_up(planes_bytes, 256) + round_up(side_bytes, 256) + partial_bytes));
  uint8_t *base = static_cast<uint8_t *>(scratch.p);
  void *planes = base;
  void *side = base + round_up(planes_bytes, 256);
  float *partial = reinterpret_cast<float *>(base + round_up(planes_bytes, 256) + round_up(side_bytes, 256));
  GemmEpilogue ep{};
  ep.y = y;
  ep.scale = 1.0f;
  ep.col_scale = alpha;
  ep.col_bias = bias;
  // the transposed product makes alpha from the partial sums itself, unless its K is split
  const int k_blocks = (int)(Kp / 64);
  bool sums_left = alpha && gemm_route(false, 3, 1, (int)M, (int)N, k_blocks, ep, N) == GemmRoute::kTransposed &&
                   k_splits_for(transposed_tiles((int)M, (int)N), k_blocks, kTransposedBlockKb) == 1;
  NB_TRY(binary_affine_operands(x, M, w, (int)K, (int)N, zero_to, wb, alpha, side, Kp, partial, planes, st, &sums_left));
  if (sums_left) {
    ep.col_scale = nullptr;
    ep.alpha_partial = partial;
    ep.alpha_parts = (int)((K + 63) / 64);
    ep.alpha_inv = (float)1 / K; // binary_weight_affine.cpp:68
    ep.alpha = alpha;
  }
  return run_gemm(false, 3, 1, planes, Kp, side, Kp, (int)M, (int)N, (int)K, ep, N, st);
}

// Fills the epilogue's destinations for a column slab [col_begin, col_begin + n)
// of row-major [rows, n_total] matrices, one per rank: y_ranks[rank] is this
// GPU's own matrix, the others are peer mappings, taken in ring order starting
// after this rank so that the ranks do not all write to the same peer first.
static int slab_destinations(GemmEpilogue &ep, float *const *y_ranks, int n_ranks, int rank, int64_t n,
                             int64_t n_total, int64_t col_begin) {
  NB_CHECK(y_ranks != nullptr, NB200_EVALUE, "y_ranks is NULL");
  NB_CHECK(n_ranks >= 1 && n_ranks <= kMaxPeers + 1, NB200_EVALUE, "n_ranks = %d outside [1, %d]", n_ranks,
           kMaxPeers + 1);
  NB_CHECK(rank >= 0 && rank < n_ranks, NB200_EVALUE, "rank %d outside [0, %d)", rank, n_ranks);
  NB_CHECK(col_begin >= 0 && n_total < (1ll << 31) && col_begin + n <= n_total, NB200_EVALUE,
           "column slab [%lld, %lld) outside [0, %lld)", (long long)col_begin, (long long)(col_begin + n),
           (long long)n_total);
  for (int r = 0; r < n_ranks; ++r)
    NB_CHECK(y_ranks[r] != nullptr, NB200_EVALUE, "y_ranks[%d] is NULL", r);
  ep.y = y_ranks[rank] + col_begin;
  ep.n_peers = n_ranks - 1;
  for (int j = 1; j < n_ranks; ++j)
    ep.peer_y[j - 1] = y_ranks[(rank + j) % n_ranks] + col_begin;
  return NB200_OK;
}

// w_kmajor: w_codes already holds the K-major layout [w_col][w_pitch] (nb200_transpose_codes_i8), so the
// re-layout pass is skipped (weights are parameters: their codes can be laid out once and reused).
static int affine_codes(const int8_t *x_codes, const int8_t *w_codes, float delta_x, float delta_w, const float *bias,
                        float *const *y_ranks, int n_ranks, int rank, int64_t rows, int64_t w_row, int64_t w_col,
                        int64_t n_total, int64_t col_begin, cudaStream_t st, bool w_kmajor = false,
                        int64_t w_pitch = 0) {
  const int64_t M = rows, K = w_row, N = w_col;
  NB_CHECK(M > 0 && K > 0 && N > 0, NB200_EVALUE, "empty operand");
  NB_CHECK(M < (1ll << 31) && K < (1ll << 31) && N < (1ll << 31), NB200_EVALUE, "extent exceeds 2^31");
  NB_CHECK(x_codes && w_codes, NB200_EVALUE, "null data pointer");
  // |acc| <= K * 127 * 127 must fit int32
  NB_CHECK(K <= 133000, NB200_ENOTIMPL, "K = %lld could overflow the int32 accumulator", (long long)K);
  GemmEpilogue ep{};
  NB_TRY(slab_destinations(ep, y_ranks, n_ranks, rank, N, n_total, col_begin));
  const int64_t Kp = round_up(K, 128);
  const bool x_direct = (K % 16 == 0) && ((reinterpret_cast<uintptr_t>(x_codes) & 15) == 0);
  if (w_kmajor)
    NB_CHECK(w_pitch >= K && w_pitch % 16 == 0 && (reinterpret_cast<uintptr_t>(w_codes) & 15) == 0, NB200_EVALUE,
             "K-major weight codes need a 16-byte aligned base and a pitch >= w_row that is a multiple of 16 (got %lld)",
             (long long)w_pitch);
  AsyncScratch scratch(st);
  NB_TRY(scratch.alloc((w_kmajor ? 0 : (size_t)N * Kp) + (x_direct ? 0 : (size_t)M * Kp) + 16));
  int8_t *wt = static_cast<int8_t *>(scratch.p);
  const int8_t *wk = w_codes;
  int64_t pitch_b = w_pitch;
  if (!w_kmajor) {
    NB_TRY(transpose_i8(w_codes, (int)K, (int)N, wt, Kp, st));
    wk = wt;
    pitch_b = Kp;
  }
  const int8_t *xa = x_codes;
  int64_t pitch_a = K;
  if (!x_direct) {
    int8_t *xc = wt + (w_kmajor ? 0 : (size_t)N * Kp);
    NB_CUDA(cudaMemcpy2DAsync(xc, (size_t)Kp, x_codes, (size_t)K, (size_t)K, (size_t)M, cudaMemcpyDeviceToDevice, st));
    xa = xc;
    pitch_a = Kp;
  }
  ep.scale = delta_x * delta_w;
  ep.col_bias = bias;
  return run_gemm(true, 1, 1, xa, pitch_a, wk, pitch_b, (int)M, (int)N, (int)K, ep, n_total, st);
}

static int affine_fxp8(const float *xq, const float *wq, float delta_x, float delta_w, const float *bias,
                       float *const *y_ranks, int n_ranks, int rank, int64_t rows, int64_t w_row, int64_t w_col,
                       int64_t n_total, int64_t col_begin, cudaStream_t st) {
  const int64_t M = rows, K = w_row, N = w_col;
  NB_CHECK(M > 0 && K > 0 && N > 0, NB200_EVALUE, "empty operand");
  NB_CHECK(M < (1ll << 31) && K < (1ll << 31) && N < (1ll << 31), NB200_EVALUE, "extent exceeds 2^31");
  NB_CHECK(xq && wq, NB200_EVALUE, "null data pointer");
  NB_CHECK(delta_x > 0.f && delta_w > 0.f, NB200_EVALUE, "step sizes must be positive");
  NB_CHECK(K <= 133000, NB200_ENOTIMPL, "K = %lld could overflow the int32 accumulator", (long long)K);
  GemmEpilogue ep{};
  NB_TRY(slab_destinations(ep, y_ranks, n_ranks, rank, N, n_total, col_begin));
  const int64_t Kp = round_up(K, 128);
  AsyncScratch scratch(st);
  NB_TRY(scratch.alloc((size_t)(M + N) * Kp));
  int8_t *xc = static_cast<int8_t *>(scratch.p);
  int8_t *wt = xc + (size_t)M * Kp;
  NB_TRY(fxp8_operands(xq, M, (int)K, Kp, delta_x, xc, wq, (int)N, delta_w, wt, st));
  ep.scale = delta_x * delta_w;
  ep.col_bias = bias;
  return run_gemm(true, 1, 1, xc, Kp, wt, Kp, (int)M, (int)N, (int)K, ep, n_total, st);
}

// Backward of y = x . W (+ b) for row-major x [M, K], W [K, N], dy [M, N]
// (Affine::backward_impl, src/nbla/function/generic/affine.cpp:98-138):
//   dx (+)= dy . W^T     A = dy [M][N], B = W [K][N]: both already contraction-major
//   dW (+)= x^T . dy     A = x^T [K][M], B = dy^T [N][M]: transposed while they are split
//   db (+)= column sums of dy
// `w_exact_bf16`: W holds values that are exact in bf16 (the +-1 / zero_to
// weights of the binary layers); it is then used as one bf16 plane and
// `w_col_scale` (alpha, per column of W, may be NULL) is folded into dy before
// the split, which reproduces the reference's products dy * (wb * alpha)
// rounding for rounding. Otherwise W is split into three pieces like x.
static int affine_backward(const float *x, const float *w, const float *w_col_scale, bool w_exact_bf16,
                           const float *dy, float *dx, float *dw, float *db, int64_t M, int64_t K, int64_t N,
                           int accum_dx, int accum_dw, int accum_db, cudaStream_t st) {
  NB_CHECK(M > 0 && K > 0 && N > 0, NB200_EVALUE, "empty operand (M=%lld K=%lld N=%lld)", (long long)M, (long long)K,
           (long long)N);
  NB_CHECK(M < (1ll << 31) && K < (1ll << 31) && N < (1ll << 31), NB200_EVALUE, "extent exceeds 2^31");
  NB_CHECK(dy != nullptr, NB200_EVALUE, "dy is NULL");
  NB_CHECK(!dx || w, NB200_EVALUE, "the gradient w.r.t. x needs the weights");
  NB_CHECK(!dw || x, NB200_EVALUE, "the gradient w.r.t. the weights needs x");
  SmallGemm sx{}, sw{};
  sx.a = dy, sx.b = w, sx.y = dx;
  sx.M = (int)M, sx.N = (int)K, sx.K = (int)N;
  sx.a_scale = w_col_scale;
  sx.accumulate = accum_dx;
  sw.a = x, sw.b = dy, sw.y = dw;
  sw.M = (int)K, sw.N = (int)N, sw.K = (int)M;
  sw.accumulate = accum_dw;
  sw.sums = db;
  sw.accumulate_sums = accum_db;
  const bool small_dx = dx && (w_exact_bf16 ? small_gemm_scaled(M, K, N) : small_gemm_plain(M, K, N));
  const bool small_dw = dw && small_gemm_transposed(K, N, M);
  if (small_dx && small_dw)
    NB_TRY(launch_small_gradients(sx, sw, st));
  else if (small_dx)
    NB_TRY((launch_small_gemm<false, true, SmallB::kPlain>(sx, st)));
  else if (small_dw && db)
    NB_TRY((launch_small_gemm<true, false, SmallB::kColumnSums>(sw, st)));
  else if (small_dw)
    NB_TRY((launch_small_gemm<true, false, SmallB::kPlain>(sw, st)));
  if (small_dx)
    dx = nullptr;
  if (small_dw)
    dw = db = nullptr;
  if (dx) {
    const int64_t Np = round_up(N, 64);
    const int planes_w = w_exact_bf16 ? 1 : 3;
    const size_t a_bytes = round_up((size_t)3 * M * Np * 2, 256), b_bytes = (size_t)planes_w * K * Np * 2;
    AsyncScratch scratch(st);
    NB_TRY(scratch.alloc(a_bytes + b_bytes));
    uint8_t *base = static_cast<uint8_t *>(scratch.p);
    NB_TRY(split_rows_bf16(SplitRows{dy, w_col_scale, base, M, (int)N, 3},
                           SplitRows{w, nullptr, base + a_bytes, K, (int)N, planes_w}, Np, st));
    GemmEpilogue ep{};
    ep.y = dx;
    ep.scale = 1.0f;
    ep.accumulate = accum_dx;
    NB_TRY(run_gemm(false, 3, planes_w, base, Np, base + a_bytes, Np, (int)M, (int)K, (int)N, ep, K, st));
  }
  if (dw) {
    const int64_t Mp = round_up(M, 64);
    const size_t a_bytes = round_up((size_t)3 * K * Mp * 2, 256), b_bytes = round_up((size_t)3 * N * Mp * 2, 256);
    const bool with_sums = db && Mp / 64 <= 256; // (one thread adds up a column's)
    AsyncScratch scratch(st);
    NB_TRY(scratch.alloc(a_bytes + b_bytes + (with_sums ? (size_t)(Mp / 64) * N * sizeof(float) : 0)));
    uint8_t *pa = static_cast<uint8_t *>(scratch.p), *pb = pa + a_bytes;
    float *sums = with_sums ? reinterpret_cast<float *>(pb + b_bytes) : nullptr;
    NB_TRY(split_columns_bf16(SplitColumns{x, pa, nullptr, M, (int)K, 3}, SplitColumns{dy, pb, sums, M, (int)N, 3}, Mp, st));
    if (with_sums) {
      NB_TRY(column_sums_finish(sums, (int)N, (int)(Mp / 64), db, accum_db, st));
      db = nullptr;
    }
    GemmEpilogue ep{};
    ep.y = dw;
    ep.scale = 1.0f;
    ep.accumulate = accum_dw;
    NB_TRY(run_gemm(false, 3, 3, pa, Mp, pb, Mp, (int)K, (int)N, (int)M, ep, N, st));
  }
  if (db) {
    int splits = (int)((M + 255) / 256);
    splits = splits > 64 ? 64 : splits;
    AsyncScratch scratch(st);
    NB_TRY(scratch.alloc((size_t)splits * N * 4));
    NB_TRY(column_sums(dy, M, (int)N, db, accum_db, static_cast<float *>(scratch.p), splits, st));
  }
  return NB200_OK;
}

} // namespace nb200

using namespace nb200;

extern "C" {

int nb200_take_device_status(int *code, void *stream) {
  NB_CHECK(code != nullptr, NB200_EVALUE, "code is NULL");
  int *word = nullptr;
  NB_TRY(device_status_word(&word));
  NB_CUDA(cudaStreamSynchronize(as_stream(stream)));
  NB_CUDA(cudaMemcpy(code, word, sizeof(int), cudaMemcpyDeviceToHost));
  if (*code != 0)
    NB_CUDA(cudaMemset(word, 0, sizeof(int)));
  return NB200_OK;
}

int nb200_binary_weight_affine_f32(const float *x, const float *w, float *wb, float *alpha, const float *bias,
                                   float *y, int64_t rows, int64_t w_row, int64_t w_col, float quantize_zero_to,
                                   void *stream) {
  NB_CHECK(alpha != nullptr, NB200_EVALUE, "alpha is NULL");
  return binary_affine(x, w, wb, alpha, bias, y, rows, w_row, w_col, quantize_zero_to, as_stream(stream));
}

int nb200_binary_connect_affine_f32(const float *x, const float *w, float *wb, const float *bias, float *y,
                                    int64_t rows, int64_t w_row, int64_t w_col, float quantize_zero_to,
                                    void *stream) {
  return binary_affine(x, w, wb, nullptr, bias, y, rows, w_row, w_col, quantize_zero_to, as_stream(stream));
}

int nb200_affine_codes_i8_f32(const int8_t *x_codes, const int8_t *w_codes, float delta_x, float delta_w,
                              const float *bias, float *y, int64_t rows, int64_t w_row, int64_t w_col,
                              void *stream) {
  NB_CHECK(y != nullptr, NB200_EVALUE, "null data pointer");
  float *const ys[1] = {y};
  return affine_codes(x_codes, w_codes, delta_x, delta_w, bias, ys, 1, 0, rows, w_row, w_col, w_col, 0,
                      as_stream(stream));
}

int nb200_affine_codes_i8_gather_f32(const int8_t *x_codes, const int8_t *w_codes, float delta_x, float delta_w,
                                     const float *bias, float *const *y_ranks, int n_ranks, int rank, int64_t rows,
                                     int64_t w_row, int64_t w_col, int64_t w_col_total, int64_t col_begin,
                                     void *stream) {
  return affine_codes(x_codes, w_codes, delta_x, delta_w, bias, y_ranks, n_ranks, rank, rows, w_row, w_col,
                      w_col_total, col_begin, as_stream(stream));
}

int nb200_affine_fxp8_f32(const float *xq, const float *wq, float delta_x, float delta_w, const float *bias, float *y,
                          int64_t rows, int64_t w_row, int64_t w_col, void *stream) {
  NB_CHECK(y != nullptr, NB200_EVALUE, "null data pointer");
  float *const ys[1] = {y};
  return affine_fxp8(xq, wq, delta_x, delta_w, bias, ys, 1, 0, rows, w_row, w_col, w_col, 0, as_stream(stream));
}

int nb200_affine_fxp8_gather_f32(const float *xq, const float *wq, float delta_x, float delta_w, const float *bias,
                                 float *const *y_ranks, int n_ranks, int rank, int64_t rows, int64_t w_row,
                                 int64_t w_col, int64_t w_col_total, int64_t col_begin, void *stream) {
  return affine_fxp8(xq, wq, delta_x, delta_w, bias, y_ranks, n_ranks, rank, rows, w_row, w_col, w_col_total,
                     col_begin, as_stream(stream));
}

int nb200_affine_f32(const float *x, const float *w, const float *bias, float *y, int64_t rows, int64_t w_row,
                     int64_t w_col, void *stream) {
  const int64_t M = rows, K = w_row, N = w_col;
  NB_CHECK(M > 0 && K > 0 && N > 0, NB200_EVALUE, "empty operand");
  NB_CHECK(M < (1ll << 31) && K < (1ll << 31) && N < (1ll << 31), NB200_EVALUE, "extent exceeds 2^31");
  NB_CHECK(x && w && y, NB200_EVALUE, "null data pointer");
  cudaStream_t st = as_stream(stream);
  if (small_gemm_plain(M, N, K)) {
    SmallGemm P{};
    P.a = x, P.b = w, P.y = y;
    P.M = (int)M, P.N = (int)N, P.K = (int)K;
    P.col_bias = bias;
    return launch_small_gemm<false, false, SmallB::kPlain>(P, st);
  }
  const int64_t Kp = round_up(K, 64);
  AsyncScratch scratch(st);
  const size_t xa = round_up((size_t)3 * M * Kp * 2, 256), wa = round_up((size_t)3 * N * Kp * 2, 256);
  NB_TRY(scratch.alloc(xa + wa));
  uint8_t *base = static_cast<uint8_t *>(scratch.p);
  NB_TRY(split_rows_bf16(SplitRows{x, nullptr, base, M, (int)K, 3}, SplitRows{}, Kp, st));
  NB_TRY(split_columns_bf16(SplitColumns{w, base + xa, nullptr, K, (int)N, 3}, SplitColumns{}, Kp, st));
  GemmEpilogue ep{};
  ep.y = y;
  ep.scale = 1.0f;
  ep.col_bias = bias;
  return run_gemm(false, 3, 3, base, Kp, base + xa, Kp, (int)M, (int)N, (int)K, ep, N, st);
}

int nb200_affine_backward_f32(const float *x, const float *w, const float *dy, float *dx, float *dw, float *db,
                              int64_t rows, int64_t w_row, int64_t w_col, int accum_dx, int accum_dw, int accum_db,
                              void *stream) {
  return affine_backward(x, w, nullptr, false, dy, dx, dw, db, rows, w_row, w_col, accum_dx, accum_dw, accum_db,
                         as_stream(stream));
}

int nb200_binary_weight_affine_backward_f32(const float *x, const float *wb, const float *alpha, const float *dy,
                                            float *dx, float *dw, float *db, int64_t rows, int64_t w_row,
                                            int64_t w_col, int accum_dx, int accum_dw, int accum_db, void *stream) {
  NB_CHECK(alpha != nullptr || dx == nullptr, NB200_EVALUE, "alpha is NULL");
  return affine_backward(x, wb, alpha, true, dy, dx, dw, db, rows, w_row, w_col, accum_dx, accum_dw, accum_db,
                         as_stream(stream));
}

int nb200_binary_connect_affine_backward_f32(const float *x, const float *wb, const float *dy, float *dx, float *dw,
                                             float *db, int64_t rows, int64_t w_row, int64_t w_col, int accum_dx,
                                             int accum_dw, int accum_db, void *stream) {
  return affine_backward(x, wb, nullptr, true, dy, dx, dw, db, rows, w_row, w_col, accum_dx, accum_dw, accum_db,
                         as_stream(stream));
}

int nb200_transpose_codes_i8(const int8_t *w_codes, int8_t *w_codes_kmajor, int64_t w_row, int64_t w_col,
                             int64_t pitch, void *stream) {
  NB_CHECK(w_codes && w_codes_kmajor, NB200_EVALUE, "null data pointer");
  NB_CHECK(w_row > 0 && w_col > 0 && w_row < (1ll << 31) && w_col < (1ll << 31), NB200_EVALUE, "bad extents");
  NB_CHECK(pitch >= w_row, NB200_EVALUE, "pitch %lld is smaller than w_row %lld", (long long)pitch, (long long)w_row);
  if (pitch > w_row) // the padding must read as zero codes
    NB_CUDA(cudaMemsetAsync(w_codes_kmajor, 0, (size_t)w_col * pitch, as_stream(stream)));
  return transpose_i8(w_codes, (int)w_row, (int)w_col, w_codes_kmajor, pitch, as_stream(stream));
}

int nb200_affine_codes_i8_kmajor_f32(const int8_t *x_codes, const int8_t *w_codes_kmajor, int64_t w_pitch,
                                     float delta_x, float delta_w, const float *bias, float *y, int64_t rows,
                                     int64_t w_row, int64_t w_col, void *stream) {
  NB_CHECK(y != nullptr, NB200_EVALUE, "null data pointer");
  float *const ys[1] = {y};
  return affine_codes(x_codes, w_codes_kmajor, delta_x, delta_w, bias, ys, 1, 0, rows, w_row, w_col, w_col, 0,
                      as_stream(stream), true, w_pitch);
}
}
