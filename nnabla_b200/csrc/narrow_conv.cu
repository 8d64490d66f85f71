// Full-precision convolution of an input with FEW channels (the 7x7 / stride 2
// stem of a residual network: 3 channels) on the tcgen05 tensor cores.
//
// Convolution<float>::forward_impl (src/nbla/function/generic/convolution.cpp:160-197)
// unfolds every sample to patches and multiplies. Here the product is an
// implicit GEMM whose rows are the pixels of ONE output row (M = 128 >= Wo) and
// whose columns are the output maps (64 >= Ko). No patch matrix is ever built,
// neither in global nor in shared memory:
//
//   1. A pre-pass writes x channel-last in fp16, every pixel in a slot of
//      16 / stride_w bytes (4 channels at stride 2, 8 at stride 1), rows and
//      columns zero-padded. A slot group of 16 bytes then holds the stride_w
//      pixels that separate two neighbouring outputs, so "output pixel m, filter
//      taps kx = c * stride_w .. (c + 1) * stride_w - 1" is the 16-byte unit m + c
//      of the staged input row.
//   2. The tensor core reads that row in place. An un-swizzled K-major operand is
//      addressed as start + (row / 8) * 128 + (row % 8) * 16 + chunk * LBO; with
//      LBO = 16 the second K chunk of row m is the first one of row m + 1: the
//      overlapping windows of a convolution, straight from the staged row. One
//      instruction (K = 16) covers 2 * stride_w filter taps of one filter row;
//      a 7x7 / stride 2 filter takes 7 x 2 of them.
//   3. The staged rows of a persistent block form a ring in shared memory: the
//      next output row needs stride_h new input rows, fetched with one bulk copy
//      each (both pieces of a row are contiguous); the other rows are reused.
//   4. fp32 accuracy from fp16 operands: x * 2^-e = x0 + 2^-11 x1 and
//      w * 2^S = w0 + 2^-11 w1 with fp16 x0, x1, w0, w1 (e per sample from
//      max |x|, S from max |w|, so that every piece is in fp16's normal range and
//      a residual keeps 11 more bits: 22 bits in all). The weights are stacked along
//      N: x0 x [w0; w1] (N = 128) gives the main product in TMEM columns 0..63
//      and one cross product in 64..127; x1 x [w0] (N = 64) accumulates the other
//      cross product there as well. The epilogue forms
//      (main + 2^-11 cross) * 2^(e - S). The product left out, x1 w1, is 2^-22 of
//      the main one, the size of the representation error.
//
// Warps: two sets of eight for the epilogue (TMEM lanes = pixels, columns = maps; warp w of a set takes lanes 32 (w % 4)
// and maps 32 (w / 4)), two MMA issuers, each with every other tile and an accumulator of its own, and a loader. With one
// issuer and one set the tensor core waited for the issue of 28 MMAs with their addresses (each MMA is as short as its
// issue) and for the epilogue of the tile before the last: 2680 cycles per tile of 1660 cycles of MMAs, 73 us for the
// codes of 64 x 3 x 224 x 224, now 64. Every mbarrier wait is time-bounded; a wait that gives
// up stores a code in *status and raises the block's abort flag, every role then
// falls through to the common teardown.
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "pdl.cuh"
#include "narrow_conv.cuh"
#include "ptx.cuh"

namespace nb200 {

int device_status_word(int **status); // gemm.cu
int encode_tiled(CUtensorMap *map, int dtype_code, int rank, const void *base, const uint64_t *dims,
                 const uint64_t *strides_bytes, const uint32_t *box, const uint32_t *elem_strides, int swizzle_bytes);

namespace {

constexpr int kSetWarps = 8, kEpilogueWarps = 2 * kSetWarps, kMmaWarp = kEpilogueWarps, kLoadWarp = kMmaWarp + 2;
constexpr int kThreadsNC = 32 * (kLoadWarp + 1);
constexpr int kM = 128, kN = 64;
constexpr int kMaxSteps = 16;             // K steps of 16 values: kernel_h * ceil(kernel_w / (2 * stride_w))
constexpr int kStepBytes = 2 * kN * 32;   // resident weights of one K step: [w0; w1] x 16 values
constexpr int kRing = 16;                 // staged input rows kept in shared memory
constexpr int kMaxKh = 8;
constexpr int kMaxRowBytes = 2560;        // one piece of one staged row
constexpr int kInFlight = 8;              // tiles between the loader and the completed MMAs (barrier ring)
constexpr size_t kMaxSmemNC = 224 * 1024;
constexpr int kAccCols = 128;             // TMEM columns of one accumulator: main | cross

constexpr int kStatusNcMmaTimeout = 0x202;
constexpr int kStatusNcEpilogueTimeout = 0x203;
constexpr int kStatusNcLoadTimeout = 0x204;

struct NarrowConv {
  int N, C, H, W, Ko, kh, kw, ph, pw, sh, sw, Ho, Wo;
  int Hp;        // staged rows per sample: H + 2 * ph
  int row_bytes; // one piece of one staged row (a multiple of 16)
  int jsteps;    // K steps per filter row
};

// Result as int8 channel-last codes [N][Ho * Wo][slots] instead of fp32 NCHW: the epilogue applies
// ReLU (optional) and FixedPointQuantize (power-of-two step) to conv + bias and stores finished
// codes, 32 consecutive maps of a pixel per thread and chunk. codes == NULL: fp32 result.
struct NarrowCodesOut {
  int8_t *codes;
  int slots, relu, kmax, kmin;
  float two_inv; // 2 / delta
};

// Four codes in [-128, 127] (saturated) -> the four bytes of one word, a in the lowest.
__device__ __forceinline__ uint32_t pack_codes4(int a, int b, int c, int d) {
  uint32_t hi, out;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(d), "r"(c), "r"(0));
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(out) : "r"(b), "r"(a), "r"(hi));
  return out;
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// e with max * 2^-e in [2^top, 2^(top + 1)) for the largest magnitude `maxbits` (fp32 bits of a
// non-negative value); 0 for zero, denormal and non-finite maxima.
__device__ __forceinline__ int scale_exponent(uint32_t maxbits, int top) {
  const int E = (int)(maxbits >> 23);
  if (E == 0 || E >= 255)
    return 0;
  const int e = E - 127 - top;
  return e < -120 ? -120 : e;
}
__device__ __forceinline__ float pow2i(int e) { return __int_as_float((127 + e) << 23); } // -126 <= e <= 127

// v = p0 + 2^-11 p1 up to 2^-22 |v| (v within fp16's range)
__device__ __forceinline__ void split2(float v, __half &p0, __half &p1) {
  p0 = __float2half_rn(v);
  p1 = __float2half_rn(__fmul_rn(__fsub_rn(v, __half2float(p0)), 2048.0f));
}

// x [N][C][H][W] fp32 -> xs [N][Hp][piece][row_bytes] fp16: unit u of a row holds the stride_w pixels
// u * stride_w .. (padded column), 8 / stride_w channel slots each; zero outside the image and past C.
// One block per (split_rows staged rows, sample), the samples last to first, against the order that the maxima were taken
// in, so that many of them still come from L2; xscale[n] = 2^e of the sample. Bound by the latency of its loads: a thread's
// loads of kUnits units go out together, four where a block has eight rows (the whole function [64, 3, 224, 224] 96.2 us with
// one at a time, 94.6 with four; 256 images 343 and 337), one where it has two.
constexpr int kAbsmaxParts = 32; // shares of a sample, what a warp reads back at once
template <int SW, int kUnits>
__global__ void __launch_bounds__(256) narrow_conv_split_kernel(const float *__restrict__ x, NarrowConv g, int split_rows,
                                                                const uint32_t *__restrict__ maxbits, int parts,
                                                                uint8_t *__restrict__ xs, float *__restrict__ xscale) {
  pdl_wait();
  pdl_trigger();
  constexpr int cpp = 8 / SW; // channel slots per pixel
  const int n = gridDim.y - 1 - blockIdx.y;
  const int lane = threadIdx.x & 31;
  const int units = g.row_bytes >> 4;
  const int py0 = blockIdx.x * split_rows;
  const int rows = min(split_rows, g.Hp - py0);
  float down = 0.0f;
  const uint32_t part = lane < parts ? __ldg(maxbits + n * parts + lane) : 0u;
  for (int base = 0; base < rows * units; base += 256 * kUnits) {
    const int i0 = base + threadIdx.x;
    float v[kUnits][8];
#pragma unroll
    for (int q = 0; q < kUnits; ++q) {
      const int i = i0 + 256 * q, r = i / units, u = i - r * units;
      const int iy = py0 + r - g.ph;
      const bool row_in = i < rows * units && iy >= 0 && iy < g.H;
      const float *src = x + ((int64_t)n * g.C * g.H + iy) * g.W;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int t = k / cpp, c = k % cpp;
        const int ix = u * SW + t - g.pw;
        v[q][k] = row_in && c < g.C && ix >= 0 && ix < g.W ? __ldg(src + (int64_t)c * g.H * g.W + ix) : 0.0f;
      }
    }
    if (base == 0) { // (behind the first loads)
      const int e = scale_exponent(__reduce_max_sync(0xffffffffu, part), 14);
      down = pow2i(-e);
      if (blockIdx.x == 0 && threadIdx.x == 0)
        xscale[n] = pow2i(e);
    }
#pragma unroll
    for (int q = 0; q < kUnits; ++q) {
      const int i = i0 + 256 * q, r = i / units, u = i - r * units;
      if (i >= rows * units)
        break;
      __align__(16) __half p0[8], p1[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        split2(__fmul_rn(v[q][k], down), p0[k], p1[k]);
      uint8_t *row = xs + ((int64_t)n * g.Hp + py0 + r) * 2 * g.row_bytes;
      *reinterpret_cast<uint4 *>(row + (size_t)u * 16) = *reinterpret_cast<const uint4 *>(p0);
      *reinterpret_cast<uint4 *>(row + g.row_bytes + (size_t)u * 16) = *reinterpret_cast<const uint4 *>(p1);
    }
  }
}

// w [Ko][C][kh][kw] fp32 -> wprep [step][group of 8 rows][chunk][row % 8][8] fp16, rows = [w0 (64); w1 (64)]
// of w * 2^S, the layout the tensor core reads without swizzle (8 x 16-byte core matrices contiguous;
// chunk stride 128, group stride 256 bytes). Step = (ky, j); value k of chunk c2 is tap
// kx = (2 j + c2) * stride_w + k / cpp, channel k % cpp. One block per step (every block finds max |w|
// for itself: the filter is a few thousand values); wscale[0] = 2^-S.
// The blocks behind those of the weights take shares of the samples: maxbits[sample][parts] receives the fp32 bits of
// each share's largest |x| (non-negative floats order like their bits; a NaN ends above infinity).
__global__ void __launch_bounds__(256) narrow_conv_prepare_kernel(const float *__restrict__ w, NarrowConv g, int steps,
                                                                  __half *__restrict__ out, float *__restrict__ wscale,
                                                                  const float *__restrict__ x, int64_t per_sample,
                                                                  int parts, uint32_t *__restrict__ maxbits) {
  pdl_wait();
  pdl_trigger();
  __shared__ uint32_t part[8];
  uint32_t m = 0;
  if ((int)blockIdx.x >= steps) {
    const int share = blockIdx.x - steps, n = share / parts, q = share - n * parts;
    const float *xs = x + (int64_t)n * per_sample;
    const int64_t begin = per_sample / 4 * q / parts * 4;
    const int64_t end = q + 1 == parts ? per_sample : per_sample / 4 * (q + 1) / parts * 4;
    if (((reinterpret_cast<uintptr_t>(x) & 15) | (per_sample & 3)) == 0) {
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
    if ((threadIdx.x & 31) == 0)
      part[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
      m = __reduce_max_sync(0xffffffffu, threadIdx.x < 8 ? part[threadIdx.x] : 0u);
      if (threadIdx.x == 0)
        maxbits[share] = m;
    }
    return;
  }
  const int count = g.Ko * g.C * g.kh * g.kw;
#pragma unroll 8
  for (int i = threadIdx.x; i < count; i += 256)
    m = max(m, __float_as_uint(fabsf(__ldg(w + i))));
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0)
    part[threadIdx.x >> 5] = m;
  __syncthreads();
  m = part[0];
  for (int i = 1; i < 8; ++i)
    m = max(m, part[i]);
  const int e = scale_exponent(m, 13);
  const float down = pow2i(-e);
  if (threadIdx.x == 0 && blockIdx.x == 0)
    wscale[0] = pow2i(e);
  const int cpp = 8 / g.sw;
  const int s = blockIdx.x;
  for (int rem = threadIdx.x; rem < kN * 16; rem += 256) { // (map, K value); both pieces
    const int o = rem >> 4, kk = rem & 15;
    const int c2 = kk >> 3, k = kk & 7;
    const int ky = s / g.jsteps, j = s - ky * g.jsteps;
    const int t = k / cpp, c = k - t * cpp;
    const int kx = (2 * j + c2) * g.sw + t;
    float v = 0.0f;
    if (o < g.Ko && c < g.C && kx < g.kw)
      v = __fmul_rn(w[((o * g.C + c) * g.kh + ky) * g.kw + kx], down);
    __half p0, p1;
    split2(v, p0, p1);
    __half *base = out + (size_t)s * (kStepBytes / 2);
    base[(((o >> 3) * 2 + c2) * 8 + (o & 7)) * 8 + k] = p0;
    base[((((o + kN) >> 3) * 2 + c2) * 8 + (o & 7)) * 8 + k] = p1;
  }
}

// The staged rows a tile needs and where they sit in the ring. Loader and MMA issuer walk the same
// sequence of tiles and keep one of these each: rows are loaded in increasing order within a sample,
// every loaded row takes the next ring slot (count % kRing).
struct RowWalk {
  int count = 0;       // rows loaded so far by this block
  int sample = -1;     // sample of the previous tile
  int loaded_upto = 0; // first staged row of `sample` that is not in the ring
  // Advances to the tile (n, first row r0, kh rows); returns the number of rows to load, the first of
  // them in `first`, and the load count of row r0 in `s0`.
  __device__ __forceinline__ int next(int n, int r0, int kh, int &first, int &s0) {
    if (n != sample || r0 > loaded_upto) {
      sample = n;
      loaded_upto = r0;
    }
    first = loaded_upto;
    s0 = count - (loaded_upto - r0);
    const int nload = r0 + kh - first;
    count += nload;
    loaded_upto = r0 + kh;
    return nload;
  }
};

__global__ void __launch_bounds__(kThreadsNC, 1)
    narrow_conv_tcgen05_kernel(const __grid_constant__ CUtensorMap map_y, int box_store,
                               const uint8_t *__restrict__ xs, const uint8_t *__restrict__ wprep,
                               const float *__restrict__ xscale, const float *__restrict__ wscale,
                               const float *__restrict__ bias, float *__restrict__ y, NarrowConv g, int *status,
                               NarrowCodesOut co) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  const int steps = g.kh * g.jsteps;
  const uint32_t slot_bytes = 2u * (uint32_t)g.row_bytes;
  // rows past Wo of the last ring slot read up to (kM + 2 * jsteps) units of its second piece
  const uint32_t tail = (uint32_t)(kM + 2 * g.jsteps) * 16u;
  uint8_t *b_res = smem;                           // [step][16 groups][2 chunks][8 rows][16 B]
  uint8_t *ring = b_res + (size_t)steps * kStepBytes; // [slot][piece][row_bytes]
  // fp32 result: every epilogue warp stages a [32 maps][32 pixels] box for bulk stores
  float *stage = reinterpret_cast<float *>(ring + ((kRing * slot_bytes + tail + 127u) & ~127u));
  uint64_t *bars = reinterpret_cast<uint64_t *>(stage + kEpilogueWarps * 1024);
  uint64_t *full_bar = bars, *done_bar = bars + kInFlight, *tmem_full = bars + 2 * kInFlight,
           *tmem_empty = bars + 2 * kInFlight + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kInFlight + 4);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // consecutive output rows per block, so that a tile finds most of its input rows in the ring
  const int num_tiles = g.N * g.Ho;
  const int tile_first = (int)((int64_t)num_tiles * blockIdx.x / gridDim.x);
  const int tile_last = (int)((int64_t)num_tiles * (blockIdx.x + 1) / gridDim.x);
  constexpr uint32_t kTmemCols = 2 * kAccCols;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kInFlight; ++s) {
      ptx::mbar_init(full_bar + s, 1);
      ptx::mbar_init(done_bar + s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(tmem_full + s, 1);
      ptx::mbar_init(tmem_empty + s, kSetWarps);
    }
    *abort_flag = 0;
    ptx::mbar_fence_init();
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc(tmem_slot, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads(); // the block has its tensor memory before it lets the successor in
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  if (early_trigger((int64_t)g.N * g.Ko * g.Ho * g.Wo))
    pdl_trigger();
  // bias of every map (0 past Ko or without bias), times 2 / delta (ReLU: over 256) when codes are written
  __shared__ __align__(16) float bias_s[kN];
  if (threadIdx.x < kN)
    bias_s[threadIdx.x] = (bias && (int)threadIdx.x < g.Ko)
                              ? (co.codes ? __fmul_rn(bias[threadIdx.x], co.relu ? co.two_inv * 0.00390625f : co.two_inv)
                                          : bias[threadIdx.x])
                              : 0.0f;
  {
    // resident weights (already in the tensor core's layout) and zeros behind the ring
    const uint4 *src = reinterpret_cast<const uint4 *>(wprep);
    const int vecs = steps * (kStepBytes / 16);
    for (int i = threadIdx.x; i < vecs; i += kThreadsNC)
      reinterpret_cast<uint4 *>(b_res)[i] = __ldg(src + i);
    for (uint32_t i = threadIdx.x; i < tail / 16u; i += kThreadsNC)
      reinterpret_cast<uint4 *>(ring + kRing * slot_bytes)[i] = make_uint4(0, 0, 0, 0);
    fence_async_smem();
  }
  __syncthreads();

  if (warp == kLoadWarp) {
    // ------------------------------------------------------------ loader: the new rows of every tile
    if (ptx::elect_one()) {
      RowWalk walk, behind; // of the tile to load, of the oldest tile that may still be read
      int seq = 0, oldest = 0, ignored, oldest_s0;
      int n = tile_first / g.Ho, oy = tile_first - n * g.Ho, old_n = n, old_oy = oy;
      behind.next(old_n, old_oy * g.sh, g.kh, ignored, oldest_s0);
      bool ok = true;
      for (int tile = tile_first; tile < tile_last && ok; ++tile, ++seq) {
        int first, s0;
        const int count_before = walk.count;
        const int nload = walk.next(n, oy * g.sh, g.kh, first, s0);
        // ring slots about to be overwritten must have been released by the tiles that used them, and the barrier of
        // this tile by the tile seven before: an issuer also waits for the barrier of the tile before its own, which
        // must not have gone round by then
        while (oldest < seq && (oldest_s0 + kRing < walk.count || seq - oldest >= kInFlight - 1)) {
          if (!ptx::mbar_wait(done_bar + (oldest & (kInFlight - 1)), (uint32_t)(oldest / kInFlight) & 1u, abort_flag)) {
            if (*abort_flag == 0)
              atomicCAS(status, 0, kStatusNcLoadTimeout);
            *abort_flag = 1;
            ok = false;
            break;
          }
          ++oldest;
          if (++old_oy == g.Ho)
            old_oy = 0, ++old_n;
          behind.next(old_n, old_oy * g.sh, g.kh, ignored, oldest_s0);
        }
        if (!ok)
          break;
        uint64_t *bar = full_bar + (seq & (kInFlight - 1));
        ptx::mbar_expect_tx(bar, (uint32_t)nload * slot_bytes);
        const uint8_t *src = xs + ((int64_t)n * g.Hp + first) * slot_bytes;
        for (int i = 0; i < nload; ++i)
          ptx::bulk_load(ring + (uint32_t)((count_before + i) % kRing) * slot_bytes, src + (int64_t)i * slot_bytes,
                         slot_bytes, bar);
        if (++oy == g.Ho)
          oy = 0, ++n;
      }
    }
  } else if (warp >= kMmaWarp) {
    // ------------------------------------------------------------- MMA issuers
    if (ptx::elect_one()) {
      const int who = warp - kMmaWarp; // takes the tiles with seq % 2 == who
      RowWalk walk;
      int seq = 0;
      bool ok = true;
      const uint32_t idesc128 = ptx::make_idesc(1u, 0u, kM, 128), idesc64 = ptx::make_idesc(1u, 0u, kM, 64);
      // the MMAs of a tile are issued from one straight piece of code with every address at hand
      const uint64_t a_base = ptx::smem_desc_k_plain(ptx::smem_u32(ring), 16u, 128u);
      const uint64_t b_base = ptx::smem_desc_k_plain(ptx::smem_u32(b_res), 128u, 256u);
      const uint32_t slot_units = slot_bytes >> 4, piece_units = (uint32_t)g.row_bytes >> 4;
      int step_ky[kMaxSteps];
      uint32_t step_unit[kMaxSteps];
#pragma unroll
      for (int s = 0; s < kMaxSteps; ++s) {
        step_ky[s] = s / g.jsteps;
        step_unit[s] = 2u * (uint32_t)(s - step_ky[s] * g.jsteps);
      }
      int n = tile_first / g.Ho, oy = tile_first - n * g.Ho;
      for (int tile = tile_first; tile < tile_last && ok; ++tile, ++seq) {
        int first, s0;
        walk.next(n, oy * g.sh, g.kh, first, s0);
        if (++oy == g.Ho)
          oy = 0, ++n;
        if ((seq & 1) != who)
          continue;
        uint32_t a_unit[kMaxSteps]; // rows 16 bytes apart, the second K chunk 16 bytes behind the first: sliding windows
#pragma unroll
        for (int s = 0; s < kMaxSteps; ++s)
          a_unit[s] = (uint32_t)((s0 + step_ky[s]) & (kRing - 1)) * slot_units + step_unit[s];
        // rows of this tile that an earlier one asked for too came with that one's barrier
        const int before = seq == 0 ? 0 : seq - 1;
        if (!ptx::mbar_wait(tmem_empty + who, ((uint32_t)(seq >> 1) & 1u) ^ 1u, abort_flag) ||
            !ptx::mbar_wait(full_bar + (before & (kInFlight - 1)), (uint32_t)(before / kInFlight) & 1u, abort_flag) ||
            !ptx::mbar_wait(full_bar + (seq & (kInFlight - 1)), (uint32_t)(seq / kInFlight) & 1u, abort_flag)) {
          if (*abort_flag == 0)
            atomicCAS(status, 0, kStatusNcMmaTimeout);
          *abort_flag = 1;
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + (uint32_t)(who * kAccCols);
#pragma unroll
        for (int s = 0; s < kMaxSteps; ++s) {
          if (s < steps) {
            const uint64_t a0 = a_base + a_unit[s], b = b_base + (uint64_t)(s * (kStepBytes / 16));
            ptx::mma_bf16(d_tmem, a0, b, idesc128, s > 0);                  // x0 x [w0; w1] -> columns 0..127
            ptx::mma_bf16(d_tmem + kN, a0 + piece_units, b, idesc64, 1u);   // x1 x [w0]     -> columns 64..127
          }
        }
        ptx::mma_commit(done_bar + (seq & (kInFlight - 1)));
        ptx::mma_commit(tmem_full + who);
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int quarter = warp & 3; // TMEM lanes [32 * quarter, 32 * quarter + 32)
    const int half = warp >> 2 & 1; // maps [32 * half, 32 * half + 32)
    const int set = warp / kSetWarps; // tiles with seq % 2 == set, in its issuer's accumulator
    uint32_t phase = 0;
    const int px = quarter * 32 + lane;
    const int64_t plane = (int64_t)g.Ho * g.Wo;
    const float ws = __ldg(wscale);
    int n = (tile_first + set) / g.Ho, oy = tile_first + set - n * g.Ho;
    for (int tile = tile_first + set; tile < tile_last; tile += 2, phase ^= 1u) {
      const float scale = __fmul_rn(__ldg(xscale + n), ws); // 2^(e - S)
      const bool got = ptx::mbar_wait_backoff(tmem_full + set, phase, abort_flag, 20u);
      if (!__all_sync(0xffffffffu, got)) {
        if (lane == 0) {
          if (*abort_flag == 0)
            atomicCAS(status, 0, kStatusNcEpilogueTimeout);
          *abort_flag = 1;
        }
        break;
      }
      ptx::tc_fence_after_sync();
      float *yrow = y + (int64_t)n * g.Ko * plane + (int64_t)oy * g.Wo + px;
      const uint32_t t0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(set * kAccCols);
      {
        uint32_t r0[32], r1[32];
        ptx::tmem_ld_32x32(t0 + (uint32_t)(half * 32), r0);      // x0 w0
        ptx::tmem_ld_32x32(t0 + (uint32_t)(kN + half * 32), r1); // x0 w1 + x1 w0, times 2^11
        ptx::tmem_ld_wait();
        // the accumulator is in registers: the MMAs of the tile after the next may start
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0)
          ptx::mbar_arrive(tmem_empty + set);
        if (co.codes != nullptr) {
          if (px < g.Wo && half * 32 < co.slots) {
            // u = conv * (2 / delta) + bias * (2 / delta), one fused multiply-add; then ReLU and the
            // quantizer of a non-negative value, (floor(u) + 1) >> 1 capped at kmax
            uint32_t wds[8];
            if (co.relu) {
              // floor(u) + 1 on the FMA pipe: u / 256 saturated to [0, 1] (a NaN becomes 0), capped, and scaled back
              // by an addition to 2^23 + 1 that rounds down; at most 255, so four of them shift as one word. Decided
              // per value, the branch and the conversions took 30 instructions where these are five.
              const float cap = (float)(2 * co.kmax) + 0.5f;
              const float k256 = __fmul_rn(__fmul_rn(scale, co.two_inv), 0.00390625f), cap256 = __fmul_rn(cap, 0.00390625f);
#pragma unroll
              for (int j4 = 0; j4 < 8; ++j4) {
                uint32_t c[4];
                const float4 b4 = *reinterpret_cast<const float4 *>(bias_s + half * 32 + 4 * j4);
                const float b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  const int j = 4 * j4 + k;
                  const float raw = __fmaf_rn(__uint_as_float(r1[j]), 0.00048828125f, __uint_as_float(r0[j]));
                  const float u = fminf(__saturatef(__fmaf_rn(raw, k256, b[k])), cap256);
                  c[k] = __float_as_uint(__fmaf_rd(u, 256.0f, 8388609.0f));
                }
                wds[j4] = __byte_perm(__byte_perm(c[0], c[1], 0x0040), __byte_perm(c[2], c[3], 0x0040), 0x5410) >> 1 &
                          0x7f7f7f7fu;
              }
            } else {
              const float cap = (float)(2 * co.kmax) + 0.5f;
              const float k2 = __fmul_rn(scale, co.two_inv);
#pragma unroll
              for (int j4 = 0; j4 < 8; ++j4) {
                int c[4];
                const float4 b4 = *reinterpret_cast<const float4 *>(bias_s + half * 32 + 4 * j4);
                const float b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  const int j = 4 * j4 + k;
                  const float raw = __fmaf_rn(__uint_as_float(r1[j]), 0.00048828125f, __uint_as_float(r0[j]));
                  const float u = __fmaf_rn(raw, k2, b[k]);
                  const int m = (__float2int_rd(fminf(fabsf(u), cap)) + 1) >> 1;
                  c[k] = u < 0.0f ? max(-m, co.kmin) : m;
                }
                // maps past Ko have zero weights and zero bias: their code is 0 on its own
                wds[j4] = pack_codes4(c[0], c[1], c[2], c[3]);
              }
            }
            uint4 *cp = reinterpret_cast<uint4 *>(co.codes + ((int64_t)n * plane + (int64_t)oy * g.Wo + px) * co.slots +
                                                  half * 32);
            cp[0] = make_uint4(wds[0], wds[1], wds[2], wds[3]);
            if (half * 32 + 16 < co.slots)
              cp[1] = make_uint4(wds[4], wds[5], wds[6], wds[7]);
          }
        } else if (box_store) {
          // the copy engine writes the box: whole lines, clipped at Wo and Ko, while the warp goes on
          float *box = stage + warp * 1024;
          if (lane == 0)
            ptx::tma_store_wait_read<0>(); // the previous store has read the box
          __syncwarp();
          if (bias) {
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {
              const float4 b4 = *reinterpret_cast<const float4 *>(bias_s + half * 32 + 4 * j4);
              const float b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
              for (int j = 4 * j4; j < 4 * j4 + 4; ++j)
                box[j * 32 + lane] = __fadd_rn(
                    __fmul_rn(__fmaf_rn(__uint_as_float(r1[j]), 0.00048828125f, __uint_as_float(r0[j])), scale), b[j - 4 * j4]);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              box[j * 32 + lane] =
                  __fmul_rn(__fmaf_rn(__uint_as_float(r1[j]), 0.00048828125f, __uint_as_float(r0[j])), scale);
          }
          ptx::fence_async_shared();
          __syncwarp();
          if (lane == 0 && quarter * 32 < g.Wo && half * 32 < g.Ko) {
            ptx::tma_store_4d(&map_y, box, quarter * 32, oy, half * 32, n);
            ptx::tma_store_commit();
          }
        } else if (px < g.Wo) {
          float *yp = yrow + (int64_t)(half * 32) * plane;
#pragma unroll
          for (int j = 0; j < 32; ++j, yp += plane) {
            const int o = half * 32 + j;
            if (o < g.Ko) {
              float v = __fmul_rn(__fmaf_rn(__uint_as_float(r1[j]), 0.00048828125f, __uint_as_float(r0[j])), scale);
              if (bias)
                v = __fadd_rn(v, bias_s[o]);
              __stcs(yp, v);
            }
          }
        }
      }
      for (oy += 2; oy >= g.Ho; oy -= g.Ho)
        ++n;
    }
  }

  // ------------------------------------------------------------------ teardown
  if (warp < kEpilogueWarps && lane == 0)
    ptx::tma_store_wait_all(); // this thread's bulk stores have been written
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0) {
    // copies that may still be in flight must land before the shared memory is released
    const uint64_t t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 2000000ull)
      __nanosleep(1000);
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// K steps per filter row, bytes of one staged piece row, shared memory of the kernel
struct NarrowPlan {
  int jsteps, steps, row_bytes;
  size_t smem;
};

NarrowPlan narrow_plan(int width, int kernel_h, int kernel_w, int pad_w, int stride_w, int Wo) {
  NarrowPlan p;
  p.jsteps = (kernel_w + 2 * stride_w - 1) / (2 * stride_w);
  p.steps = kernel_h * p.jsteps;
  const int units_image = (width + 2 * pad_w + stride_w - 1) / stride_w;
  const int units_read = Wo - 1 + 2 * p.jsteps; // by rows that hold an output pixel
  p.row_bytes = 16 * (units_image > units_read ? units_image : units_read);
  const size_t ring = ((size_t)kRing * 2 * p.row_bytes + (size_t)(kM + 2 * p.jsteps) * 16 + 127) & ~size_t(127);
  p.smem = (size_t)p.steps * kStepBytes + ring + kEpilogueWarps * 4096 + (2 * kInFlight + 4) * 8 + 16 + 128;
  return p;
}

} // namespace

bool narrow_conv_applies(const float *x, int channels, int height, int width, int outmaps, int kernel_h,
                         int kernel_w, int pad_w, int stride_w, int dilation_h, int dilation_w, int group, int Wo) {
  static const bool off = []() {
    const char *e = std::getenv("NNABLA_B200_DIRECT_CONV");
    return e && e[0] == '1';
  }();
  if (off)
    return false;
  (void)x;
  (void)height;
  if (!(group == 1 && dilation_h == 1 && dilation_w == 1 && (stride_w == 1 || stride_w == 2) &&
        channels <= 8 / stride_w && outmaps <= kN && Wo <= kM && kernel_h <= kMaxKh))
    return false;
  const NarrowPlan p = narrow_plan(width, kernel_h, kernel_w, pad_w, stride_w, Wo);
  return p.steps <= kMaxSteps && p.row_bytes <= kMaxRowBytes && p.smem <= kMaxSmemNC;
}

int narrow_conv_tc(const float *x, const float *w, const float *bias, float *y, int batch, int channels, int height,
                   int width, int outmaps, int kernel_h, int kernel_w, int pad_h, int pad_w, int stride_h,
                   int stride_w, int Ho, int Wo, cudaStream_t st, int8_t *y_codes, int slots, int relu, int kmax,
                   int kmin, float delta) {
  NarrowCodesOut co{y_codes, slots, relu, kmax, kmin, y_codes ? 2.0f / delta : 0.0f};
  const NarrowPlan p = narrow_plan(width, kernel_h, kernel_w, pad_w, stride_w, Wo);
  NarrowConv g{batch,    channels, height, width, outmaps, kernel_h,          kernel_w,    pad_h,
               pad_w,    stride_h, stride_w, Ho,  Wo,      height + 2 * pad_h, p.row_bytes, p.jsteps};
  NB_CHECK(batch <= 65535 && g.Hp <= 65535, NB200_ENOTIMPL, "batch or padded height larger than 65535");
  // scratch: weights | staged input | per-sample maxima (bits) | per-sample 2^e | 2^-S
  const size_t w_bytes = (size_t)p.steps * kStepBytes;
  const size_t xs_bytes = (size_t)batch * g.Hp * 2 * p.row_bytes;
  const size_t tail_bytes = ((size_t)batch * 4 * (kAbsmaxParts + 1) + 16 + 255) & ~size_t(255);
  AsyncScratch scratch(st);
  NB_TRY(scratch.alloc(w_bytes + xs_bytes + tail_bytes));
  uint8_t *wprep = static_cast<uint8_t *>(scratch.p);
  uint8_t *xs = wprep + w_bytes;
  uint32_t *maxbits = reinterpret_cast<uint32_t *>(xs + xs_bytes);
  float *xscale = reinterpret_cast<float *>(maxbits + (size_t)batch * kAbsmaxParts);
  float *wscale = xscale + batch;
  const int64_t per_sample = (int64_t)channels * height * width;
  // shares of at least 4096 values, not many more than fill the chip twice (a block's start and end cost two microseconds)
  const int64_t most = std::min<int64_t>(kAbsmaxParts, 16ll * sm_count() / batch);
  const int parts = (int)std::max<int64_t>(1, std::min(per_sample / 4096, most));
  NB_CUDA(launch_dependent(narrow_conv_prepare_kernel, dim3((unsigned)(p.steps + batch * parts)), dim3(256), 0, st, w, g,
                           p.steps, reinterpret_cast<__half *>(wprep), wscale, x, per_sample, parts, maxbits));
  // eight rows per block (a few units per thread) where that gives every SM several blocks
  const int split_rows = (int64_t)batch * g.Hp >= 64ll * sm_count() ? 8 : 2;
  const dim3 split_grid((unsigned)((g.Hp + split_rows - 1) / split_rows), (unsigned)batch);
  auto split = stride_w == 2 ? (split_rows == 8 ? narrow_conv_split_kernel<2, 4> : narrow_conv_split_kernel<2, 1>)
                             : (split_rows == 8 ? narrow_conv_split_kernel<1, 4> : narrow_conv_split_kernel<1, 1>);
  NB_CUDA(launch_dependent(split, split_grid, dim3(256), 0, st, x, g, split_rows, maxbits, parts, xs, xscale));
  static std::atomic<bool> configured[64]{};
  int dev = 0;
  NB_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    NB_CUDA(cudaFuncSetAttribute(narrow_conv_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmemNC));
    configured[dev & 63] = true;
  }
  // y as (Wo, Ho, Ko, N) fp32 for the bulk stores of the fp32 result (needs 16-byte row pitch and base)
  CUtensorMap map_y;
  const bool box_store = y_codes == nullptr && (Wo % 4) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
  {
    const bool real = box_store;
    const uint64_t dims[4] = {(uint64_t)(real ? Wo : 32), (uint64_t)(real ? Ho : 1), (uint64_t)(real ? outmaps : 32),
                              (uint64_t)(real ? batch : 1)};
    const uint64_t strides[3] = {dims[0] * 4, dims[0] * dims[1] * 4, dims[0] * dims[1] * dims[2] * 4};
    const uint32_t box[4] = {32, 1, 32, 1};
    // without a usable y the map covers the (16-byte aligned) scratch and is never used
    NB_TRY(encode_tiled(&map_y, 2, 4, real ? static_cast<const void *>(y) : static_cast<const void *>(wprep), dims,
                        strides, box, nullptr, 0));
  }
  int *status = nullptr;
  NB_TRY(device_status_word(&status));
  const int tiles = batch * Ho;
  const int grid = tiles < sm_count() ? tiles : sm_count();
  NB_CUDA(launch_dependent(narrow_conv_tcgen05_kernel, dim3(grid), dim3(kThreadsNC), p.smem, st, map_y,
                           box_store ? 1 : 0, xs, wprep, xscale, wscale, bias, y, g, status, co));
  NB_LAUNCH_CHECK();
  return NB200_OK;
}

} // namespace nb200
