// Weight gradient of a convolution on tcgen05, straight from channel-last pieces:
//
//   dW[o][c][tap] = sum over images and output pixels of dy[pixel][o] * x[pixel * stride + tap][c]
//
// Both operands are read as they lie, pixels along K: a row of shared memory is one pixel's 64 channels, which is the
// MN-major operand layout (128-byte swizzle) of the tensor core, so nothing is transposed. A tap is a shift of the x
// box by whole rows (see conv_codes.cuh), so one box of x serves all taps of a task.
//
//   A (M = 128 rows)  two taps x 64 channels of x; the second tap's rows start at the leading byte offset, which is the
//                     distance between the two shifts
//   B (N columns)     the pieces of 64 maps of dy, side by side: 3 x 64 = 192 columns
//   D (TMEM)          fp32; columns 0 to 63 sum products of full magnitude, the others those 2^-8 and 2^-16 of it:
//                     x0 meets (d0, d1, d2), x1 meets (d0, d1) from column 64 on, x2 meets d0 from column 128 on
//
// Pixels run over the box's padded width; dy's box is as wide as x's with zeros (the copy engine's fill) where an
// output row has ended, and its rows up to a multiple of 16 are zeroed once.
//
// A task is (group, 64 maps, 64 channels, up to six taps that share a box; the third pair of taps has 128 columns left in
// tensor memory: column 0 to 63 as above, all other products in the rest). The tasks' boxes, weighted with their MMAs,
// are dealt out evenly to one block per SM; a block that ends a task or its share leaves its partial sums in a slot of
// its own and a second kernel adds the slots in order (deterministic). Every 96 accumulation steps the tensor memory
// is emptied into fp32 registers (gemm.cuh: the tensor core's additions truncate).
//
// What bounds it: 100 cycles per MMA of 192 columns and 16 pixels, the shared-memory traffic beside it (80 % for the
// operands, the rest for the copies), and beside both the L2: every task of up to six taps reads the boxes again. The
// previous form made the batch the K axis of an implicit GEMM (two transposing passes, K padded to 64 images per pixel):
// 216 us and 165 us of passes for 64 -> 64 maps on [128, 64, 56, 56], now 82 and a share of the preparation's 88, and
// 3 x the work at 20 images.
#pragma once
#include "gemm.cuh"

namespace nb200 {

constexpr int kWgradMaxTaps = 64;
constexpr int kWgradTaps = 6;                          // per task at most: three pairs

struct ConvWgradProblem {
  int tiles_h, boxes;               // boxes per image, in all
  int h_box, wp, hp;                // dy box: h_box rows of wp pixels; x box: hp rows of wp pixels
  int y0, x0;                       // x box origin relative to the dy box (in strided pixels)
  int sy, sx;                       // forward stride
  int groups, o_blocks, c_blocks, tap_groups;
  int k_stride, c_stride;           // channel slots between groups in dy / x
  int k16;                          // MMA steps per box
  int dy_bytes, x_bytes;            // of one plane's box in shared memory
  int x_planes;                     // 1 or 3
  int stages, flush;                // ring depth; boxes per accumulation in tensor memory
  int work, per_block;              // all boxes times their tasks' MMAs (x_planes == 1 counts), and a block's share
  int group_work;                   // work of one (group, o block, c block): boxes * pairs of all tap groups
  int task_taps;                    // taps per task at most: 4 or kWgradTaps
  int tg_tap[kWgradMaxTaps + 1];    // taps of tap group k: [tg_tap[k], tg_tap[k + 1]), at most six, by ascending shift
  int tg_pair[kWgradMaxTaps + 1];   // pairs of taps before tap group k
  int tg_ry[kWgradMaxTaps], tg_rx[kWgradMaxTaps]; // residues of a tap group's x rows and columns
  int tap_row[kWgradMaxTaps];       // shift of a tap, in rows of the box
  int tap_id[kWgradMaxTaps];        // its index in the filter
  float *slots;

  // one slot of partial sums: [tap][channel][map]
  __host__ __device__ __forceinline__ int slot_floats() const { return task_taps * 64 * 64; }
  __host__ __device__ __forceinline__ int tasks() const { return groups * o_blocks * c_blocks * tap_groups; }
  // first unit of work of a task, and its pairs
  __host__ __device__ __forceinline__ int task_begin(int task, int &pairs) const {
    const int big = task / tap_groups, tg = task - big * tap_groups;
    pairs = tg_pair[tg + 1] - tg_pair[tg];
    return big * group_work + boxes * tg_pair[tg];
  }
  // boxes [b0, b1) of a task that a block does
  __host__ __device__ __forceinline__ void share(int block, int begin, int pairs, int &b0, int &b1) const {
    const int lo = block * per_block - begin, hi = lo + per_block;
    b0 = lo <= 0 ? 0 : (lo + pairs - 1) / pairs;
    b1 = hi <= 0 ? 0 : (hi + pairs - 1) / pairs;
    b0 = b0 < boxes ? b0 : boxes;
    b1 = b1 < boxes ? b1 : boxes;
  }
};

constexpr int kWgradMaxStages = 4;

// kPx: planes of x.
template <int kPx>
__global__ void __launch_bounds__(kGemmThreads, 1)
    conv_wgrad_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_dy,
                              const __grid_constant__ ConvWgradProblem prob, int *status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full[kWgradMaxStages], empty[kWgradMaxStages], tmem_full, tmem_empty;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int *abort_flag = &abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t stage_bytes = 3u * prob.dy_bytes + (uint32_t)kPx * prob.x_bytes;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kWgradMaxStages; ++i) {
      ptx::mbar_init(full + i, 1);
      ptx::mbar_init(empty + i, 1);
    }
    ptx::mbar_init(&tmem_full, 1);
    ptx::mbar_init(&tmem_empty, kEpilogueWarps);
    abort_word = 0;
    ptx::mbar_fence_init();
    ptx::prefetch_tensormap(&map_x);
    ptx::prefetch_tensormap(&map_dy);
  }
  // rows behind the boxes are read (up to a multiple of 16 pixels, and by shifted taps) but never loaded: zero
  {
    const int dy_used = prob.h_box * prob.wp * kRowBytes, x_used = prob.hp * prob.wp * kRowBytes;
    for (int s = 0; s < prob.stages; ++s)
      for (int p = 0; p < 3 + kPx; ++p) {
        uint8_t *base = smem + s * stage_bytes + (p < 3 ? p * prob.dy_bytes : 3 * prob.dy_bytes + (p - 3) * prob.x_bytes);
        const int from = p < 3 ? dy_used : x_used, to = p < 3 ? prob.dy_bytes : prob.x_bytes;
        for (int i = from + 16 * (int)threadIdx.x; i < to; i += 16 * kGemmThreads)
          *reinterpret_cast<uint4 *>(base + i) = make_uint4(0, 0, 0, 0);
      }
    ptx::fence_async_shared();
  }
  if (warp == 1) {
    ptx::tmem_alloc(&tmem_slot, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  pdl_wait();
  if (prob.task_taps < kWgradTaps) // small problems (early_trigger's reason)
    pdl_trigger();
  auto gave_up = [&](int code) {
    if (*abort_flag == 0)
      atomicCAS(status, 0, code);
    *abort_flag = 1;
  };
  // every role walks the block's tasks in the same order
  const int tasks = prob.tasks();
  auto walk = [&](auto &&segment) {
    const int lo = (int)blockIdx.x * prob.per_block;
    int task = lo / prob.group_work;
    int tg = 0;
    while (tg + 1 < prob.tap_groups && task * prob.group_work + prob.boxes * prob.tg_pair[tg + 1] <= lo)
      ++tg;
    for (task = task * prob.tap_groups + tg; task < tasks; ++task) {
      int pairs, b0, b1;
      const int begin = prob.task_begin(task, pairs);
      if (begin >= lo + prob.per_block)
        return;
      prob.share((int)blockIdx.x, begin, pairs, b0, b1);
      if (b0 < b1 && !segment(task, pairs, b0, b1))
        return;
    }
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (ptx::elect_one()) {
      int st = 0;
      uint32_t phase = 0;
      const uint32_t tx = (uint32_t)(3 * prob.h_box + kPx * prob.hp) * prob.wp * kRowBytes;
      walk([&](int task, int, int b0, int b1) {
        const int tg = task % prob.tap_groups;
        int r = task / prob.tap_groups;
        const int cb = r % prob.c_blocks;
        r /= prob.c_blocks;
        const int ob = r % prob.o_blocks, g = r / prob.o_blocks;
        const int k_at = g * prob.k_stride + ob * 64, c_at = g * prob.c_stride + cb * 64;
        int img = b0 / prob.tiles_h, th = b0 - img * prob.tiles_h;
        for (int b = b0; b < b1; ++b) {
          if (!ptx::mbar_wait(empty + st, phase ^ 1u, abort_flag)) {
            gave_up(kStatusProducerTimeout);
            return false;
          }
          uint8_t *dst = smem + st * stage_bytes;
          ptx::mbar_expect_tx(full + st, tx);
          const int row0 = th * prob.h_box;
#pragma unroll
          for (int p = 0; p < 3; ++p)
            ptx::tma_load_5d(dst + p * prob.dy_bytes, &map_dy, full + st, k_at, 0, row0, img, p);
#pragma unroll
          for (int p = 0; p < kPx; ++p)
            ptx::tma_load_5d(dst + 3 * prob.dy_bytes + p * prob.x_bytes, &map_x, full + st, c_at,
                             prob.x0 * prob.sx + prob.tg_rx[tg], (row0 + prob.y0) * prob.sy + prob.tg_ry[tg], img, p);
          if (++st == prob.stages) {
            st = 0;
            phase ^= 1u;
          }
          if (++th == prob.tiles_h) {
            th = 0;
            ++img;
          }
        }
        return true;
      });
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    if (ptx::elect_one()) {
      int st = 0, chunk = 0;
      uint32_t phase = 0;
      // MN-major operands: bits 15 and 16
      const uint32_t idesc0 = ptx::make_idesc(1u, 1u, kTileM, 192) | (3u << 15);
      const uint32_t idesc1 = ptx::make_idesc(1u, 1u, kTileM, 128) | (3u << 15);
      const uint32_t idesc2 = ptx::make_idesc(1u, 1u, kTileM, 64) | (3u << 15);
      // start address in the low 14 bits, leading byte offset (between 64-element chunks) from bit 16 on; the high
      // word (stride between groups of eight pixels, version, swizzle) is that of smem_desc_k
      const uint32_t hi = (uint32_t)(ptx::smem_desc_k(0, kRowBytes) >> 32);
      const uint32_t smem16 = ptx::smem_u32(smem) >> 4;
      walk([&](int task, int pairs, int b0, int b1) {
        const int tg = task % prob.tap_groups, t0 = prob.tg_tap[tg], t1 = prob.tg_tap[tg + 1];
        uint32_t a_off[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int ta = t0 + 2 * q < t1 ? t0 + 2 * q : t0, tb = ta + 1 < t1 ? ta + 1 : ta;
          a_off[q] = (uint32_t)prob.tap_row[ta] * 8u + ((uint32_t)(prob.tap_row[tb] - prob.tap_row[ta]) * 8u << 16);
        }
        for (int c0 = b0; c0 < b1; c0 += prob.flush, ++chunk) {
          if (!ptx::mbar_wait(&tmem_empty, ((uint32_t)chunk & 1u) ^ 1u, abort_flag)) {
            gave_up(kStatusMmaTimeout);
            return false;
          }
          ptx::tc_fence_after_sync();
          uint32_t accumulate = 0;
          const int c1 = c0 + prob.flush < b1 ? c0 + prob.flush : b1;
          for (int b = c0; b < c1; ++b) {
            if (!ptx::mbar_wait(full + st, phase, abort_flag)) {
              gave_up(kStatusMmaTimeout);
              return false;
            }
            ptx::tc_fence_after_sync();
            const uint32_t b_lo = smem16 + ((uint32_t)st * stage_bytes >> 4);
            const uint32_t a_lo = b_lo + (3u * (uint32_t)prob.dy_bytes >> 4);
            const uint32_t b_lbo = ((uint32_t)prob.dy_bytes >> 4) << 16;
            auto step = [&](int k, int q) { // 16 pixels of one pair of taps
              const uint32_t d = tmem_base + (uint32_t)q * 192u;
              const uint64_t bd = ((uint64_t)hi << 32) | (b_lo + b_lbo + (uint32_t)k * 128u);
              if (q == 2) {
                // the third pair has 128 columns: the product of the first pieces, and all the others together
                const uint64_t plane = (uint32_t)prob.dy_bytes >> 4;
                auto ad = [&](int p) {
                  return ((uint64_t)hi << 32) | (a_lo + ((uint32_t)(p * prob.x_bytes) >> 4) + a_off[2] + (uint32_t)k * 128u);
                };
                ptx::mma_bf16(d, ad(0), bd, idesc1, accumulate);
                ptx::mma_bf16(d + 64u, ad(0), bd + 2 * plane, idesc2, 1u);
                if constexpr (kPx == 3) {
                  ptx::mma_bf16(d + 64u, ad(1), bd, idesc2, 1u);
                  ptx::mma_bf16(d + 64u, ad(1), bd + plane, idesc2, 1u);
                  ptx::mma_bf16(d + 64u, ad(2), bd, idesc2, 1u);
                }
                return;
              }
#pragma unroll
              for (int p = 0; p < kPx; ++p) {
                const uint64_t ad =
                    ((uint64_t)hi << 32) | (a_lo + ((uint32_t)(p * prob.x_bytes) >> 4) + a_off[q] + (uint32_t)k * 128u);
                // later pieces only ever add to columns that the first one has written in this step
                ptx::mma_bf16(d + 64u * p, ad, bd, p == 0 ? idesc0 : (p == 1 ? idesc1 : idesc2),
                              p == 0 ? accumulate : 1u);
              }
            };
            auto steps = [&](auto count) { // all pairs of the task, four steps of straight code at a time
              int k = 0;
              for (; k + 4 <= prob.k16; k += 4)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
#pragma unroll
                  for (int q = 0; q < decltype(count)::value; ++q)
                    step(k + u, q);
                  accumulate = 1;
                }
              for (; k < prob.k16; ++k) {
#pragma unroll
                for (int q = 0; q < decltype(count)::value; ++q)
                  step(k, q);
                accumulate = 1;
              }
            };
            if (pairs == 3)
              steps(std::integral_constant<int, 3>{});
            else if (pairs == 2)
              steps(std::integral_constant<int, 2>{});
            else
              steps(std::integral_constant<int, 1>{});
            ptx::mma_commit(empty + st);
            if (++st == prob.stages) {
              st = 0;
              phase ^= 1u;
            }
          }
          ptx::mma_commit(&tmem_full);
        }
        return true;
      });
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int quarter = warp & 3, set = (warp - 2) >> 2; // TMEM lanes; maps [32 * set, + 32)
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + 32u * set;
    int chunk = 0;
    walk([&](int task, int pairs, int b0, int b1) {
      float acc[3][32];
#pragma unroll
      for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int j = 0; j < 32; ++j)
          acc[q][j] = 0.0f;
      for (int c0 = b0; c0 < b1; c0 += prob.flush, ++chunk) {
        const bool got = ptx::mbar_wait(&tmem_full, (uint32_t)chunk & 1u, abort_flag);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0)
            gave_up(kStatusEpilogueTimeout);
          return false;
        }
        ptx::tc_fence_after_sync();
#pragma unroll
        for (int q = 0; q < 3; ++q)
          if (q < pairs) {
            uint32_t r0[32], r1[32];
            float low[32]; // the products of the smaller pieces
            ptx::tmem_ld_32x32(lane_base + 192u * q + 64u, r1);
            if (q < 2)
              ptx::tmem_ld_32x32(lane_base + 192u * q + 128u, r0);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j)
              low[j] = q < 2 ? __fadd_rn(__uint_as_float(r1[j]), __uint_as_float(r0[j])) : __uint_as_float(r1[j]);
            ptx::tmem_ld_32x32(lane_base + 192u * q, r0);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j)
              acc[q][j] = __fadd_rn(acc[q][j], __fadd_rn(__uint_as_float(r0[j]), low[j]));
          }
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0)
          ptx::mbar_arrive(&tmem_empty);
      }
      // slot of this (block, task): [tap][channel][map]
      float *slot = prob.slots + (int64_t)((int)blockIdx.x + task) * prob.slot_floats();
#pragma unroll
      for (int q = 0; q < 3; ++q)
        if (q < pairs) {
          float4 *dst = reinterpret_cast<float4 *>(slot + (2 * q * 64 + quarter * 32 + lane) * 64 + 32 * set);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            dst[j] = make_float4(acc[q][4 * j], acc[q][4 * j + 1], acc[q][4 * j + 2], acc[q][4 * j + 3]);
        }
      return true;
    });
  }

  // ------------------------------------------------------------------ teardown
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0) {
    const uint64_t t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 2000000ull)
      __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, 512);
  }
}

// What the sums were made of, as the caller holds it.
struct ConvWgradOperands {
  const float *x, *dy;
  int N, C, H, W, Ko, Ho, Wo, kw, sh, sw, ph, pw, dh, dw;
};

// One element of dW from the fp32 operands, by the lanes of a warp. Pixels outside the image count as zeros, like in the
// reference's unfolded patches.
__device__ __forceinline__ float conv_wgrad_element(const ConvWgradOperands &G, int o, int c, int tap) {
  const int ky = tap / G.kw, kx = tap - ky * G.kw, plane = G.Ho * G.Wo;
  float s = 0.0f;
  for (int64_t i = threadIdx.x & 31; i < (int64_t)G.N * plane; i += 32) {
    const int n = (int)(i / plane), p = (int)(i - (int64_t)n * plane), oy = p / G.Wo;
    const int iy = oy * G.sh - G.ph + ky * G.dh, ix = (p - oy * G.Wo) * G.sw - G.pw + kx * G.dw;
    const bool in = iy >= 0 && iy < G.H && ix >= 0 && ix < G.W;
    const float xv = in ? __ldg(G.x + (((int64_t)n * G.C + c) * G.H + iy) * G.W + ix) : 0.0f;
    s = __fmaf_rn(__ldg(G.dy + ((int64_t)n * G.Ko + o) * plane + p), xv, s);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1)
    s += __shfl_xor_sync(0xffffffffu, s, d);
  return s;
}

// dW[o][c][tap] (+)= the slots of a task in block order; one thread block per (task, channel), the maps of a slot are
// contiguous. Only the first and the last slot can be missing (per_block >= 2 pairs).
//
// Sums that are not finite are made again from the operands: the padded columns pair zeros of dy with pixels of x that the
// tap does not reach there, and a NaN or an infinity of x would spread to taps that have no output pixel with it (and an
// infinity of either operand to a NaN, through its pieces).
__global__ void __launch_bounds__(64 * kWgradTaps, 5)
    conv_wgrad_finish_kernel(const __grid_constant__ ConvWgradProblem prob, const __grid_constant__ ConvWgradOperands G,
                             int Kog, int Cg, int taps, float *__restrict__ dw, int accumulate) {
  pdl_wait();
  pdl_trigger();
  const int task = blockIdx.x;
  const int tg = task % prob.tap_groups;
  int r = task / prob.tap_groups;
  const int cb = r % prob.c_blocks;
  r /= prob.c_blocks;
  const int ob = r % prob.o_blocks, g = r / prob.o_blocks;
  const int t0 = prob.tg_tap[tg], n_taps = prob.tg_tap[tg + 1] - t0;
  const int o = ob * 64 + (threadIdx.x & 63), c = cb * 64 + blockIdx.y, t = threadIdx.x >> 6;
  if (t >= n_taps || c >= Cg) // (whole warps: a warp's threads have one tap, and maps in a row)
    return;
  const bool live = o < Kog;
  float s = 0.0f;
  if (live) {
    int pairs, b0, b1;
    const int begin = prob.task_begin(task, pairs);
    int first = begin / prob.per_block, last = (begin + prob.boxes * pairs - 1) / prob.per_block;
    prob.share(first, begin, pairs, b0, b1);
    first += b0 < b1 ? 0 : 1;
    prob.share(last, begin, pairs, b0, b1);
    last -= b0 < b1 ? 0 : 1;
    const float *src =
        prob.slots + (int64_t)(first + task) * prob.slot_floats() + (t * 64 + blockIdx.y) * 64 + (threadIdx.x & 63);
    int b = first;
    for (; b + 8 <= last + 1; b += 8, src += (int64_t)8 * prob.slot_floats()) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        v[u] = __ldcs(src + (int64_t)u * prob.slot_floats());
#pragma unroll
      for (int u = 0; u < 8; ++u)
        s = __fadd_rn(s, v[u]);
    }
    for (; b <= last; ++b, src += prob.slot_floats())
      s = __fadd_rn(s, __ldcs(src));
  }
  const int tap = prob.tap_id[t0 + t], lane = threadIdx.x & 31;
  for (uint32_t again = __ballot_sync(0xffffffffu, !(fabsf(s) < __int_as_float(0x7f800000))); again; again &= again - 1) {
    const int l = __ffs(again) - 1;
    const float v = conv_wgrad_element(G, g * Kog + o - lane + l, g * Cg + c, tap);
    s = lane == l ? v : s;
  }
  if (live) {
    float *dst = dw + ((int64_t)(g * Kog + o) * Cg + c) * taps + tap;
    *dst = accumulate ? __fadd_rn(*dst, s) : s;
  }
}

} // namespace nb200
