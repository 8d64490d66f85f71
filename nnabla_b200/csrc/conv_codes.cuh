// Implicit-GEMM convolution of int8 channel-last activation codes with +-1
// (int8) weights on tcgen05, with the layer's whole inference tail in the
// epilogue:
//
//   u      = fma(acc, scale[o] * f, bias[o] * f)    (BN folded into scale / bias; f = 2 / delta, exact)
//   u      = fma(residual, step * f, u)             (codes with their step, or fp32; optional)
//   code   = min((floor(max(u, 0)) + 1) >> 1, kmax) -> int8, channel-last
//
// i.e. code * delta = FixedPointQuantize(ReLU(acc * scale + bias + residual)) with one rounding per
// fused multiply-add (the quantizer rounds |x| / delta + 0.5 down, which is (floor(2x / delta) + 1) >> 1).
//
// The PIXELS of a tile are the rows of the MMA (TMEM lanes), the output maps
// its columns: thread t of an epilogue warp owns one pixel and reads 32
// consecutive maps of it from TMEM, which are 32 consecutive bytes of the
// channel-last result, so the tile leaves as 128-bit stores of finished codes,
// one byte per value, with no transpose through shared memory.
//
//   A (M = 128 rows)  activation box: n_box images x h_box output rows x Wo
//                     pixels, one K block = one filter tap x E channel slots,
//                     fetched by a 5-D TMA box shifted by the tap (stride via
//                     element strides, padding = zero fill)
//   B (N columns)     weights [Ko][taps * c_slots], K-major, as
//                     nb200_binary_weights_prepare_i8 lays them out
//   D (TMEM)          int32, 128 lanes x N columns, double buffered
//
// Warp roles as in the plain contraction kernel: warp 0 TMA producer, warp 1
// MMA issuer and TMEM owner, eight epilogue warps (two per lane quarter,
// alternating 32-column chunks). Every wait is bounded (ptx::mbar_wait); a wait
// that gives up records a status code and all roles fall through to the
// teardown, which always frees TMEM.
#pragma once
#include "gemm.cuh"

namespace nb200 {

struct ConvCodesProblem {
  int Nimg, Ko, Ho, Wo;
  int h_box, n_box, tiles_h, tiles_n, n_tiles; // pixel boxes and column tiles
  int bn;                                      // UMMA N: columns per tile (multiple of 16)
  int kw, taps, cblocks;
  int sh, sw, ph, pw, dh, dw;
  int pixels;    // n_box * h_box * Wo (<= 128)
  int slots_out; // bytes per pixel of the code result / floats per pixel of the fp32 result
  // halo form (stride 1): one box of hp x wp input pixels per tile and channel block
  int wp, hp;          // wp = Wo + (kw - 1) * dw, hp = h_box + (kh - 1) * dh
  int h_half;          // output rows of one MMA row block (h_box, or half of it with two row blocks per tile)
  int a_tile_bytes;    // bytes of one channel block's pixel tile in shared memory (readable rows included)
  int a_bufs;          // pixel-tile buffers: 2 to kTileBufs, or 1 where every block has one tile
  __device__ __forceinline__ int num_tiles() const { return n_tiles * tiles_h * tiles_n; }
  __device__ __forceinline__ int k_blocks() const { return taps * cblocks; }
};

struct ConvCodesEpilogue {
  const float *scale, *bias;   // per output map
  const int8_t *res_codes;     // residual as codes in the result's own layout (or NULL)
  const float *res_f32;        // residual as fp32, channel-last [pixels][slots_out] (or NULL)
  float res_scale;             // factor of the residual: (its step, or 1 for fp32) * out_scale
  int8_t *y_codes;             // result as codes (or NULL)
  float *y_f32;                // result as fp32 channel-last, before ReLU / quantizer (or NULL)
  float *y_nchw;               // result as fp32 [batch][maps][pixels]: acc * scale (+ bias), each operation rounded
                               // on its own like the reference's product followed by its bias addition (or NULL)
  int has_bias;
  int relu;
  float out_scale;             // factor of scale: 2 / delta when codes are written (delta: the quantizer's step, a
                               // power of two), the activations' step for the plain fp32 result, else 1
  float bias_scale;            // factor of bias: 2 / delta when codes are written, else 1
  int kmax, kmin;              // code range
  int saturate;                // codes with ReLU and kmax = 127: out_scale, bias_scale and res_scale hold
                               // 1 / (128 * delta) instead of 2 / delta
  int small_acc;               // every accumulator is below 2^22 in magnitude (see int_to_float)
#ifdef NB200_CC_TRACE
  long long *trace; // timing experiments: block 0 writes %globaltimer at its phase boundaries
#endif
};

#ifdef NB200_CC_TRACE
#define NB_CC_STAMP(slot, tile_local)                                                                                 \
  do {                                                                                                                 \
    if (ep.trace && blockIdx.x == 0 && (tile_local) < 64)                                                              \
      ep.trace[(tile_local) * 16 + (slot)] = (long long)ptx::globaltimer_ns();                                         \
  } while (0)
#define NB_CC_WAITED(slot, tile_local, expr)                                                                          \
  do {                                                                                                                 \
    const long long w0_ = (long long)ptx::globaltimer_ns();                                                            \
    expr;                                                                                                              \
    if (ep.trace && blockIdx.x == 0 && (tile_local) < 64)                                                              \
      ep.trace[(tile_local) * 16 + (slot)] += (long long)ptx::globaltimer_ns() - w0_;                                  \
  } while (0)
#else
#define NB_CC_WAITED(slot, tile_local, expr) expr
#define NB_CC_STAMP(slot, tile_local)                                                                                 \
  do {                                                                                                                 \
  } while (0)
#endif

// Exact for |a| < 2^22 (the accumulators of this kernel stay below 2^21 in magnitude for K <= 16384).
__device__ __forceinline__ float int_to_float(int a) {
  return __fsub_rn(__int_as_float(a + 0x4B400000), 12582912.0f);
}

// Four int32 codes -> four int8 lanes of one word (a in the lowest byte), each saturated to [-128, 127].
__device__ __forceinline__ uint32_t pack_s8x4(int a, int b, int c, int d) {
  uint32_t hi, out;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(d), "r"(c), "r"(0));
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(out) : "r"(b), "r"(a), "r"(hi));
  return out;
}

constexpr int kCodesMaxMaps = 512;
// a * b + c with one rounding, clamped to [0, 1] (NaN: 0).
__device__ __forceinline__ float fma_sat(float a, float b, float c) {
  float d;
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

constexpr int kTileBufs = 4;       // barriers of the halo form's pixel tiles
constexpr int kWeightParts = 4;    // barriers of the resident weights
constexpr int kCodesKTable = 64; // K blocks whose coordinates are tabulated once per block

// kResidentB: all tiles use the same weights (one column tile) and all their K blocks fit in
// shared memory beside the ring: the weights are loaded once per CTA and only the activation
// boxes stream. The copy engine spends about four cycles on every box row whatever its width,
// so a stage's weight rows (as many as its pixel rows, or more) are the larger part of its cost.
//
// kHalo (stride 1, with kResidentB): the filter taps of a stride-1 convolution read the SAME input
// pixels shifted by whole pixels, so a tile fetches its input once, as one box of hp x wp pixels
// per channel block (rows = pixels in raster order of the padded width wp), instead of once per
// tap. Output pixel (y, x) of the tile is MMA row y * wp + x (rows with x >= Wo are not stored),
// and tap (ky, kx) reads the same tile through a descriptor whose start is moved by
// (ky * dh * wp + kx * dw) rows. That works because the swizzle is a function of the shared-memory
// ADDRESS bits, for the copy engine's writes and the tensor core's reads alike: a start address
// that is a whole number of rows further on reads exactly the rows further on (no base-offset
// field is needed; setting one breaks it). This cuts the copy engine's rows per tile by the number
// of taps.
//
// Several column tiles (more maps than BN) in the halo form: every block then has one tile, with the weights of its own
// columns (launch_conv_codes checks it). For the few pixels of late stages and small batches this takes an image's pixels
// once instead of once per tap, and narrow tiles spread the weights, which one SM's port brings in at 64 bytes a cycle:
// 512 -> 512 maps of 7 x 7 pixels, one image, 10.4 us with a box per tap and 64 columns, now 8.4 (launch and wait included).
//
// kHalves = 2 (halo form, at most 64 maps): a tile is two MMA row blocks, rows [0, 128) and the 128 rows from
// h_half * wp on, of ONE input box of 2 * h_half output rows; their accumulators lie side by side in tensor memory.
// With one block of 18 small MMAs per tile the hand-over between the roles (four barriers, the commits, the
// descriptors' way into uniform registers) took as long as the MMAs themselves.
template <int BN, int STAGES, int RB, bool kResidentB = false, bool kHalo = false, int kHalves = 1>
__global__ void __launch_bounds__(kGemmThreads, 1)
    conv_codes_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                              const ConvCodesProblem prob, const ConvCodesEpilogue ep, int *status) {
  static_assert(RB == 128 || RB == 64, "operand rows are one 128-byte or 64-byte swizzle span");
  static_assert(BN % 16 == 0 && BN >= 16 && BN <= 256, "UMMA N for M = 128");
  static_assert(!kHalo || kResidentB, "the halo form streams pixel tiles only");
  static_assert(kHalves == 1 || (kHalo && kHalves == 2 && BN == 64), "two row blocks only with 64 maps");
  constexpr int kSets = kEpilogueWarps / 4; // sets of four epilogue warps, one per TMEM lane quarter
  constexpr int kCols = kHalves * BN;       // accumulator columns of a tile
  // The halo forms keep the maps' scale and bias in tensor memory, the same in every lane, and read them like the
  // accumulators. MMAs of 64 and 128 columns take 94 % of the shared-memory bandwidth (6 of 6.4 KB, 8 of 8.6 KB a
  // call), and sixteen 128-bit broadcast reads per chunk took the rest and more: the MMAs and the epilogue of a tile
  // ran one after the other.
  constexpr int kScaleCol = 2 * kCols; // scale at [kScaleCol, + BN), bias behind it
  constexpr int kElems = RB;              // int8: K elements per operand row of one K block
  constexpr int kMmasPerBlock = RB / 32;  // 32 bytes of K per MMA
  constexpr uint32_t kABytes = kTileM * RB;
  constexpr uint32_t kBBytes = BN * RB;
  constexpr uint32_t kStageBytes = kABytes + (kResidentB ? 0u : kBBytes);
  constexpr int kUsedCols = 2 * kCols + (kHalo ? 2 * BN : 0);
  constexpr uint32_t kTmemCols = (kUsedCols <= 64) ? 64 : (kUsedCols <= 128) ? 128 : (kUsedCols <= 256) ? 256 : 512;

  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // resident weights (kResidentB): [k block][BN rows] behind the ring
  const uint32_t resident_bytes = kResidentB ? (uint32_t)(prob.taps * prob.cblocks) * kBBytes : 0u;
  // halo form: the ring's place is taken by prob.a_bufs buffers (1, or 2 to kTileBufs) of cblocks pixel tiles each
  const uint32_t ring_bytes =
      kHalo ? (uint32_t)(prob.a_bufs * prob.cblocks * prob.a_tile_bytes) : (uint32_t)STAGES * kStageBytes;
  uint8_t *b_resident = smem + ring_bytes;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + ring_bytes + resident_bytes);
  uint64_t *full_bar = bars;
  uint64_t *empty_bar = bars + STAGES;
  uint64_t *tmem_full = bars + 2 * STAGES;
  uint64_t *tmem_empty = bars + 2 * STAGES + 2;
  uint64_t *b_full = bars + 2 * STAGES + 4; // resident weights, kWeightParts runs of K blocks
  uint64_t *a_full = b_full + kWeightParts; // halo form: pixel-tile buffers
  uint64_t *a_empty = a_full + kTileBufs;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(a_empty + kTileBufs);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  // (scale, bias) of every output map, times out_scale; read as float4 pairs, so 16-byte aligned
  float2 *sb = reinterpret_cast<float2 *>((reinterpret_cast<uintptr_t>(tmem_slot + 4) + 15) & ~uintptr_t(15));
  const float4 *sb2 = reinterpret_cast<const float4 *>(sb);
  // per K block (filter tap x channel block): x = halo form's operand offset in 16-byte units, y = channel
  // coordinate, z / w = the tap's column / row shift. One thread issues all copies and all MMAs of a tile;
  // the two integer divisions per K block that these take cost it more than the instruction they feed.
  int4 *kb_table = reinterpret_cast<int4 *>(sb + kCodesMaxMaps);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_tiles = prob.num_tiles();
  const int k_blocks = prob.k_blocks();

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(full_bar + s, 1);
      ptx::mbar_init(empty_bar + s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(tmem_full + b, 1);
      ptx::mbar_init(tmem_empty + b, 4 * kSets);
    }
    for (int q = 0; q < kWeightParts; ++q)
      ptx::mbar_init(b_full + q, 1);
    for (int b = 0; b < kTileBufs; ++b) {
      ptx::mbar_init(a_full + b, 1);
      ptx::mbar_init(a_empty + b, 1);
    }
    *abort_flag = 0;
    ptx::mbar_fence_init();
    ptx::prefetch_tensormap(&map_x);
    ptx::prefetch_tensormap(&map_w);
  }
  auto kb_entry = [&](int kb) {
    const int tap = kb / prob.cblocks, cb = kb - tap * prob.cblocks;
    const int ky = tap / prob.kw, kx = tap - ky * prob.kw;
    return make_int4((cb * prob.a_tile_bytes + (ky * prob.dh * prob.wp + kx * prob.dw) * RB) >> 4, cb * kElems,
                     kx * prob.dw, ky * prob.dh);
  };
  const bool tabulated = k_blocks <= kCodesKTable;
  for (int kb = threadIdx.x; kb < k_blocks && kb < kCodesKTable; kb += kGemmThreads)
    kb_table[kb] = kb_entry(kb);
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads(); // the block has its tensor memory before it lets the successor in
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  // (codes and channel-last results are read by convolutions)
  if (!ep.y_nchw || early_trigger((int64_t)prob.Nimg * prob.Ko * prob.Ho * prob.Wo))
    pdl_trigger();
  // K blocks of one part of the resident weights
  const int part_blocks = (k_blocks + kWeightParts - 1) / kWeightParts;

  // tile -> (column tile, pixel box); the column tiles of one box are neighbours in time (the box stays in L2)
  auto decode = [&](int tile, int &n0, int &img0, int &oy0) {
    const int nt = tile % prob.n_tiles;
    const int r = tile / prob.n_tiles;
    n0 = nt * BN;
    oy0 = (r % prob.tiles_h) * prob.h_box;
    img0 = (r / prob.tiles_h) * prob.n_box;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      const uint32_t tx_bytes = (uint32_t)(prob.pixels * RB) + (kResidentB ? 0u : kBBytes);
      // the weights behind the first pixels: the first MMAs need both, the others the rest of the weights
      auto load_weights = [&](int n0) {
        for (int q = 0; q < kWeightParts; ++q) {
          const int kb0 = q * part_blocks, kb1 = min(kb0 + part_blocks, k_blocks);
          if (kb0 < kb1)
            ptx::mbar_expect_tx(b_full + q, (uint32_t)(kb1 - kb0) * kBBytes);
          for (int kb = kb0; kb < kb1; ++kb)
            ptx::tma_load_3d(b_resident + (size_t)kb * kBBytes, &map_w, b_full + q, kb * kElems, n0, 0);
        }
      };
      if (kResidentB && !kHalo && (int)blockIdx.x < num_tiles)
        load_weights(0);
      int alocal = 0, ab = 0;
      uint32_t ab_phase = 0;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++alocal) {
        int n0, img0, oy0;
        decode(tile, n0, img0, oy0);
        NB_CC_STAMP(0, (tile - (int)blockIdx.x) / (int)gridDim.x);
        if constexpr (kHalo) {
          if (!ptx::mbar_wait(a_empty + ab, ab_phase ^ 1u, abort_flag)) {
            if (*abort_flag == 0)
              atomicCAS(status, 0, kStatusProducerTimeout);
            *abort_flag = 1;
            break;
          }
          ptx::mbar_expect_tx(a_full + ab, (uint32_t)(prob.cblocks * prob.hp * prob.wp * RB));
          for (int cb = 0; cb < prob.cblocks; ++cb)
            ptx::tma_load_5d(smem + (size_t)(ab * prob.cblocks + cb) * prob.a_tile_bytes, &map_x, a_full + ab,
                             cb * kElems, -prob.pw, oy0 - prob.ph, img0, 0);
          if (alocal == 0)
            load_weights(n0);
          if (++ab == prob.a_bufs) {
            ab = 0;
            ab_phase ^= 1u;
          }
        } else {
        for (int kb = 0; kb < k_blocks; ++kb) {
          bool got_slot;
          NB_CC_WAITED(9, (tile - (int)blockIdx.x) / (int)gridDim.x,
                       got_slot = ptx::mbar_wait(empty_bar + stage, phase ^ 1u, abort_flag));
          if (!got_slot) {
            if (*abort_flag == 0)
              atomicCAS(status, 0, kStatusProducerTimeout);
            *abort_flag = 1;
            ok = false;
            break;
          }
          uint8_t *st = smem + stage * kStageBytes;
          ptx::mbar_expect_tx(full_bar + stage, tx_bytes);
          const int4 e = tabulated ? kb_table[kb] : kb_entry(kb);
          ptx::tma_load_5d(st, &map_x, full_bar + stage, e.y, e.z - prob.pw, oy0 * prob.sh - prob.ph + e.w, img0, 0);
          if (!kResidentB)
            ptx::tma_load_3d(st + kABytes, &map_w, full_bar + stage, kb * kElems, n0, 0);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        }
        NB_CC_STAMP(1, (tile - (int)blockIdx.x) / (int)gridDim.x);
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    if (ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      int local = 0, ab = 0;
      uint32_t ab_phase = 0;
      bool ok = true;
      const uint32_t idesc = ptx::make_idesc(2u, 1u, kTileM, BN); // s32 accumulator, s8 operands
      // resident weights: waited for part by part, as the first tile's MMAs come to them (a block with one tile spent
      // as long on the wait for all of them as on its MMAs)
      int weights_here = kResidentB ? 0 : 0x3fffffff; // K blocks
      auto weights = [&](int kb_end) {
        while (weights_here < kb_end) {
          if (!ptx::mbar_wait(b_full + weights_here / part_blocks, 0u, abort_flag)) {
            if (*abort_flag == 0)
              atomicCAS(status, 0, kStatusMmaTimeout);
            *abort_flag = 1;
            ok = false;
            return false;
          }
          ptx::tc_fence_after_sync();
          weights_here += part_blocks;
        }
        return true;
      };
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++local) {
        const int buf = local & 1;
        const uint32_t buf_phase = (uint32_t)(local >> 1) & 1u;
        NB_CC_STAMP(2, local);
        if (!ptx::mbar_wait(tmem_empty + buf, buf_phase ^ 1u, abort_flag)) {
          if (*abort_flag == 0)
            atomicCAS(status, 0, kStatusMmaTimeout);
          *abort_flag = 1;
          break;
        }
        ptx::tc_fence_after_sync();
        NB_CC_STAMP(3, local);
        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * kCols);
        uint32_t accumulate = 0;
        if constexpr (kHalo) {
          if (!ptx::mbar_wait(a_full + ab, ab_phase, abort_flag)) {
            if (*abort_flag == 0)
              atomicCAS(status, 0, kStatusMmaTimeout);
            *abort_flag = 1;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t a_base = ptx::smem_u32(smem) + (uint32_t)(ab * prob.cblocks * prob.a_tile_bytes);
          // (start addresses are 16-byte units in the low 14 bits of a descriptor; shared memory ends below 2^18)
          const uint64_t adesc0 = ptx::smem_desc_k(a_base, RB), bdesc0 = ptx::smem_desc_k(ptx::smem_u32(b_resident), RB);
          const uint32_t hi = (uint32_t)(adesc0 >> 32), alo = (uint32_t)adesc0, blo = (uint32_t)bdesc0;
          const uint32_t half_step = (uint32_t)(prob.h_half * prob.wp * RB) >> 4;
          auto issue = [&](uint32_t a_off, int kb) {
#pragma unroll
            for (int h = 0; h < kHalves; ++h)
#pragma unroll
              for (int k = 0; k < kMmasPerBlock; ++k)
                ptx::mma_i8(d_tmem + h * BN, ((uint64_t)hi << 32) | (alo + a_off + h * half_step + 2 * k),
                            ((uint64_t)hi << 32) | (blo + (uint32_t)kb * (kBBytes >> 4) + 2 * k), idesc,
                            k == 0 ? accumulate : 1u);
            accumulate = 1;
          };
          // Offsets of kBatch K blocks first, then their MMAs back to back: descriptors reach the tensor core
          // through uniform registers, and a loop that makes one K block's at a time spent 45 cycles an iteration
          // on that (an MMA of 64 columns takes 51).
          constexpr int kBatch = 4;
          int kb = 0;
          if (tabulated)
            for (; kb + kBatch <= k_blocks && weights(kb + kBatch); kb += kBatch) {
              uint32_t off[kBatch];
#pragma unroll
              for (int u = 0; u < kBatch; ++u)
                off[u] = (uint32_t)kb_table[kb + u].x;
#pragma unroll
              for (int u = 0; u < kBatch; ++u)
                issue(off[u], kb + u);
            }
          for (; kb < k_blocks && weights(kb + 1); ++kb)
            issue((uint32_t)(tabulated ? kb_table[kb].x : kb_entry(kb).x), kb);
          if (!ok)
            break;
          ptx::mma_commit(a_empty + ab); // the pixel tile is free once these MMAs have read it
          if (++ab == prob.a_bufs) {
            ab = 0;
            ab_phase ^= 1u;
          }
          ptx::mma_commit(tmem_full + buf);
        } else {
        for (int kb = 0; kb < k_blocks; ++kb) {
          bool got_data;
          NB_CC_WAITED(10, local, got_data = ptx::mbar_wait(full_bar + stage, phase, abort_flag));
          if (!got_data) {
            if (*abort_flag == 0)
              atomicCAS(status, 0, kStatusMmaTimeout);
            *abort_flag = 1;
            ok = false;
            break;
          }
          if (!weights(kb + 1))
            break;
          ptx::tc_fence_after_sync();
          const uint32_t st = ptx::smem_u32(smem + stage * kStageBytes);
          const uint64_t adesc = ptx::smem_desc_k(st, RB);
          const uint64_t bdesc = kResidentB ? ptx::smem_desc_k(ptx::smem_u32(b_resident) + (uint32_t)kb * kBBytes, RB)
                                            : ptx::smem_desc_k(st + kABytes, RB);
#pragma unroll
          for (int k = 0; k < kMmasPerBlock; ++k) {
            ptx::mma_i8(d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc, accumulate);
            accumulate = 1;
          }
          ptx::mma_commit(empty_bar + stage);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok)
          ptx::mma_commit(tmem_full + buf);
        }
        NB_CC_STAMP(4, local);
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int quarter = warp & 3;      // TMEM lanes [32 * quarter, +32) are visible to this warp
    const int first_col = 32 * ((warp - 2) >> 2); // this warp's first 32-column chunk of a tile's accumulators
    const float cap = (float)(2 * ep.kmax) + 0.5f;
    // scale and bias are the epilogue's alone: the copies and MMAs do not wait for their loads (0.7 us of a launch that
    // has one tile per block)
    for (int c = threadIdx.x - 64; c < prob.n_tiles * BN; c += 32 * kEpilogueWarps)
      sb[c] = c < prob.Ko ? make_float2(ep.scale ? __fmul_rn(ep.scale[c], ep.out_scale) : ep.out_scale,
                                        ep.bias ? __fmul_rn(ep.bias[c], ep.bias_scale) : 0.0f)
                          : make_float2(0.0f, 0.0f);
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpilogueWarps) : "memory");
    // this thread's pixel of every tile: image of the box, row and column (the divisions stay out of the loop)
    const int row = quarter * 32 + lane;
    const int per_img = prob.h_box * prob.Wo, pitch = kHalo ? prob.wp : prob.Wo;
    const int box_img = kHalo ? 0 : row / per_img, in_img = row - box_img * per_img;
    const int box_y = in_img / pitch, box_x = in_img - box_y * pitch;
    const bool box_ok = box_img < prob.n_box && box_x < prob.Wo && box_y < prob.h_half;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
    if constexpr (kHalo) {
      // one column tile, or one tile for this block: this warp's maps are the same for every tile
      const int own = (int)(blockIdx.x % (unsigned)prob.n_tiles) * BN;
      for (int c = first_col; c < BN; c += 32 * kSets) {
        uint32_t t[32];
#pragma unroll
        for (int j = 0; j < 32; ++j)
          t[j] = __float_as_uint(sb[own + c + j].x);
        ptx::tmem_st_32x32(lane_base + kScaleCol + c, t);
#pragma unroll
        for (int j = 0; j < 32; ++j)
          t[j] = __float_as_uint(sb[own + c + j].y);
        ptx::tmem_st_32x32(lane_base + kScaleCol + BN + c, t);
      }
      ptx::tmem_st_wait();
    }
    int local = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++local) {
      int n0, img0, oy0;
      decode(tile, n0, img0, oy0);
      const int buf = local & 1;
      const uint32_t buf_phase = (uint32_t)(local >> 1) & 1u;
      const int img = img0 + box_img;
      // the residual of this warp's first chunk, and of its second where it has two, is requested before the accumulator is
      // waited for: the second's load inside its chunk was a latency per tile. [256, 64, 56, 56] 68.3 us, now 58.5, [256,
      // 128, 28, 28] 34.5 and 33.1; batch 64 17.1 and 16.5, 13.3 and 12.5. (Requested a tile ahead: 53.5 and 30.6, but
      // batch 64 17.9 and 13.0, since a launch of few tiles waits for its instructions.)
      constexpr bool kTwo = kCols == 64 * kSets;
      uint4 ra = make_uint4(0, 0, 0, 0), rb = ra, ra2 = ra, rb2 = ra;
      auto load_residual = [&](int64_t off, bool upper, uint4 &a, uint4 &b) {
        a = __ldg(reinterpret_cast<const uint4 *>(ep.res_codes + off));
        b = upper ? __ldg(reinterpret_cast<const uint4 *>(ep.res_codes + off) + 1) : make_uint4(0, 0, 0, 0);
      };
      auto pixel_ok = [&](int half) {
        const int y = box_y + half * prob.h_half;
        return box_ok && img < prob.Nimg && y < prob.h_box && oy0 + y < prob.Ho;
      };
      auto in_plane_of = [&](int half) { return (oy0 + box_y + half * prob.h_half) * prob.Wo + box_x; };
      const int64_t plane0 = (int64_t)img * prob.Ho * prob.Wo; // pixels before this image
      if (ep.res_codes && pixel_ok(0) && n0 + first_col < prob.slots_out)
        load_residual((plane0 + in_plane_of(0)) * prob.slots_out + n0 + first_col, n0 + first_col + 16 < prob.slots_out, ra, rb);
      if (kTwo && ep.res_codes) {
        constexpr int kNext = 32 * kSets;
        const int half = kNext / BN, col = n0 + first_col + kNext % BN;
        if (pixel_ok(half) && col < prob.slots_out)
          load_residual((plane0 + in_plane_of(half)) * prob.slots_out + col, col + 16 < prob.slots_out, ra2, rb2);
      }
      if (threadIdx.x == 64)
        NB_CC_STAMP(5, local);
      const bool got = ptx::mbar_wait(tmem_full + buf, buf_phase, abort_flag);
      if (!__all_sync(0xffffffffu, got)) {
        if (lane == 0) {
          if (*abort_flag == 0)
            atomicCAS(status, 0, kStatusEpilogueTimeout);
          *abort_flag = 1;
        }
        break;
      }
      ptx::tc_fence_after_sync();
      if (threadIdx.x == 64)
        NB_CC_STAMP(6, local);
#pragma unroll 1
      for (int c0 = first_col; c0 < kCols; c0 += 32 * kSets) {
        const int col = n0 + c0 % BN; // first output map of the chunk
        const int half = c0 / BN; // row block
        const bool live = pixel_ok(half) && col < (ep.y_nchw ? prob.Ko : prob.slots_out);
        const int in_plane = in_plane_of(half); // inside the image's plane
        const int64_t off = (plane0 + in_plane) * prob.slots_out + col;
        const bool upper = col + 16 < prob.slots_out; // the pixel's row ends in the middle of this chunk otherwise
        if (kTwo && c0 != first_col)
          ra = ra2, rb = rb2;
        else if (!kTwo && c0 != first_col && ep.res_codes && live) // later chunks: fetched here
          load_residual(off, upper, ra, rb);
        uint32_t r[32];
        ptx::tmem_ld_32x32(lane_base + (uint32_t)(buf * kCols + c0), r);
        float scale[32], bias[32]; // (maps past Ko have scale = bias = 0)
        if constexpr (kHalo) {
          uint32_t (&us)[32] = reinterpret_cast<uint32_t (&)[32]>(scale), (&ub)[32] = reinterpret_cast<uint32_t (&)[32]>(bias);
          ptx::tmem_ld_32x32(lane_base + kScaleCol + (uint32_t)(c0 % BN), us);
          ptx::tmem_ld_32x32(lane_base + kScaleCol + BN + (uint32_t)(c0 % BN), ub);
          ptx::tmem_ld_wait();
        } else {
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j2 = 0; j2 < 16; ++j2) {
            const float4 k = sb2[(col >> 1) + j2]; // (scale, bias) of two neighbouring maps
            scale[2 * j2] = k.x;
            bias[2 * j2] = k.y;
            scale[2 * j2 + 1] = k.z;
            bias[2 * j2 + 1] = k.w;
          }
        }
        if (threadIdx.x == 64)
          NB_CC_STAMP(7, local);
        if (!live)
          continue;
        if (ep.y_nchw) {
          // fp32 [batch][maps][pixels]: the 32 lanes of a store are 32 neighbouring pixels of one map
          const int64_t plane = (int64_t)prob.Ho * prob.Wo;
          float *yp = ep.y_nchw + ((int64_t)img * prob.Ko + col) * plane + in_plane;
          // all 32 values first, without branches (maps past Ko have scale = bias = 0), then the stores:
          // with a test per map in between, the maps went through the pipes one after the other
          float val[32];
          if (ep.small_acc) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              val[j] = int_to_float((int)r[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              val[j] = (float)(int)r[j];
          }
#pragma unroll
          for (int j = 0; j < 32; ++j)
            val[j] = __fmul_rn(val[j], scale[j]);
          if (ep.has_bias) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              val[j] = __fadd_rn(val[j], bias[j]);
          }
          if (col + 32 <= prob.Ko) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              yp[(int64_t)j * plane] = val[j];
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (col + j < prob.Ko)
                yp[(int64_t)j * plane] = val[j];
          }
          continue;
        }
        // Integers become floats on the add / multiply pipes instead of the (much narrower) conversion
        // pipe: for |a| < 2^22, the bit pattern of 1.5 * 2^23 plus a IS the float 1.5 * 2^23 + a.
        // code + 128 of a residual (one XOR per word) lands in the low mantissa byte of 1.5 * 2^23
        const uint32_t rw[8] = {ra.x ^ 0x80808080u, ra.y ^ 0x80808080u, ra.z ^ 0x80808080u, ra.w ^ 0x80808080u,
                                rb.x ^ 0x80808080u, rb.y ^ 0x80808080u, rb.z ^ 0x80808080u, rb.w ^ 0x80808080u};
        auto residual = [&](int j) {
          return __fsub_rn(__uint_as_float(__byte_perm(rw[j >> 2], 0x4B400000u, 0x7650 + (j & 3))), 12582912.0f + 128.0f);
        };
        uint32_t w[8];
        if (ep.saturate) {
          // ReLU and a quantizer with codes up to 127: scale, bias and residual carry 1 / (128 * delta), so that the
          // last fused multiply-add saturated to [0, 1] is the ReLU, the upper limit and a NaN's 0 at once. Adding
          // 256.00390625 = 2^8 + 2^-8 rounded DOWN leaves floor(128 v + 0.5), 0 to 128, in mantissa bits 8 to 15,
          // and of four codes in a word a 128 becomes 127 by subtracting its top bit: 8.5 instructions a value with a
          // residual, where limits, conversion and packing one by one took 14.
          // (one test of the residual's kind per chunk: a test per value keeps the values from overlapping)
          float v[32];
          if (ep.res_codes) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              v[j] = fma_sat(residual(j), ep.res_scale, __fmaf_rn(int_to_float((int)r[j]), scale[j], bias[j]));
          } else if (ep.res_f32) {
            const float4 *rp = reinterpret_cast<const float4 *>(ep.res_f32 + off);
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {
              const float4 t = (j4 < 4 || upper) ? __ldg(rp + j4) : make_float4(0.f, 0.f, 0.f, 0.f);
              const float f[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int j = 4 * j4 + i;
                v[j] = fma_sat(f[i], ep.res_scale, __fmaf_rn(int_to_float((int)r[j]), scale[j], bias[j]));
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              v[j] = fma_sat(int_to_float((int)r[j]), scale[j], bias[j]);
          }
#pragma unroll
          for (int j4 = 0; j4 < 8; ++j4) {
            uint32_t c[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              c[i] = __float_as_uint(__fadd_rd(v[4 * j4 + i], 256.00390625f));
            const uint32_t packed = __byte_perm(__byte_perm(c[0], c[1], 0x0051), __byte_perm(c[2], c[3], 0x0051), 0x5410);
            w[j4] = packed - ((packed >> 7) & 0x01010101u);
          }
        } else {
          // u = acc * scale + bias, one fused multiply-add (scale and bias already carry the factor
          // 2 / delta when codes are written, so u is twice the quantizer's argument)
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j)
            v[j] = __fmaf_rn(int_to_float((int)r[j]), scale[j], bias[j]);
          if (ep.res_codes) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              v[j] = __fmaf_rn(residual(j), ep.res_scale, v[j]);
          } else if (ep.res_f32) {
            const float4 *rp = reinterpret_cast<const float4 *>(ep.res_f32 + off);
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {
              const float4 t = (j4 < 4 || upper) ? __ldg(rp + j4) : make_float4(0.f, 0.f, 0.f, 0.f);
              v[4 * j4 + 0] = __fmaf_rn(t.x, ep.res_scale, v[4 * j4 + 0]);
              v[4 * j4 + 1] = __fmaf_rn(t.y, ep.res_scale, v[4 * j4 + 1]);
              v[4 * j4 + 2] = __fmaf_rn(t.z, ep.res_scale, v[4 * j4 + 2]);
              v[4 * j4 + 3] = __fmaf_rn(t.w, ep.res_scale, v[4 * j4 + 3]);
            }
          }
          if (ep.y_f32) {
            float4 *yp = reinterpret_cast<float4 *>(ep.y_f32 + off);
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4)
              if (j4 < 4 || upper)
                yp[j4] = make_float4(v[4 * j4], v[4 * j4 + 1], v[4 * j4 + 2], v[4 * j4 + 3]);
            continue;
          }
#pragma unroll
          for (int j4 = 0; j4 < 8; ++j4) {
            uint32_t packed = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float x = v[4 * j4 + k];
              int code;
              if (ep.relu) {
                code = (__float2int_rd(fminf(fmaxf(x, 0.0f), cap)) + 1) >> 1;
              } else {
                const int m = (__float2int_rd(fminf(fabsf(x), cap)) + 1) >> 1;
                code = x < 0.0f ? max(-m, ep.kmin) : m;
              }
              packed |= ((uint32_t)code & 0xffu) << (8 * k);
            }
            w[j4] = packed;
          }
        }
        if (ep.y_codes == nullptr)
          continue; // no result configured (the host refuses this; never store through a null pointer)
        uint4 *yp = reinterpret_cast<uint4 *>(ep.y_codes + off);
        yp[0] = make_uint4(w[0], w[1], w[2], w[3]);
        if (upper)
          yp[1] = make_uint4(w[4], w[5], w[6], w[7]);
      }
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0)
        ptx::mbar_arrive(tmem_empty + buf);
      if (threadIdx.x == 64)
        NB_CC_STAMP(8, local);
    }
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
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// without the resident weights (k blocks * BN * RB bytes more when kResidentB)
// (in the halo form the ring is replaced by the pixel-tile buffers, counted by the caller)
template <int BN, int STAGES, int RB, bool kResidentB = false, bool kHalo = false>
constexpr size_t conv_codes_smem_bytes() {
  return (kHalo ? 0 : (size_t)STAGES * (kTileM * RB + (kResidentB ? 0 : BN * RB))) +
         (2 * STAGES + 4 + 2 * kTileBufs + kWeightParts) * 8 + 32 + kCodesMaxMaps * sizeof(float2) + kCodesKTable * sizeof(int4) + 1024;
}

} // namespace nb200
