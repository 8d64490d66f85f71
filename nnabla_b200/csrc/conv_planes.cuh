// Stride-1 convolution of channel-last floating-point planes on tcgen05, pixels on the MMA rows, each input pixel
// fetched once per tile for all filter taps (the halo form of conv_codes.cuh, for operands split into 16-bit pieces).
//
//   y[n, o, pixel] = scale[o] * sum over taps, channels and planes of A[plane][n, pixel + tap][c] * B[o][tap][c] + bias[o]
//
// Two uses:
//  * the input gradient of a convolution: A = dy in three bf16 pieces, B = the +-1 weights. A forward stride s makes
//    s * s classes of input pixels (row and column residues mod s): each class is a stride-1 convolution of dy with
//    the taps that reach it, so that no zeros are multiplied (spreading dy over the input grid multiplied s * s times
//    as much and stored it first);
//  * the forward convolution of fp32 activations: A = two fp16 pieces of the scaled activations, B = +-1 weights. A
//    stride s makes s * s classes of taps, each reading one of the s * s interleaved images of x.
//
// A column tile has as many maps as spread them evenly (160 as 80 + 80, not as 128 + 32 and 96 empty columns): an MMA's
// time follows its columns (a [24, 96, 35, 29] layer of 160 maps 29.6 us forward, 26.6 with even tiles; its input gradient,
// 96 columns, 31.9 and 29.3).
//
// What bounds it: the tensor core (an MMA of 128 rows takes 51 / 67 cycles for 64 / 128 columns, limited by the
// shared-memory reads of A). The previous form put the maps on the 128 MMA rows, half of them empty for 64 maps, and
// fetched a box of pixels per filter tap: 540 us for the input gradient of a 64 -> 64 3 x 3 layer on [128, 64, 56, 56],
// now 95 to 120, 71 of them MMAs at the rates above; the forward of 256 -> 256 maps on [128, 256, 28, 28] 183 us, now 169.
//
// A tile is a part of an image, or several small images: the box then holds them one behind the other, n_box deep,
// each with the halo along its columns only (a box per filter row) or with none (a box per tap), see
// choose_planes_span. A box and its place in the weights are tables in the problem, and all three roles walk them by
// counters: divisions per box took longer than the MMAs of one tap (512 -> 512 maps of 8 x 8, a box per tap, 256
// images: 207 us, 175 without them).
//
// Warp 0 loads (TMA), two warps issue the MMAs, eight epilogue warps store. The issuing warps take alternate tiles
// (kResident) or alternate weight tiles into accumulators of their own: a thread that decodes a tile, waits for
// barriers and comes back to the head of its unrolled loop leaves the tensor core idle, 27 % of the time with one. A
// stage of the pixel ring is the input box of PG planes of one 64-channel block; the weights of one tap and channel
// block come through a second ring
// (kResident: all of them are loaded once). With kResident the planes come one after the other, smallest pieces
// first, which also keeps the number of accumulation steps at full magnitude down; otherwise the planes of a box are
// multiplied with a weight tile together, so that each weight tile is fetched once per box.
#pragma once
#include "gemm.cuh"
#include "prepare.cuh"

namespace nb200 {

constexpr int kPlanesMaxTaps = 64;
constexpr int kPlanesMaxStages = 8;
constexpr int kPlanesThreads = kGemmThreads + 32; // the second issuing warp stands behind the epilogue warps

struct ConvPlanesProblem {
  int Nimg, maps, total_maps, groups; // output maps per group and in all
  int H, W;                           // output image
  int sy, sx;                         // output pixel (sy * u + ry, sx * v + rx) belongs to class ry * sx + rx
  int in_sy, in_sx;                   // step between the input pixels of a box
  int Wu;                             // columns of a class's grid: ceil(W / sx)
  int h_box, tiles_h, n_tiles;        // class rows per tile, tiles per class and image, column tiles
  int bn;                             // columns of a tile, a multiple of 16 up to BN: the maps spread evenly over the tiles
  int n_box, img_rows;                // images per tile (1 with tiles_h > 1) and MMA rows from one to the next
  int wp, hp;                         // input box: hp rows of wp pixels
  int cblocks;                        // 64-channel blocks of one group
  int c_group_stride;                 // channel slots between groups in A
  int k_slots;                        // weight slots per tap
  int plane_bytes;                    // of one plane's box in shared memory
  int planes;                         // planes of A
  int chunk;                          // weight tiles (tap, channel block) per accumulation in tensor memory, even; 0 = all
  int a_stages, b_stages;
  int class_box[17];                  // boxes that a tile of output class k sums: [class_box[k], class_box[k + 1])
  int box_tap[kPlanesMaxTaps + 1];    // taps that read box b: [box_tap[b], box_tap[b + 1]); may be none
  int16_t box_y[kPlanesMaxTaps], box_x[kPlanesMaxTaps]; // first input row (of a tile at row 0) and column
  int tap_row[kPlanesMaxTaps];        // first row of the box that tap reads
  int tap_k[kPlanesMaxTaps];          // its index in the weights
  const float *scale, *bias;          // per output map, may be NULL
  const uint32_t *image_max;          // per image: bits of the magnitude that its scaling was chosen from, may be NULL
  float *y;
  int accumulate;
  __host__ __device__ __forceinline__ int num_tiles() const {
    return n_tiles * sy * sx * groups * tiles_h * ((Nimg + n_box - 1) / n_box);
  }
};

template <int BN, int PG, bool kResident, bool kF16>
__global__ void __launch_bounds__(kPlanesThreads, 1)
    conv_planes_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                               const __grid_constant__ ConvPlanesProblem prob, int *status) {
  static_assert(BN == 64 || BN == 128, "column tiles of 64 or 128 maps");
  constexpr uint32_t kBBytes = BN * kRowBytes;
  constexpr int kAccs = kResident ? 1 : 2; // accumulators of a chunk: one per issuing warp, which share its tiles
  constexpr uint32_t kTmemCols = 2 * kAccs * BN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t stage_bytes = (uint32_t)PG * prob.plane_bytes;
  uint8_t *b_base = smem; // weights first: MMAs may read up to 128 rows past a box (rows of no stored pixel)
  const uint32_t b_tiles = kResident ? (uint32_t)(prob.box_tap[prob.class_box[prob.sy * prob.sx]] * prob.cblocks)
                                     : (uint32_t)prob.b_stages;
  uint8_t *a_base = smem + b_tiles * kBBytes;

  __shared__ __align__(8) uint64_t a_full[kPlanesMaxStages], a_empty[kPlanesMaxStages], b_full[kPlanesMaxStages],
      b_empty[kPlanesMaxStages], tmem_full[2], tmem_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int *abort_flag = &abort_word;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_tiles = prob.num_tiles();
  const int plane_groups = prob.planes / PG;
  const uint32_t b_bytes = (uint32_t)prob.bn * kRowBytes; // of a weight tile, in kBBytes of shared memory

  if (threadIdx.x == 0) {
    for (int i = 0; i < kPlanesMaxStages; ++i) {
      ptx::mbar_init(a_full + i, 1);
      ptx::mbar_init(a_empty + i, 2); // both issuers: a barrier's phase must not run past one that has not seen it
      ptx::mbar_init(b_full + i, 1);
      ptx::mbar_init(b_empty + i, 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(tmem_full + b, kAccs);
      ptx::mbar_init(tmem_empty + b, kEpilogueWarps);
    }
    abort_word = 0;
    ptx::mbar_fence_init();
    ptx::prefetch_tensormap(&map_a);
    ptx::prefetch_tensormap(&map_b);
  }
  if (warp == 1) {
    ptx::tmem_alloc(&tmem_slot, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  pdl_wait();
  if (early_trigger((int64_t)prob.Nimg * prob.total_maps * prob.H * prob.W))
    pdl_trigger();

  struct TileAt {
    int n0, cls, group, row0, img;
  };
  // the column tiles of a box are neighbours in time, then the classes: the box stays in L2
  auto decode = [&](int tile) {
    TileAt t;
    t.n0 = (tile % prob.n_tiles) * prob.bn;
    tile /= prob.n_tiles;
    t.cls = tile % (prob.sy * prob.sx);
    tile /= prob.sy * prob.sx;
    t.group = tile % prob.groups;
    tile /= prob.groups;
    t.row0 = (tile % prob.tiles_h) * prob.h_box;
    t.img = tile / prob.tiles_h * prob.n_box;
    return t;
  };
  // the boxes of a tile, in the order of the ring: (channel block, box of its class, plane group)
  struct BoxWalk {
    int first, end, cb, box, pg; // box counts from first, the first of the class, to end
  };
  auto boxes_of = [&](const TileAt &t) {
    const int first = prob.class_box[t.cls];
    return BoxWalk{first, prob.class_box[t.cls + 1], 0, first, 0};
  };
  auto next_box = [&](BoxWalk &b) {
    if (++b.pg == plane_groups) {
      b.pg = 0;
      if (++b.box == b.end) {
        b.box = b.first;
        ++b.cb;
      }
    }
  };
  auto taps_of = [&](const TileAt &t) { // 0: an output class that no tap reaches
    return prob.box_tap[prob.class_box[t.cls + 1]] - prob.box_tap[prob.class_box[t.cls]];
  };
  auto gave_up = [&](int code) {
    if (*abort_flag == 0)
      atomicCAS(status, 0, code);
    *abort_flag = 1;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (ptx::elect_one()) {
      int as = 0, bs = 0;
      uint32_t aphase = 0, bphase = 0;
      bool ok = true;
      if (kResident && (int)blockIdx.x < num_tiles) { // one group, one column tile
        ptx::mbar_expect_tx(b_full, b_tiles * b_bytes);
        for (uint32_t i = 0; i < b_tiles; ++i) {
          const int tap = (int)i / prob.cblocks, cb = (int)i - tap * prob.cblocks;
          ptx::tma_load_3d(b_base + i * kBBytes, &map_b, b_full, prob.tap_k[tap] * prob.k_slots + cb * 64, 0, 0);
        }
      }
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        const TileAt t = decode(tile);
        if (taps_of(t) == 0)
          continue;
        for (BoxWalk at = boxes_of(t); at.cb < prob.cblocks && ok; next_box(at)) {
          const int cb = at.cb, pg = at.pg, tap0 = prob.box_tap[at.box], tap1 = prob.box_tap[at.box + 1];
          if (tap0 == tap1)
            continue;
          if (!ptx::mbar_wait(a_empty + as, aphase ^ 1u, abort_flag)) {
            gave_up(kStatusProducerTimeout);
            ok = false;
            break;
          }
          ptx::mbar_expect_tx(a_full + as, (uint32_t)(PG * prob.n_box * prob.hp * prob.wp * kRowBytes));
#pragma unroll
          for (int p = 0; p < PG; ++p)
            ptx::tma_load_5d(a_base + as * stage_bytes + p * prob.plane_bytes, &map_a, a_full + as,
                             t.group * prob.c_group_stride + cb * 64, prob.box_x[at.box],
                             t.row0 * prob.in_sy + prob.box_y[at.box], t.img,
                             prob.planes - 1 - (pg * PG + p)); // smallest pieces first
          if (++as == prob.a_stages) {
            as = 0;
            aphase ^= 1u;
          }
          if (!kResident)
            for (int tap = tap0; tap < tap1; ++tap) {
              if (!ptx::mbar_wait(b_empty + bs, bphase ^ 1u, abort_flag)) {
                gave_up(kStatusProducerTimeout);
                ok = false;
                break;
              }
              ptx::mbar_expect_tx(b_full + bs, b_bytes);
              ptx::tma_load_3d(b_base + bs * kBBytes, &map_b, b_full + bs, prob.tap_k[tap] * prob.k_slots + cb * 64,
                               t.group * prob.maps + t.n0, 0);
              if (++bs == prob.b_stages) {
                bs = 0;
                bphase ^= 1u;
              }
            }
        }
      }
    }
  } else if (warp == 1 || warp == 2 + kEpilogueWarps) {
    // ------------------------------------------------------------- MMA issuers
    const int who = warp == 1 ? 0 : 1;
    if (ptx::elect_one()) {
      int as = 0, bs = 0, local = 0; // stages and chunk (or tile) counted over both issuers' work
      uint32_t aphase = 0, bphase = 0;
      bool ok = true;
      const uint32_t idesc = ptx::make_idesc(1u, kF16 ? 0u : 1u, kTileM, (uint32_t)prob.bn);
      const uint32_t hi = (uint32_t)(ptx::smem_desc_k(0, kRowBytes) >> 32);
      const uint32_t a_lo = ptx::smem_u32(a_base) >> 4, b_lo = ptx::smem_u32(b_base) >> 4; // below 2^14
      auto next_a = [&]() {
        if (++as == prob.a_stages) {
          as = 0;
          aphase ^= 1u;
        }
      };
      uint32_t accumulate = 0, d_tmem = 0;
      auto open_chunk = [&]() { // waits for the accumulator of the next chunk
        const int buf = local & 1;
        if (!ptx::mbar_wait(tmem_empty + buf, ((uint32_t)(local >> 1) & 1u) ^ 1u, abort_flag)) {
          gave_up(kStatusMmaTimeout);
          return false;
        }
        ptx::tc_fence_after_sync();
        d_tmem = tmem_base + (uint32_t)((buf * kAccs + (kResident ? 0 : who)) * BN);
        accumulate = 0;
        return true;
      };
      auto wait = [&](uint64_t *bar, uint32_t phase) {
        if (!ptx::mbar_wait(bar, phase, abort_flag)) {
          gave_up(kStatusMmaTimeout);
          return false;
        }
        ptx::tc_fence_after_sync();
        return true;
      };
      auto issue = [&](uint32_t a_row16, uint32_t b16) {
#pragma unroll
        for (int p = 0; p < PG; ++p)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            ptx::mma_bf16(d_tmem, ((uint64_t)hi << 32) | (a_row16 + p * ((uint32_t)prob.plane_bytes >> 4) + 2 * k),
                          ((uint64_t)hi << 32) | (b16 + 2 * k), idesc, accumulate);
            accumulate = 1;
          }
      };
      if (kResident && (int)blockIdx.x < num_tiles)
        ok = wait(b_full, 0u);
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        const TileAt t = decode(tile);
        if (taps_of(t) == 0)
          continue;
        if constexpr (kResident) {
          if ((local & 1) != who) { // the other issuer's tile: its boxes are released as soon as they have come
            for (BoxWalk at = boxes_of(t); at.cb < prob.cblocks; next_box(at)) {
              if (prob.box_tap[at.box] == prob.box_tap[at.box + 1])
                continue;
              if (!(ok = wait(a_full + as, aphase)))
                break;
              ptx::mbar_arrive(a_empty + as);
              next_a();
            }
            ++local;
            continue;
          }
          ok = open_chunk();
          for (BoxWalk at = boxes_of(t); at.cb < prob.cblocks && ok; next_box(at)) {
            const int cb = at.cb, tap0 = prob.box_tap[at.box], tap1 = prob.box_tap[at.box + 1];
            if (tap0 == tap1)
              continue;
            if (!(ok = wait(a_full + as, aphase)))
              break;
            const uint32_t a_stage = a_lo + ((uint32_t)as * stage_bytes >> 4);
            // in batches: the descriptors of three taps before their MMAs
            int tap = tap0;
            for (; tap + 3 <= tap1; tap += 3) {
              uint32_t off[3];
#pragma unroll
              for (int u = 0; u < 3; ++u)
                off[u] = a_stage + (uint32_t)prob.tap_row[tap + u] * (kRowBytes >> 4);
#pragma unroll
              for (int u = 0; u < 3; ++u)
                issue(off[u], b_lo + (uint32_t)((tap + u) * prob.cblocks + cb) * (kBBytes >> 4));
            }
            for (; tap < tap1; ++tap)
              issue(a_stage + (uint32_t)prob.tap_row[tap] * (kRowBytes >> 4),
                    b_lo + (uint32_t)(tap * prob.cblocks + cb) * (kBBytes >> 4));
            ptx::mma_commit(a_empty + as); // the boxes are free once these MMAs have read them
            next_a();
          }
        } else {
          // Weight stages alternate between the issuers (their number is even), so that each sees every phase of its own.
          int in_chunk = 0;
          ok = open_chunk();
          for (BoxWalk at = boxes_of(t); at.cb < prob.cblocks && ok; next_box(at)) {
            const int tap0 = prob.box_tap[at.box], tap1 = prob.box_tap[at.box + 1];
            if (tap0 == tap1)
              continue;
            if (!(ok = wait(a_full + as, aphase)))
              break;
            const uint32_t a_stage = a_lo + ((uint32_t)as * stage_bytes >> 4);
            for (int tap = tap0; tap < tap1; ++tap) {
              if (prob.chunk > 0 && in_chunk == prob.chunk) {
                ptx::mma_commit(tmem_full + (local & 1));
                ++local;
                in_chunk = 0;
                if (!(ok = open_chunk()))
                  break;
              }
              if ((bs & 1) == who) {
                if (!(ok = wait(b_full + bs, bphase)))
                  break;
                issue(a_stage + (uint32_t)prob.tap_row[tap] * (kRowBytes >> 4), b_lo + (uint32_t)bs * (kBBytes >> 4));
                ptx::mma_commit(b_empty + bs);
              }
              ++in_chunk;
              if (++bs == prob.b_stages) {
                bs = 0;
                bphase ^= 1u;
              }
            }
            ptx::mma_commit(a_empty + as);
            next_a();
          }
        }
        if (ok) {
          ptx::mma_commit(tmem_full + (local & 1));
          ++local;
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int quarter = warp & 3, set = (warp - 2) >> 2; // TMEM lanes [32 * quarter, + 32); even / odd column chunks
    const int row = quarter * 32 + lane, box_img = row / prob.img_rows, in_img = row - box_img * prob.img_rows;
    const int box_y = in_img / prob.wp, box_x = in_img - box_y * prob.wp;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int64_t plane = (int64_t)prob.H * prob.W;
    constexpr int kMine = BN / 64; // chunks of 32 columns per warp
    int local = 0, b_at = 0;       // chunks, weight tiles so far
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      const TileAt t = decode(tile);
      const int taps = taps_of(t);
      const int ry = t.cls / prob.sx, rx = t.cls - ry * prob.sx;
      const int iy = (t.row0 + box_y) * prob.sy + ry, ix = box_x * prob.sx + rx;
      const int img = t.img + box_img;
      const bool pix_ok = box_img < prob.n_box && img < prob.Nimg && box_y < prob.h_box && box_x < prob.Wu &&
                          iy < prob.H && ix < prob.W;
      const int tiles_k = kResident ? 1 : taps * prob.cblocks;
      const int chunks = taps == 0 ? 0 : (kResident || prob.chunk == 0 ? 1 : (tiles_k + prob.chunk - 1) / prob.chunk);
      float acc[kMine][32];
#pragma unroll
      for (int ci = 0; ci < kMine; ++ci)
#pragma unroll
        for (int j = 0; j < 32; ++j)
          acc[ci][j] = 0.0f;
      // With one chunk of maps per warp the values to add to are fetched before the accumulator is waited for: behind the
      // wait, eight at a time, a tile's epilogue took longer than its MMAs (input gradient of a 64 -> 64 3 x 3 layer on
      // [128, 64, 56, 56] added to dx 121 us, now 96; not added 91). With two chunks there are no registers for them.
      constexpr int kAhead = kMine == 1 ? 32 : 1;
      float ahead[kAhead];
      auto chunk_left = [&](int ci) { // maps of this chunk that the tile has
        const int c = 32 * set + 64 * ci;
        return min(prob.maps - t.n0, prob.bn) - c;
      };
      auto chunk_y = [&](int ci) {
        return prob.y + ((int64_t)img * prob.total_maps + t.group * prob.maps + t.n0 + 32 * set + 64 * ci) * plane +
               (int64_t)iy * prob.W + ix;
      };
      if (kMine == 1 && prob.accumulate && pix_ok) {
        const float *yp = chunk_y(0);
        const int left = chunk_left(0);
#pragma unroll
        for (int j = 0; j < kAhead; ++j)
          ahead[j] = j < left ? yp[(int64_t)j * plane] : 0.0f;
      }
      for (int kc = 0; kc < chunks; ++kc, ++local) {
        const int buf = local & 1;
        const bool got = ptx::mbar_wait(tmem_full + buf, (uint32_t)(local >> 1) & 1u, abort_flag);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0)
            gave_up(kStatusEpilogueTimeout);
          ok = false;
          break;
        }
        ptx::tc_fence_after_sync();
        // a chunk of one weight tile lies in the accumulator of the issuer that had it
        const int in_chunk = prob.chunk == 0 || tiles_k - kc * prob.chunk < prob.chunk ? tiles_k - kc * prob.chunk : prob.chunk;
        const bool both = kAccs == 2 && in_chunk > 1;
        const int only = kAccs == 2 && in_chunk == 1 ? b_at & 1 : 0;
        b_at += in_chunk;
#pragma unroll
        for (int ci = 0; ci < kMine; ++ci) {
          const uint32_t at = lane_base + (uint32_t)((buf * kAccs + only) * BN + 32 * set + 64 * ci);
          uint32_t r[32], r2[32];
          ptx::tmem_ld_32x32(at, r);
          if (both)
            ptx::tmem_ld_32x32(at + BN, r2);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) // chunk sums in fp32, round to nearest (the first addend is 0)
            acc[ci][j] = __fadd_rn(acc[ci][j], __uint_as_float(r[j]));
          if (both)
#pragma unroll
            for (int j = 0; j < 32; ++j)
              acc[ci][j] = __fadd_rn(acc[ci][j], __uint_as_float(r2[j]));
        }
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0)
          ptx::mbar_arrive(tmem_empty + buf);
      }
      if (!ok)
        break;
#pragma unroll
      for (int ci = 0; ci < kMine; ++ci) {
        const int left = chunk_left(ci);
        if (left <= 0)
          continue;
        const int map0 = t.group * prob.maps + t.n0 + 32 * set + 64 * ci;
        float *yp = chunk_y(ci);
        if (prob.scale || prob.bias || prob.image_max) {
          // one rounding per operation, like the reference's product and bias addition (the image's factor is a power
          // of two)
          const float up = prob.image_max && pix_ok
                               ? __int_as_float((127 + half_pair_exponent(__ldg(prob.image_max + img))) << 23)
                               : 1.0f;
          const float ls = prob.scale && lane < left ? __ldg(prob.scale + map0 + lane) : 1.0f;
          const float lb = prob.bias && lane < left ? __ldg(prob.bias + map0 + lane) : 0.0f;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            acc[ci][j] = __fmul_rn(acc[ci][j], __fmul_rn(__shfl_sync(0xffffffffu, ls, j), up));
            if (prob.bias)
              acc[ci][j] = __fadd_rn(acc[ci][j], __shfl_sync(0xffffffffu, lb, j));
          }
        }
        if (!pix_ok)
          continue;
        if (prob.accumulate) {
#pragma unroll
          for (int j0 = 0; j0 < 32; j0 += 8) {
            float old[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
              old[j] = kMine == 1 ? ahead[(j0 + j) % kAhead] : j0 + j < left ? yp[(int64_t)(j0 + j) * plane] : 0.0f;
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (j0 + j < left)
                yp[(int64_t)(j0 + j) * plane] = __fadd_rn(old[j], acc[ci][j0 + j]);
          }
        } else if (left >= 32) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            yp[(int64_t)j * plane] = acc[ci][j];
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (j < left)
              yp[(int64_t)j * plane] = acc[ci][j];
        }
      }
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

} // namespace nb200
