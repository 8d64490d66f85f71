// Training side of the companion functions of a binary-weight ResNet:
// batch-statistics BatchNormalization (forward), and the backward passes of
// BatchNormalization, ReLU, Add2, MaxPooling and GlobalAveragePooling.
//
// The elementwise parts follow the reference's operation order, every operation
// rounded separately, so that given the same per-channel statistics the results
// are bit-identical to its CPU code. The per-channel SUMS (batch mean and
// variance, parameter gradients) are block partials added in a fixed order in
// double precision: deterministic, and closer to the exact sums than the
// reference's sequential fp32 accumulation, so those agree to rounding only.
#include <cmath>

#include "common.cuh"
#include "pdl.cuh"

namespace nb200 {
namespace {

constexpr int kThreads = 256;

inline unsigned grid_for(size_t items, int per_thread = 1) {
  size_t b = (items + (size_t)kThreads * per_thread - 1) / ((size_t)kThreads * per_thread);
  const size_t cap = (size_t)sm_count() * 64;
  if (b > cap)
    b = cap;
  return (unsigned)(b < 1 ? 1 : b);
}

// ---------------------------------------------------------------- elementwise backward passes

// relu.cpp:41-49: dx (+)= y > 0 ? dy : 0; add2.cpp: dx (+)= dy.
// A block takes kThreads * kPer consecutive vectors (values where a tensor is not 16-byte aligned), the last block's first
// (st_result); block 0 the remainder of a vector.
template <int kOp, bool kAccum, bool kVec, int kPer>
__global__ void __launch_bounds__(kThreads) grad_pass_kernel(const float *__restrict__ y, const float *__restrict__ dy,
                                                             float *__restrict__ dx, size_t total) {
  pdl_wait();
  pdl_trigger();
  auto one = [](float yv, float g, float old) {
    const float v = kOp == 0 ? (yv > 0.0f ? g : 0.0f) : g;
    return kAccum ? __fadd_rn(old, v) : v;
  };
  const size_t first = block_descending() * (kThreads * kPer) + threadIdx.x;
  const size_t total4 = kVec ? total / 4 : 0;
  if (kVec) {
    const bool keep = total * sizeof(float) <= kKeepBytes;
    float4 g[kPer], yv[kPer], o[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u)
      if (first + u * kThreads < total4) {
        g[u] = ld_stream(reinterpret_cast<const float4 *>(dy) + first + u * kThreads);
        yv[u] = kOp == 0 ? ld_stream(reinterpret_cast<const float4 *>(y) + first + u * kThreads) : g[u];
        o[u] = kAccum ? reinterpret_cast<const float4 *>(dx)[first + u * kThreads] : g[u];
      }
#pragma unroll
    for (int u = 0; u < kPer; ++u)
      if (first + u * kThreads < total4)
        st_result(reinterpret_cast<float4 *>(dx) + first + u * kThreads,
                  make_float4(one(yv[u].x, g[u].x, o[u].x), one(yv[u].y, g[u].y, o[u].y), one(yv[u].z, g[u].z, o[u].z),
                              one(yv[u].w, g[u].w, o[u].w)),
                  keep);
    if (blockIdx.x == 0 && threadIdx.x < total - total4 * 4) {
      const size_t i = total4 * 4 + threadIdx.x;
      dx[i] = one(kOp == 0 ? y[i] : 0.0f, dy[i], kAccum ? dx[i] : 0.0f);
    }
  } else {
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const size_t i = first + u * kThreads;
      if (i < total)
        dx[i] = one(kOp == 0 ? y[i] : 0.0f, dy[i], kAccum ? dx[i] : 0.0f);
    }
  }
}

// Vectors (or values, unaligned) of a thread: four, or one while that leaves every SM room for all its blocks at once.
template <int kOp, bool kAccum>
int launch_grad_pass(const float *y, const float *dy, float *dx, size_t size, cudaStream_t st) {
  const bool vec = ((reinterpret_cast<uintptr_t>(kOp == 0 ? y : dy) | reinterpret_cast<uintptr_t>(dy) |
                     reinterpret_cast<uintptr_t>(dx)) & 15) == 0;
  const size_t items = vec ? size / 4 : size;
  const bool few = items <= (size_t)sm_count() * 4 * kThreads;
  const size_t per = (size_t)kThreads * (few ? 1 : 4);
  const size_t blocks = items ? (items + per - 1) / per : 1;
  auto kernel = vec ? (few ? grad_pass_kernel<kOp, kAccum, true, 1> : grad_pass_kernel<kOp, kAccum, true, 4>)
                    : (few ? grad_pass_kernel<kOp, kAccum, false, 1> : grad_pass_kernel<kOp, kAccum, false, 4>);
  NB_CUDA(launch_dependent(kernel, dim3((unsigned)blocks), dim3(kThreads), 0, st, y, dy, dx, size));
  return NB200_OK;
}

// global_average_pooling.cpp:75-117: every pixel of map m receives dy[m] / (H W).
template <bool kAccum>
__global__ void __launch_bounds__(kThreads) gap_backward_kernel(const float *__restrict__ dy, float *__restrict__ dx,
                                                                size_t total, unsigned S) {
  pdl_wait();
  pdl_trigger();
  const size_t stride = (size_t)gridDim.x * kThreads;
  for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < total; i += stride) {
    const float g = __fdiv_rn(__ldg(dy + i / S), (float)S);
    dx[i] = kAccum ? __fadd_rn(dx[i], g) : g;
  }
}

// max_pooling.cpp:44-77, :134-139, :194-228. The reference stores the index of the first maximum of
// every clipped window and then runs dx[index] += dy over the outputs in order. Two passes here: the
// first writes that index map (one thread per output, the reference's scan with its strict compare);
// in the second every INPUT pixel walks the windows that contain it in ascending output order and adds
// dy of those whose index is its own: the same additions in the same order, without atomics.
__global__ void __launch_bounds__(kThreads)
    max_pooling_index_kernel(const float *__restrict__ x, int *__restrict__ index, size_t outputs, int H, int W,
                             int Ho, int Wo, int kh, int kw, int sh, int sw, int ph, int pw) {
  pdl_wait();
  pdl_trigger();
  const size_t stride = (size_t)gridDim.x * kThreads;
  for (size_t o = (size_t)blockIdx.x * kThreads + threadIdx.x; o < outputs; o += stride) {
    const int ox = (int)(o % Wo);
    const size_t t = o / Wo;
    const int oy = (int)(t % Ho);
    const float *xm = x + (t / Ho) * H * W;
    int y0 = oy * sh - ph, x0 = ox * sw - pw;
    const int y1 = min(y0 + kh, H), x1 = min(x0 + kw, W);
    y0 = max(y0, 0);
    x0 = max(x0, 0);
    int best_i = y0 * W + x0;
    float best = __ldg(xm + best_i);
    for (int yy = y0; yy < y1; ++yy)
      for (int xx = x0; xx < x1; ++xx) {
        const float v = __ldg(xm + yy * W + xx);
        if (best < v) {
          best = v;
          best_i = yy * W + xx;
        }
      }
    index[o] = best_i;
  }
}

template <bool kAccum>
__global__ void __launch_bounds__(kThreads)
    max_pooling_backward_kernel(const int *__restrict__ index, const float *__restrict__ dy, float *__restrict__ dx,
                                size_t total, int H, int W, int Ho, int Wo, int kh, int kw, int sh, int sw, int ph,
                                int pw) {
  pdl_wait();
  pdl_trigger();
  const size_t stride = (size_t)gridDim.x * kThreads;
  for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < total; i += stride) {
    const int ix = (int)(i % W);
    const size_t t = i / W;
    const int iy = (int)(t % H);
    const size_t m = t / H;
    const int *im = index + m * Ho * Wo;
    const float *dym = dy + m * Ho * Wo;
    float acc = kAccum ? dx[i] : 0.0f;
    // windows oy with oy * sh - ph <= iy < oy * sh - ph + kh
    int oy0 = iy + ph - kh + 1;
    oy0 = oy0 <= 0 ? 0 : (oy0 + sh - 1) / sh;
    int oy1 = (iy + ph) / sh;
    oy1 = oy1 < Ho - 1 ? oy1 : Ho - 1;
    int ox0 = ix + pw - kw + 1;
    ox0 = ox0 <= 0 ? 0 : (ox0 + sw - 1) / sw;
    int ox1 = (ix + pw) / sw;
    ox1 = ox1 < Wo - 1 ? ox1 : Wo - 1;
    const int mine = iy * W + ix;
    for (int oy = oy0; oy <= oy1; ++oy)
      for (int ox = ox0; ox <= ox1; ++ox)
        if (__ldg(im + oy * Wo + ox) == mine)
          acc = __fadd_rn(acc, __ldg(dym + oy * Wo + ox));
    dx[i] = acc;
  }
}

// ---------------------------------------------------------------- per-channel sums

// Walks the values of channel c of an [N, C, S] tensor: item j of the channel (j = n * S + s, counted in
// units of kW values) lives at ((n * C + c) * S + s). Start and step are split once; no division per item.
struct ChannelItems {
  unsigned n, s, dn, ds, S, N;
  __device__ __forceinline__ ChannelItems(size_t first, size_t step, unsigned S_, unsigned N_) : S(S_), N(N_) {
    n = (unsigned)(first / S_);
    s = (unsigned)(first - (size_t)n * S_);
    dn = (unsigned)(step / S_);
    ds = (unsigned)(step - (size_t)dn * S_);
  }
  __device__ __forceinline__ bool valid() const { return n < N; }
  __device__ __forceinline__ void next() {
    s += ds;
    const unsigned carry = s >= S ? 1u : 0u;
    s -= carry ? S : 0u;
    n += dn + carry;
  }
};

// (v)^-0.5 and (v)^-1.5 rounded from double precision: what a correctly rounded powf returns
__device__ __forceinline__ float inv_sqrt_rn(float v) { return (float)(1.0 / sqrt((double)v)); }
__device__ __forceinline__ float inv_sqrt_cubed_rn(float v) { return (float)(1.0 / ((double)v * sqrt((double)v))); }

template <int K> __device__ __forceinline__ void block_sums(float (&v)[K], float *out) {
  __shared__ float part[K][kThreads / 32];
#pragma unroll
  for (int k = 0; k < K; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if ((threadIdx.x & 31) == 0)
      part[k][threadIdx.x >> 5] = v[k];
  }
  __syncthreads();
  if (threadIdx.x < K) {
    float t = 0.0f;
    for (int w = 0; w < kThreads / 32; ++w)
      t += part[threadIdx.x][w];
    out[threadIdx.x] = t;
  }
}

// Calls use(loaded value, sum) for this block's items of channel c, four at a time with their loads before their use:
// the sums are HBM-bound and one load in flight per thread reached half of the copy bandwidth. use adds to a sum of the
// four, which is then added to v_sum: a quarter of the additions at the sum's full magnitude.
template <int kW, int K, typename Load, typename Use>
__device__ __forceinline__ void channel_sum_loop(unsigned N, unsigned C, unsigned S, float (&v_sum)[K], Load load, Use use) {
  const unsigned c = blockIdx.y, P = gridDim.x, Su = S / kW;
  ChannelItems it((size_t)blockIdx.x * kThreads + threadIdx.x, (size_t)P * kThreads, Su, N);
  while (it.valid()) {
    decltype(load((size_t)0)) v[4];
    bool live[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      live[u] = it.valid();
      if (live[u])
        v[u] = load(((size_t)it.n * C + c) * S + (size_t)kW * it.s);
      it.next();
    }
    float four[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
      four[k] = 0.0f;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (live[u])
        use(v[u], four);
#pragma unroll
    for (int k = 0; k < K; ++k)
      v_sum[k] += four[k];
  }
}

// partial sums of x and x^2 of channel blockIdx.y over the items of block blockIdx.x: partial[c][p][2]
template <bool kVec>
__global__ void __launch_bounds__(kThreads) bn_stats_kernel(const float *__restrict__ x, unsigned N, unsigned C,
                                                            unsigned S, float *__restrict__ partial) {
  pdl_wait();
  pdl_trigger();
  float v[2] = {0.0f, 0.0f};
  if constexpr (kVec) {
    channel_sum_loop<4>(N, C, S, v, [&](size_t i) { return __ldg(reinterpret_cast<const float4 *>(x + i)); },
                        [](float4 a, float (&s)[2]) {
                          s[0] += (a.x + a.y) + (a.z + a.w);
                          s[1] += (a.x * a.x + a.y * a.y) + (a.z * a.z + a.w * a.w);
                        });
  } else {
    channel_sum_loop<1>(N, C, S, v, [&](size_t i) { return __ldg(x + i); },
                        [](float a, float (&s)[2]) {
                          s[0] += a;
                          s[1] += a * a;
                        });
  }
  block_sums<2>(v, partial + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 2);
}

// Sums over the P blocks of a channel's K partial sums, by kLanes neighbouring lanes: each adds every kLanes-th block's,
// then the lanes' sums are added pairwise; a fixed order, in double precision. One lane per channel is a chain of P loads
// and additions ([128, 64, 56, 56], 13 blocks a channel: 3.4 us, now 2.6), a warp per channel is slower where P is 4.
constexpr int kLanes = 8, kFinishThreads = 128;
template <int K> __device__ __forceinline__ void channel_total(const float *__restrict__ partial, unsigned P, double (&t)[K]) {
#pragma unroll
  for (int k = 0; k < K; ++k)
    t[k] = 0.0;
  for (unsigned p = threadIdx.x % kLanes; p < P; p += kLanes)
#pragma unroll
    for (int k = 0; k < K; ++k)
      t[k] += (double)partial[(size_t)p * K + k];
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1)
      t[k] += __shfl_down_sync(0xffffffffu, t[k], o, kLanes);
}

// batch_normalization.cpp:191-205 given the channel's sums: mean, variance, running statistics.
__global__ void bn_stats_finish_kernel(const float *__restrict__ partial, unsigned P, unsigned C, float count,
                                       float decay, int update, float *__restrict__ m, float *__restrict__ v,
                                       float *__restrict__ rm, float *__restrict__ rv) {
  pdl_wait();
  pdl_trigger();
  const unsigned c = (blockIdx.x * kFinishThreads + threadIdx.x) / kLanes;
  double t[2]; // (all lanes of a warp add and shuffle together)
  channel_total<2>(partial + (size_t)c * P * 2, c < C ? P : 0u, t);
  if (c >= C || threadIdx.x % kLanes != 0)
    return;
  const float mean = __fdiv_rn((float)t[0], count);
  const float var = __fsub_rn(__fdiv_rn((float)t[1], count), __fmul_rn(mean, mean));
  m[c] = mean;
  v[c] = var;
  if (update) {
    const float keep = __fsub_rn(1.0f, decay);
    rm[c] = __fadd_rn(__fmul_rn(decay, rm[c]), __fmul_rn(keep, mean));
    rv[c] = __fadd_rn(__fmul_rn(decay, rv[c]),
                      __fdiv_rn(__fmul_rn(__fmul_rn(keep, var), count), __fsub_rn(count, 1.0f)));
  }
}

// partial[c][p][3]: sum dy, sum dy * (x - m), sum (x - m) (the last for batch statistics only). The reference's sums
// over dy * scale * (x - m), dy * scale and dy * (x - m) / sqrt(v + eps) are these times a constant of the channel.
template <bool kVec, bool kBatch>
__global__ void __launch_bounds__(kThreads)
    bn_backward_sums_kernel(const float *__restrict__ x, const float *__restrict__ dy, const float *__restrict__ mean,
                            unsigned N, unsigned C, unsigned S, float *__restrict__ partial) {
  pdl_wait();
  pdl_trigger();
  const float m = mean[blockIdx.y];
  float v[3] = {0.0f, 0.0f, 0.0f};
  auto one = [&](float xv, float g, float (&s)[3]) {
    const float cx = __fsub_rn(xv, m);
    s[0] += g;
    s[1] += __fmul_rn(g, cx);
    if (kBatch)
      s[2] += cx;
  };
  if constexpr (kVec) {
    struct Pair {
      float4 a, g;
    };
    channel_sum_loop<4>(N, C, S, v,
                        [&](size_t i) {
                          return Pair{__ldg(reinterpret_cast<const float4 *>(x + i)),
                                      __ldg(reinterpret_cast<const float4 *>(dy + i))};
                        },
                        [&](const Pair &p, float (&s)[3]) {
                          one(p.a.x, p.g.x, s);
                          one(p.a.y, p.g.y, s);
                          one(p.a.z, p.g.z, s);
                          one(p.a.w, p.g.w, s);
                        });
  } else {
    channel_sum_loop<1>(N, C, S, v, [&](size_t i) { return make_float2(__ldg(x + i), __ldg(dy + i)); },
                        [&](float2 p, float (&s)[3]) { one(p.x, p.y, s); });
  }
  block_sums<3>(v, partial + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 3);
}

// coef[c][4] for the dx pass: {dvar * 2, dmean / n, gamma * (v + eps)^-0.5, -}. Batch mode
// (batch_normalization.cpp:326-334): dvar = s0 * -0.5 * (v + eps)^-1.5 + dv;
// dmean = s1 * (-1 / sqrt(v + eps)) + dvar * -2 * s2 / n + dm. `partial` may be NULL (no sums were needed).
__global__ void bn_backward_finish_kernel(const float *__restrict__ partial, unsigned P, unsigned C, float count,
                                          const float *__restrict__ gamma, const float *__restrict__ var, float eps,
                                          const float *__restrict__ dm, const float *__restrict__ dv, int batch,
                                          float *__restrict__ coef, float *__restrict__ dbeta, int accum_dbeta,
                                          float *__restrict__ dgamma, int accum_dgamma) {
  pdl_wait();
  pdl_trigger();
  const unsigned c = (blockIdx.x * kFinishThreads + threadIdx.x) / kLanes;
  double t[3]; // (all lanes of a warp add and shuffle together)
  channel_total<3>(partial + (size_t)c * P * 3, partial && c < C ? P : 0u, t);
  if (c >= C || threadIdx.x % kLanes != 0)
    return;
  const float ve = __fadd_rn(var[c], eps);
  const double scale = gamma ? (double)gamma[c] : 1.0;
  // sum dy*scale*(x-m), sum dy*scale, sum (x-m), sum dy, sum dy*(x-m)/sqrt(v+eps)
  const double s[5] = {scale * t[1], scale * t[0], t[2], t[0], t[1] / sqrt((double)ve)};
  {
    const float r = inv_sqrt_rn(ve);
    coef[c * 4 + 2] = gamma ? __fmul_rn(gamma[c], r) : r;
  }
  if (batch) {
    const float dvar = __fadd_rn(__fmul_rn(__fmul_rn((float)s[0], -0.5f), inv_sqrt_cubed_rn(ve)), dv ? dv[c] : 0.0f);
    float dmean = __fmul_rn((float)s[1], __fdiv_rn(-1.0f, __fsqrt_rn(ve)));
    dmean = __fadd_rn(dmean, __fdiv_rn(__fmul_rn(__fmul_rn(dvar, -2.0f), (float)s[2]), count));
    dmean = __fadd_rn(dmean, dm ? dm[c] : 0.0f);
    coef[c * 4 + 0] = __fmul_rn(dvar, 2.0f);
    coef[c * 4 + 1] = __fdiv_rn(dmean, count);
  }
  if (dbeta)
    dbeta[c] = accum_dbeta ? __fadd_rn(dbeta[c], (float)s[3]) : (float)s[3];
  if (dgamma)
    dgamma[c] = accum_dgamma ? __fadd_rn(dgamma[c], (float)s[4]) : (float)s[4];
}

// batch (batch_normalization.cpp:336-349): dx (+)= dy * scale / sqrt(v + eps) + dvar * 2 * (x - m) / n + dmean / n
// global (:413-440):                       dx (+)= dy * (gamma * (v + eps)^-0.5)
template <bool kBatch, bool kAccum>
__global__ void __launch_bounds__(kThreads)
    bn_backward_dx_kernel(const float *__restrict__ x, const float *__restrict__ dy, const float *__restrict__ gamma,
                          const float *__restrict__ mean, const float *__restrict__ var, float eps,
                          const float *__restrict__ coef, float count, size_t total, unsigned C, unsigned S,
                          float *__restrict__ dx) {
  pdl_wait();
  pdl_trigger();
  const size_t stride = (size_t)gridDim.x * kThreads;
  const size_t first = (size_t)blockIdx.x * kThreads + threadIdx.x;
  ChannelWalk walk(first, stride, S, C);
  for (size_t i = first; i < total; i += stride, walk.next()) {
    const unsigned c = walk.c;
    const float scale = gamma ? __ldg(gamma + c) : 1.0f;
    const float ve = __fadd_rn(__ldg(var + c), eps);
    float g;
    if (kBatch) {
      const float a = __fdiv_rn(__fmul_rn(dy[i], scale), __fsqrt_rn(ve));
      const float b = __fdiv_rn(__fmul_rn(__ldg(coef + c * 4), __fsub_rn(x[i], __ldg(mean + c))), count);
      g = __fadd_rn(__fadd_rn(a, b), __ldg(coef + c * 4 + 1));
    } else {
      g = __fmul_rn(dy[i], __ldg(coef + c * 4 + 2));
    }
    dx[i] = kAccum ? __fadd_rn(dx[i], g) : g;
  }
}

// a / d for many a and one d > 0: a times 1 / d held in two floats, hi rounded toward zero and lo > 0 (an infinite a stays
// infinite). Within 2^-23 ulp of the quotient before its one rounding, in two instructions instead of a division's dozen.
struct Quotient {
  float hi, lo;
  __device__ __forceinline__ explicit Quotient(float d) {
    hi = __frcp_rz(d);
    if (__fmaf_rn(-hi, d, 1.0f) == 0.0f)
      hi = __int_as_float(__float_as_int(hi) - 1);
    lo = isinf(hi) ? hi : __fmul_rn(__fmaf_rn(-hi, d, 1.0f), hi);
  }
  __device__ __forceinline__ float operator()(float a) const { return __fmaf_rn(a, hi, __fmul_rn(a, lo)); }
};

// The same for planes of whole float4: a warp takes a run of up to 32 * kRun float4 of one plane, `runs` of them per
// plane, with all its loads in flight before the channel's constants are made. The run length is chosen so that the last
// run of a plane is nearly full (a block per 512 float4 left 784-float4 planes a quarter idle: 66 us for
// [128, 64, 56, 56] against 47 us of traffic).
template <int kRun, bool kBatch, bool kAccum>
__global__ void __launch_bounds__(kThreads)
    bn_backward_dx_plane_kernel(const float *__restrict__ x, const float *__restrict__ dy,
                                const float *__restrict__ gamma, const float *__restrict__ mean,
                                const float *__restrict__ var, float eps, const float *__restrict__ coef, float count,
                                unsigned C, int S4, unsigned runs, size_t total_runs, float *__restrict__ dx) {
  pdl_wait();
  pdl_trigger();
  const size_t run = block_descending() * (kThreads / 32) + (threadIdx.x >> 5);
  if (run >= total_runs)
    return;
  const bool keep = total_runs / runs * S4 * sizeof(float4) <= kKeepBytes;
  const size_t plane = run / runs;
  const int c = (int)(plane % C), i0 = (int)(run - plane * runs) * (32 * kRun) + (int)(threadIdx.x & 31);
  const float4 *xp = reinterpret_cast<const float4 *>(x) + plane * S4;
  const float4 *gp = reinterpret_cast<const float4 *>(dy) + plane * S4;
  float4 *op = reinterpret_cast<float4 *>(dx) + plane * S4;
  float4 g[kRun], xv[kRun], o[kRun];
#pragma unroll
  for (int u = 0; u < kRun; ++u) {
    const int i = i0 + 32 * u;
    if (i < S4) {
      g[u] = __ldcs(gp + i);
      if (kBatch)
        xv[u] = __ldcs(xp + i);
      if (kAccum)
        o[u] = op[i];
    }
  }
  const float scale = gamma ? __ldg(gamma + c) : 1.0f;
  const Quotient by_sd(__fsqrt_rn(__fadd_rn(__ldg(var + c), eps))), by_count(count);
  const float m = __ldg(mean + c), k0 = __ldg(coef + c * 4), k1 = __ldg(coef + c * 4 + 1), k2 = __ldg(coef + c * 4 + 2);
  auto one = [&](float xe, float ge, float old) {
    float r;
    if (kBatch) {
      const float a = by_sd(__fmul_rn(ge, scale));
      const float b = by_count(__fmul_rn(k0, __fsub_rn(xe, m)));
      r = __fadd_rn(__fadd_rn(a, b), k1);
    } else {
      r = __fmul_rn(ge, k2);
    }
    return kAccum ? __fadd_rn(old, r) : r;
  };
#pragma unroll
  for (int u = 0; u < kRun; ++u) {
    const int i = i0 + 32 * u;
    if (i < S4) {
      const float4 a = kBatch ? xv[u] : make_float4(0, 0, 0, 0), b = kAccum ? o[u] : make_float4(0, 0, 0, 0);
      st_result(op + i, make_float4(one(a.x, g[u].x, b.x), one(a.y, g[u].y, b.y), one(a.z, g[u].z, b.z),
                                    one(a.w, g[u].w, b.w)), keep);
    }
  }
}

template <int kRun>
int bn_backward_dx_planes(const float *x, const float *dy, const float *gamma, const float *mean, const float *var,
                          float eps, const float *coef, float count, size_t planes, unsigned C, int S4, float *dx,
                          bool batch, bool accum, cudaStream_t st) {
  const unsigned runs = (unsigned)((S4 + 32 * kRun - 1) / (32 * kRun));
  const size_t total = planes * runs, blocks = (total + kThreads / 32 - 1) / (kThreads / 32);
  NB_CHECK(blocks < (1ull << 31), NB200_ENOTIMPL, "tensor too large");
  auto kernel = batch ? (accum ? bn_backward_dx_plane_kernel<kRun, true, true> : bn_backward_dx_plane_kernel<kRun, true, false>)
                      : (accum ? bn_backward_dx_plane_kernel<kRun, false, true> : bn_backward_dx_plane_kernel<kRun, false, false>);
  NB_CUDA(launch_dependent(kernel, dim3((unsigned)blocks), dim3(kThreads), 0, st, x, dy, gamma, mean, var, eps, coef,
                           count,
                           C, S4, runs, total, dx));
  return NB200_OK;
}

// Blocks per channel of a pass that sums over channels. All blocks have the same share, so it takes as long as its rounds
// of resident blocks: the counts that fill one to four rounds exactly are compared by how full their rounds are, more
// rounds only where they are 5 % fuller (8 blocks per SM whatever the kernel's registers allow made 3 rounds of 592 blocks
// of the gradients' 1216: [128, 64, 56, 56] 44 us, now 38).
template <typename Kernel>
int channel_blocks(Kernel kernel, std::atomic<int> (&resident)[64], int64_t outer, int64_t channels, int64_t inner, bool vec,
                   int *out) {
  int dev = 0;
  NB_CUDA(cudaGetDevice(&dev));
  int per_sm = resident[dev & 63]; // the same value whichever thread stores it
  if (per_sm == 0) {
    NB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, 0));
    resident[dev & 63] = per_sm;
  }
  const int64_t slots = (int64_t)per_sm * sm_count();
  int64_t best = 1;
  double best_full = 0.0;
  for (int64_t rounds = 1; rounds <= 4; ++rounds) {
    const int64_t p = rounds * slots / channels;
    const double full = (double)(p * channels) / (double)(rounds * slots);
    if (p >= 1 && full > best_full + 0.05)
      best = p, best_full = full;
  }
  const int64_t items = outer * (vec ? inner / 4 : inner), most = (items + kThreads - 1) / kThreads;
  // short channels, a thread's share at most one set of four loads: as many blocks as 8 per SM give (fewer loads in a row)
  if (items <= best * kThreads * 4)
    best = (8ll * sm_count() + channels - 1) / channels;
  best = best > most ? most : best;
  *out = (int)(best < 1 ? 1 : best);
  return NB200_OK;
}

} // namespace
} // namespace nb200

using namespace nb200;

extern "C" {

int nb200_batch_normalization_inference_f32(const float *x, const float *beta, const float *gamma, const float *mean,
                                            const float *var, float *y, int64_t outer, int64_t channels,
                                            int64_t inner, float eps, void *stream);

int nb200_batch_normalization_batch_f32(const float *x, const float *beta, const float *gamma, float *running_mean,
                                        float *running_var, float *y, float *batch_mean, float *batch_var,
                                        int64_t outer, int64_t channels, int64_t inner, float eps, float decay_rate,
                                        int update_running, void *stream) {
  NB_CHECK(outer > 0 && channels > 0 && inner > 0, NB200_EVALUE, "bad extents");
  NB_CHECK(channels <= 65535 && inner < (1ll << 31) && outer < (1ll << 31), NB200_EVALUE, "extent too large");
  NB_CHECK(x && y && batch_mean && batch_var, NB200_EVALUE, "null data pointer");
  NB_CHECK(!update_running || (running_mean && running_var), NB200_EVALUE, "running statistics are needed");
  cudaStream_t st = as_stream(stream);
  const bool vec = (inner % 4 == 0) && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  auto stats = vec ? bn_stats_kernel<true> : bn_stats_kernel<false>;
  static std::atomic<int> resident[2][64]{};
  int P = 0;
  NB_TRY(channel_blocks(stats, resident[vec], outer, channels, inner, vec, &P));
  AsyncScratch scratch(st);
  NB_TRY(scratch.alloc((size_t)channels * P * 2 * sizeof(float)));
  float *partial = static_cast<float *>(scratch.p);
  const dim3 grid((unsigned)P, (unsigned)channels), finish_grid((unsigned)((channels * kLanes + kFinishThreads - 1) / kFinishThreads));
  NB_CUDA(launch_dependent(stats, grid, dim3(kThreads), 0, st, x,
                           (unsigned)outer, (unsigned)channels, (unsigned)inner, partial));
  NB_CUDA(launch_dependent(bn_stats_finish_kernel, finish_grid, dim3(kFinishThreads), 0, st, partial,
                           (unsigned)P, (unsigned)channels, (float)(outer * inner), decay_rate, update_running,
                           batch_mean, batch_var, running_mean, running_var));
  return nb200_batch_normalization_inference_f32(x, beta, gamma, batch_mean, batch_var, y, outer, channels, inner,
                                                 eps, stream);
}

int nb200_batch_normalization_backward_f32(const float *x, const float *dy, const float *gamma, const float *mean,
                                           const float *var, const float *dmean, const float *dvar, float *dx,
                                           float *dbeta, float *dgamma, int64_t outer, int64_t channels,
                                           int64_t inner, float eps, int batch_stat, int accum_dx, int accum_dbeta,
                                           int accum_dgamma, void *stream) {
  NB_CHECK(outer > 0 && channels > 0 && inner > 0, NB200_EVALUE, "bad extents");
  NB_CHECK(channels <= 65535 && inner < (1ll << 31) && outer < (1ll << 31), NB200_EVALUE, "extent too large");
  NB_CHECK(x && dy && mean && var, NB200_EVALUE, "null data pointer");
  if (!dx && !dbeta && !dgamma)
    return NB200_OK;
  cudaStream_t st = as_stream(stream);
  const bool vec = (inner % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy)) & 15) == 0;
  auto sums_kernel = vec ? (batch_stat ? bn_backward_sums_kernel<true, true> : bn_backward_sums_kernel<true, false>)
                         : (batch_stat ? bn_backward_sums_kernel<false, true> : bn_backward_sums_kernel<false, false>);
  static std::atomic<int> resident[4][64]{};
  int P = 0;
  NB_TRY(channel_blocks(sums_kernel, resident[2 * vec + (batch_stat != 0)], outer, channels, inner, vec, &P));
  AsyncScratch scratch(st);
  NB_TRY(scratch.alloc((size_t)channels * (P * 3 + 4) * sizeof(float)));
  float *partial = static_cast<float *>(scratch.p);
  float *coef = partial + (size_t)channels * P * 3;
  const bool sums = (batch_stat && dx) || dbeta || dgamma;
  const dim3 finish_grid((unsigned)((channels * kLanes + kFinishThreads - 1) / kFinishThreads));
  if (sums) {
    const dim3 grid((unsigned)P, (unsigned)channels);
    NB_CUDA(launch_dependent(sums_kernel, grid, dim3(kThreads), 0, st, x, dy, mean, (unsigned)outer, (unsigned)channels,
                             (unsigned)inner, partial));
  }
  NB_CUDA(launch_dependent(bn_backward_finish_kernel, finish_grid, dim3(kFinishThreads), 0, st,
                           sums ? partial : nullptr, (unsigned)P, (unsigned)channels, (float)(outer * inner), gamma, var,
                           eps, dmean, dvar, batch_stat, coef, sums ? dbeta : nullptr, accum_dbeta,
                           sums ? dgamma : nullptr, accum_dgamma));
  if (dx) {
    const size_t total = (size_t)outer * channels * inner;
    const unsigned grid = grid_for(total, 4);
    // runs of float4 from planes of 32 values on (below that a warp would be mostly idle)
    if (vec && inner >= 32 && (reinterpret_cast<uintptr_t>(dx) & 15) == 0) {
      const int S4 = (int)(inner / 4);
      const size_t planes = (size_t)outer * channels;
      auto idle = [&](int run) { return (double)((S4 + 32 * run - 1) / (32 * run) * (32 * run)) / S4; };
      int best = 2;
      for (int run : {4, 5, 7})
        if (idle(run) <= idle(best) + 1e-9)
          best = run;
      auto launch = best == 2 ? bn_backward_dx_planes<2>
                              : (best == 4 ? bn_backward_dx_planes<4> : (best == 5 ? bn_backward_dx_planes<5> : bn_backward_dx_planes<7>));
      return launch(x, dy, gamma, mean, var, eps, coef, (float)(outer * inner), planes, (unsigned)channels, S4, dx,
                    batch_stat != 0, accum_dx != 0, st);
    }
    auto kernel = batch_stat ? (accum_dx ? bn_backward_dx_kernel<true, true> : bn_backward_dx_kernel<true, false>)
                             : (accum_dx ? bn_backward_dx_kernel<false, true> : bn_backward_dx_kernel<false, false>);
    NB_CUDA(launch_dependent(kernel, dim3(grid), dim3(kThreads), 0, st, x, dy, gamma, mean, var, eps, coef,
                             (float)(outer * inner), total, (unsigned)channels, (unsigned)inner, dx));
  }
  return NB200_OK;
}

int nb200_relu_backward_f32(const float *y, const float *dy, float *dx, size_t size, int accum, void *stream) {
  if (size == 0)
    return NB200_OK;
  NB_CHECK(y && dy && dx, NB200_EVALUE, "null data pointer");
  return accum ? launch_grad_pass<0, true>(y, dy, dx, size, as_stream(stream))
               : launch_grad_pass<0, false>(y, dy, dx, size, as_stream(stream));
}

int nb200_add2_backward_f32(const float *dy, float *dx, size_t size, int accum, void *stream) {
  if (size == 0)
    return NB200_OK;
  NB_CHECK(dy && dx, NB200_EVALUE, "null data pointer");
  return accum ? launch_grad_pass<1, true>(nullptr, dy, dx, size, as_stream(stream))
               : launch_grad_pass<1, false>(nullptr, dy, dx, size, as_stream(stream));
}

int nb200_global_average_pooling_backward_f32(const float *dy, float *dx, int64_t maps, int64_t spatial, int accum,
                                              void *stream) {
  NB_CHECK(maps >= 0 && spatial > 0 && spatial < (1ll << 31), NB200_EVALUE, "bad extents");
  const size_t total = (size_t)maps * spatial;
  if (total == 0)
    return NB200_OK;
  NB_CHECK(dy && dx, NB200_EVALUE, "null data pointer");
  NB_CUDA(launch_dependent(accum ? gap_backward_kernel<true> : gap_backward_kernel<false>, dim3(grid_for(total, 4)),
                           dim3(kThreads), 0, as_stream(stream), dy, dx, total, (unsigned)spatial));
  return NB200_OK;
}

int nb200_max_pooling_backward_f32(const float *x, const float *dy, float *dx, int64_t maps, int height, int width,
                                   int kernel_h, int kernel_w, int stride_h, int stride_w, int pad_h, int pad_w,
                                   int ignore_border, int accum, void *stream) {
  NB_CHECK(maps >= 0 && height > 0 && width > 0 && kernel_h > 0 && kernel_w > 0 && stride_h > 0 && stride_w > 0 &&
               pad_h >= 0 && pad_w >= 0,
           NB200_EVALUE, "bad pooling geometry");
  // Output extent: src/nbla/function/utils/base_pooling.cpp:59.
  const int Ho = (height + pad_h - (ignore_border ? kernel_h - pad_h : 1)) / stride_h + 1;
  const int Wo = (width + pad_w - (ignore_border ? kernel_w - pad_w : 1)) / stride_w + 1;
  NB_CHECK(Ho > 0 && Wo > 0, NB200_EVALUE, "pooling output would be empty");
  const size_t total = (size_t)maps * height * width;
  if (total == 0)
    return NB200_OK;
  NB_CHECK(x && dy && dx, NB200_EVALUE, "null data pointer");
  NB_CHECK((int64_t)height * width < (1ll << 31), NB200_EVALUE, "map larger than 2^31 pixels");
  cudaStream_t st = as_stream(stream);
  const size_t outputs = (size_t)maps * Ho * Wo;
  AsyncScratch scratch(st);
  NB_TRY(scratch.alloc(outputs * sizeof(int)));
  int *index = static_cast<int *>(scratch.p);
  NB_CUDA(launch_dependent(max_pooling_index_kernel, dim3(grid_for(outputs, 1)), dim3(kThreads), 0, st, x, index,
                           outputs,
                           height, width, Ho, Wo, kernel_h, kernel_w, stride_h, stride_w, pad_h, pad_w));
  NB_CUDA(launch_dependent(accum ? max_pooling_backward_kernel<true> : max_pooling_backward_kernel<false>,
                           dim3(grid_for(total, 1)), dim3(kThreads), 0, st, index, dy, dx, total, height, width, Ho, Wo,
                           kernel_h, kernel_w, stride_h, stride_w, pad_h, pad_w));
  return NB200_OK;
}

} // extern "C"
