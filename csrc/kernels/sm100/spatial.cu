// Convolution helpers, pooling and batch normalisation for sm_100a (NCHW, bf16 or fp32 io, fp32 arithmetic).
//
// Counterparts in the reference: im2col / col2im (crates/incin-backends/src/cuda/ops/kernels/conv.cu:5-181, fold
// with atomicAdd), pooling (pool.cu:7-248, backward with atomics) and the inference-only per-element batch norm
// (crates/incin-backends/src/kernel.rs:1345-1389).  Differences here:
//   * im2col writes the [N*OH*OW, C*KH*KW] matrix the tcgen05 GEMM consumes directly (K-major rows), and col2im
//     GATHERS the contributions of each input pixel, so the data gradient needs no atomics and is deterministic;
//   * max pooling keeps the argmax (int32 offset inside the plane) so its backward is a gather as well;
//   * batch norm has a training forward (per-channel mean / biased variance in one pass over the channel with
//     one CTA or a small cluster per channel, running statistics updated in the same kernel) and a full backward.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cooperative_groups.h>
#include <stdint.h>
#include <type_traits>

#include "incin_b200.h"

namespace {

template <typename T> __device__ __forceinline__ float ldf(const T* p, long long i);
template <> __device__ __forceinline__ float ldf<float>(const float* p, long long i) { return p[i]; }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p, long long i) { return __bfloat162float(p[i]); }
template <typename T> __device__ __forceinline__ void stf(T* p, long long i, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, long long i, float v) { p[i] = v; }
template <> __device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, long long i, float v) { p[i] = __float2bfloat16(v); }

struct ConvGeom {
  int N, C, H, W, KH, KW, OH, OW, sh, sw, ph, pw, dh, dw;
};

// A divisor known before the launch.  I, here and below, is the type of a flat index: 32 bits wherever the tensor has fewer
// than 2^31 elements, and then a quotient is one multiplication, because dividing (64-bit indices above all) was most of the
// time of these kernels.  With 2^(s - 1) < d <= 2^s and mul = ceil(2^(31 + s) / d), which is below 2^32, mul * d exceeds
// 2^(31 + s) by less than 2^s, so n * mul / 2^(31 + s) exceeds n / d by less than 1 / d for n < 2^31: the floors agree.
template <typename I>
struct Divisor {
  I d;
  explicit Divisor(long long v) : d((I)v) {}
  __device__ __forceinline__ I of(I n) const { return n / d; }
};
template <>
struct Divisor<unsigned> {
  unsigned d, mul;
  int shift = 31;
  explicit Divisor(long long v) : d((unsigned)v) {
    while (shift < 62 && (1ull << (shift - 31)) < d) ++shift;
    mul = (unsigned)(((1ull << shift) + d - 1) / d);
  }
  __device__ __forceinline__ unsigned of(unsigned n) const { return (unsigned)(((unsigned long long)n * mul) >> shift); }
};
using Div = Divisor<unsigned>;   // of values below 2^31

// cols[(n*OH+oh)*OW+ow][(c*KH+kh)*KW+kw] = x[n][c][oh*sh-ph+kh*dh][ow*sw-pw+kw*dw] (0 outside)
template <typename T, typename I>
__global__ void im2col_kernel(const T* __restrict__ x, T* __restrict__ cols, ConvGeom g, I total, Divisor<I> K, Divisor<I> OW, Divisor<I> OH,
                              Div KW, Div KH) {
  for (I t = (I)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (I)gridDim.x * blockDim.x) {
    const I row = K.of(t), line = OW.of(row), image = OH.of(line);
    const unsigned k = (unsigned)(t - row * K.d), q = KW.of(k);
    const int ow = (int)(row - line * OW.d), oh = (int)(line - image * OH.d);
    const int c = (int)KH.of(q), kw = (int)(k - q * KW.d), kh = (int)q - c * g.KH;
    const int ih = oh * g.sh - g.ph + kh * g.dh, iw = ow * g.sw - g.pw + kw * g.dw;
    T v = T(0.0f);
    if (ih >= 0 && ih < g.H && iw >= 0 && iw < g.W) v = x[(((long long)image * g.C + c) * g.H + ih) * g.W + iw];
    cols[t] = v;
  }
}

// Tiled form.  A block writes one output row (n, oh) for CT channels: the KH input rows of those channels, padding
// included, are brought into shared memory with coalesced reads, and every thread assembles 16 bytes of the column
// matrix from them.  tab[k] is where element k of the block's channels lies for ow = 0, so the inner loop has no index
// arithmetic.  A warp takes 2 units of a row by 16 output columns: whole sectors on the way out, few bank conflicts on
// the way in.  Bound by the column matrix it writes (K / C times the input).  N 64, C 64, 3 x 3, bf16,
// 32 x 32 and 16 x 16 together (75 and 19 MB): 390 -> 70 us.
template <typename T>
__global__ void __launch_bounds__(256) im2col_tile_kernel(const T* __restrict__ x, T* __restrict__ cols, ConvGeom g, int CT, int SW) {
  extern __shared__ __align__(16) unsigned char im2col_smem[];
  constexpr int V = 16 / sizeof(T);
  const int KK = g.KH * g.KW, kt = CT * KK;
  int* tab = reinterpret_cast<int*>(im2col_smem);                     // [kt]
  T* tile = reinterpret_cast<T*>(tab + ((kt + 3) & ~3));              // [CT][KH][SW]
  const int n = blockIdx.x / g.OH, oh = blockIdx.x % g.OH;
  const int c0 = blockIdx.y * CT, nc = min(CT, g.C - c0), nk = nc * KK;
  for (int k = threadIdx.x; k < nk; k += 256) {
    const int c = k / KK, r = k % KK;
    tab[k] = (c * g.KH + r / g.KW) * SW + (r % g.KW) * g.dw;
  }
  const int lines = nc * g.KH, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int l0 = warp; l0 < lines; l0 += 32) {                         // four lines a warp in flight
    for (int i = lane; i < SW; i += 32) {
      const int iw = i - g.pw;
      const bool col_ok = iw >= 0 && iw < g.W;
      T v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int l = l0 + q * 8, c = l / g.KH, ih = oh * g.sh - g.ph + (l - c * g.KH) * g.dh;
        v[q] = T(0.0f);
        if (l < lines && col_ok && ih >= 0 && ih < g.H) v[q] = x[(((long long)n * g.C + c0 + c) * g.H + ih) * g.W + iw];
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (l0 + q * 8 < lines) tile[(l0 + q * 8) * SW + i] = v[q];
    }
  }
  __syncthreads();
  const int units = nk / V;                                           // the host has checked that K and CT * KK are multiples of V
  const long long K = (long long)g.C * KK;
  T* dst = cols + ((long long)n * g.OH + oh) * g.OW * K + (long long)c0 * KK;
  for (int u = warp * 2 + (lane & 1); u < units; u += 16) {           // 2 units of a row by 16 output columns a warp
    int off[V];
#pragma unroll
    for (int i = 0; i < V; ++i) off[i] = tab[u * V + i];
    for (int ow = lane >> 1; ow < g.OW; ow += 16) {
      alignas(16) T e[V];
      const int base = ow * g.sw;
#pragma unroll
      for (int i = 0; i < V; ++i) e[i] = tile[off[i] + base];
      *reinterpret_cast<uint4*>(dst + (long long)ow * K + u * V) = *reinterpret_cast<const uint4*>(e);
    }
  }
}

// dx[n][c][ih][iw] = sum over the (kh, kw, oh, ow) that read this pixel: a gather, no atomics
template <typename T, typename I>
__global__ void col2im_kernel(const T* __restrict__ cols, T* __restrict__ dx, ConvGeom g, I total, Divisor<I> W, Divisor<I> H, Divisor<I> C,
                              Div SH, Div SW) {
  const int K = g.C * g.KH * g.KW;
  for (I t = (I)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (I)gridDim.x * blockDim.x) {
    const I line = W.of(t), plane = H.of(line), image = C.of(plane);
    const int iw = (int)(t - line * W.d), ih = (int)(line - plane * H.d), c = (int)(plane - image * C.d);
    const T* from = cols + (long long)image * g.OH * g.OW * K;
    float acc = 0.0f;
    for (int kh = 0; kh < g.KH; ++kh) {
      const int hh = ih + g.ph - kh * g.dh;
      if (hh < 0) continue;
      const int oh = (int)SH.of((unsigned)hh);
      if (oh * g.sh != hh || oh >= g.OH) continue;
      for (int kw = 0; kw < g.KW; ++kw) {
        const int ww = iw + g.pw - kw * g.dw;
        if (ww < 0) continue;
        const int ow = (int)SW.of((unsigned)ww);
        if (ow * g.sw != ww || ow >= g.OW) continue;
        acc += ldf(from, ((long long)oh * g.OW + ow) * K + (c * g.KH + kh) * g.KW + kw);
      }
    }
    stf(dx, (long long)t, acc);
  }
}

// Tiled form.  A block owns RB input rows of CT channels of one image: the part of the column matrix that reaches them
// (every output row that reads them, OW columns, CT * KH * KW elements) is staged in shared memory, 16 bytes a load, and
// each thread gathers its pixels from there, in the same order of kh and kw as the general kernel.  The pitch is one
// word more than the data, so that neighbouring pixels lie in different banks.  Strides of 1 only: with larger ones few of
// the staged elements belong to a pixel's row (the dispatch has figures).  Bound by the column matrix it reads;
// the same two layers: 191 -> 88 us.
template <typename T>
__global__ void __launch_bounds__(256) col2im_tile_kernel(const T* __restrict__ cols, T* __restrict__ dx, ConvGeom g, int CT, int RB) {
  extern __shared__ __align__(16) unsigned char col2im_smem[];
  constexpr int V = 16 / sizeof(T), WV = 4 / sizeof(T);               // elements per 16-byte load, per 4-byte word
  T* tile = reinterpret_cast<T*>(col2im_smem);                        // [rows][OW][pitch]
  const int KK = g.KH * g.KW, pitch = CT * KK + WV;
  const int bands = (g.H + RB - 1) / RB;
  const int n = blockIdx.x / bands, i0 = (blockIdx.x % bands) * RB, i1 = min(i0 + RB, g.H);
  const int c0 = blockIdx.y * CT, nc = min(CT, g.C - c0), units = nc * KK / V;
  const int oh0 = max(0, i0 + g.ph - (g.KH - 1) * g.dh), oh1 = min(g.OH - 1, i1 - 1 + g.ph);   // output rows that reach the band
  const long long K = (long long)g.C * KK;
  const T* src = cols + ((long long)n * g.OH + oh0) * g.OW * K + (long long)c0 * KK;
  const unsigned total = (unsigned)(max(0, oh1 - oh0 + 1) * g.OW * units);
  for (unsigned t0 = threadIdx.x; t0 < total; t0 += 1024) {            // four loads a thread in flight
    uint4 v[4];
    unsigned row[4], u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned t = t0 + q * 256;
      row[q] = t / (unsigned)units;
      u[q] = t - row[q] * (unsigned)units;
      if (t < total) v[q] = *reinterpret_cast<const uint4*>(src + row[q] * K + u[q] * V);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (t0 + q * 256 >= total) break;
      uint32_t* d = reinterpret_cast<uint32_t*>(tile + (long long)row[q] * pitch + u[q] * V);
      d[0] = v[q].x; d[1] = v[q].y; d[2] = v[q].z; d[3] = v[q].w;
    }
  }
  __syncthreads();
  const int lines = nc * (i1 - i0), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // lanes beyond a narrow image take the next line
  const int lw = g.W >= 32 ? 32 : (g.W > 16 ? 32 : (g.W > 8 ? 16 : 8)), per = 32 / lw;
  for (int l = warp * per + lane / lw; l < lines; l += 8 * per) {
    const int c = l / (i1 - i0), ih = i0 + l % (i1 - i0);
    T* out = dx + (((long long)n * g.C + c0 + c) * g.H + ih) * g.W;
    for (int iw = lane % lw; iw < g.W; iw += lw) {
      float acc = 0.0f;
      for (int kh = 0; kh < g.KH; ++kh) {
        const int oh = ih + g.ph - kh * g.dh;
        if (oh < 0 || oh >= g.OH) continue;
        const T* line = tile + (oh - oh0) * g.OW * pitch + (c * g.KH + kh) * g.KW;
        for (int kw = 0; kw < g.KW; ++kw) {
          const int ow = iw + g.pw - kw * g.dw;
          if (ow < 0 || ow >= g.OW) continue;
          acc += ldf(line, ow * pitch + kw);
        }
      }
      stf(out, iw, acc);
    }
  }
}

// ---- pooling ---------------------------------------------------------------------------------------------------
// One thread an element, whatever the shape of a plane
template <typename I>
struct Place {
  int x, y;
  long long plane;
  __device__ __forceinline__ Place(I t, const Divisor<I>& width, const Divisor<I>& height) {
    const I row = width.of(t), p = height.of(row);
    x = (int)(t - row * width.d);
    y = (int)(row - p * height.d);
    plane = (long long)p;
  }
};

template <typename T, typename I>
__global__ void maxpool_fwd_kernel(const T* __restrict__ x, T* __restrict__ y, int* __restrict__ arg, ConvGeom g, I total, Divisor<I> OW, Divisor<I> OH) {
  for (I t = (I)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (I)gridDim.x * blockDim.x) {
    const Place<I> o(t, OW, OH);
    const T* p = x + o.plane * g.H * g.W;
    float best = -INFINITY;
    int best_i = -1;
    for (int kh = 0; kh < g.KH; ++kh) {
      const int ih = o.y * g.sh - g.ph + kh;
      if (ih < 0 || ih >= g.H) continue;
      for (int kw = 0; kw < g.KW; ++kw) {
        const int iw = o.x * g.sw - g.pw + kw;
        if (iw < 0 || iw >= g.W) continue;
        const float v = ldf(p, (long long)ih * g.W + iw);
        if (v > best || v != v || best_i < 0) {
          best = v;
          best_i = ih * g.W + iw;
        }
      }
    }
    stf(y, (long long)t, best);
    if (arg) arg[t] = best_i;
  }
}

// dx[plane][i] = sum of dy over the windows whose argmax is i: gather over the windows that cover pixel i (N 64, C 64,
// 32 x 32 bf16, 2 x 2 windows: 38 us with divisions of 64-bit indices -> 20; a row at a time per group of threads took 25
// there and 24 ms on one row of 10^6)
template <typename T, typename I>
__global__ void maxpool_bwd_kernel(const T* __restrict__ dy, const int* __restrict__ arg, T* __restrict__ dx, ConvGeom g, I total,
                                   Divisor<I> W, Divisor<I> H, Div SH, Div SW) {
  for (I t = (I)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (I)gridDim.x * blockDim.x) {
    const Place<I> i(t, W, H);
    const int me = i.y * g.W + i.x;
    const int oh_lo = (int)SH.of((unsigned)max(0, i.y + g.ph - g.KH + g.sh)), oh_hi = min(g.OH - 1, (int)SH.of((unsigned)(i.y + g.ph)));
    const int ow_lo = (int)SW.of((unsigned)max(0, i.x + g.pw - g.KW + g.sw)), ow_hi = min(g.OW - 1, (int)SW.of((unsigned)(i.x + g.pw)));
    const T* dyp = dy + i.plane * g.OH * g.OW;
    const int* ap = arg + i.plane * g.OH * g.OW;
    float acc = 0.0f;
    for (int oh = oh_lo; oh <= oh_hi; ++oh)
      for (int ow = ow_lo; ow <= ow_hi; ++ow) {
        const long long o = (long long)oh * g.OW + ow;
        if (ap[o] == me) acc += ldf(dyp, o);
      }
    stf(dx, (long long)t, acc);
  }
}

// average pooling (padding counted in the divisor, like the CPU oracle); backward when `bwd`
template <typename T>
__global__ void avgpool_kernel(const T* __restrict__ in, T* __restrict__ out, ConvGeom g, long long total, int bwd) {
  const float inv = 1.0f / (float)(g.KH * g.KW);
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    float acc = 0.0f;
    if (!bwd) {
      const int ow = (int)(t % g.OW), oh = (int)((t / g.OW) % g.OH);
      const long long plane = t / ((long long)g.OW * g.OH);
      for (int kh = 0; kh < g.KH; ++kh) {
        const int ih = oh * g.sh - g.ph + kh;
        if (ih < 0 || ih >= g.H) continue;
        for (int kw = 0; kw < g.KW; ++kw) {
          const int iw = ow * g.sw - g.pw + kw;
          if (iw >= 0 && iw < g.W) acc += ldf(in, (plane * g.H + ih) * g.W + iw);
        }
      }
    } else {
      const int iw = (int)(t % g.W), ih = (int)((t / g.W) % g.H);
      const long long plane = t / ((long long)g.W * g.H);
      const int oh_lo = max(0, (ih + g.ph - g.KH + g.sh) / g.sh), oh_hi = min(g.OH - 1, (ih + g.ph) / g.sh);
      const int ow_lo = max(0, (iw + g.pw - g.KW + g.sw) / g.sw), ow_hi = min(g.OW - 1, (iw + g.pw) / g.sw);
      for (int oh = oh_lo; oh <= oh_hi; ++oh)
        for (int ow = ow_lo; ow <= ow_hi; ++ow) acc += ldf(in, (plane * g.OH + oh) * g.OW + ow);
    }
    stf(out, t, acc * inv);
  }
}

// ---- batch norm (a block, or a cluster of up to eight, per channel) -------------------------------------------------------------------------
__device__ __forceinline__ float2 block_sum2(float a, float b) {
  __shared__ float sa[32], sb[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    sa[threadIdx.x >> 5] = a;
    sb[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  float ra = 0.0f, rb = 0.0f;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    ra += sa[w];
    rb += sb[w];
  }
  return make_float2(ra, rb);
}

// Training forward and backward: one CTA per channel, or (CL) a thread-block cluster of 2 to 8, whose partial sums meet in
// distributed shared memory (fixed order, so results repeat to the bit).  The two passes over the channel are the work;
// one CTA per channel left most SMs idle at 64 to 128 channels and split a 64-bit index per element.  With VEC 16 bytes
// are read and written at a time (HW a multiple of that, aligned bases).  N 64, C 64, 32 x 32 and
// N 64, C 128, 16 x 16 in bf16, average: forward 53 -> 9.5 us, backward 60 -> 10 us.  Channels of one CTA do without the
// cluster and its barriers, and short ones (fewer than 512 16-byte pieces, a piece a thread) take an element a thread:
// (one cluster kernel for all | this) N 32, C 4096, HW 4 forward 30 -> 17 us, backward 46 -> 27; N 2, C 1000, HW 64 10.1 -> 6.1 and
// 14.8 -> 10.9.
__device__ __forceinline__ float2 cluster_sum2(float2 mine) {
  __shared__ float2 part;
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  if (threadIdx.x == 0) part = mine;
  cl.sync();
  float2 r = make_float2(0.0f, 0.0f);
  for (unsigned k = 0; k < cl.num_blocks(); ++k) {
    const float2 o = *cl.map_shared_rank(&part, k);
    r.x += o.x;
    r.y += o.y;
  }
  cl.sync();   // nobody leaves (or reuses part) while others still read it
  return r;
}

// calls f(offset of V consecutive elements of channel c) for this CTA's share of them
template <int V, typename I, typename F>
__device__ __forceinline__ void channel_loop(int N, int C, long long HW, int c, int slice, int slices, F f) {
  const I hwv = (I)(HW / V), count = (I)N * hwv;
#pragma unroll V == 1 ? 4 : 1
  for (I i = (I)slice * blockDim.x + threadIdx.x; i < count; i += (I)slices * blockDim.x) {
    const I n = i / hwv, j = i - n * hwv;
    f(((long long)n * C + c) * HW + (long long)j * V);
  }
}
template <int V, typename T> __device__ __forceinline__ void load_v(const T* p, float (&v)[V]) {
  alignas(16) T e[V];
  if constexpr (V > 1) *reinterpret_cast<uint4*>(e) = *reinterpret_cast<const uint4*>(p);
  else e[0] = p[0];
#pragma unroll
  for (int k = 0; k < V; ++k) v[k] = ldf(e, k);
}
template <int V, typename T> __device__ __forceinline__ void store_v(T* p, const float (&v)[V]) {
  alignas(16) T e[V];
#pragma unroll
  for (int k = 0; k < V; ++k) stf(e, k, v[k]);
  if constexpr (V > 1) *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(e);
  else p[0] = e[0];
}

template <bool CL, typename T, int V, typename I>
__global__ void __launch_bounds__(512) batchnorm_train_fwd_kernel(const T* __restrict__ x, const float* __restrict__ gamma,
                                                                  const float* __restrict__ beta, T* __restrict__ y,
                                                                  float* __restrict__ save_mean, float* __restrict__ save_rstd,
                                                                  float* __restrict__ run_mean, float* __restrict__ run_var, int N, int C,
                                                                  long long HW, float eps, float momentum) {
  const int slices = CL ? (int)cooperative_groups::this_cluster().num_blocks() : 1;
  const int c = blockIdx.x / slices, slice = blockIdx.x % slices;
  const long long count = (long long)N * HW;
  // shifted sums (shift = first element of the channel) keep the one-pass variance accurate for large means
  const float shift = ldf(x, (long long)c * HW);
  float s = 0.0f, ss = 0.0f;
  channel_loop<V, I>(N, C, HW, c, slice, slices, [&](long long o) {
    float v[V];
    load_v<V>(x + o, v);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const float d = v[k] - shift;
      s += d;
      ss += d * d;
    }
  });
  float2 r = block_sum2(s, ss);
  if constexpr (CL) r = cluster_sum2(r);
  const float m_sh = r.x / (float)count;
  const float var = fmaxf(r.y / (float)count - m_sh * m_sh, 0.0f);
  const float mean = m_sh + shift, rstd = rsqrtf(var + eps);
  if (threadIdx.x == 0 && slice == 0) {
    save_mean[c] = mean;
    save_rstd[c] = rstd;
    if (run_mean) run_mean[c] = (1.0f - momentum) * run_mean[c] + momentum * mean;
    if (run_var) run_var[c] = (1.0f - momentum) * run_var[c] + momentum * var * ((float)count / (float)(count > 1 ? count - 1 : 1));
  }
  const float ga = gamma ? gamma[c] : 1.0f, be = beta ? beta[c] : 0.0f;
  channel_loop<V, I>(N, C, HW, c, slice, slices, [&](long long o) {
    float v[V];
    load_v<V>(x + o, v);
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = (v[k] - mean) * rstd * ga + be;
    store_v<V>(y + o, v);
  });
}

template <typename T>
__global__ void batchnorm_eval_kernel(const T* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                                      const float* __restrict__ mean, const float* __restrict__ var, T* __restrict__ y, int C,
                                      long long HW, float eps, long long total) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const int c = (int)((t / HW) % C);
    const float ga = gamma ? gamma[c] : 1.0f, be = beta ? beta[c] : 0.0f;
    stf(y, t, (ldf(x, t) - mean[c]) * rsqrtf(var[c] + eps) * ga + be);
  }
}

// dx = gamma*rstd/M * (M*dy - sum(dy) - xhat*sum(dy*xhat)); dgamma += sum(dy*xhat); dbeta += sum(dy)
template <bool CL, typename T, int V, typename I>
__global__ void __launch_bounds__(512) batchnorm_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                            const float* __restrict__ gamma, const float* __restrict__ save_mean,
                                                            const float* __restrict__ save_rstd, T* __restrict__ dx,
                                                            float* __restrict__ dgamma, float* __restrict__ dbeta, int N, int C,
                                                            long long HW) {
  const int slices = CL ? (int)cooperative_groups::this_cluster().num_blocks() : 1;
  const int c = blockIdx.x / slices, slice = blockIdx.x % slices;
  const long long count = (long long)N * HW;
  const float mean = save_mean[c], rstd = save_rstd[c];
  float s1 = 0.0f, s2 = 0.0f;
  channel_loop<V, I>(N, C, HW, c, slice, slices, [&](long long o) {
    float g[V], v[V];
    load_v<V>(dy + o, g);
    load_v<V>(x + o, v);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      s1 += g[k];
      s2 += g[k] * (v[k] - mean) * rstd;
    }
  });
  float2 r = block_sum2(s1, s2);
  if constexpr (CL) r = cluster_sum2(r);
  if (threadIdx.x == 0 && slice == 0) {
    if (dgamma) dgamma[c] += r.y;
    if (dbeta) dbeta[c] += r.x;
  }
  const float ga = gamma ? gamma[c] : 1.0f;
  const float k0 = ga * rstd / (float)count;
  channel_loop<V, I>(N, C, HW, c, slice, slices, [&](long long o) {
    float g[V], v[V];
    load_v<V>(dy + o, g);
    load_v<V>(x + o, v);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const float xh = (v[k] - mean) * rstd;
      g[k] = k0 * ((float)count * g[k] - r.x - xh * r.y);
    }
    store_v<V>(dx + o, g);
  });
}

// ---- adaptive average pooling: output cell (oh, ow) averages rows [floor(oh*H/OH), ceil((oh+1)*H/OH)) x the same in w
// (crates/incin-backends/src/cuda/ops/kernels/pool.cu adaptive_avg_pool2d_{fwd,bwd}; the backward there scatters with
// atomics, here every input pixel gathers from the output cells whose window contains it)
// (products below 2^31 are divided in 32 bits)
__device__ __forceinline__ int ad_div(long long a, const Div& b) {
  return a <= 0x7fffffffLL ? (int)b.of((unsigned)a) : (int)(a / b.d);
}
__device__ __forceinline__ int ad_start(int o, int in, const Div& out) { return ad_div((long long)o * in, out); }
__device__ __forceinline__ int ad_end(int o, int in, const Div& out) { return ad_div(((long long)o + 1) * in + out.d - 1, out); }

template <typename T, typename I>
__global__ void adaptive_avgpool_fwd_kernel(const T* __restrict__ x, T* __restrict__ y, Div H, Div W, Div OH, Div OW, I total, Divisor<I> oh_,
                                            Divisor<I> ow_) {
  for (I t = (I)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (I)gridDim.x * blockDim.x) {
    const Place<I> o(t, ow_, oh_);
    const int h0 = ad_start(o.y, H.d, OH), h1 = ad_end(o.y, H.d, OH), w0 = ad_start(o.x, W.d, OW), w1 = ad_end(o.x, W.d, OW);
    const T* p = x + o.plane * H.d * W.d;
    float acc = 0.0f;
    for (int h = h0; h < h1; ++h)
      for (int w = w0; w < w1; ++w) acc += ldf(p, (long long)h * W.d + w);
    stf(y, (long long)t, acc / (float)((h1 - h0) * (w1 - w0)));
  }
}

// Input index i lies in cell o, [start(o), end(o)), if and only if o * in < (i + 1) * out and (o + 1) * in > i * out: the
// cells floor(i * out / in) .. ceil((i + 1) * out / in) - 1.  N 64, C 128, 16 x 16 -> 4 x 4 bf16: 47 -> 20 us.
template <typename T, typename I>
__global__ void adaptive_avgpool_bwd_kernel(const T* __restrict__ dy, T* __restrict__ dx, Div H, Div W, Div OH, Div OW, I total, Divisor<I> h_,
                                            Divisor<I> w_) {
  for (I t = (I)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (I)gridDim.x * blockDim.x) {
    const Place<I> i(t, w_, h_);
    const T* p = dy + i.plane * OH.d * OW.d;
    const int oh_lo = ad_start(i.y, OH.d, H), oh_hi = ad_end(i.y, OH.d, H), ow_lo = ad_start(i.x, OW.d, W), ow_hi = ad_end(i.x, OW.d, W);
    float acc = 0.0f;
    for (int oh = oh_lo; oh < oh_hi; ++oh) {
      const int eh = ad_end(oh, H.d, OH) - ad_start(oh, H.d, OH);
      for (int ow = ow_lo; ow < ow_hi; ++ow) {
        const int ew = ad_end(ow, W.d, OW) - ad_start(ow, W.d, OW);
        acc += ldf(p, (long long)oh * OW.d + ow) / (float)(eh * ew);
      }
    }
    stf(dx, (long long)t, acc);
  }
}

inline unsigned grid_for(long long n) {
  long long g = (n + 255) / 256;
  return (unsigned)(g < 1 ? 1 : (g > 148LL * 16 ? 148LL * 16 : g));
}

// calls f with the element count in the narrowest type that the kernels' flat index can have (a step past the end fits too)
template <typename F> void with_index(long long total, F f) {
  if (total < 0x7fffffffLL) f((unsigned)total);
  else f(total);
}

ConvGeom geom(const incin_conv_geom* d) {
  ConvGeom g;
  g.N = d->N; g.C = d->C; g.H = d->H; g.W = d->W; g.KH = d->KH; g.KW = d->KW;
  g.sh = d->stride_h; g.sw = d->stride_w; g.ph = d->pad_h; g.pw = d->pad_w;
  g.dh = d->dil_h > 0 ? d->dil_h : 1; g.dw = d->dil_w > 0 ? d->dil_w : 1;
  g.OH = (g.H + 2 * g.ph - g.dh * (g.KH - 1) - 1) / g.sh + 1;
  g.OW = (g.W + 2 * g.pw - g.dw * (g.KW - 1) - 1) / g.sw + 1;
  return g;
}

bool valid(const incin_conv_geom* d) {
  return d && d->N > 0 && d->C > 0 && d->H > 0 && d->W > 0 && d->KH > 0 && d->KW > 0 && d->stride_h > 0 && d->stride_w > 0 &&
         d->pad_h >= 0 && d->pad_w >= 0 && (d->H + 2 * d->pad_h - (d->dil_h > 0 ? d->dil_h : 1) * (d->KH - 1) - 1) >= 0 &&
         (d->W + 2 * d->pad_w - (d->dil_w > 0 ? d->dil_w : 1) * (d->KW - 1) - 1) >= 0;
}

}  // namespace

template <typename... KArgs, typename... Args>
static int launch_channels(void (*kern)(KArgs...), int C, int slices, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)C * (unsigned)slices);
  cfg.blockDim = dim3(512);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)slices;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = slices > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...) == cudaSuccess && cudaGetLastError() == cudaSuccess ? INCIN_OK : INCIN_ERR_LAUNCH;
}

// CTAs per channel: enough for four on every SM, at least 4096 elements each, 8 at most
static int channel_slices(long long C, long long count) {
  int s = 1;
  while (s < 8 && C * s < 4 * 148 && count / (2 * s) >= 4096) s *= 2;
  return s;
}

#define DISPATCH(is_bf16, CALL_BF16, CALL_F32) \
  do {                                         \
    if (is_bf16) { CALL_BF16; } else { CALL_F32; } \
  } while (0)

extern "C" int incin_conv_out_hw(const incin_conv_geom* d, int* oh, int* ow) {
  if (!valid(d) || !oh || !ow) return INCIN_ERR_ARGUMENT;
  const ConvGeom g = geom(d);
  *oh = g.OH;
  *ow = g.OW;
  return INCIN_OK;
}

// Both take the tiled kernel where the column matrix can be moved 16 bytes at a time (K a multiple of that, aligned base)
// and the tile fits the 48 KB of shared memory a kernel gets without asking; the general kernel otherwise (very wide
// images, K = 27 and the like).  Channels go in eights: 8 * KH * KW elements are always whole 16-byte units.
constexpr long long kTileBytes = 48 * 1024;

template <typename T>
static int im2col_t(const void* x, void* cols, const ConvGeom& g, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  const long long KK = (long long)g.KH * g.KW, total = (long long)g.N * g.OH * g.OW * g.C * KK;
  const long long SW = (long long)(g.OW - 1) * g.sw + (long long)(g.KW - 1) * g.dw + 1;
  auto bytes = [&](long long ct) { return (ct * KK + 3) / 4 * 16 + ct * g.KH * SW * (long long)sizeof(T); };
  const long long c8 = (g.C + 7) / 8 * 8;
  long long CT = 8;
  while (CT * 2 <= c8 && CT < 64 && bytes(CT * 2) <= kTileBytes / 2) CT *= 2;
  // The tile pays where a row fills a warp's 16 columns and there is enough to write (bf16, tile | general: N 64, C 64, 32 x 32,
  // 3 x 3 49 | 90 us; N 64, C 256, 8 x 8 37 | 25; N 1, C 64, 32 x 32 8.0 | 4.4; N 16, C 64, 8 x 8 patches 17 | 2.9).
  if (g.OW >= 16 && total >= 3 << 19 && g.C * KK % V == 0 && (reinterpret_cast<uintptr_t>(cols) & 15) == 0 && KK <= 4096 && SW <= 65536 && bytes(CT) <= kTileBytes &&
      (long long)g.N * g.OH <= 0x7fffffffLL && c8 / CT <= 65535) {
    const dim3 grid((unsigned)(g.N * g.OH), (unsigned)((g.C + CT - 1) / CT));
    im2col_tile_kernel<T><<<grid, 256, (size_t)bytes(CT), s>>>(static_cast<const T*>(x), static_cast<T*>(cols), g, (int)CT, (int)SW);
  } else {
    with_index(total, [&](auto n) {
      using I = decltype(n);
      im2col_kernel<T><<<grid_for(total), 256, 0, s>>>(static_cast<const T*>(x), static_cast<T*>(cols), g, n, Divisor<I>(g.C * KK), Divisor<I>(g.OW),
                                                       Divisor<I>(g.OH), Div(g.KW), Div(g.KH));
    });
  }
  return cudaGetLastError() == cudaSuccess ? INCIN_OK : INCIN_ERR_LAUNCH;
}

template <typename T>
static int col2im_t(const void* cols, void* dx, const ConvGeom& g, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T), WV = 4 / sizeof(T), CT = 8;
  const long long KK = (long long)g.KH * g.KW, total = (long long)g.N * g.C * g.H * g.W;
  auto bytes = [&](long long rb) {   // output rows that reach rb input rows, at most
    long long oh = rb + (long long)(g.KH - 1) * g.dh;
    if (oh > g.OH) oh = g.OH;
    return oh * g.OW * (CT * KK + WV) * (long long)sizeof(T);
  };
  long long RB = g.H < 8 ? g.H : 8;
  while (RB > 1 && bytes(RB) > kTileBytes) --RB;
  const long long bands = (g.H + RB - 1) / RB;
  const long long groups = (g.C + CT - 1) / CT;
  // The tile pays where its rows are read KH times and there are blocks enough (bf16, tile | general: N 64, C 64, 32 x 32, 3 x 3
  // 67 | 151 us; N 64, C 16, 14 x 14, 256 blocks, 9.6 | 7.1; N 8, C 16, 40 x 40, 128 blocks, 18 | 7.1; 1 x 1, N 8, C 256, 28 x 28
  // 14 | 11).  Strides: 2 x 128 x 128, C 32, 3 x 3 by 4 42 | 10; 8 x 56 x 56, C 64, 3 x 3 by 2 51 | 25.
  if (g.sh == 1 && g.sw == 1 && KK > 1 && g.N * bands * groups >= 256 && g.C * KK % V == 0 && (reinterpret_cast<uintptr_t>(cols) & 15) == 0 &&
      KK <= 4096 && bytes(RB) <= kTileBytes && g.N * bands <= 0x7fffffffLL && groups <= 65535) {
    const dim3 grid((unsigned)(g.N * bands), (unsigned)groups);
    col2im_tile_kernel<T><<<grid, 256, (size_t)bytes(RB), s>>>(static_cast<const T*>(cols), static_cast<T*>(dx), g, CT, (int)RB);
  } else {
    with_index(total, [&](auto n) {
      using I = decltype(n);
      col2im_kernel<T><<<grid_for(total), 256, 0, s>>>(static_cast<const T*>(cols), static_cast<T*>(dx), g, n, Divisor<I>(g.W), Divisor<I>(g.H),
                                                       Divisor<I>(g.C), Div(g.sh), Div(g.sw));
    });
  }
  return cudaGetLastError() == cudaSuccess ? INCIN_OK : INCIN_ERR_LAUNCH;
}

extern "C" int incin_im2col(const void* x, void* cols, const incin_conv_geom* d, int is_bf16, void* stream) {
  if (!x || !cols || !valid(d)) return INCIN_ERR_ARGUMENT;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return is_bf16 ? im2col_t<__nv_bfloat16>(x, cols, geom(d), s) : im2col_t<float>(x, cols, geom(d), s);
}

extern "C" int incin_col2im(const void* cols, void* dx, const incin_conv_geom* d, int is_bf16, void* stream) {
  if (!cols || !dx || !valid(d)) return INCIN_ERR_ARGUMENT;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return is_bf16 ? col2im_t<__nv_bfloat16>(cols, dx, geom(d), s) : col2im_t<float>(cols, dx, geom(d), s);
}

template <typename T>
static void maxpool_fwd_t(const void* x, void* y, int* argmax, const ConvGeom& g, cudaStream_t s) {
  with_index((long long)g.N * g.C * g.OH * g.OW, [&](auto total) {
    maxpool_fwd_kernel<T><<<grid_for((long long)total), 256, 0, s>>>(static_cast<const T*>(x), static_cast<T*>(y), argmax, g, total,
                                                                  Divisor<decltype(total)>(g.OW), Divisor<decltype(total)>(g.OH));
  });
}
template <typename T>
static void maxpool_bwd_t(const void* dy, const int* argmax, void* dx, const ConvGeom& g, cudaStream_t s) {
  with_index((long long)g.N * g.C * g.H * g.W, [&](auto total) {
    maxpool_bwd_kernel<T><<<grid_for((long long)total), 256, 0, s>>>(static_cast<const T*>(dy), argmax, static_cast<T*>(dx), g, total,
                                                                  Divisor<decltype(total)>(g.W), Divisor<decltype(total)>(g.H), Div(g.sh), Div(g.sw));
  });
}

extern "C" int incin_maxpool2d_fwd(const void* x, void* y, int* argmax, const incin_conv_geom* d, int is_bf16, void* stream) {
  if (!x || !y || !valid(d)) return INCIN_ERR_ARGUMENT;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  DISPATCH(is_bf16, maxpool_fwd_t<__nv_bfloat16>(x, y, argmax, geom(d), s), maxpool_fwd_t<float>(x, y, argmax, geom(d), s));
  return cudaGetLastError() == cudaSuccess ? INCIN_OK : INCIN_ERR_LAUNCH;
}

extern "C" int incin_maxpool2d_bwd(const void* dy, const int* argmax, void* dx, const incin_conv_geom* d, int is_bf16,
                                   void* stream) {
  if (!dy || !argmax || !dx || !valid(d)) return INCIN_ERR_ARGUMENT;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  DISPATCH(is_bf16, maxpool_bwd_t<__nv_bfloat16>(dy, argmax, dx, geom(d), s), maxpool_bwd_t<float>(dy, argmax, dx, geom(d), s));
  return cudaGetLastError() == cudaSuccess ? INCIN_OK : INCIN_ERR_LAUNCH;
}

extern "C" int incin_avgpool2d(const void* in, void* out, const incin_conv_geom* d, int backward, int is_bf16, void* stream) {
  if (!in || !out || !valid(d)) return INCIN_ERR_ARGUMENT;
  const ConvGeom g = geom(d);
  const long long total = backward ? (long long)g.N * g.C * g.H * g.W : (long long)g.N * g.C * g.OH * g.OW;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  DISPATCH(is_bf16, (avgpool_kernel<__nv_bfloat16><<<grid_for(total), 256, 0, s>>>(static_cast<const __nv_bfloat16*>(in), static_cast<__nv_bfloat16*>(out), g, total, backward)),
           (avgpool_kernel<float><<<grid_for(total), 256, 0, s>>>(static_cast<const float*>(in), static_cast<float*>(out), g, total, backward)));
  return cudaGetLastError() == cudaSuccess ? INCIN_OK : INCIN_ERR_LAUNCH;
}

template <typename T>
static int batchnorm_train_fwd_t(const void* x, const float* gamma, const float* beta, void* y, float* save_mean, float* save_rstd,
                                 float* running_mean, float* running_var, int N, int C, long long HW, float eps, float momentum,
                                 cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  const long long count = (long long)N * HW;
  const bool vec = HW % V == 0 && count >= 512 * V && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
  const int slices = channel_slices(C, count);
  auto pick = [&](auto cl) {
    constexpr bool CL = decltype(cl)::value;
    return count > 0x40000000LL ? batchnorm_train_fwd_kernel<CL, T, 1, long long>
                                : (vec ? batchnorm_train_fwd_kernel<CL, T, V, unsigned> : batchnorm_train_fwd_kernel<CL, T, 1, unsigned>);
  };
  auto kern = slices > 1 ? pick(std::true_type{}) : pick(std::false_type{});
  return launch_channels(kern, C, slices, s, static_cast<const T*>(x), gamma, beta, static_cast<T*>(y), save_mean,
                         save_rstd, running_mean, running_var, N, C, HW, eps, momentum);
}

template <typename T>
static int batchnorm_bwd_t(const void* dy, const void* x, const float* gamma, const float* save_mean, const float* save_rstd, void* dx,
                           float* dgamma, float* dbeta, int N, int C, long long HW, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  const long long count = (long long)N * HW;
  const bool vec = HW % V == 0 && count >= 512 * V &&
                   ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dx)) & 15) == 0;
  const int slices = channel_slices(C, count);
  auto pick = [&](auto cl) {
    constexpr bool CL = decltype(cl)::value;
    return count > 0x40000000LL ? batchnorm_bwd_kernel<CL, T, 1, long long>
                                : (vec ? batchnorm_bwd_kernel<CL, T, V, unsigned> : batchnorm_bwd_kernel<CL, T, 1, unsigned>);
  };
  auto kern = slices > 1 ? pick(std::true_type{}) : pick(std::false_type{});
  return launch_channels(kern, C, slices, s, static_cast<const T*>(dy), static_cast<const T*>(x), gamma, save_mean,
                         save_rstd, static_cast<T*>(dx), dgamma, dbeta, N, C, HW);
}

extern "C" int incin_batchnorm_train_fwd(const void* x, const float* gamma, const float* beta, void* y, float* save_mean,
                                         float* save_rstd, float* running_mean, float* running_var, int N, int C, long long HW,
                                         float eps, float momentum, int is_bf16, void* stream) {
  if (!x || !y || !save_mean || !save_rstd || N <= 0 || C <= 0 || HW <= 0) return INCIN_ERR_ARGUMENT;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return is_bf16 ? batchnorm_train_fwd_t<__nv_bfloat16>(x, gamma, beta, y, save_mean, save_rstd, running_mean, running_var, N, C, HW, eps, momentum, s)
                 : batchnorm_train_fwd_t<float>(x, gamma, beta, y, save_mean, save_rstd, running_mean, running_var, N, C, HW, eps, momentum, s);
}

extern "C" int incin_batchnorm_eval(const void* x, const float* gamma, const float* beta, const float* mean, const float* var,
                                    void* y, int N, int C, long long HW, float eps, int is_bf16, void* stream) {
  if (!x || !y || !mean || !var || N <= 0 || C <= 0 || HW <= 0) return INCIN_ERR_ARGUMENT;
  const long long total = (long long)N * C * HW;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  DISPATCH(is_bf16, (batchnorm_eval_kernel<__nv_bfloat16><<<grid_for(total), 256, 0, s>>>(static_cast<const __nv_bfloat16*>(x), gamma, beta, mean, var, static_cast<__nv_bfloat16*>(y), C, HW, eps, total)),
           (batchnorm_eval_kernel<float><<<grid_for(total), 256, 0, s>>>(static_cast<const float*>(x), gamma, beta, mean, var, static_cast<float*>(y), C, HW, eps, total)));
  return cudaGetLastError() == cudaSuccess ? INCIN_OK : INCIN_ERR_LAUNCH;
}

extern "C" int incin_batchnorm_bwd(const void* dy, const void* x, const float* gamma, const float* save_mean,
                                   const float* save_rstd, void* dx, float* dgamma, float* dbeta, int N, int C, long long HW,
                                   int is_bf16, void* stream) {
  if (!dy || !x || !dx || !save_mean || !save_rstd || N <= 0 || C <= 0 || HW <= 0) return INCIN_ERR_ARGUMENT;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return is_bf16 ? batchnorm_bwd_t<__nv_bfloat16>(dy, x, gamma, save_mean, save_rstd, dx, dgamma, dbeta, N, C, HW, s)
                 : batchnorm_bwd_t<float>(dy, x, gamma, save_mean, save_rstd, dx, dgamma, dbeta, N, C, HW, s);
}

extern "C" int incin_adaptive_avgpool2d(const void* in, void* out, long long planes, int H, int W, int OH, int OW, int backward,
                                        int is_bf16, void* stream) {
  if (!in || !out || planes <= 0 || H <= 0 || W <= 0 || OH <= 0 || OW <= 0) return INCIN_ERR_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  const long long total = planes * (backward ? (long long)H * W : (long long)OH * OW);
  const Div h(H), w(W), oh(OH), ow(OW);
  with_index(total, [&](auto n) {
    using I = decltype(n);
    if (backward)
      DISPATCH(is_bf16,
               (adaptive_avgpool_bwd_kernel<<<grid_for(total), 256, 0, s>>>((const __nv_bfloat16*)in, (__nv_bfloat16*)out, h, w, oh, ow, n, Divisor<I>(H), Divisor<I>(W))),
               (adaptive_avgpool_bwd_kernel<<<grid_for(total), 256, 0, s>>>((const float*)in, (float*)out, h, w, oh, ow, n, Divisor<I>(H), Divisor<I>(W))));
    else
      DISPATCH(is_bf16,
               (adaptive_avgpool_fwd_kernel<<<grid_for(total), 256, 0, s>>>((const __nv_bfloat16*)in, (__nv_bfloat16*)out, h, w, oh, ow, n, Divisor<I>(OH), Divisor<I>(OW))),
               (adaptive_avgpool_fwd_kernel<<<grid_for(total), 256, 0, s>>>((const float*)in, (float*)out, h, w, oh, ow, n, Divisor<I>(OH), Divisor<I>(OW))));
  });
  return cudaGetLastError() == cudaSuccess ? INCIN_OK : INCIN_ERR_LAUNCH;
}
