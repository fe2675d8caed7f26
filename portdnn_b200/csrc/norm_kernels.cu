// Softmax and batchnorm (NHWC): the operators the reference's network wrappers need beside the
// convolution path (tools/layer.h:128-205, 284-310).  HBM-bound; arithmetic in fp32, one rounding on
// store.  The reference composes both from reduce / binaryop / pointwise launches
// (include/portdnn/internal/softmax/launch_internal.h:45-275,
// include/portdnn/internal/batchnorm/launch_internal.h:95-640); here each is one to three kernels.
#include "column_sums.cuh"
#include "common.cuh"

#include <algorithm>
#include <cfloat>

namespace pdnn {
namespace {

constexpr int kBlock = 256;
// Blocks to an SM of the kernels whose grids are one wave: the launch bound that the compiler keeps and the size of the grid.
constexpr int kMomentBlocks = 3, kApplyBlocks = 4;
constexpr int gradient_blocks(int packet) { return packet == 8 ? 3 : 4; }  // (80 and 63 registers)

template <typename F>
int dispatch(int dtype, F&& f) {
  switch (dtype) {
    case PDNN_F32: return f(float{});
    case PDNN_F16: return f(__half{});
    case PDNN_BF16: return f(__nv_bfloat16{});
  }
  return fail(PDNN_INVALID_PARAMETER, "unknown dtype %d", dtype);
}

__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  return v;
}

// V consecutive elements as floats (one 16-byte access when V > 1).
template <typename T, int V>
__device__ __forceinline__ void load_v(const T* p, float (&v)[V]) {
  if constexpr (V == 1) {
    v[0] = to_f32(*p);
  } else {
    const Vec16<T> pk = load16(p);
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = to_f32(pk.get(i));
  }
}
template <typename T, int V>
__device__ __forceinline__ void store_v(T* p, const float (&v)[V]) {
  if constexpr (V == 1) {
    p[0] = from_f32<T>(v[0]);
  } else {
    Vec16<T> pk;
#pragma unroll
    for (int i = 0; i < V; ++i) pk.set(i, from_f32<T>(v[i]));
    store16(p, pk);
  }
}

// One warp per pixel, packets of V channels, at most R packets per lane (C <= 32 * R * V): the
// pixel is read once and stays in registers through the three steps.
template <typename T, int V, int R>
__global__ void __launch_bounds__(kBlock) softmax_forward_vec_kernel(const T* x, T* __restrict__ y,
                                                                     size_t rows, int C) {
  overlap_wait();
  const int lane = threadIdx.x & 31, packets = C / V;
  const size_t warps = (size_t)gridDim.x * (kBlock / 32);
  for (size_t row = (size_t)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); row < rows; row += warps) {
    const T* xr = x + row * C;
    float v[R][V];
    float m = -INFINITY;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int pk = lane + 32 * r;
      if (pk < packets) {
        load_v<T, V>(xr + pk * V, v[r]);
#pragma unroll
        for (int k = 0; k < V; ++k) m = fmaxf(m, v[r][k]);
      }
    }
    m = warp_max(m);
    float sum = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (lane + 32 * r < packets) {
        float packet = 0.f;
#pragma unroll
        for (int k = 0; k < V; ++k) {
          v[r][k] = expf(v[r][k] - m);
          packet += v[r][k];
        }
        sum += packet;
      }
    sum = warp_sum(sum);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int pk = lane + 32 * r;
      if (pk < packets) {
#pragma unroll
        for (int k = 0; k < V; ++k) v[r][k] = v[r][k] / sum;
        store_v<T, V>(y + row * C + pk * V, v[r]);
      }
    }
  }
}

// Few pixels of many channels: a block of four warps per pixel, a packet to a thread, so that a quarter of the exponentials and
// divisions stand one after another in a thread.  The sums of the packets are added up in the order of
// softmax_forward_vec_kernel, whose lane has packets lane, lane + 32, ...: a pixel's result does not depend on how many there are.
// us, a warp to a pixel / here, 250, 700, 1024, 2000 pixels: f16 1000 channels 2.95 1.65, 3.00 2.05, 3.03 2.38, 3.77 3.72; 264 channels 2.13 1.61,
// 2.16 1.76, 2.18 2.33, 2.55 2.61; f32 500 channels 2.10 1.48, 2.15 1.71, 2.19 2.23, 2.65 2.73; 132 channels 1.71 1.44, 1.74 1.56, 1.76 1.88,
// 1.98 2.36.  So up to six blocks to an SM, and up to a whole wave of them where a warp has more than 64 packets of 16 bits.
constexpr int kSoftmaxRow = 128;
bool softmax_by_rows(size_t rows, int packets, bool wide, int sms) {
  return rows <= (size_t)sms * (wide && packets > 64 ? 2048 / kSoftmaxRow : 6);
}
template <typename T, int V>
__global__ void __launch_bounds__(kSoftmaxRow) softmax_forward_row_kernel(const T* x, T* __restrict__ y, int C) {
  overlap_wait();
  __shared__ float red[kSoftmaxRow / 32], packet[kSoftmaxRow];
  const int warp = threadIdx.x >> 5;
  const bool here = (int)threadIdx.x < C / V;
  const size_t at = (size_t)blockIdx.x * C + (size_t)threadIdx.x * V;
  float v[V], m = -INFINITY, sum = 0.f;
  if (here) {
    load_v<T, V>(x + at, v);
#pragma unroll
    for (int k = 0; k < V; ++k) m = fmaxf(m, v[k]);
  }
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) red[warp] = m;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kSoftmaxRow / 32; ++i) m = fmaxf(m, red[i]);
  if (here) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      v[k] = expf(v[k] - m);
      sum += v[k];
    }
  }
  packet[threadIdx.x] = sum;
  __syncthreads();
  sum = 0.f;
#pragma unroll
  for (int i = 0; i < kSoftmaxRow / 32; ++i) sum += packet[(threadIdx.x & 31) + 32 * i];
  sum = warp_sum(sum);
  if (!here) return;
#pragma unroll
  for (int k = 0; k < V; ++k) v[k] = v[k] / sum;
  store_v<T, V>(y + at, v);
}

// One warp per pixel: y = exp(x - max) / sum exp(x - max) over the pixel's C channels.
template <typename T>
__global__ void __launch_bounds__(kBlock) softmax_forward_kernel(const T* __restrict__ x, T* __restrict__ y, size_t rows,
                                                                 int C) {
  const int lane = threadIdx.x & 31;
  const size_t warps = (size_t)gridDim.x * (kBlock / 32);
  for (size_t row = (size_t)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); row < rows; row += warps) {
    const T* xr = x + row * C;
    T* yr = y + row * C;
    float m = -INFINITY;
    for (int c = lane; c < C; c += 32) m = fmaxf(m, to_f32(xr[c]));
    m = warp_max(m);
    float sum = 0.f;
    for (int c = lane; c < C; c += 32) sum += expf(to_f32(xr[c]) - m);
    sum = warp_sum(sum);
    for (int c = lane; c < C; c += 32) yr[c] = from_f32<T>(expf(to_f32(xr[c]) - m) / sum);
  }
}

// dx = (dy - sum_c(dy * y)) * y, y = the forward output, on packets: both rows are read once and stay in
// registers.  The form below reads them twice, a value at a time.  250 x 1000 f16: 13.3 -> 3.7 us.
template <typename T, int V, int R>
__global__ void __launch_bounds__(kBlock) softmax_grad_vec_kernel(const T* y, const T* dy,
                                                                  T* __restrict__ dx, size_t rows, int C) {
  overlap_wait();
  const int lane = threadIdx.x & 31, packets = C / V;
  const size_t warps = (size_t)gridDim.x * (kBlock / 32);
  for (size_t row = (size_t)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); row < rows; row += warps) {
    const T *yr = y + row * C, *gr = dy + row * C;
    Vec16<T> yv[R], gv[R];
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (lane + 32 * r < packets) {
        yv[r] = load16(yr + (lane + 32 * r) * V);
        gv[r] = load16(gr + (lane + 32 * r) * V);
      }
    float sum = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (lane + 32 * r < packets) {
#pragma unroll
        for (int k = 0; k < V; ++k) sum += to_f32(gv[r].get(k)) * to_f32(yv[r].get(k));
      }
    sum = warp_sum(sum);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (lane + 32 * r < packets) {
        Vec16<T> o;
#pragma unroll
        for (int k = 0; k < V; ++k) o.set(k, from_f32<T>((to_f32(gv[r].get(k)) - sum) * to_f32(yv[r].get(k))));
        store16(dx + row * C + (lane + 32 * r) * V, o);
      }
  }
}

// dx = (dy - sum_c(dy * y)) * y, y = the forward output.
template <typename T>
__global__ void __launch_bounds__(kBlock) softmax_grad_kernel(const T* __restrict__ y, const T* __restrict__ dy,
                                                              T* __restrict__ dx, size_t rows, int C) {
  const int lane = threadIdx.x & 31;
  const size_t warps = (size_t)gridDim.x * (kBlock / 32);
  for (size_t row = (size_t)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); row < rows; row += warps) {
    const T* yr = y + row * C;
    const T* gr = dy + row * C;
    float sum = 0.f;
    for (int c = lane; c < C; c += 32) sum += to_f32(gr[c]) * to_f32(yr[c]);
    sum = warp_sum(sum);
    for (int c = lane; c < C; c += 32) dx[row * C + c] = from_f32<T>((to_f32(gr[c]) - sum) * to_f32(yr[c]));
  }
}

// The elementwise steps on packets of V channels (C % V == 0, 16-byte aligned tensors): n counts
// packets.  The per-channel operands are read as packets too (they stay in L1).
template <typename T, int V>
__global__ void __launch_bounds__(kBlock, kApplyBlocks)
    batchnorm_apply_vec_kernel(const T* x, const T* beta, const T* gamma,
                               const T* mean, const T* var, T* __restrict__ out, size_t n,
                               int C, float eps) {
  overlap_wait();
  const size_t cvecs = (size_t)(C / V);
  const size_t step = (size_t)gridDim.x * kBlock;
  size_t i = (size_t)blockIdx.x * kBlock + threadIdx.x;
  if (step % cvecs == 0) {
    // every packet of this thread belongs to the same channels (the host sizes the grid for
    // this): the per-channel operands and the square root are taken once
    if (i >= n) return;
    const int c = (int)(i % cvecs) * V;
    float b[V], g[V], m[V], sd[V];
    load_v<T, V>(beta + c, b);
    load_v<T, V>(gamma + c, g);
    load_v<T, V>(mean + c, m);
    load_v<T, V>(var + c, sd);
    // 1 / sqrt(var + eps) once per channel: the division per element would make the kernel
    // instruction-bound; the product differs from the quotient by at most one ulp of fp32
#pragma unroll
    for (int k = 0; k < V; ++k) sd[k] = 1.f / sqrtf(sd[k] + eps);
    auto put = [&](size_t at, const Vec16<T>& xv) {
      float o[V];
#pragma unroll
      for (int k = 0; k < V; ++k) o[k] = (to_f32(xv.get(k)) - m[k]) * sd[k] * g[k] + b[k];
      store_v<T, V>(out + at * V, o);
    };
    for (; i + 3 * step < n; i += 4 * step) {  // four packets requested together
      Vec16<T> xv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) xv[u] = load16(x + (i + u * step) * V);
#pragma unroll
      for (int u = 0; u < 4; ++u) put(i + u * step, xv[u]);
    }
    for (; i < n; i += step) put(i, load16(x + i * V));
    return;
  }
  for (; i < n; i += step) {
    const int c = (int)(i % cvecs) * V;
    float xv[V], b[V], g[V], m[V], v[V], o[V];
    load_v<T, V>(x + i * V, xv);
    load_v<T, V>(beta + c, b);
    load_v<T, V>(gamma + c, g);
    load_v<T, V>(mean + c, m);
    load_v<T, V>(var + c, v);
#pragma unroll
    for (int k = 0; k < V; ++k) o[k] = (xv[k] - m[k]) / sqrtf(v[k] + eps) * g[k] + b[k];
    store_v<T, V>(out + i * V, o);
  }
}

// A thread has five packets of 50176 x 256 f16 or so: with the square root and the two divisions of its eight channels
// to do, as long as the packets took it, it ran at 3.5 TB/s of L2 (21.8 us).  The merging kernel does them once per
// channel: terms[c] = mean x, mean dy, sum dy * xc / rows / variance, gamma / deviation.  (Where a thread's channels change,
// below, the division by the deviation used to come after the multiplication by gamma; the last factor is now
// rounded first, as it always was where they do not.)
template <typename T, int V>
__global__ void __launch_bounds__(kBlock, gradient_blocks(V))
    batchnorm_grad_training_vec_kernel(const T* x, const T* dy, const float4* terms, T* __restrict__ out, size_t n, int C) {
  overlap_wait();
  const size_t cvecs = (size_t)(C / V);
  const size_t step = (size_t)gridDim.x * kBlock;
  size_t i = (size_t)blockIdx.x * kBlock + threadIdx.x;
  if (step % cvecs == 0) {  // the thread's channels never change: per-channel terms taken once
    if (i >= n) return;
    const int c = (int)(i % cvecs) * V;
    float mx[V], mdy[V], kk[V], sd[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const float4 t = terms[c + k];
      mx[k] = t.x, mdy[k] = t.y, kk[k] = t.z, sd[k] = t.w;
    }
    auto put = [&](size_t at, const Vec16<T>& xv, const Vec16<T>& gv) {
      float o[V];
#pragma unroll
      for (int k = 0; k < V; ++k) o[k] = ((to_f32(gv.get(k)) - mdy[k]) - (to_f32(xv.get(k)) - mx[k]) * kk[k]) * sd[k];
      store_v<T, V>(out + at * V, o);
    };
    for (; i + 3 * step < n; i += 4 * step) {  // four packets of either tensor requested together
      Vec16<T> xv[4], gv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        xv[u] = load16(x + (i + u * step) * V);
        gv[u] = load16(dy + (i + u * step) * V);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) put(i + u * step, xv[u], gv[u]);
    }
    for (; i < n; i += step) put(i, load16(x + i * V), load16(dy + i * V));
    return;
  }
  for (; i < n; i += step) {
    const int c = (int)(i % cvecs) * V;
    float xv[V], gv[V], o[V];
    load_v<T, V>(x + i * V, xv);
    load_v<T, V>(dy + i * V, gv);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const float4 t = terms[c + k];
      o[k] = ((gv[k] - t.y) - (xv[k] - t.x) * t.z) * t.w;
    }
    store_v<T, V>(out + i * V, o);
  }
}

template <typename T, int V>
__global__ void __launch_bounds__(kBlock)
    batchnorm_grad_frozen_vec_kernel(const T* __restrict__ dy, const T* __restrict__ gamma,
                                     const T* __restrict__ pop_var, T* __restrict__ out, size_t n, int C, float eps) {
  const size_t cvecs = (size_t)(C / V);
  const size_t step = (size_t)gridDim.x * kBlock;
  size_t i = (size_t)blockIdx.x * kBlock + threadIdx.x;
  if (step % cvecs == 0) {  // the thread's channels never change: scale taken once
    if (i >= n) return;
    const int c = (int)(i % cvecs) * V;
    float g[V], v[V];
    load_v<T, V>(gamma + c, g);
    load_v<T, V>(pop_var + c, v);
#pragma unroll
    for (int k = 0; k < V; ++k) g[k] = g[k] / sqrtf(v[k] + eps);
#pragma unroll 4
    for (; i < n; i += step) {
      float gv[V], o[V];
      load_v<T, V>(dy + i * V, gv);
#pragma unroll
      for (int k = 0; k < V; ++k) o[k] = gv[k] * g[k];
      store_v<T, V>(out + i * V, o);
    }
    return;
  }
  for (; i < n; i += step) {
    const int c = (int)(i % cvecs) * V;
    float gv[V], g[V], v[V], o[V];
    load_v<T, V>(dy + i * V, gv);
    load_v<T, V>(gamma + c, g);
    load_v<T, V>(pop_var + c, v);
#pragma unroll
    for (int k = 0; k < V; ++k) o[k] = gv[k] * (g[k] / sqrtf(v[k] + eps));
    store_v<T, V>(out + i * V, o);
  }
}

// The sums of the frozen gradient on packets (MODE 2 below): lane tx of the block owns V channels; 32 lanes x 8
// row lanes.
template <typename T, int V>
__global__ void __launch_bounds__(kBlock)
    batchnorm_frozen_sums_vec_kernel(const T* __restrict__ x, const T* __restrict__ dy, const float* __restrict__ shift,
                                     const float* __restrict__ scale, float* __restrict__ partial, size_t rows, int C,
                                     size_t rows_per_slice) {
  __shared__ float red[2][8][32][V];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = (blockIdx.y * 32 + tx) * V;
  const size_t begin = (size_t)blockIdx.x * rows_per_slice;
  const size_t end = begin + rows_per_slice < rows ? begin + rows_per_slice : rows;
  float a[V], b[V], sh[V], sc[V];
#pragma unroll
  for (int k = 0; k < V; ++k) a[k] = b[k] = 0.f, sh[k] = 0.f, sc[k] = 1.f;
  if (c < C) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      sh[k] = shift[c + k];
      sc[k] = scale[c + k];
    }
    for (size_t r = begin + ty; r < end; r += 8) {
      float xv[V], gv[V];
      load_v<T, V>(x + r * C + c, xv);
      load_v<T, V>(dy + r * C + c, gv);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        a[k] += gv[k];
        b[k] += (xv[k] - sh[k]) * gv[k] / sc[k];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < V; ++k) {
    red[0][ty][tx][k] = a[k];
    red[1][ty][tx][k] = b[k];
  }
  __syncthreads();
  if (ty < 2 && c < C) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      float sum = 0.f;
#pragma unroll
      for (int l = 0; l < 8; ++l) sum += red[ty][l][tx][k];
      partial[((size_t)blockIdx.x * 2 + ty) * C + c + k] = sum;
    }
  }
}

// out = (x - mean[c]) / sqrt(var[c] + eps) * gamma[c] + beta[c]
template <typename T>
__global__ void __launch_bounds__(kBlock)
    batchnorm_apply_kernel(const T* __restrict__ x, const T* __restrict__ beta, const T* __restrict__ gamma,
                           const T* __restrict__ mean, const T* __restrict__ var, T* __restrict__ out, size_t n, int C,
                           float eps) {
  for (size_t i = (size_t)blockIdx.x * kBlock + threadIdx.x; i < n; i += (size_t)gridDim.x * kBlock) {
    const int c = (int)(i % C);
    const float v = (to_f32(x[i]) - to_f32(mean[c])) / sqrtf(to_f32(var[c]) + eps) * to_f32(gamma[c]) + to_f32(beta[c]);
    out[i] = from_f32<T>(v);
  }
}

// Per-channel sums over the rows of one slice: partial[slice][0][c], partial[slice][1][c].
//   MODE 0: sum x,                 sum dy
//   MODE 1: sum (x - shift)^2,     sum dy * (x - shift)         shift = per-channel float
//   MODE 2: sum dy,                sum (x - shift) * dy / scale shift, scale = per-channel float
// dy may be NULL (its sums are then zero).  Block: 32 channel lanes x 8 row lanes.
template <typename T, int MODE>
__global__ void __launch_bounds__(kBlock)
    batchnorm_sums_kernel(const T* __restrict__ x, const T* __restrict__ dy, const float* __restrict__ shift,
                          const float* __restrict__ scale, float* __restrict__ partial, size_t rows, int C,
                          size_t rows_per_slice) {
  __shared__ float red[2][8][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = blockIdx.y * 32 + tx;
  const size_t begin = (size_t)blockIdx.x * rows_per_slice;
  const size_t end = begin + rows_per_slice < rows ? begin + rows_per_slice : rows;
  float a = 0.f, b = 0.f;
  if (c < C) {
    const float sh = MODE == 0 ? 0.f : shift[c];
    const float sc = MODE == 2 ? scale[c] : 1.f;
    for (size_t r = begin + ty; r < end; r += 8) {
      const float xv = to_f32(x[r * C + c]);
      const float gv = dy != nullptr ? to_f32(dy[r * C + c]) : 0.f;
      if (MODE == 0) {
        a += xv;
        b += gv;
      } else if (MODE == 1) {
        const float d = xv - sh;
        a += d * d;
        b += gv * d;
      } else {
        a += gv;
        b += (xv - sh) * gv / sc;
      }
    }
  }
  red[0][ty][tx] = a;
  red[1][ty][tx] = b;
  __syncthreads();
  if (ty < 2 && c < C) {
    float sum = 0.f;
#pragma unroll
    for (int l = 0; l < 8; ++l) sum += red[ty][l][tx];
    partial[((size_t)blockIdx.x * 2 + ty) * C + c] = sum;
  }
}

// totals[k][c] = sum over slices of partial[slice][k][c], divided by divide0 (k = 0) or divide1.
struct StoreTotals {
  float* totals;
  int C;
  float divide0, divide1;
  __device__ __forceinline__ void operator()(size_t i, float sum) const {
    totals[i] = sum / (i < (size_t)C ? divide0 : divide1);
  }
};

// Training forward, last step: running = batch * (1 - m) + given * m.
template <typename T>
__global__ void __launch_bounds__(kBlock)
    batchnorm_running_kernel(const float* __restrict__ batch_mean, const float* __restrict__ batch_var,
                             const T* __restrict__ mean, const T* __restrict__ var, T* __restrict__ run_mean,
                             T* __restrict__ run_var, int C, float momentum) {
  const int c = blockIdx.x * kBlock + threadIdx.x;
  if (c >= C) return;
  run_mean[c] = from_f32<T>(batch_mean[c] * (1.f - momentum) + to_f32(mean[c]) * momentum);
  run_var[c] = from_f32<T>(batch_var[c] * (1.f - momentum) + to_f32(var[c]) * momentum);
}

// Training gradient, elementwise step.  stats0 = [mean x | mean dy], stats1 = [var | sum dy * xc].
template <typename T>
__global__ void __launch_bounds__(kBlock)
    batchnorm_grad_training_kernel(const T* __restrict__ x, const T* __restrict__ dy, const T* __restrict__ gamma,
                                   const float* __restrict__ stats0, const float* __restrict__ stats1,
                                   T* __restrict__ out, size_t n, int C, float rows, float eps) {
  for (size_t i = (size_t)blockIdx.x * kBlock + threadIdx.x; i < n; i += (size_t)gridDim.x * kBlock) {
    const int c = (int)(i % C);
    const float v = stats1[c] + eps, sd = sqrtf(v);
    const float k = stats1[C + c] / rows / v;
    const float d = to_f32(x[i]) - stats0[c];
    out[i] = from_f32<T>(((to_f32(dy[i]) - stats0[C + c]) - d * k) * to_f32(gamma[c]) / sd);
  }
}

// Per-channel results of the gradients.  Training: beta_grad = mean dy * rows, gamma_grad =
// sum(dy * xc) / sqrt(var + eps).  Frozen: the two sums as they are.
template <typename T>
__global__ void __launch_bounds__(kBlock)
    batchnorm_param_grads_kernel(const float* __restrict__ stats0, const float* __restrict__ stats1,
                                 T* __restrict__ beta_grad, T* __restrict__ gamma_grad, int C, float rows, float eps,
                                 int training) {
  const int c = blockIdx.x * kBlock + threadIdx.x;
  if (c >= C) return;
  if (training) {
    beta_grad[c] = from_f32<T>(stats0[C + c] * rows);
    gamma_grad[c] = from_f32<T>(stats1[C + c] / sqrtf(stats1[c] + eps));
  } else {
    beta_grad[c] = from_f32<T>(stats0[c]);
    gamma_grad[c] = from_f32<T>(stats0[C + c]);
  }
}

// Frozen gradient, elementwise step: out = dy * gamma / sqrt(pop_var + eps).
template <typename T>
__global__ void __launch_bounds__(kBlock)
    batchnorm_grad_frozen_kernel(const T* __restrict__ dy, const T* __restrict__ gamma, const T* __restrict__ pop_var,
                                 T* __restrict__ out, size_t n, int C, float eps) {
  for (size_t i = (size_t)blockIdx.x * kBlock + threadIdx.x; i < n; i += (size_t)gridDim.x * kBlock) {
    const int c = (int)(i % C);
    out[i] = from_f32<T>(to_f32(dy[i]) * (to_f32(gamma[c]) / sqrtf(to_f32(pop_var[c]) + eps)));
  }
}

// Channel vectors of T as float (shift / scale operands of the sums kernel).
template <typename T>
__global__ void __launch_bounds__(kBlock)
    batchnorm_prepare_frozen_kernel(const T* __restrict__ pop_mean, const T* __restrict__ pop_var,
                                    float* __restrict__ shift, float* __restrict__ scale, int C, float eps) {
  const int c = blockIdx.x * kBlock + threadIdx.x;
  if (c >= C) return;
  shift[c] = to_f32(pop_mean[c]);
  scale[c] = sqrtf(to_f32(pop_var[c]) + eps);
}

// ---- batch statistics in one pass -------------------------------------------------------------------
// Per-channel moments of the rows, without a first pass for the mean.  A thread subtracts a value of its own,
// the mean of its first kBatch rows (in the gradient, from kSettled rows on, the mean of those), from the rows it reads, so that
// what it adds up is of the size of the deviations however far the channel lies from zero; sets of rows are then merged pairwise (Chan, Golub and
// LeVeque: the sums of two sets around their own means, plus the product of the means' differences weighted
// n_a n_b / (n_a + n_b)), the difference of two means being that of the subtracted values plus that of what is
// left.  So a large mean enters no sum: in fp32 the variance is off by 6e-8 of itself at a mean of 1000 deviations
// (two passes 5e-8 to 1.5e-7, growing with the rows).  Threads, then slices of rows are merged in a fixed order.
// Bound by HBM: one pass over the tensors where sums around a mean that is known beforehand take two, and in
// the forward pass the one that writes the output.  Convolution, normalisation and ReLU in training, 64 x 28x28,
// 128 -> 256, f16: 128.0 us with sums that follow the mean, 122.6 here.
constexpr int kBatch = 4;          // rows a thread has in flight
constexpr float kSettled = 16.f;   // rows after which a thread subtracts their mean
constexpr int kMomentChannels = 4; // channels per thread: 8 or 16 bytes

// A set of rows: its means as hx + lx and hy + ly, sum (x - mean x)^2, sum (x - mean x)(dy - mean dy), and the
// sums as they are.  (The means of the results come from those: an infinity then stays one.)
template <bool DY>
struct Moments {
  static constexpr int N = DY ? 8 : 4;
  float v[N];  // hx, lx, sxx, sx, then hy, ly, sxy, sy
  // Adds a set of nb rows to one of na.
  __device__ __forceinline__ void merge(const Moments& b, float na, float nb) {
    if (na == 0.f) *this = b;
    if (na == 0.f || nb == 0.f) return;
    const float share = nb / (na + nb), weight = na * share;
    const float dx = (b.v[0] - v[0]) + (b.v[1] - v[1]);
    v[1] += dx * share;
    v[2] += b.v[2] + dx * dx * weight;
    v[3] += b.v[3];
    if constexpr (DY) {
      const float dy = (b.v[4] - v[4]) + (b.v[5] - v[5]);
      v[5] += dy * share;
      v[6] += b.v[6] + dx * dy * weight;
      v[7] += b.v[7];
    }
  }
};

template <typename T>
__device__ __forceinline__ void load_four(const T* p, float (&v)[kMomentChannels]) {
  if constexpr (sizeof(T) == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  } else {
    const uint2 q = *reinterpret_cast<const uint2*>(p);
    const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = to_f32(e[k]);
  }
}

// Block: 32 lanes x 4 channels, 8 row lanes; blockIdx.x the channel tile (the extent of a grid that has no practical
// limit), blockIdx.y the slice of rows.
// partial[slice][value of the set][c].  APPLY: the forward output is written on the way,
// out = (x - mean) / sqrt(var + eps) * gamma + beta with the given mean and variance.
template <typename T, bool DY, bool APPLY>
__global__ void __launch_bounds__(kBlock, kMomentBlocks)
    batchnorm_moments_kernel(const T* x, const T* dy, const T* beta,
                             const T* gamma, const T* mean, const T* var,
                             T* __restrict__ out, float* __restrict__ partial, size_t rows, int C, size_t rows_per_slice, float eps) {
  overlap_wait();
  constexpr int NC = kMomentChannels, NS = Moments<DY>::N;
  __shared__ float red[8][NS][NC][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = (blockIdx.x * 32 + tx) * NC;
  const size_t begin = (size_t)blockIdx.y * rows_per_slice;
  const size_t end = begin + rows_per_slice < rows ? begin + rows_per_slice : rows;
  // the subtracted values, and sums of d, d^2 and x (h, d h and dy), d = x - hx, h = dy - hy
  float hx[NC] = {}, s1[NC] = {}, s2[NC] = {}, sx[NC] = {}, hy[NC] = {}, t1[NC] = {}, sxy[NC] = {}, sy[NC] = {};
  float n = 0.f;
  if (c < C) {
    float am[NC], as[NC], ag[NC], ab[NC];
    if (APPLY) {
      load_four(mean + c, am);
      load_four(var + c, as);
      load_four(gamma + c, ag);
      load_four(beta + c, ab);
#pragma unroll
      for (int k = 0; k < NC; ++k) as[k] = 1.f / sqrtf(as[k] + eps);
    }
    auto apply = [&](const float (&v)[NC], T* to) {
      float o[NC];
#pragma unroll
      for (int k = 0; k < NC; ++k) o[k] = (v[k] - am[k]) * as[k] * ag[k] + ab[k];
      if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(to) = make_float4(o[0], o[1], o[2], o[3]);
      } else {
        uint2 q;
#pragma unroll
        for (int k = 0; k < NC; ++k) reinterpret_cast<T*>(&q)[k] = from_f32<T>(o[k]);
        *reinterpret_cast<uint2*>(to) = q;
      }
    };
    auto add = [&](int k, float xv, float gv) {
      const float d = xv - hx[k];
      s1[k] += d;
      s2[k] = fmaf(d, d, s2[k]);
      if (DY) {
        const float h = gv - hy[k];
        t1[k] += h;
        sxy[k] = fmaf(d, h, sxy[k]);
      }
    };
    // one offset moves through the tensors; eight rows further down is the row lane's next one
    size_t at = (begin + ty) * C + c;
    const unsigned next = 8u * (unsigned)C;
    int left = (int)(end - begin) - ty;  // rows from the lane's next one on
    auto batch = [&](auto first) {
      float xv[kBatch][NC], gv[kBatch][NC];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        load_four(x + at + (size_t)i * next, xv[i]);
        if (DY) load_four(dy + at + (size_t)i * next, gv[i]);
      }
      if (APPLY) {
#pragma unroll
        for (int i = 0; i < kBatch; ++i) apply(xv[i], out + at + (size_t)i * next);
      }
      if (decltype(first)::value && n == 0.f) {
        constexpr float inv_batch = 1.f / (float)kBatch;
#pragma unroll
        for (int k = 0; k < NC; ++k) {
          hx[k] = ((xv[0][k] + xv[1][k]) + (xv[2][k] + xv[3][k])) * inv_batch;
          if (DY) hy[k] = ((gv[0][k] + gv[1][k]) + (gv[2][k] + gv[3][k])) * inv_batch;
        }
      }
      static_assert(kBatch == 4, "sums of four");
#pragma unroll
      for (int k = 0; k < NC; ++k) {
#pragma unroll
        for (int i = 0; i < kBatch; ++i) add(k, xv[i][k], DY ? gv[i][k] : 0.f);
        sx[k] += (xv[0][k] + xv[1][k]) + (xv[2][k] + xv[3][k]);
        if (DY) sy[k] += (gv[0][k] + gv[1][k]) + (gv[2][k] + gv[3][k]);
      }
      n += (float)kBatch;
      left -= 8 * kBatch, at += (size_t)kBatch * next;
    };
    if constexpr (DY) {
#pragma unroll 1
      while (left > 8 * (kBatch - 1) && n < kSettled) batch(std::true_type{});
      if (n == kSettled && left > 0) {
        // From here on the sums are about the means of all rows so far.  Four rows leave a mean half a deviation off, and
        // the sum of n products 0.25 n off the one around the means: the gradient of gamma, a sum of random signs, showed its
        // rounding.  Relative error against float64, fp32, 100x56x56x256 / 128x56x56x64: 1.2e-6 / 8.6e-7 without, 4.0e-7 / 2.7e-7 so
        // (6.0e-7 / 5.7e-7 with two waves of blocks, whose threads have half the rows).
#pragma unroll
        for (int k = 0; k < NC; ++k) {
          const float ox = hx[k], oy = hy[k], px = ox + s1[k] * (1.f / kSettled), py = oy + t1[k] * (1.f / kSettled);
          const float mx = px - ox, my = py - oy;  // (what is added is what the new values differ by)
          if (!(fabsf(mx) < INFINITY && fabsf(my) < INFINITY)) continue;
          const float rx = fmaf(-kSettled, mx, s1[k]);
          s2[k] = fmaf(-mx, s1[k] + rx, s2[k]);
          sxy[k] = fmaf(-mx, t1[k], fmaf(-my, rx, sxy[k]));
          t1[k] = fmaf(-kSettled, my, t1[k]);
          s1[k] = rx, hx[k] = px, hy[k] = py;
        }
      }
#pragma unroll 1
      while (left > 8 * (kBatch - 1)) batch(std::false_type{});
    } else {
#pragma unroll 1
      while (left > 8 * (kBatch - 1)) batch(std::true_type{});
    }
    for (; left > 0; left -= 8, at += next) {
      float xv[NC], gv[NC];
      load_four(x + at, xv);
      if (DY) load_four(dy + at, gv);
      if (APPLY) apply(xv, out + at);
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        if (n == 0.f) {
          hx[k] = xv[k];
          if (DY) hy[k] = gv[k];
        }
        add(k, xv[k], DY ? gv[k] : 0.f);
        sx[k] += xv[k];
        if (DY) sy[k] += gv[k];
      }
      n += 1.f;
    }
  }
  const float inv_n = n > 0.f ? 1.f / n : 0.f;
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    const float lx = s1[k] * inv_n, sxx = fmaf(-s1[k], lx, s2[k]);
    red[ty][0][k][tx] = hx[k];
    red[ty][1][k][tx] = lx;
    red[ty][2][k][tx] = sxx < 0.f ? 0.f : sxx;  // (a NaN stays)
    red[ty][3][k][tx] = sx[k];
    if constexpr (DY) {
      const float ly = t1[k] * inv_n;
      red[ty][4][k][tx] = hy[k];
      red[ty][5][k][tx] = ly;
      red[ty][6][k][tx] = fmaf(-s1[k], ly, sxy[k]);
      red[ty][7][k][tx] = sy[k];
    }
  }
  __syncthreads();
  // thread (tx, k): channel c + k, its eight row lanes one after another
  if (ty < NC && c < C && begin < end) {
    const size_t here = end - begin;
    Moments<DY> t;
    float nt = 0.f;
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      if ((size_t)l >= here) break;
      const float nb = (float)((here - l + 7) / 8);
      Moments<DY> b;
#pragma unroll
      for (int i = 0; i < NS; ++i) b.v[i] = red[l][i][ty][tx];
      t.merge(b, nt, nb);
      nt += nb;
    }
    float* to = partial + (size_t)blockIdx.y * NS * C + c + ty;
#pragma unroll
    for (int i = 0; i < NS; ++i) to[(size_t)i * C] = t.v[i];
  }
}

// Merges the slices of a channel: 8 channels to a block, 64 threads to a channel.  Bound by latency: with four
// slices' values requested together, and a few slices to a thread, the block waits for L2 twice.
// A channel whose sums overflowed, or that holds an infinity, is added up again around its mean, row by row: the
// deviations of an infinite gradient and the like then come out as infinities or NaN by the formula itself,
// not by the way the rows were cut into sets.
// finish(c, moments): what becomes of channel c.
constexpr int kMergeChannels = 8, kMergeLanes = 64, kMergeWarps = kMergeChannels * kMergeLanes / 32;
template <typename T, bool DY, typename Finish>
__global__ void __launch_bounds__(kMergeChannels * kMergeLanes)
    batchnorm_merge_kernel(const float* partial, const T* x, const T* dy, int slices, int C,
                           size_t rows, size_t rows_per_slice, Finish finish) {
  overlap_wait();
  constexpr int NS = Moments<DY>::N;
  __shared__ float red[kMergeWarps][NS + 1][kMergeChannels];
  const int tx = threadIdx.x % kMergeChannels, ty = threadIdx.x / kMergeChannels, c = blockIdx.x * kMergeChannels + tx;
  Moments<DY> t{};
  float n = 0.f;
  if (c < C) {
#pragma unroll 1
    for (int s0 = ty; s0 < slices; s0 += 4 * kMergeLanes) {
      Moments<DY> b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float* at = partial + (size_t)min(s0 + kMergeLanes * i, slices - 1) * NS * C + c;
#pragma unroll
        for (int j = 0; j < NS; ++j) b[i].v[j] = at[(size_t)j * C];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int s = s0 + kMergeLanes * i;
        if (s >= slices) break;
        const size_t left = rows - (size_t)s * rows_per_slice;
        const float nb = (float)(left < rows_per_slice ? left : rows_per_slice);
        t.merge(b[i], n, nb);
        n += nb;
      }
    }
  }
  // neighbours first, the lower lane's set before the upper one's: the lanes of a warp that share a channel,
  // then the warps
  auto merge_down = [&](int o, bool here) {
    Moments<DY> b;
#pragma unroll
    for (int j = 0; j < NS; ++j) b.v[j] = __shfl_down_sync(0xFFFFFFFFu, t.v[j], o);
    const float nb = __shfl_down_sync(0xFFFFFFFFu, n, o);
    if (here) {
      t.merge(b, n, nb);
      n += nb;
    }
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = kMergeChannels; o < 32; o <<= 1) merge_down(o, (lane & (2 * o - kMergeChannels)) == 0);
  if (lane < kMergeChannels) {
#pragma unroll
    for (int j = 0; j < NS; ++j) red[warp][j][lane] = t.v[j];
    red[warp][NS][lane] = n;
  }
  __syncthreads();
  if (warp >= kMergeChannels) return;
  const int set = min(lane, kMergeWarps - 1);  // a lane takes a warp's set
#pragma unroll
  for (int j = 0; j < NS; ++j) t.v[j] = red[set][j][warp];
  n = red[set][NS][warp];
#pragma unroll
  for (int o = 1; o < kMergeWarps; o <<= 1) merge_down(o, (lane & (2 * o - 1)) == 0);
  const int mine = blockIdx.x * kMergeChannels + warp;
  if (mine >= C) return;
  const bool finite = fabsf(t.v[2]) <= FLT_MAX && (!DY || fabsf(t.v[NS - 2]) <= FLT_MAX);
  if (!__shfl_sync(0xFFFFFFFFu, (int)finite, 0)) {
    const float around = __shfl_sync(0xFFFFFFFFu, t.v[3], 0) / (float)rows;
    float a = 0.f, b = 0.f;
    for (size_t r = lane; r < rows; r += 32) {
      const float d = to_f32(x[r * C + mine]) - around;
      a += d * d;
      if (DY) b += to_f32(dy[r * C + mine]) * d;
    }
    t.v[2] = warp_sum(a);
    if (DY) t.v[NS - 2] = warp_sum(b);
  }
  if (lane == 0) finish(mine, t);
}

// Training forward: running = batch * (1 - m) + given * m.
template <typename T>
struct StoreRunning {
  const T *mean, *var;
  T *run_mean, *run_var;
  float rows, momentum;
  __device__ __forceinline__ void operator()(int c, const Moments<false>& t) const {
    run_mean[c] = from_f32<T>(t.v[3] / rows * (1.f - momentum) + to_f32(mean[c]) * momentum);
    run_var[c] = from_f32<T>(t.v[2] / rows * (1.f - momentum) + to_f32(var[c]) * momentum);
  }
};

// Training gradient: the parameters' gradients, and the per-channel terms its elementwise step reads.
template <typename T>
struct StoreGradStats {
  float4* terms;
  const T* gamma;
  T *beta_grad, *gamma_grad;
  float rows, eps;
  __device__ __forceinline__ void operator()(int c, const Moments<true>& t) const {
    const float variance = t.v[2] / rows, v = variance + eps;
    terms[c] = make_float4(t.v[3] / rows, t.v[7] / rows, t.v[6] / rows / v, to_f32(gamma[c]) / sqrtf(v));
    beta_grad[c] = from_f32<T>(t.v[7]);
    gamma_grad[c] = from_f32<T>(t.v[6] / sqrtf(variance + eps));
  }
};

// Slices of the moments kernel, a multiple of 32 rows each (whole batches of every row lane): one wave of three blocks per SM,
// all of which then end together, and half as many sets to merge as with two (us, forward / gradient, two waves / one: 64x28x28x256
// f16 16.1 / 12.8 and 36.3 / 32.8, 128x56x56x64 41.9 / 37.3 and 75.2 / 70.5).  No block more than that: one of a second wave
// takes as long as the first (64x28x28x2048 f16, 28 slices of 16 tiles for 444 places 119.5 and 209.6, 27 slices 84.4 and 172.9).
// `waves` 2: the forward pass in fp32 on tensors well beyond the L2 cache (30x56x56x640 90.3 in one, 84.6 in two; 110x24x24x752 73.8 / 69.7;
// 64x28x28x640, 128 MB, 48.5 / 50.4).
int moment_slices(size_t rows, int C, int sms, int waves, size_t* rows_per_slice) {
  const size_t ctiles = (size_t)(C + 32 * kMomentChannels - 1) / (32 * kMomentChannels);
  const size_t want = std::max<size_t>((size_t)sms * kMomentBlocks * waves / ctiles, 1);
  size_t per = (rows + want - 1) / want;
  per = (per + 8 * kBatch - 1) / (8 * kBatch) * (8 * kBatch);
  if (per < 64) per = 64;
  *rows_per_slice = per;
  return (int)((rows + per - 1) / per);
}

// Row slices of the per-channel reductions: enough blocks to fill the device a few times over
// (a block covers `block_channels` channels), at least 64 rows per slice.
int slices_for(size_t rows, int C, int sms, int block_channels) {
  const size_t ctiles = (size_t)(C + block_channels - 1) / block_channels;
  size_t want = ((size_t)sms * 8 + ctiles - 1) / ctiles;
  const size_t cap = (rows + 63) / 64;
  if (want > cap) want = cap;
  if (want < 1) want = 1;
  if (want > 4096) want = 4096;
  return (int)want;
}

// Grid of an elementwise packet kernel whose threads should keep their channels: the number of
// threads is made a multiple of the packets per pixel when that costs little, and no more of them than the
// device holds at once (blocks_per_sm), so that what a thread prepares for its channels serves several packets and no
// second wave is left over.  us, 8 blocks to an SM / as they fit: training gradient, three kernels, 64x28x28x256 f16 (3) 32.9 / 26.0,
// 128x56x56x64 69.7 / 62.1, f32 (4) 42.3 / 41.4; frozen forward (4) 8.4 / 7.0.  The frozen gradient is no better for it.
unsigned channel_stable_grid(size_t packets, int cvecs, int sms, unsigned blocks_per_sm) {
  unsigned grid = std::min(grid_for(packets, kBlock, sms), (unsigned)sms * blocks_per_sm);
  // threads = grid * kBlock must be a multiple of cvecs: grid a multiple of cvecs / gcd(cvecs, kBlock)
  int a = cvecs, b = kBlock;
  while (b != 0) {
    const int t = a % b;
    a = b;
    b = t;
  }
  const unsigned unit = (unsigned)(cvecs / a);
  // (a wave with room for no more than four units: several waves.  Training gradient, bf16, one wave whose threads change their
  // channels / threads that keep them, three kernels: 118x8x8x904 41.1 / 27.7, 29x10x10x1000 24.0 / 21.2)
  if (grid <= 4 * unit) grid = std::min(grid_for(packets, kBlock, sms), (unsigned)sms * (2048u / kBlock));
  if (unit > 1 && grid > 4 * unit) grid -= grid % unit;
  return grid;
}

bool params_ok(int batch, int rows, int cols, int channels) { return batch > 0 && rows > 0 && cols > 0 && channels > 0; }

// Scratch of one call: [partial: slices * 2 * C][stats0: 2C][stats1: 2C][shift: C][scale: C] floats.  terms: C float4 from
// the first 16-byte boundary of stats0 on, in the place of all that follows it (the training gradient in packets,
// which has no other statistics).
struct Scratch {
  float *partial, *stats0, *stats1, *shift, *scale;
  float4* terms;
  void* base;
};

int get_scratch(Scratch* sc, int slices, int C, cudaStream_t s) {
  const size_t floats = (size_t)slices * 2 * C + 6 * (size_t)C + 3;  // (terms begin up to three floats later)
  if (cudaMallocAsync(&sc->base, floats * sizeof(float), s) != cudaSuccess) {
    cudaGetLastError();
    return fail(PDNN_ALLOCATION_PROBLEM, "batchnorm: cannot allocate %zu bytes of scratch", floats * sizeof(float));
  }
  sc->partial = static_cast<float*>(sc->base);
  sc->stats0 = sc->partial + (size_t)slices * 2 * C;
  sc->stats1 = sc->stats0 + 2 * C;
  sc->shift = sc->stats1 + 2 * C;
  sc->scale = sc->shift + C;
  sc->terms = reinterpret_cast<float4*>((reinterpret_cast<uintptr_t>(sc->stats0) + 15) & ~(uintptr_t)15);
  return PDNN_OK;
}

}  // namespace

int launch_softmax(int direction, int dtype, const void* input, const void* gradient, void* output,
                   const PdnnSoftmaxParams& p, cudaStream_t s) {
  // validate_params, include/portdnn/softmax/launch.h:40-50
  if (!params_ok(p.batch, p.rows, p.cols, p.channels))
    return fail(PDNN_INVALID_PARAMETER, "softmax: batch, rows, cols and channels must be positive");
  if (p.input_format != 0) return fail(PDNN_INVALID_PARAMETER, "softmax: only NHWC is implemented");
  if (input == nullptr || output == nullptr || (direction == 1 && gradient == nullptr))
    return fail(PDNN_INVALID_PARAMETER, "softmax: null tensor");
  const int sms = device_sm_count();
  if (sms <= 0) return fail(PDNN_ALLOCATION_PROBLEM, "no CUDA device");
  const size_t rows = (size_t)p.batch * p.rows * p.cols;
  const unsigned grid = grid_for(rows * 32, kBlock, sms);
  return dispatch(dtype, [&](auto tag) {
    using T = decltype(tag);
    constexpr int VN = Vec16<T>::N;
    const bool vec = p.channels % VN == 0 && aligned16(input) && aligned16(output);
    if (direction == 0 && vec && p.channels <= 32 * VN)
      launch_overlapped(softmax_forward_vec_kernel<T, VN, 1>, grid, kBlock, s, static_cast<const T*>(input),
                        static_cast<T*>(output), rows, p.channels);
    else if (direction == 0 && vec && p.channels <= kSoftmaxRow * VN && softmax_by_rows(rows, p.channels / VN, VN == 8, sms))
      launch_overlapped(softmax_forward_row_kernel<T, VN>, (unsigned)rows, kSoftmaxRow, s, static_cast<const T*>(input),
                        static_cast<T*>(output), p.channels);
    else if (direction == 0 && vec && p.channels <= 128 * VN)
      launch_overlapped(softmax_forward_vec_kernel<T, VN, 4>, grid, kBlock, s, static_cast<const T*>(input),
                        static_cast<T*>(output), rows, p.channels);
    else if (direction == 0)
      softmax_forward_kernel<T><<<grid, kBlock, 0, s>>>(static_cast<const T*>(input), static_cast<T*>(output), rows,
                                                        p.channels);
    else if (vec && aligned16(gradient) && p.channels <= 32 * VN)
      launch_overlapped(softmax_grad_vec_kernel<T, VN, 1>, grid, kBlock, s, static_cast<const T*>(input),
                        static_cast<const T*>(gradient), static_cast<T*>(output), rows, p.channels);
    else if (vec && aligned16(gradient) && p.channels <= 128 * VN)
      launch_overlapped(softmax_grad_vec_kernel<T, VN, 4>, grid, kBlock, s, static_cast<const T*>(input),
                        static_cast<const T*>(gradient), static_cast<T*>(output), rows, p.channels);
    else
      softmax_grad_kernel<T><<<grid, kBlock, 0, s>>>(static_cast<const T*>(input), static_cast<const T*>(gradient),
                                                     static_cast<T*>(output), rows, p.channels);
    return check_launch(direction == 0 ? "softmax forward" : "softmax gradient");
  });
}

int launch_batchnorm_forward(int dtype, const void* input, const void* beta, const void* gamma, const void* mean,
                             const void* variance, void* running_mean, void* running_variance, void* output,
                             const PdnnBatchNormParams& p, cudaStream_t s) {
  if (!params_ok(p.batch, p.rows, p.cols, p.channels))
    return fail(PDNN_INVALID_PARAMETER, "batchnorm: batch, rows, cols and channels must be positive");
  if (p.input_format != 0) return fail(PDNN_INVALID_PARAMETER, "batchnorm: only NHWC is implemented");
  if (!(p.epsilon > 0.f)) return fail(PDNN_INVALID_PARAMETER, "batchnorm: epsilon must be positive");
  if (input == nullptr || beta == nullptr || gamma == nullptr || mean == nullptr || variance == nullptr ||
      output == nullptr || (p.is_training && (running_mean == nullptr || running_variance == nullptr)))
    return fail(PDNN_INVALID_PARAMETER, "batchnorm: null tensor");
  const int sms = device_sm_count();
  if (sms <= 0) return fail(PDNN_ALLOCATION_PROBLEM, "no CUDA device");
  const size_t rows = (size_t)p.batch * p.rows * p.cols, n = rows * p.channels;
  const int C = p.channels;
  return dispatch(dtype, [&](auto tag) -> int {
    using T = decltype(tag);
    constexpr int VN = Vec16<T>::N;
    const bool vec = C % VN == 0 && aligned16(input) && aligned16(output) && aligned16(beta) && aligned16(gamma) &&
                     aligned16(mean) && aligned16(variance);
    if (vec && p.is_training) {
      // output, batch moments and running statistics in two kernels
      size_t per = 0;
      const int slices = moment_slices(rows, C, sms, sizeof(T) == 4 && 2 * n * sizeof(T) > 5 * kStreamedBytes ? 2 : 1, &per);
      Scratch sc;
      const int st = get_scratch(&sc, Moments<false>::N / 2 * slices, C, s);
      if (st != PDNN_OK) return st;
      const dim3 grid((unsigned)((C / kMomentChannels + 31) / 32), (unsigned)slices);
      const T *mt = static_cast<const T*>(mean), *vt = static_cast<const T*>(variance);
      launch_overlapped(batchnorm_moments_kernel<T, false, true>, grid, kBlock, s, static_cast<const T*>(input), nullptr,
                        static_cast<const T*>(beta), static_cast<const T*>(gamma), mt, vt, static_cast<T*>(output),
                        sc.partial, rows, C, per, p.epsilon);
      launch_overlapped(batchnorm_merge_kernel<T, false, StoreRunning<T>>, (C + kMergeChannels - 1) / kMergeChannels,
                        kMergeChannels * kMergeLanes, s, sc.partial, static_cast<const T*>(input), nullptr, slices, C, rows,
                        per,
                        StoreRunning<T>{mt, vt, static_cast<T*>(running_mean), static_cast<T*>(running_variance), (float)rows, p.momentum});
      count_launch();
      cudaFreeAsync(sc.base, s);
      return check_launch("batchnorm forward (training)");
    }
    if (vec)
      // (fp32 tensors that stream through L2 are ahead with two waves, us, one / two: 116x39x39x280 70.1 / 64.8, 43x82x82x112 45.7 / 43.5)
      launch_overlapped(batchnorm_apply_vec_kernel<T, VN>, channel_stable_grid(n / VN, C / VN, sms, VN == 4 && n * sizeof(T) > kStreamedBytes ? 2 * kApplyBlocks : kApplyBlocks), kBlock, s,
                        static_cast<const T*>(input), static_cast<const T*>(beta), static_cast<const T*>(gamma),
                        static_cast<const T*>(mean), static_cast<const T*>(variance), static_cast<T*>(output), n / VN, C,
                        p.epsilon);
    else
      batchnorm_apply_kernel<T><<<grid_for(n, kBlock, sms), kBlock, 0, s>>>(
          static_cast<const T*>(input), static_cast<const T*>(beta), static_cast<const T*>(gamma),
          static_cast<const T*>(mean), static_cast<const T*>(variance), static_cast<T*>(output), n, C, p.epsilon);
    int st = check_launch("batchnorm forward");
    if (st != PDNN_OK || !p.is_training) return st;
    // batch mean, then the biased batch variance around it, then the running statistics
    const int slices = slices_for(rows, C, sms, 32);
    const size_t per_slice = (rows + slices - 1) / slices;
    Scratch sc;
    st = get_scratch(&sc, slices, C, s);
    if (st != PDNN_OK) return st;
    const dim3 grid(slices, (C + 31) / 32);
    batchnorm_sums_kernel<T, 0><<<grid, kBlock, 0, s>>>(static_cast<const T*>(input), nullptr, nullptr, nullptr,
                                                       sc.partial, rows, C, per_slice);
    launch_column_sums(sc.partial, slices, 2 * (size_t)C, sms, s, StoreTotals{sc.stats0, C, (float)rows, (float)rows});
    batchnorm_sums_kernel<T, 1><<<grid, kBlock, 0, s>>>(static_cast<const T*>(input), nullptr, sc.stats0, nullptr,
                                                       sc.partial, rows, C, per_slice);
    launch_column_sums(sc.partial, slices, 2 * (size_t)C, sms, s, StoreTotals{sc.stats1, C, (float)rows, 1.f});
    batchnorm_running_kernel<T><<<(C + kBlock - 1) / kBlock, kBlock, 0, s>>>(
        sc.stats0, sc.stats1, static_cast<const T*>(mean), static_cast<const T*>(variance),
        static_cast<T*>(running_mean), static_cast<T*>(running_variance), C, p.momentum);
    st = check_launch("batchnorm forward (batch statistics)");
    count_launch(4);
    cudaFreeAsync(sc.base, s);
    return st;
  });
}

int launch_batchnorm_gradient(int dtype, const void* input, const void* gradient, const void* gamma,
                              const void* pop_mean, const void* pop_variance, void* beta_grad, void* gamma_grad,
                              void* output, const PdnnBatchNormParams& p, cudaStream_t s) {
  if (!params_ok(p.batch, p.rows, p.cols, p.channels))
    return fail(PDNN_INVALID_PARAMETER, "batchnorm: batch, rows, cols and channels must be positive");
  if (p.input_format != 0) return fail(PDNN_INVALID_PARAMETER, "batchnorm: only NHWC is implemented");
  if (!(p.epsilon > 0.f)) return fail(PDNN_INVALID_PARAMETER, "batchnorm: epsilon must be positive");
  if (input == nullptr || gradient == nullptr || gamma == nullptr || beta_grad == nullptr || gamma_grad == nullptr ||
      output == nullptr || (!p.is_training && (pop_mean == nullptr || pop_variance == nullptr)))
    return fail(PDNN_INVALID_PARAMETER, "batchnorm gradient: null tensor");
  const int sms = device_sm_count();
  if (sms <= 0) return fail(PDNN_ALLOCATION_PROBLEM, "no CUDA device");
  const size_t rows = (size_t)p.batch * p.rows * p.cols, n = rows * p.channels;
  const int C = p.channels;
  return dispatch(dtype, [&](auto tag) -> int {
    using T = decltype(tag);
    constexpr int VN = Vec16<T>::N;
    const bool vec = C % VN == 0 && aligned16(input) && aligned16(gradient) && aligned16(output) && aligned16(gamma) &&
                     (p.is_training || aligned16(pop_variance));
    const bool one_pass = vec && p.is_training;
    size_t per_slice = 0;
    const int slices = one_pass ? moment_slices(rows, C, sms, 1, &per_slice) : slices_for(rows, C, sms, vec ? 32 * VN : 32);
    if (!one_pass) per_slice = (rows + slices - 1) / slices;
    Scratch sc;
    int st = get_scratch(&sc, one_pass ? Moments<true>::N / 2 * slices : slices, C, s);
    if (st != PDNN_OK) return st;
    const dim3 grid(slices, (C + 31) / 32), vgrid(slices, (C / VN + 31) / 32);
    const unsigned c1grid = (C + kBlock - 1) / kBlock;
    const T *x = static_cast<const T*>(input), *dy = static_cast<const T*>(gradient), *g = static_cast<const T*>(gamma);
    if (one_pass) {
      const dim3 mgrid((unsigned)((C / kMomentChannels + 31) / 32), (unsigned)slices);
      launch_overlapped(batchnorm_moments_kernel<T, true, false>, mgrid, kBlock, s, x, dy, nullptr, nullptr, nullptr,
                        nullptr, nullptr, sc.partial, rows, C, per_slice, 0.f);
      launch_overlapped(batchnorm_merge_kernel<T, true, StoreGradStats<T>>, (C + kMergeChannels - 1) / kMergeChannels,
                        kMergeChannels * kMergeLanes, s, sc.partial, x, dy, slices, C, rows, per_slice,
                        StoreGradStats<T>{sc.terms, g, static_cast<T*>(beta_grad), static_cast<T*>(gamma_grad), (float)rows, p.epsilon});
      launch_overlapped(batchnorm_grad_training_vec_kernel<T, VN>, channel_stable_grid(n / VN, C / VN, sms, gradient_blocks(VN)), kBlock, s, x,
                        dy, static_cast<const float4*>(sc.terms), static_cast<T*>(output), n / VN, C);
      count_launch(2);
      cudaFreeAsync(sc.base, s);
      return check_launch("batchnorm gradient (training)");
    }
    if (p.is_training) {
      batchnorm_sums_kernel<T, 0><<<grid, kBlock, 0, s>>>(x, dy, nullptr, nullptr, sc.partial, rows, C, per_slice);
      launch_column_sums(sc.partial, slices, 2 * (size_t)C, sms, s, StoreTotals{sc.stats0, C, (float)rows, (float)rows});
      batchnorm_sums_kernel<T, 1><<<grid, kBlock, 0, s>>>(x, dy, sc.stats0, nullptr, sc.partial, rows, C, per_slice);
      launch_column_sums(sc.partial, slices, 2 * (size_t)C, sms, s, StoreTotals{sc.stats1, C, (float)rows, 1.f});
      batchnorm_grad_training_kernel<T><<<grid_for(n, kBlock, sms), kBlock, 0, s>>>(
          x, dy, g, sc.stats0, sc.stats1, static_cast<T*>(output), n, C, (float)rows, p.epsilon);
      count_launch(4);
    } else {
      batchnorm_prepare_frozen_kernel<T><<<c1grid, kBlock, 0, s>>>(static_cast<const T*>(pop_mean),
                                                                 static_cast<const T*>(pop_variance), sc.shift, sc.scale,
                                                                 C, p.epsilon);
      if (vec) batchnorm_frozen_sums_vec_kernel<T, VN><<<vgrid, kBlock, 0, s>>>(x, dy, sc.shift, sc.scale, sc.partial, rows, C, per_slice);
      else batchnorm_sums_kernel<T, 2><<<grid, kBlock, 0, s>>>(x, dy, sc.shift, sc.scale, sc.partial, rows, C, per_slice);
      launch_column_sums(sc.partial, slices, 2 * (size_t)C, sms, s, StoreTotals{sc.stats0, C, 1.f, 1.f});
      if (vec)
        batchnorm_grad_frozen_vec_kernel<T, VN><<<channel_stable_grid(n / VN, C / VN, sms, 2048 / kBlock), kBlock, 0, s>>>(
            dy, g, static_cast<const T*>(pop_variance), static_cast<T*>(output), n / VN, C, p.epsilon);
      else
        batchnorm_grad_frozen_kernel<T><<<grid_for(n, kBlock, sms), kBlock, 0, s>>>(
            dy, g, static_cast<const T*>(pop_variance), static_cast<T*>(output), n, C, p.epsilon);
      count_launch(3);
    }
    batchnorm_param_grads_kernel<T><<<c1grid, kBlock, 0, s>>>(sc.stats0, sc.stats1, static_cast<T*>(beta_grad),
                                                             static_cast<T*>(gamma_grad), C, (float)rows, p.epsilon,
                                                             p.is_training);
    st = check_launch("batchnorm gradient");
    cudaFreeAsync(sc.base, s);
    return st;
  });
}

}  // namespace pdnn
