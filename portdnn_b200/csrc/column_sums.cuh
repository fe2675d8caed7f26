// Second stage of the split reductions (filter gradients over pixel splits or slices, batch statistics
// over row slices): the columns of a rows x n fp32 matrix of partial sums are added in a fixed order.
#pragma once

#include "common.cuh"

namespace pdnn {
namespace {

constexpr int kSumLanes = 32;  // row lanes of a block: 32 columns x 32 lanes
constexpr int kSumFlat = 256;  // threads of a block without row lanes

// Bound by latency: the matrix is in L2 and a thread that walks a column alone waits for one load after
// another (784 x 512 sums of batch statistics: 60 us on two blocks).  Here a block takes 32 columns with
// 32 threads to a column, each with four loads in flight, and adds the 32 partial results in order through
// shared memory: 60 -> 3.4 us, 444 x 1296 (depthwise filter gradient) 20 -> 3.3 us.
// finish(i, sum): what becomes of column i.
template <typename Finish>
__global__ void __launch_bounds__(32 * kSumLanes)
    column_sums_kernel(const float* __restrict__ m, int rows, size_t n, Finish finish) {
  __shared__ float red[kSumLanes][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (size_t first = (size_t)blockIdx.x * 32; first < n; first += (size_t)gridDim.x * 32) {
    const size_t i = first + tx;
    float sum = 0.f;
    if (i < n) {
      int r = ty;
      for (; r + 3 * kSumLanes < rows; r += 4 * kSumLanes) {
        const float a = __ldg(m + (size_t)r * n + i), b = __ldg(m + (size_t)(r + kSumLanes) * n + i);
        const float c = __ldg(m + (size_t)(r + 2 * kSumLanes) * n + i), d = __ldg(m + (size_t)(r + 3 * kSumLanes) * n + i);
        sum += (a + b) + (c + d);
      }
      for (; r < rows; r += kSumLanes) sum += __ldg(m + (size_t)r * n + i);
    }
    red[ty][tx] = sum;
    __syncthreads();
    // warp ty adds the lanes of column ty
    float v = red[tx][ty];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if (tx == 0 && first + ty < n) finish(first + ty, v);
    __syncthreads();
  }
}

// One thread per column, for matrices of few rows or so many columns that they fill the device.
template <typename Finish>
__global__ void __launch_bounds__(kSumFlat)
    column_sums_flat_kernel(const float* __restrict__ m, int rows, size_t n, Finish finish) {
  for (size_t i = (size_t)blockIdx.x * kSumFlat + threadIdx.x; i < n; i += (size_t)gridDim.x * kSumFlat) {
    float sum = 0.f;
#pragma unroll 4
    for (int r = 0; r < rows; ++r) sum += __ldg(m + (size_t)r * n + i);
    finish(i, sum);
  }
}

// Row lanes pay as soon as a column has more rows than a thread has loads in flight; a matrix of
// several columns for every thread the device holds (sms * 2048) is bound by its bytes either way.
template <typename Finish>
void launch_column_sums(const float* m, int rows, size_t n, int sms, cudaStream_t s, Finish finish) {
  if (rows <= 8 || n > (size_t)sms * 8192)
    column_sums_flat_kernel<<<grid_for(n, kSumFlat, sms), kSumFlat, 0, s>>>(m, rows, n, finish);
  else
    column_sums_kernel<<<grid_for(n, 32, sms), 32 * kSumLanes, 0, s>>>(m, rows, n, finish);
}

// The plain finish: out[i] = sum, or out[i] += sum.
template <typename T>
struct StoreSum {
  T* out;
  bool accumulate;
  __device__ __forceinline__ void operator()(size_t i, float sum) const {
    out[i] = from_f32<T>(accumulate ? to_f32(out[i]) + sum : sum);
  }
};

}  // namespace
}  // namespace pdnn
