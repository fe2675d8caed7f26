// Second stage of the split reductions (filter gradients over pixel splits or slices; batch statistics over row
// slices where the tensors are not in 16-byte packets, and with frozen parameters): the columns of a
// rows x n fp32 matrix of partial sums are added in a fixed order.
#pragma once

#include "common.cuh"

namespace pdnn {
namespace {

constexpr int kSumFlat = 256;  // threads of a block without row lanes

// Bound by latency: the matrix is in L2 and a thread that walks a column alone waits for one load after
// another.  Here a block takes 32 columns with LANES (8 or 32) threads to a column, each with four loads
// in flight, and adds their results through shared memory, in a fixed order.  Four sums of 784 x 512 of a batch
// normalisation, on two blocks before: 36 us less each; depthwise filter gradient of 56x56x144 at 128 images
// (444 x 1296): 8 us less.
// finish(i, sum): what becomes of column i.
template <int LANES, typename Finish>
__global__ void __launch_bounds__(32 * LANES)
    column_sums_kernel(const float* m, int rows, size_t n, Finish finish) {
  overlap_wait();
  __shared__ float red[LANES][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (size_t first = (size_t)blockIdx.x * 32; first < n; first += (size_t)gridDim.x * 32) {
    const size_t i = first + tx;
    float sum = 0.f;
    if (i < n) {
      int r = ty;
      for (; r + 3 * LANES < rows; r += 4 * LANES) {
        const float a = m[(size_t)r * n + i], b = m[(size_t)(r + LANES) * n + i];
        const float c = m[(size_t)(r + 2 * LANES) * n + i], d = m[(size_t)(r + 3 * LANES) * n + i];
        sum += (a + b) + (c + d);
      }
      float rest[3];  // the last ones requested together, too (7x45x61 104 -> 152 3x3 filter gradient: 40.8 -> 39.0 us)
#pragma unroll
      for (int u = 0; u < 3; ++u) rest[u] = r + u * LANES < rows ? m[(size_t)(r + u * LANES) * n + i] : 0.f;
#pragma unroll
      for (int u = 0; u < 3; ++u)
        if (r + u * LANES < rows) sum += rest[u];
    }
    red[ty][tx] = sum;
    __syncthreads();
    // LANES neighbouring threads add the lanes of a column
    const int col = (int)threadIdx.x / LANES;
    float v = red[(int)threadIdx.x % LANES][col];
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if ((int)threadIdx.x % LANES == 0 && first + col < n) finish(first + col, v);
    __syncthreads();
  }
}

// One thread per column, for matrices of few rows or so many columns that they fill the device.
template <typename Finish>
__global__ void __launch_bounds__(kSumFlat)
    column_sums_flat_kernel(const float* m, int rows, size_t n, Finish finish) {
  overlap_wait();
  for (size_t i = (size_t)blockIdx.x * kSumFlat + threadIdx.x; i < n; i += (size_t)gridDim.x * kSumFlat) {
    float sum = 0.f;
#pragma unroll 8
    for (int r = 0; r < rows; ++r) sum += m[(size_t)r * n + i];
    finish(i, sum);
  }
}

// Row lanes pay where one thread per column leaves the device idle and a column has more rows than a
// thread has loads in flight; 32 of them where there are few columns or many rows, so that a thread keeps
// rows of its own to add.
template <typename Finish>
void launch_column_sums(const float* m, int rows, size_t n, int sms, cudaStream_t s, Finish finish) {
  if (rows <= 8 || n >= (size_t)sms * 1024)
    launch_overlapped(column_sums_flat_kernel<Finish>, grid_for(n, kSumFlat, sms), kSumFlat, s, m, rows, n, finish);
  else if (rows >= 256 || n < 4096)
    launch_overlapped(column_sums_kernel<32, Finish>, grid_for(n, 32, sms), 32 * 32, s, m, rows, n, finish);
  else
    launch_overlapped(column_sums_kernel<8, Finish>, grid_for(n, 32, sms), 32 * 8, s, m, rows, n, finish);
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
