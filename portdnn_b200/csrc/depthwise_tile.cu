// Depthwise 3x3 convolutions, all three passes, on tiles that TMA brings into shared memory.
#include "column_sums.cuh"
#include "depthwise_tile.cuh"
#include "tc_gemm.cuh"
#include "umma.cuh"

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace pdnn {

using namespace umma;

namespace {

// ---- a 32-bit word of channels in fp32 -----------------------------------------------------------
// One fp32 channel, or two 16-bit ones as a pair that the packed multiply-add takes in one instruction.  (The
// product of two 16-bit values is exact in fp32, so a packed multiply-add rounds once, as fmaf does.)
template <typename T>
struct Lanes {
  static constexpr int E = 2;
  using V = unsigned long long;
  static __device__ __forceinline__ V zero() { return 0ull; }
  static __device__ __forceinline__ V unpack(unsigned w);
  static __device__ __forceinline__ unsigned pack(V v);
  static __device__ __forceinline__ void fma(V& acc, V a, V b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
  static __device__ __forceinline__ void add(V& acc, V a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(a)); }
  static __device__ __forceinline__ float get(V v, int e) { return __uint_as_float(e ? (unsigned)(v >> 32) : (unsigned)v); }
};
template <>
__device__ __forceinline__ unsigned long long Lanes<__half>::unpack(unsigned w) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(f.x), "f"(f.y));
  return v;
}
template <>
__device__ __forceinline__ unsigned long long Lanes<__nv_bfloat16>::unpack(unsigned w) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(w << 16), "r"(w & 0xFFFF0000u));
  return v;
}
template <>
__device__ __forceinline__ unsigned Lanes<__half>::pack(unsigned long long v) {
  const __half2 h = __floats2half2_rn(__uint_as_float((unsigned)v), __uint_as_float((unsigned)(v >> 32)));
  return *reinterpret_cast<const unsigned*>(&h);
}
template <>
__device__ __forceinline__ unsigned Lanes<__nv_bfloat16>::pack(unsigned long long v) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float((unsigned)v), __uint_as_float((unsigned)(v >> 32)));
  return *reinterpret_cast<const unsigned*>(&h);
}
template <>
struct Lanes<float> {
  static constexpr int E = 1;
  using V = float;
  static __device__ __forceinline__ V zero() { return 0.f; }
  static __device__ __forceinline__ V unpack(unsigned w) { return __uint_as_float(w); }
  static __device__ __forceinline__ unsigned pack(V v) { return __float_as_uint(v); }
  static __device__ __forceinline__ void fma(V& acc, V a, V b) { acc = fmaf(a, b, acc); }
  static __device__ __forceinline__ void add(V& acc, V a) { acc += a; }
  static __device__ __forceinline__ float get(V v, int) { return v; }
};

// Two fp16 channels summed in fp16, tap by tile column, as window3_strip_kernel does: the same bits.
struct HalfSums {
  static constexpr int E = 2;
  using V = __half2;
  static __device__ __forceinline__ V zero() { return __float2half2_rn(0.f); }
  static __device__ __forceinline__ V unpack(unsigned w) { return *reinterpret_cast<const __half2*>(&w); }
  static __device__ __forceinline__ unsigned pack(V v) { return *reinterpret_cast<const unsigned*>(&v); }
  static __device__ __forceinline__ void fma(V& acc, V a, V b) { acc = __hfma2(a, b, acc); }
  static __device__ __forceinline__ float get(V v, int e) { return e ? __high2float(v) : __low2float(v); }
};

// One block to an SM.  Filter gradient, us, 128 images, f16, 56x56x144 / 112x112x32 / 28x28x192 / 7x7x960: two blocks of
// two stages of 54 KB 67 / 47 / 22 / 16, one block of three of 72 KB 49 / 45 / 21 / 13, four of 54 KB 57 / 49 / 22 /
// 13: larger tiles read fewer rows twice, and a block's stages are filled one after another, not in bursts.
constexpr int kTileThreads = 512;            // most threads that multiply; one warp more requests the tiles
constexpr int kTileStages = 3;
constexpr int kTileStageBytes = 72 * 1024;
constexpr unsigned kTileHead = 128;          // barriers and the abort flag

struct Tiles {
  int words, strips;       // 32-bit words of channels to a block, strips of two output rows
  int chunks, slices;      // blocks along the channels, blocks that share the tiles of a chunk
  int tw, tiles_w, tiles_h;
  unsigned tiles;          // of one chunk: tiles_w * tiles_h * images
  int channels, in_rows, in_cols, out_rows, out_cols, pad_rows, pad_cols;
  int mirrored;            // the filter's taps in reverse order (input gradient)
  int down;                // the last images first (reads_from_the_end)
  unsigned x_bytes, dy_off, dy_bytes, stage_bytes;
  unsigned* error_record;
};

// dW[r][s][c] = sum of x[h * ST + r][w * ST + s][c] * dy[h][w][c].  What bounds the nine multiply-adds per word
// is everything around them: loads, conversions and bounds checks (56x56x144, 128 images, f16: 71 million warp
// instructions with the rows in registers, 24 million here).  A warp of its own has TMA bring tiles of TW columns x
// 2 * strips rows with their halo, zeros outside the image, so that the multiplying warps check nothing and only read
// shared memory; a thread owns a word of channels and a strip of two output rows, walks the columns of the tile with
// a window of 3 columns x (ST + 3) rows in registers, converts every word once, and multiplies two channels to an
// instruction.  Its 9 sums are taken tile by tile and added up in registers over the tiles of the block (one chain of up
// to 1800 products had four times the error: 56x56x144, 128 images, fp32, products of random sign, 7.5e-7 -> 1.9e-7 of the
// root of the number of terms, at the same time); the block's partial sums go to partial[slice][tap][channel].  What is left is the bytes: 5.3 TB/s of the
// tensors, 5.8 with the halo.
// us with the second stage, before / now, 128 images, f16: 56x56x144 86 / 44, 112x112x96 / 2 85 / 60, 112x112x32 69 / 42,
// 14x14x384 20 / 13, 7x7x960 19 / 14.
template <typename T, int ST, int TW>
__global__ void __launch_bounds__(kTileThreads + 32, 1)
    depthwise_filter_tile_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap dy_map,
                                 const unsigned* x, const unsigned* dy, float* partial, const Tiles g) {
  using L = Lanes<T>;
  using V = typename L::V;
  constexpr int E = L::E, XW = (TW - 1) * ST + 3, ROWS = ST + 3;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 127u) & ~127u;
  uint8_t* smem = smem_raw + (base - raw);
  const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = (int)(threadIdx.x & 31);
  const int workers = (int)(blockDim.x >> 5) - 1;  // warps that multiply; the last one requests
  auto full_bar = [&](int s) { return base + 8u * (uint32_t)s; };
  auto empty_bar = [&](int s) { return base + 8u * (uint32_t)(kTileStages + s); };
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 16 * kTileStages);
  if (threadIdx.x < 2 * kTileStages) {
    mbar_init(base + 8u * threadIdx.x, threadIdx.x < kTileStages ? 1u : (unsigned)workers);
    if (threadIdx.x == 0) *abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();
  overlap_wait();
  const int chunk = (int)blockIdx.x % g.chunks, slice = (int)blockIdx.x / g.chunks;
  const int words = g.words, strips = g.strips;
  const int word = (int)threadIdx.x % words, strip = (int)threadIdx.x / words;
  const bool live = strip < strips && warp < workers;
  V acc[9];
#pragma unroll
  for (int t = 0; t < 9; ++t) acc[t] = L::zero();

  int s = 0;
  uint32_t ph = 0;
  if (warp == workers) {
    if (lane == 0) {
      prefetch_tensormap(&x_map);
      prefetch_tensormap(&dy_map);
    }
#pragma unroll 1
    for (unsigned tile = (unsigned)slice; tile < g.tiles; tile += (unsigned)g.slices) {
      const int tw = (int)(tile % (unsigned)g.tiles_w);
      const unsigned rest = tile / (unsigned)g.tiles_w;
      const int w0 = tw * TW, h0 = (int)(rest % (unsigned)g.tiles_h) * 2 * strips, n = (int)(rest / (unsigned)g.tiles_h);
      if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, g.error_record, kWaitLimitNs, 0x1500u + (unsigned)s)) break;
      const uint32_t at = base + kTileHead + (uint32_t)s * g.stage_bytes;
      warp_arrive_expect_tx(full_bar(s), g.x_bytes + g.dy_bytes);
      warp_tma_load_4d(at, &x_map, full_bar(s), chunk * words * E, w0 * ST - g.pad_cols, h0 * ST - g.pad_rows, n);
      warp_tma_load_4d(at + g.dy_off, &dy_map, full_bar(s), chunk * words * E, w0, h0, n);
      if (++s == kTileStages) {
        s = 0;
        ph ^= 1u;
      }
    }
  } else {
    const int row = XW * words;  // words of a row of the x tile
#pragma unroll 1
    for (unsigned tile = (unsigned)slice; tile < g.tiles; tile += (unsigned)g.slices) {
      if (!mbar_wait(full_bar(s), ph, abort_flag, g.error_record, kWaitLimitNs, 0x1600u + (unsigned)s)) break;
      if (live) {
        const uint8_t* at = smem + kTileHead + (size_t)s * g.stage_bytes;
        const unsigned* xp = reinterpret_cast<const unsigned*>(at) + 2 * ST * strip * row + word;
        const unsigned* dp = reinterpret_cast<const unsigned*>(at + g.dy_off) + 2 * strip * TW * words + word;
        const int tw = (int)(tile % (unsigned)g.tiles_w), th = (int)(tile / (unsigned)g.tiles_w % (unsigned)g.tiles_h);
        const int cols_left = g.out_cols - tw * TW, rows_left = g.out_rows - 2 * (th * strips + strip);
        V sum[9];  // of this tile
#pragma unroll
        for (int t = 0; t < 9; ++t) sum[t] = L::zero();
        auto walk = [&](auto whole) {  // (false: without the products of outputs that do not exist)
          V win[3][ROWS];  // column c of the tile in win[c % 3]
#pragma unroll
          for (int c = 0; c < 3 - ST; ++c)
#pragma unroll
            for (int r = 0; r < ROWS; ++r) win[c][r] = L::unpack(xp[r * row + c * words]);
#pragma unroll
          for (int j = 0; j < TW; ++j) {
#pragma unroll
            for (int c = j * ST + 3 - ST; c < j * ST + 3; ++c)
#pragma unroll
              for (int r = 0; r < ROWS; ++r) win[c % 3][r] = L::unpack(xp[r * row + c * words]);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const V d = L::unpack(dp[(k * TW + j) * words]);
              if (!decltype(whole)::value && (j >= cols_left || k >= rows_left)) continue;
#pragma unroll
              for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c) L::fma(sum[r * 3 + c], win[(j * ST + c) % 3][k * ST + r], d);
            }
          }
        };
        if (cols_left >= TW && rows_left >= 2) walk(std::true_type{});
        else walk(std::false_type{});
#pragma unroll
        for (int t = 0; t < 9; ++t) L::add(acc[t], sum[t]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty_bar(s));
      if (++s == kTileStages) {
        s = 0;
        ph ^= 1u;
      }
    }
  }
  // The zeros that stand for pixels outside the image and for outputs that do not exist are no terms of the sums, and
  // make NaNs of infinities: a thread with a NaN takes its products once more, from memory and only those that there are.
  // (56x56x144, 128 images, f16: 43.5 us, and 1060 with a NaN in every sum.  A look at every tile's sums while it is in
  // shared memory took 48.5 us without any, a second walk over the tiles 48.9 and 300, loads in batches here, or a
  // function of its own, 45.4 and 810, 46.2 and 620: the sums of a network that works come first.)
  V all[9];  // their sum is a NaN if one of them is
#pragma unroll
  for (int t = 0; t < 9; ++t) all[t] = acc[t];
#pragma unroll
  for (int step = 1; step < 9; step *= 2)
#pragma unroll
    for (int t = 0; t + step < 9; t += 2 * step) L::add(all[t], all[t + step]);
  const int pixel_words = g.channels / E, channel_word = chunk * words + word;
  if ((isnan(L::get(all[0], 0)) || isnan(L::get(all[0], E - 1))) && live && channel_word < pixel_words) {
#pragma unroll
    for (int t = 0; t < 9; ++t) acc[t] = L::zero();
#pragma unroll 1
    for (unsigned tile = (unsigned)slice; tile < g.tiles; tile += (unsigned)g.slices) {
      const unsigned rest = tile / (unsigned)g.tiles_w;
      const int w0 = (int)(tile % (unsigned)g.tiles_w) * TW, n = (int)(rest / (unsigned)g.tiles_h);
      const int h0 = 2 * ((int)(rest % (unsigned)g.tiles_h) * strips + strip);
      V sum[9];
#pragma unroll
      for (int t = 0; t < 9; ++t) sum[t] = L::zero();
#pragma unroll 1
      for (int j = 0; j < min(TW, g.out_cols - w0); ++j)
#pragma unroll 1
        for (int k = 0; k < min(2, g.out_rows - h0); ++k) {
          const V d = L::unpack(dy[(((size_t)n * g.out_rows + h0 + k) * g.out_cols + w0 + j) * pixel_words + channel_word]);
#pragma unroll
          for (int t = 0; t < 9; ++t) {
            const int ih = (h0 + k) * ST - g.pad_rows + t / 3, iw = (w0 + j) * ST - g.pad_cols + t % 3;
            if (ih >= 0 && ih < g.in_rows && iw >= 0 && iw < g.in_cols)
              L::fma(sum[t], L::unpack(x[(((size_t)n * g.in_rows + ih) * g.in_cols + iw) * pixel_words + channel_word]), d);
          }
        }
#pragma unroll
      for (int t = 0; t < 9; ++t) L::add(acc[t], sum[t]);
    }
  }
  __syncthreads();
  if (*abort_flag) {  // copies already requested may still be landing in shared memory
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) {
    }
    return;
  }
  // the block's strips in a fixed order; every tile has been read, its place takes the sums
  float* red = reinterpret_cast<float*>(smem + kTileHead);
  if (live) {
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
      for (int e = 0; e < E; ++e) red[((t * strips + strip) * words + word) * E + e] = L::get(acc[t], e);
  }
  __syncthreads();
  const int cols = words * E;
  for (int i = (int)threadIdx.x; i < 9 * cols; i += (int)blockDim.x) {
    const int t = i / cols, col = i - t * cols, ch = chunk * cols + col;
    if (ch >= g.channels) continue;
    float sum = 0.f;
    for (int k = 0; k < strips; ++k) sum += red[(t * strips + k) * cols + col];
    partial[((size_t)slice * 9 + t) * g.channels + ch] = sum;
  }
}

// Forward pass, and the input gradient of stride 1 as the forward pass of dy with the filter mirrored and the padding
// complemented, on the same tiles and walk: nine multiply-adds in fp32 to a pair of channels, one rounding.  Bound by
// HBM; one thread to an output packet with nine loads of it, as these layers ran before, by the loads.  bf16, us, 128
// images: 56x56x144 forward 184 -> 44, input gradient 285 -> 44; 112x112x96 / 2 forward 134 -> 64; 7x7x960 20 -> 8.5.
// fp16 sums in fp16 (HalfSums), against the strips of depthwise3_async_kernel, whose 111 instructions to a 16-byte packet -
// copies, slots, addresses - are twice what is left here; us, strips / tiles: 128 images 112x112x32 43.7 / 35.1, 56x56x144 45.9 /
// 40.2 (5.8 TB/s), 14x14x576 16.3 / 11.9, 7x7x960 9.7 / 7.5; 64 images 112x112x96 / 2 38.5 / 34.2, 28x28x192 10.3 / 9.2.
// (fp32 has the strips.)
template <typename T, typename L, int ST, int TW>
__global__ void __launch_bounds__(kTileThreads + 32, 1)
    depthwise_forward_tile_kernel(const __grid_constant__ CUtensorMap x_map, const T* filter, T* out, const Tiles g) {
  using V = typename L::V;
  constexpr int E = L::E, XW = (TW - 1) * ST + 3, ROWS = ST + 3;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 127u) & ~127u;
  uint8_t* smem = smem_raw + (base - raw);
  const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = (int)(threadIdx.x & 31);
  const int workers = (int)(blockDim.x >> 5) - 1;
  auto full_bar = [&](int s) { return base + 8u * (uint32_t)s; };
  auto empty_bar = [&](int s) { return base + 8u * (uint32_t)(kTileStages + s); };
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 16 * kTileStages);
  if (threadIdx.x < 2 * kTileStages) {
    mbar_init(base + 8u * threadIdx.x, threadIdx.x < kTileStages ? 1u : (unsigned)workers);
    if (threadIdx.x == 0) *abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();
  overlap_wait();
  const int chunk = (int)blockIdx.x % g.chunks, slice = (int)blockIdx.x / g.chunks;
  const int words = g.words, strips = g.strips;
  const int word = (int)threadIdx.x % words, strip = (int)threadIdx.x / words;
  const int pixel_words = g.channels / E, channel_word = chunk * words + word;

  int s = 0;
  uint32_t ph = 0;
  if (warp == workers) {
    if (lane == 0) prefetch_tensormap(&x_map);
#pragma unroll 1
    for (unsigned i = (unsigned)slice; i < g.tiles; i += (unsigned)g.slices) {
      const unsigned tile = g.down ? g.tiles - 1u - i : i;
      const int tw = (int)(tile % (unsigned)g.tiles_w);
      const unsigned rest = tile / (unsigned)g.tiles_w;
      const int w0 = tw * TW, h0 = (int)(rest % (unsigned)g.tiles_h) * 2 * strips, n = (int)(rest / (unsigned)g.tiles_h);
      if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, g.error_record, kWaitLimitNs, 0x1700u + (unsigned)s)) break;
      warp_arrive_expect_tx(full_bar(s), g.x_bytes);
      warp_tma_load_4d(base + kTileHead + (uint32_t)s * g.stage_bytes, &x_map, full_bar(s), chunk * words * E, w0 * ST - g.pad_cols,
                       h0 * ST - g.pad_rows, n);
      if (++s == kTileStages) {
        s = 0;
        ph ^= 1u;
      }
    }
  } else {
    const bool live = strip < strips && channel_word < pixel_words;
    V f[9];
    bool finite = true;
#pragma unroll
    for (int t = 0; t < 9; ++t) {
      f[t] = live ? L::unpack(reinterpret_cast<const unsigned*>(filter)[(g.mirrored ? 8 - t : t) * pixel_words + channel_word]) : L::zero();
#pragma unroll
      for (int e = 0; e < E; ++e) finite = finite && isfinite(L::get(f[t], e));
    }
    const int row = XW * words;
    const size_t image_words = (size_t)g.out_rows * g.out_cols * pixel_words;
#pragma unroll 1
    for (unsigned i = (unsigned)slice; i < g.tiles; i += (unsigned)g.slices) {
      const unsigned tile = g.down ? g.tiles - 1u - i : i;
      if (!mbar_wait(full_bar(s), ph, abort_flag, g.error_record, kWaitLimitNs, 0x1800u + (unsigned)s)) break;
      const int tw = (int)(tile % (unsigned)g.tiles_w);
      const unsigned rest = tile / (unsigned)g.tiles_w;
      const int w0 = tw * TW, h0 = ((int)(rest % (unsigned)g.tiles_h) * strips + strip) * 2, n = (int)(rest / (unsigned)g.tiles_h);
      if (live && h0 < g.out_rows) {
        const unsigned* xp = reinterpret_cast<const unsigned*>(smem + kTileHead + (size_t)s * g.stage_bytes) + 2 * ST * strip * row + word;
        unsigned* yp = reinterpret_cast<unsigned*>(out) + (size_t)n * image_words + ((size_t)h0 * g.out_cols + w0) * pixel_words + channel_word;
        const int cols_left = g.out_cols - w0, y_row = g.out_cols * pixel_words;
        const bool second = h0 + 1 < g.out_rows;
        auto walk = [&](auto every_tap) {
          V win[3][ROWS];  // column c of the tile in win[c % 3]
#pragma unroll
          for (int c = 0; c < 3 - ST; ++c)
#pragma unroll
            for (int r = 0; r < ROWS; ++r) win[c][r] = L::unpack(xp[r * row + c * words]);
#pragma unroll
          for (int j = 0; j < TW; ++j) {
#pragma unroll
            for (int c = j * ST + 3 - ST; c < j * ST + 3; ++c)
#pragma unroll
              for (int r = 0; r < ROWS; ++r) win[c % 3][r] = L::unpack(xp[r * row + c * words]);
            if (j < cols_left) {
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                V acc = L::zero();
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                  constexpr bool by_column = std::is_same<L, HalfSums>::value;
                  const int r = by_column ? t % 3 : t / 3, c = by_column ? t / 3 : t % 3;
                  // a tap outside the image is no term of the sum: the zero there and an infinite weight would be one
                  if (!decltype(every_tap)::value) {
                    const int ih = (h0 + k) * ST - g.pad_rows + r, iw = (w0 + j) * ST - g.pad_cols + c;
                    if (ih < 0 || ih >= g.in_rows || iw < 0 || iw >= g.in_cols) continue;
                  }
                  L::fma(acc, win[(j * ST + c) % 3][k * ST + r], f[r * 3 + c]);
                }
                if (k == 0 || second) yp[k * y_row + j * pixel_words] = L::pack(acc);
              }
            }
          }
        };
        if (finite) walk(std::true_type{});
        else walk(std::false_type{});
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty_bar(s));
      if (++s == kTileStages) {
        s = 0;
        ph ^= 1u;
      }
    }
  }
  __syncthreads();
  if (*abort_flag) {  // copies already requested may still be landing in shared memory
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) {
    }
  }
}

int up(int v, int to) { return (v + to - 1) / to * to; }

// Words and strips of a block: the split of the channels into equal chunks (of whole 16-byte packets, for TMA) and
// of the rows into equal tiles that takes the least time by the estimate below, with tiles of at most
// kTileStageBytes.  p: the geometry as the walk sees it; filter_gradient: a stage holds a tile of dy, too.
bool plan_tiles(const PdnnDepthwiseConv2DParams& p, int elems, bool filter_gradient, Tiles* out) {
  const int sms = device_sm_count(), total = p.channels / elems, row_pairs = (p.out_rows + 1) / 2, st = p.stride_rows;
  // 14 columns (the sizes of networks for 224 x 224 pixels are its multiples) or 8, whichever leaves less of the last
  // tile empty; two columns of the window are read again for every tile.  56x56x144, 128 images: 44 and 49 us; 7x7x960: 19 and 13.
  const int tw = st == 2 ? 4 : (p.out_cols + 13) / 14 * 16 < (p.out_cols + 7) / 8 * 10 ? 14 : 8;
  const int xw = (tw - 1) * st + 3;
  double best = 1e30;
  for (int chunks = 1; chunks <= total / 4; ++chunks) {
    const int words = up((total + chunks - 1) / chunks, 4);
    if (words > 256 / elems || (chunks - 1) * words >= total) continue;  // (a box has at most 256 elements)
    if (words < 16 && chunks > 1) break;  // rows of less than 64 bytes: only where a pixel has no more
    auto bytes = [&](int strips) {
      const int x = up(((2 * strips - 1) * st + 3) * xw * words * 4, 128);
      return filter_gradient ? up(x + 2 * strips * tw * words * 4, 128) : x;
    };
    int most = std::min(kTileThreads / words, row_pairs);
    while (most > 1 && (bytes(most) > kTileStageBytes || (2 * most - 1) * st + 3 > 256)) --most;
    if (most < 1 || bytes(most) > kTileStageBytes) continue;
    const int slices = std::max(1, sms / chunks), least_h = (row_pairs + most - 1) / most;
    for (int tiles_h = least_h; tiles_h <= std::min(8 * least_h, row_pairs); tiles_h *= 2) {
      const int strips = (row_pairs + tiles_h - 1) / tiles_h;
      const long long tiles = (long long)((p.out_cols + tw - 1) / tw) * tiles_h * p.batch;
      // tiles one block after another works off, each its warps' instructions and what a tile costs besides (about six
      // warps' worth: its barriers, the first reads), and the rows above and below a tile that are read again
      const double rounds = tiles > 8ll * slices ? (double)tiles / slices : (double)((tiles + slices - 1) / slices);
      // (rows of a box that are no multiple of 64 bytes share their memory sectors with the next chunk's block)
      const double split_rows = chunks == 1 || words % 16 == 0 ? 1.0 : words % 8 == 0 ? 1.08 : 1.15;
      const double cost = rounds * (up(words * strips, 32) / 32 + 6) * (1.0 + 0.1 / strips) * split_rows;
      if (cost < best - 1e-9) {
        best = cost;
        out->words = words;
        out->strips = strips;
        out->chunks = chunks;
        out->tiles_h = (row_pairs + strips - 1) / strips;
        out->x_bytes = (unsigned)(((2 * strips - 1) * st + 3) * xw * words * 4);
        out->dy_bytes = (unsigned)(2 * strips * tw * words * 4);
        out->dy_off = (unsigned)up((int)out->x_bytes, 128);
        out->stage_bytes = (unsigned)bytes(strips);
      }
    }
  }
  if (best > 1e29) return false;
  out->tw = tw;
  out->tiles_w = (p.out_cols + tw - 1) / tw;
  const unsigned long long tiles = (unsigned long long)out->tiles_w * out->tiles_h * p.batch;
  if (tiles > 0x3FFFFFFFull) return false;
  out->tiles = (unsigned)tiles;
  out->channels = p.channels;
  out->in_rows = p.in_rows;
  out->in_cols = p.in_cols;
  out->out_rows = p.out_rows;
  out->out_cols = p.out_cols;
  out->pad_rows = p.pad_rows;
  out->pad_cols = p.pad_cols;
  out->mirrored = out->down = 0;
  out->error_record = tc_error_record_address();
  return out->error_record != nullptr;
}

bool tile_layer(const PdnnDepthwiseConv2DParams& p, int es) {
  return p.window_rows == 3 && p.window_cols == 3 && p.channel_multiplier == 1 && p.stride_rows == p.stride_cols && p.stride_rows <= 2 &&
         p.channels * es % 16 == 0;
}

bool x_tile_map(CUtensorMap* map, int dtype, const void* x, const PdnnDepthwiseConv2DParams& p, const Tiles& g, int elems) {
  const int st = p.stride_rows;
  const uint32_t box[4] = {(uint32_t)(g.words * elems), (uint32_t)((g.tw - 1) * st + 3), (uint32_t)((2 * g.strips - 1) * st + 3), 1};
  return tc_dense_nhwc_map(map, dtype, x, p.batch, p.in_rows, p.in_cols, p.channels, box);
}

template <typename... Params>
bool opt_in(void (*kernel)(Params...), std::mutex& mu, bool (&done)[kMaxDevices]) {
  const int dev = current_device();
  if (dev < 0 || dev >= kMaxDevices) return false;
  std::lock_guard<std::mutex> lock(mu);
  if (!done[dev]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 256 + kTileStages * kTileStageBytes) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    done[dev] = true;
  }
  return true;
}

template <typename... Params, typename... Args>
bool launch_tiles(void (*kernel)(Params...), const Tiles& g, size_t least_smem, cudaStream_t s, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(g.slices * g.chunks));
  cfg.blockDim = dim3((unsigned)up(g.words * g.strips, 32) + 32);
  cfg.dynamicSmemBytes = 128 + kTileHead + std::max((size_t)kTileStages * g.stage_bytes, least_smem);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess;
}

template <typename T, int ST, int TW>
int launch_filter_tiles(const CUtensorMap& x_map, const CUtensorMap& dy_map, const void* x, const void* dy, float* partial,
                        const Tiles& g, cudaStream_t s) {
  static std::mutex mu;
  static bool done[kMaxDevices] = {};
  if (!opt_in(depthwise_filter_tile_kernel<T, ST, TW>, mu, done)) return 0;
  const size_t sums = (size_t)9 * g.words * g.strips * Lanes<T>::E * 4;
  launch_tiles(depthwise_filter_tile_kernel<T, ST, TW>, g, sums, s, x_map, dy_map, static_cast<const unsigned*>(x),
               static_cast<const unsigned*>(dy), partial, g);  // (the caller's check_launch() reads the error)
  return g.slices;
}

template <typename T, typename L, int ST, int TW>
bool launch_forward_tiles(const CUtensorMap& x_map, const void* filter, void* out, const Tiles& g, cudaStream_t s) {
  static std::mutex mu;
  static bool done[kMaxDevices] = {};
  if (!opt_in(depthwise_forward_tile_kernel<T, L, ST, TW>, mu, done)) return false;
  launch_tiles(depthwise_forward_tile_kernel<T, L, ST, TW>, g, 0, s, x_map, static_cast<const T*>(filter), static_cast<T*>(out), g);
  return true;
}

// f(stride, columns) as integral constants
template <typename F>
auto with_tile_shape(int stride, int tw, F f) {
  if (stride == 2) return f(std::integral_constant<int, 2>{}, std::integral_constant<int, 4>{});
  if (tw == 14) return f(std::integral_constant<int, 1>{}, std::integral_constant<int, 14>{});
  return f(std::integral_constant<int, 1>{}, std::integral_constant<int, 8>{});
}

}  // namespace

int launch_depthwise_filter_tiles(int dtype, const void* x, const void* dy, float* partial, const PdnnDepthwiseConv2DParams& p,
                                  int max_slices, cudaStream_t s) {
  const int es = (int)dtype_size(dtype), elems = 4 / es;
  Tiles g;
  if (!tile_layer(p, es) || !aligned16(x) || !aligned16(dy) || !plan_tiles(p, elems, true, &g)) return 0;
  // Few tiles leave all but a few SMs idle, which the kernel that spreads rows over warps does not (3 images, 7x7x960:
  // 8.1 us on three tiles, 7.2 there; 4 images, 14x14x384, eight tiles: 6.6 and 8.3).
  if (g.tiles < 8) return 0;
  g.slices = std::max(1, std::min<int>({max_slices, device_sm_count() / g.chunks, (int)std::min<unsigned>(g.tiles, 1u << 20)}));
  const uint32_t dy_box[4] = {(uint32_t)(g.words * elems), (uint32_t)g.tw, (uint32_t)(2 * g.strips), 1};
  CUtensorMap x_map, dy_map;
  if (!x_tile_map(&x_map, dtype, x, p, g, elems) ||
      !tc_dense_nhwc_map(&dy_map, dtype, dy, p.batch, p.out_rows, p.out_cols, p.channels, dy_box))
    return 0;
  return with_tile_shape(p.stride_rows, g.tw, [&](auto st, auto tw) {
    constexpr int ST = decltype(st)::value, TW = decltype(tw)::value;
    return dtype == PDNN_F32   ? launch_filter_tiles<float, ST, TW>(x_map, dy_map, x, dy, partial, g, s)
           : dtype == PDNN_F16 ? launch_filter_tiles<__half, ST, TW>(x_map, dy_map, x, dy, partial, g, s)
                               : launch_filter_tiles<__nv_bfloat16, ST, TW>(x_map, dy_map, x, dy, partial, g, s);
  });
}

bool launch_depthwise_forward_tiles(int dtype, const void* x, const void* filter, void* out, const PdnnDepthwiseConv2DParams& p,
                                    bool mirrored, cudaStream_t s) {
  Tiles g;
  if (!tile_layer(p, 2) || !aligned16(x) || !aligned16(filter) || !aligned16(out) || !plan_tiles(p, 2, false, &g)) return false;
  // (offsets in a strip's two rows are 32-bit words in an int: in 64 bits 56x56x144, 128 images, took 44.4 us, not 43.2)
  if ((long long)p.out_cols * p.channels > 0x7FFFFFFFll) return false;
  g.mirrored = mirrored ? 1 : 0;
  g.down = reads_from_the_end((size_t)p.batch * p.in_rows * p.in_cols * p.channels * 2);
  g.slices = std::max(1, std::min<int>(device_sm_count() / g.chunks, (int)std::min<unsigned>(g.tiles, 1u << 20)));
  CUtensorMap x_map;
  if (!x_tile_map(&x_map, dtype, x, p, g, 2)) return false;
  return with_tile_shape(p.stride_rows, g.tw, [&](auto st, auto tw) {
    constexpr int ST = decltype(st)::value, TW = decltype(tw)::value;
    return dtype == PDNN_F16 ? launch_forward_tiles<__half, HalfSums, ST, TW>(x_map, filter, out, g, s)
                             : launch_forward_tiles<__nv_bfloat16, Lanes<__nv_bfloat16>, ST, TW>(x_map, filter, out, g, s);
  });
}

}  // namespace pdnn
