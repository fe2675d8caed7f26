// Depthwise 3x3 filter gradient on tiles that TMA brings into shared memory.
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
  static __device__ __forceinline__ void fma(V& acc, V a, V b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
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
struct Lanes<float> {
  static constexpr int E = 1;
  using V = float;
  static __device__ __forceinline__ V zero() { return 0.f; }
  static __device__ __forceinline__ V unpack(unsigned w) { return __uint_as_float(w); }
  static __device__ __forceinline__ void fma(V& acc, V a, V b) { acc = fmaf(a, b, acc); }
  static __device__ __forceinline__ float get(V v, int) { return v; }
};

constexpr int kTileThreads = 288;            // most threads that multiply; one warp more requests the tiles
constexpr int kTileStages = 2;
constexpr int kTileStageBytes = 54 * 1024;   // two blocks of two stages to an SM
constexpr unsigned kTileHead = 128;          // barriers and the abort flag
template <int ST>
struct TileCols { static constexpr int value = ST == 1 ? 8 : 4; };  // output columns of a tile

struct FilterTiles {
  int words, strips;       // 32-bit words of channels to a block, strips of two output rows
  int chunks, slices;      // blocks along the channels, blocks that share the tiles of a chunk
  int tiles_w, tiles_h;
  unsigned tiles;          // of one chunk: tiles_w * tiles_h * images
  int channels, out_rows, out_cols, pad_rows, pad_cols;
  unsigned x_bytes, dy_off, dy_bytes, stage_bytes;
  unsigned* error_record;
};

// dW[r][s][c] = sum of x[h * ST + r][w * ST + s][c] * dy[h][w][c].  What bounds the nine multiply-adds per word
// is everything around them: loads, conversions and bounds checks.  Here a
// warp of its own has TMA bring tiles of TW columns x 2 * strips rows with their halo, zeros outside the image, so
// that the multiplying warps check nothing and only read shared memory; a thread owns a word of channels and
// a strip of two output rows, walks the columns of the tile with a window of 3 columns x (ST + 3) rows in
// registers, converts every word once, and multiplies two channels to an instruction.  Its 9 sums stay in
// registers over all tiles of the block; the block's partial sums go to partial[slice][tap][channel].
template <typename T, int ST>
__global__ void __launch_bounds__(kTileThreads + 32, 2)
    depthwise_filter_tile_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap dy_map,
                                 float* partial, const FilterTiles g) {
  using L = Lanes<T>;
  using V = typename L::V;
  constexpr int E = L::E, TW = TileCols<ST>::value, XW = (TW - 1) * ST + 3, ROWS = ST + 3;
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
        auto walk = [&](auto whole) {
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
              // (where there is no such output, the zero that stands for dy meets values of x that are not its own:
              // an infinity among them must not become a NaN)
              if (!decltype(whole)::value && (j >= cols_left || k >= rows_left)) continue;
#pragma unroll
              for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c) L::fma(acc[r * 3 + c], win[(j * ST + c) % 3][k * ST + r], d);
            }
          }
        };
        if (cols_left >= TW && rows_left >= 2) walk(std::true_type{});
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

int up(int v, int to) { return (v + to - 1) / to * to; }

// Words and strips of a block: the split of the channels into equal chunks (of whole 16-byte packets, for TMA) and
// of the rows into equal tiles that leaves the fewest threads without work, with tiles of at most
// kTileStageBytes.
bool plan_filter_tiles(const PdnnDepthwiseConv2DParams& p, int elems, FilterTiles* out) {
  const int total = p.channels / elems, row_pairs = (p.out_rows + 1) / 2, st = p.stride_rows;
  const int tw = st == 1 ? TileCols<1>::value : TileCols<2>::value, xw = (tw - 1) * st + 3;
  double best = 1e30;
  for (int chunks = 1; chunks <= total / 4; ++chunks) {
    const int words = up((total + chunks - 1) / chunks, 4);
    if (words > 256 / elems || (chunks - 1) * words >= total) continue;  // (a box has at most 256 elements)
    if (words < 16 && chunks > 1) break;  // rows of less than 64 bytes: only where a pixel has no more
    auto bytes = [&](int strips) {
      const int x = up(((2 * strips - 1) * st + 3) * xw * words * 4, 128);
      return up(x + 2 * strips * tw * words * 4, 128);
    };
    int most = std::min(kTileThreads / words, row_pairs);
    while (most > 1 && (bytes(most) > kTileStageBytes || (2 * most - 1) * st + 3 > 256)) --most;
    if (most < 1 || bytes(most) > kTileStageBytes) continue;
    const int tiles_h = (row_pairs + most - 1) / most, strips = (row_pairs + tiles_h - 1) / tiles_h;
    // thread slots spent on a column of the image, and the rows above and below a tile that are read again
    const double cost = (double)chunks * tiles_h * (up(words * strips, 32) + 32) * (1.0 + 0.1 / strips);
    if (cost < best - 1e-9) {
      best = cost;
      out->words = words;
      out->strips = strips;
      out->chunks = chunks;
      out->tiles_h = tiles_h;
      out->x_bytes = (unsigned)(((2 * strips - 1) * st + 3) * xw * words * 4);
      out->dy_bytes = (unsigned)(2 * strips * tw * words * 4);
      out->dy_off = (unsigned)up((int)out->x_bytes, 128);
      out->stage_bytes = (unsigned)bytes(strips);
    }
  }
  if (best > 1e29) return false;
  out->tiles_w = (p.out_cols + tw - 1) / tw;
  const unsigned long long tiles = (unsigned long long)out->tiles_w * out->tiles_h * p.batch;
  if (tiles > 0x3FFFFFFFull) return false;
  out->tiles = (unsigned)tiles;
  out->channels = p.channels;
  out->out_rows = p.out_rows;
  out->out_cols = p.out_cols;
  out->pad_rows = p.pad_rows;
  out->pad_cols = p.pad_cols;
  return true;
}

template <typename T, int ST>
int launch_filter_tiles(const CUtensorMap& x_map, const CUtensorMap& dy_map, float* partial, const FilterTiles& g, cudaStream_t s) {
  auto kernel = depthwise_filter_tile_kernel<T, ST>;
  const size_t sums = (size_t)9 * g.words * g.strips * Lanes<T>::E * 4;
  const size_t smem = 128 + kTileHead + std::max((size_t)kTileStages * g.stage_bytes, sums);
  {
    static std::mutex mu;
    static bool opted_in[kMaxDevices] = {};
    const int dev = current_device();
    if (dev < 0 || dev >= kMaxDevices) return 0;
    std::lock_guard<std::mutex> lock(mu);
    if (!opted_in[dev]) {
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 256 + kTileStages * kTileStageBytes) != cudaSuccess) {
        cudaGetLastError();
        return 0;
      }
      opted_in[dev] = true;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(g.slices * g.chunks));
  cfg.blockDim = dim3((unsigned)up(g.words * g.strips, 32) + 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, x_map, dy_map, partial, g);  // (the caller's check_launch() reads the error)
  return g.slices;
}

}  // namespace

int launch_depthwise_filter_tiles(int dtype, const void* x, const void* dy, float* partial, const PdnnDepthwiseConv2DParams& p,
                                  int max_slices, cudaStream_t s) {
  const int es = (int)dtype_size(dtype), elems = 4 / es;
  if (p.window_rows != 3 || p.window_cols != 3 || p.channel_multiplier != 1 || p.stride_rows != p.stride_cols || p.stride_rows > 2 ||
      p.channels * es % 16 != 0 || !aligned16(x) || !aligned16(dy))
    return 0;
  FilterTiles g;
  if (!plan_filter_tiles(p, elems, &g)) return 0;
  g.error_record = tc_error_record_address();
  if (g.error_record == nullptr) return 0;
  const int st = p.stride_rows, tw = st == 1 ? TileCols<1>::value : TileCols<2>::value;
  // two blocks to an SM, all channels of a tile side by side
  g.slices = std::max(1, std::min<int>({max_slices, 2 * device_sm_count() / g.chunks, (int)std::min<unsigned>(g.tiles, 1u << 20)}));
  const uint32_t x_box[4] = {(uint32_t)(g.words * elems), (uint32_t)((tw - 1) * st + 3), (uint32_t)((2 * g.strips - 1) * st + 3), 1};
  const uint32_t dy_box[4] = {(uint32_t)(g.words * elems), (uint32_t)tw, (uint32_t)(2 * g.strips), 1};
  CUtensorMap x_map, dy_map;
  if (!tc_dense_nhwc_map(&x_map, dtype, x, p.batch, p.in_rows, p.in_cols, p.channels, x_box) ||
      !tc_dense_nhwc_map(&dy_map, dtype, dy, p.batch, p.out_rows, p.out_cols, p.channels, dy_box))
    return 0;
  if (dtype == PDNN_F32)
    return st == 1 ? launch_filter_tiles<float, 1>(x_map, dy_map, partial, g, s) : launch_filter_tiles<float, 2>(x_map, dy_map, partial, g, s);
  if (dtype == PDNN_F16)
    return st == 1 ? launch_filter_tiles<__half, 1>(x_map, dy_map, partial, g, s) : launch_filter_tiles<__half, 2>(x_map, dy_map, partial, g, s);
  return st == 1 ? launch_filter_tiles<__nv_bfloat16, 1>(x_map, dy_map, partial, g, s)
                 : launch_filter_tiles<__nv_bfloat16, 2>(x_map, dy_map, partial, g, s);
}

}  // namespace pdnn
