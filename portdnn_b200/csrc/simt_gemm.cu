// Matrix products and convolutions in fp32 arithmetic on the CUDA cores, for what the tensor-core kernels cannot tile: fp32
// convolutions whose channel or feature count is not a multiple of 4, small 16-bit layers of odd counts, and
// products whose rows are not whole 16-byte packets.  The products are fp32 multiply-adds, as in the kernels of one thread
// per output (direct_conv.cu, simt_matmul_kernel), so the results are theirs but for the order of the sums.
//
// Those kernels load two words for each multiply-add and walk a sum in one thread.  Here a block of 256 threads
// takes a tile of BM x BN outputs, four rows by four columns to a thread, and the operands pass through shared
// memory sixteen terms at a time, the next sixteen being on their way in registers meanwhile: 8 words of shared memory for
// 16 multiply-adds, two to an instruction.  Where the tiles are fewer than the device takes, up to
// eight blocks of a cluster share the terms of a tile and add up their sums through distributed shared memory, in the
// order of the terms; a filter gradient that is one long sum is also cut into slices, added up by a second launch.
#include "simt_gemm.cuh"

#include <cooperative_groups.h>

#include "column_sums.cuh"

namespace pdnn {
namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 256;
constexpr int kTerms = 16;     // terms of a step
constexpr int kOutputs = 4096;  // of a tile
constexpr int kMaxSplits = 8;   // portable cluster size
constexpr int kBlocksPerSm = 3;

// How the terms of a sum are found.
enum ATerms {
  kRows = 0,    // a row of A is one or several runs of neighbouring terms: a product's row, the taps of a pixel
  kPixels = 1,  // a term is a pixel, a row a tap and a channel: filter gradients
  kColumns = 2  // A is stored transposed
};

struct SimtArgs {
  const void *a, *b, *bias;
  void* out;
  float* partial;  // where not null: sums of slices instead of results
  long long a_batch, b_batch, out_batch;
  int n, inner;      // columns; terms of a run
  int lda;           // kRows of a product, kColumns
  int bs, bk, bn;    // strides of B: tap, term, column
  long long om, on;  // strides of the output: row, column
  // Rows of A that are pixels: a pixel of the grid rows x cols (of batch images) with phases of step pixels, its runs at
  // (ah + dir * i, aw + dir * j) of the tensor that is read.
  int batch, rows, cols, m;
  int a_rows, a_cols, a_channels, dir;
  int step_rows, step_cols, pad_rows, pad_cols, window_rows, window_cols;
  int conv, m_tiles, n_tiles, splits, slices;
  int misses;  // some tap of some pixel lies outside the tensor that is read
  int act, staged;  // staged: the epilogue rounds to the tensors' type between its steps, as the direct kernel does
  float alpha, beta;
  int out_f32;
};

template <typename T>
__device__ __forceinline__ float load(const void* p, long long at) {
  return to_f32(static_cast<const T*>(p)[at]);
}

// Two fp32 multiply-adds, each rounded once as fmaf() is, in one instruction.
__device__ __forceinline__ void fma_two(float2& c, float2 a, float2 b) {
  unsigned long long& to = reinterpret_cast<unsigned long long&>(c);
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(to)
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
}

// Bound by shared memory in large layers (28x45x61 101 -> 150 3x3 fp32: 85 % of its wavefronts, multiply-add pipe 52 %), by the latency
// of a step's loads in small ones.  Times of both
// this and a thread to an output: thread_to_an_output and simt_matmul_tiled.
template <typename T, int A, bool B_RUNS, int BN>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) simt_gemm_kernel(const SimtArgs g) {
  overlap_wait();
  constexpr int BM = kOutputs / BN, kLdA = BM + 4, kLdB = BN + 4;
  constexpr int kA = BM * kTerms / kThreads, kB = BN * kTerms / kThreads;  // elements a thread brings in a step
  constexpr bool kARuns = A == kRows;
  constexpr int kTiles = 2 * kTerms * (kLdA + kLdB);
  __shared__ __align__(16) float shared[kTiles > kOutputs ? kTiles : kOutputs];
  __shared__ int4 table[A == kRows ? BM : A == kPixels ? 2 * kTerms : 1];
  __shared__ int out_row[A == kRows ? BM : 1];  // of the pixel that is a row
  auto as = [&](int buf, int k) { return shared + (buf * kTerms + k) * kLdA; };
  auto bs = [&](int buf, int k) { return shared + 2 * kTerms * kLdA + (buf * kTerms + k) * kLdB; };
  const int t = threadIdx.x;

  unsigned id = blockIdx.x;
  const int rank = (int)(id % (unsigned)g.splits);
  id /= (unsigned)g.splits;
  const int m0 = (int)(id % (unsigned)g.m_tiles) * BM;
  id /= (unsigned)g.m_tiles;
  const int n0 = (int)(id % (unsigned)g.n_tiles) * BN;
  id /= (unsigned)g.n_tiles;
  const int slice = (int)(id % (unsigned)g.slices), outer = (int)(id / (unsigned)g.slices);  // a product of a batch, a phase

  const T* pa = static_cast<const T*>(g.a) + (g.conv ? 0 : outer * g.a_batch);
  const T* pb = static_cast<const T*>(g.b) + (g.conv ? 0 : outer * g.b_batch);
  // the taps that meet the pixels of this phase: first_r + step * i, first_s + step * j
  int M = g.m, runs_r = 1, runs_s = 1, first_r = 0, first_s = 0, rows = g.rows, cols = g.cols, phase_r = 0, phase_s = 0;
  if (A == kRows && g.conv) {
    if (g.dir < 0) {
      phase_r = outer / g.step_cols, phase_s = outer - phase_r * g.step_cols;
      rows = (g.rows - phase_r + g.step_rows - 1) / g.step_rows, cols = (g.cols - phase_s + g.step_cols - 1) / g.step_cols;
      first_r = (phase_r + g.pad_rows) % g.step_rows, first_s = (phase_s + g.pad_cols) % g.step_cols;
      runs_r = first_r < g.window_rows ? (g.window_rows - first_r + g.step_rows - 1) / g.step_rows : 0;
      runs_s = first_s < g.window_cols ? (g.window_cols - first_s + g.step_cols - 1) / g.step_cols : 0;
    } else {
      runs_r = g.window_rows, runs_s = g.window_cols;
    }
    M = g.batch * rows * cols;
  }
  if (m0 >= M) return;  // (a later phase is smaller; the whole cluster leaves)
  const int tap_r = g.dir < 0 ? g.step_rows : 1, tap_s = g.dir < 0 ? g.step_cols : 1;

  if (A == kRows) {
    for (int i = t; i < BM; i += kThreads) {
      int4 e = make_int4(0, -(1 << 30), 0, 0);  // base, row, column of the run of tap 0
      const int m = m0 + i;
      int o = m;
      if (m < M) {
        if (!g.conv) {
          e.x = m * g.lda, e.y = 0;
        } else {
          const int c = m % cols, rest = m / cols, r = rest % rows, n = rest / rows;
          if (g.dir > 0) {
            e.y = r * g.step_rows - g.pad_rows, e.z = c * g.step_cols - g.pad_cols;
          } else {
            e.y = (r * g.step_rows + phase_r + g.pad_rows - first_r) / g.step_rows;
            e.z = (c * g.step_cols + phase_s + g.pad_cols - first_s) / g.step_cols;
            o = (n * g.rows + r * g.step_rows + phase_r) * g.cols + c * g.step_cols + phase_s;
          }
          e.x = ((n * g.a_rows + e.y) * g.a_cols + e.z) * g.a_channels;
        }
      }
      table[i] = e, out_row[i] = o;
    }
    __syncthreads();
  }
  // where a row's run of tap (i, j) begins, or -1 where the tap misses the image
  auto run_at = [&](const int4& e, int i, int j) -> int {
    const int r = e.y + g.dir * i, c = e.z + g.dir * j;
    if ((unsigned)r >= (unsigned)g.a_rows || (unsigned)c >= (unsigned)g.a_cols) return -1;
    return e.x + g.dir * (i * g.a_cols + j) * g.a_channels;
  };
  // row and column of a pixel's window, and the element there
  auto pixel = [&](int p) -> int4 {
    int4 e = make_int4(0, -(1 << 30), 0, 0);
    if (p < g.inner) {
      const int c = p % g.cols, rest = p / g.cols, r = rest % g.rows, n = rest / g.rows;
      e.y = r * g.step_rows - g.pad_rows, e.z = c * g.step_cols - g.pad_cols;
      e.x = ((n * g.a_rows + e.y) * g.a_cols + e.z) * g.a_channels;
    }
    return e;
  };

  const int chunks = (g.inner + kTerms - 1) / kTerms, steps = runs_r * runs_s * chunks;
  const long long parts = (long long)g.splits * g.slices;
  auto part_at = [&](int part) { return (int)(steps * (long long)part / parts); };
  const int begin = part_at(slice * g.splits + rank), end = part_at(slice * g.splits + rank + 1);

  // the elements of A and B that this thread brings
  const int ak = kARuns ? t % kTerms : t / BM, am = kARuns ? t / kTerms : t % BM;
  const int bk = B_RUNS ? t % kTerms : t / BN, bn = B_RUNS ? t / kTerms : t % BN;
  constexpr int kStepA = kARuns ? kThreads / kTerms : kThreads / BM, kStepB = B_RUNS ? kThreads / kTerms : kThreads / BN;
  int tap_h = 0, tap_w = 0, tap_at = 0;  // kPixels: this thread's row of A
  bool row_ok = false;
  if (A == kPixels) {
    const int m = m0 + am;
    row_ok = m < M;
    const int c = m % g.a_channels, tap = m / g.a_channels;
    tap_h = tap / g.window_cols, tap_w = tap - tap_h * g.window_cols;
    tap_at = (tap_h * g.a_cols + tap_w) * g.a_channels + c;
  } else if (A == kColumns) {
    row_ok = m0 + am < M;
  }

  // the step that is fetched next
  int run, k0, ri, si;
  bool new_run;
  int at[kARuns ? kA : 1];
  int b_tap = 0;
  auto first_step = [&] {
    run = begin / max(chunks, 1), k0 = (begin - run * chunks) * kTerms;
    ri = runs_s > 0 ? run / runs_s : 0, si = run - ri * runs_s;
    new_run = true;
  };
  const int b_first = bk * g.bk + (n0 + bn) * g.bn, b_step = kStepB * (B_RUNS ? g.bn : g.bk);
  float ra[kA], rb[kB];
  unsigned inside = 0;  // which of ra are elements of the tensor
  auto fetch = [&](int buf) {
    if (new_run) {
      if constexpr (A == kRows) {
#pragma unroll
        for (int i = 0; i < kA; ++i) at[i] = run_at(table[am + i * kStepA], ri, si);
      }
      b_tap = ((first_r + ri * tap_r) * g.window_cols + first_s + si * tap_s) * g.bs;
      new_run = false;
    }
    if constexpr (A == kRows) {
      const bool k_ok = k0 + ak < g.inner;
      inside = 0;
#pragma unroll
      for (int i = 0; i < kA; ++i) {
        const bool ok = k_ok && at[i] >= 0;
        ra[i] = ok ? to_f32(pa[at[i] + k0 + ak]) : 0.f;
        inside |= (unsigned)ok << i;
      }
    } else if constexpr (A == kPixels) {
      inside = 0;
#pragma unroll
      for (int i = 0; i < kA; ++i) {
        const int4 e = table[buf * kTerms + ak + i * kStepA];
        const bool ok = row_ok && (unsigned)(e.y + tap_h) < (unsigned)g.a_rows && (unsigned)(e.z + tap_w) < (unsigned)g.a_cols;
        ra[i] = ok ? to_f32(pa[e.x + tap_at]) : 0.f;
        inside |= (unsigned)ok << i;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kA; ++i) {
        const int k = k0 + ak + i * kStepA;
        ra[i] = row_ok && k < g.inner ? to_f32(pa[k * g.lda + m0 + am]) : 0.f;
      }
    }
    const int b_at = b_tap + k0 * g.bk;
#pragma unroll
    for (int i = 0; i < kB; ++i) {
      const bool ok = k0 + bk + (B_RUNS ? 0 : i * kStepB) < g.inner && n0 + bn + (B_RUNS ? i * kStepB : 0) < g.n;
      rb[i] = ok ? to_f32(pb[b_at + b_first + i * b_step]) : 0.f;
    }
    k0 += kTerms;
    if (k0 >= g.inner) {
      k0 = 0, new_run = true;
      if (++si == runs_s) si = 0, ++ri;
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int i = 0; i < kA; ++i) {
      if (kARuns) as(buf, ak)[am + i * kStepA] = ra[i];
      else as(buf, ak + i * kStepA)[am] = ra[i];
    }
#pragma unroll
    for (int i = 0; i < kB; ++i) {
      if (B_RUNS) bs(buf, bk)[bn + i * kStepB] = rb[i];
      else bs(buf, bk + i * kStepB)[bn] = rb[i];
    }
  };
  // the pixels of a step, for everyone: written while the preceding step is computed, read in the next
  auto look_up = [&](int step) {
    if (A == kPixels && t < kTerms) table[(step & 1) * kTerms + t] = pixel(step * kTerms + t);
  };

  const int tm = t / (BN / 4), tn = t % (BN / 4);
  float2 acc[2][4] = {};  // rows tm * 4 + 2 i and the next, columns tn * 4 + j
  if (begin < end) {
    if (A == kPixels) {
      look_up(begin);
      look_up(begin + 1);
      __syncthreads();
    }
    first_step();
    fetch(begin & 1);
    put(0);
    __syncthreads();
    for (int step = begin; step < end; ++step) {
      const int buf = (step - begin) & 1;
      if (step + 1 < end) fetch((step + 1) & 1);
      look_up(step + 2);  // (the place of this step's pixels, which were read before the last barrier)
#pragma unroll 8
      for (int k = 0; k < kTerms; ++k) {
        const float4 av = *reinterpret_cast<const float4*>(as(buf, k) + tm * 4), bv = *reinterpret_cast<const float4*>(bs(buf, k) + tn * 4);
        const float2 a[2] = {make_float2(av.x, av.y), make_float2(av.z, av.w)};
        const float b[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) fma_two(acc[i][j], a[i], make_float2(b[j], b[j]));
      }
      if (step + 1 < end) put(buf ^ 1);
      __syncthreads();
    }
  }

  // A tap outside the image has no term, whatever the other operand is there, but the tiles multiply it by zero: a block with a
  // sum that is not a number forms its sums again from the terms that there are.  us, all numbers finite / one NaN in dy or the
  // filter, fp32, forward, input gradient, filter gradient: 24x60x61 66 -> 97 3x3 532 / 845, 599 / 892, 630 / 1176; when the thread that
  // stores a sum walked its terms alone, the NaN took 3564, 2886, 34876.
  if constexpr (A != kColumns) {
    if (g.misses) {
      bool bad = false;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) bad = bad || acc[i][j].x != acc[i][j].x || acc[i][j].y != acc[i][j].y;
      if (__syncthreads_or(bad)) {
        first_step();
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int step = begin; step < end; ++step) {
          look_up(step);
          __syncthreads();  // (everyone has read the step before)
          fetch(step & 1);
          put(0);
#pragma unroll
          for (int i = 0; i < kA; ++i) {  // where the elements are, in the second buffer
            const float there = (inside >> i) & 1u ? 1.f : 0.f;
            if (kARuns) as(1, ak)[am + i * kStepA] = there;
            else as(1, ak + i * kStepA)[am] = there;
          }
          __syncthreads();
#pragma unroll 1
          for (int k = 0; k < kTerms; ++k) {
            const float4 av = *reinterpret_cast<const float4*>(as(0, k) + tm * 4), bv = *reinterpret_cast<const float4*>(bs(0, k) + tn * 4);
            const float4 there = *reinterpret_cast<const float4*>(as(1, k) + tm * 4);
            const float b[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (there.x != 0.f) acc[0][j].x = fmaf(av.x, b[j], acc[0][j].x);
              if (there.y != 0.f) acc[0][j].y = fmaf(av.y, b[j], acc[0][j].y);
              if (there.z != 0.f) acc[1][j].x = fmaf(av.z, b[j], acc[1][j].x);
              if (there.w != 0.f) acc[1][j].y = fmaf(av.w, b[j], acc[1][j].y);
            }
          }
        }
        __syncthreads();
      }
    }
  }
  const float bias = g.staged && g.bias != nullptr && n0 + t % BN < g.n ? load<T>(g.bias, n0 + t % BN) : 0.f;

  // the sums of the cluster's blocks, in the order of their terms, each block a share of the rows
  cg::cluster_group cluster = cg::this_cluster();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float* to = shared + (tm * 4 + 2 * i) * BN + tn * 4;
    *reinterpret_cast<float4*>(to) = make_float4(acc[i][0].x, acc[i][1].x, acc[i][2].x, acc[i][3].x);
    *reinterpret_cast<float4*>(to + BN) = make_float4(acc[i][0].y, acc[i][1].y, acc[i][2].y, acc[i][3].y);
  }
  cluster.sync();
  const int share = BM / g.splits, last = (rank + 1) * share, col = t % BN, n = n0 + col;
  constexpr int kRowStep = kThreads / BN, kBatch = 8;
  for (int row0 = rank * share + t / BN; row0 < last && m0 + row0 < M && n < g.n; row0 += kBatch * kRowStep) {
    float sums[kBatch] = {};
    if (g.splits == 1) {
#pragma unroll
      for (int u = 0; u < kBatch; ++u)
        if (row0 + u * kRowStep < last) sums[u] = shared[(row0 + u * kRowStep) * BN + col];
    } else {
      for (int q = 0; q < g.splits; ++q) {
        const float* peer = cluster.map_shared_rank(shared, q);
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
          if (row0 + u * kRowStep < last) sums[u] += peer[(row0 + u * kRowStep) * BN + col];
      }
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int row = row0 + u * kRowStep, m = m0 + row;
      if (row >= last || m >= M) break;
      float v = sums[u];
      long long o = n * g.on;
      if (g.partial != nullptr) {
        g.partial[(long long)slice * M * g.n + m * g.om + o] = v;
        continue;
      }
      o += (A == kRows ? out_row[row] : m) * g.om;
      if (!g.conv) o += outer * g.out_batch;
      if (g.staged) {
        v *= g.alpha;
        if (g.bias != nullptr) v = to_f32(from_f32<T>(v)) + bias;
        if (g.act != PDNN_ACT_NONE) v = apply_activation(to_f32(from_f32<T>(v)), g.act);
        if (g.beta != 0.f) v = to_f32(from_f32<T>(v)) + to_f32(from_f32<T>(g.beta * load<T>(g.out, o)));
        static_cast<T*>(g.out)[o] = from_f32<T>(v);
      } else if (g.out_f32) {
        if (g.beta != 0.f) v += g.beta * static_cast<const float*>(g.out)[o];
        static_cast<float*>(g.out)[o] = v;
      } else {
        if (g.beta != 0.f) v += g.beta * load<T>(g.out, o);
        static_cast<T*>(g.out)[o] = from_f32<T>(v);
      }
    }
  }
  cluster.sync();  // (nobody leaves while its sums are read)
}

template <typename T, int A, bool B_RUNS, int BN>
int launch(const SimtArgs& g, unsigned blocks, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)g.splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // (not with slices, whose second launch is a few blocks: 60x26x25 55 -> 61 1x1/2 filter gradient, replayed from a graph with the caller's
  // scratch, 19.4 us overlapped, 15.7 not; called 19.8 and 18.4)
  cfg.numAttrs = g.partial == nullptr && (unsigned long long)blocks * kThreads < 4ull * 2048ull * (unsigned long long)device_sm_count() ? 2 : 1;  // as launch_overlapped()
  cudaLaunchKernelEx(&cfg, simt_gemm_kernel<T, A, B_RUNS, BN>, g);
  return check_launch("fp32 tiles");
}

template <int A, bool B_RUNS>
int launch_typed(int dtype, int bn, const SimtArgs& g, unsigned blocks, cudaStream_t s) {
  auto run = [&](auto tag) {
    using T = decltype(tag);
    return bn == 32 ? launch<T, A, B_RUNS, 32>(g, blocks, s) : launch<T, A, B_RUNS, 64>(g, blocks, s);
  };
  switch (dtype) {
    case PDNN_F32: return run(float{});
    case PDNN_F16: return run(__half{});
    case PDNN_BF16: return run(__nv_bfloat16{});
  }
  return fail(PDNN_INVALID_PARAMETER, "unknown dtype %d", dtype);
}

struct Tiling {
  int bn, m_tiles, n_tiles, splits, slices;
};

// Half-width tiles where the columns end in the first half of a tile.  Blocks of a cluster share a tile while the device has room
// for kBlocksPerSm blocks to an SM and four steps are left to each; slices follow where even that
// leaves half of them idle and a slice has 64 steps.  `counted`: the rows that decide, which may be fewer than there are.
Tiling choose(long long m, long long counted, int n, long long inner, long long runs, long long outer, bool slices, int sms) {
  Tiling t;
  const int over = n % 64;
  t.bn = over != 0 && over <= 32 && n < 128 ? 32 : 64;
  const int bm = kOutputs / t.bn;
  t.m_tiles = (int)((m + bm - 1) / bm), t.n_tiles = (n + t.bn - 1) / t.bn;
  const long long tiles = ((counted + bm - 1) / bm) * t.n_tiles * outer, steps = runs * ((inner + kTerms - 1) / kTerms);
  const long long room = (long long)kBlocksPerSm * sms;
  t.splits = 1, t.slices = 1;
  // (a filter gradient's pixels have always been added up in eight parts at least: fewer are longer sums, and larger errors)
  while (t.splits < kMaxSplits && (slices || (2 * tiles * t.splits <= room && steps >= 8ll * t.splits))) t.splits *= 2;
  if (slices) {
    const long long fit = room / (tiles * t.splits), most = steps / 64;
    t.slices = (int)(fit < most ? fit : most);
    if (t.slices < 2) t.slices = 1;
  }
  return t;
}

constexpr long long kMostElements = 0x7FFFFF00ll;

Tiling conv_tiling(int pass, const PdnnConv2DParams& p, bool any_order, int sms) {
  const long long taps = (long long)p.window_rows * p.window_cols, px_out = (long long)p.out_rows * p.out_cols;
  if (pass == PDNN_FORWARD)  // an image has the same result alone and in any batch, unless the caller does not ask for it
    return choose(p.batch * px_out, any_order ? p.batch * px_out : px_out, p.features, p.channels, taps, 1, false, sms);
  if (pass == PDNN_INPUT_BACKPROP) {
    const int phases = p.stride_rows * p.stride_cols;
    const long long m = (long long)p.batch * ((p.in_rows + p.stride_rows - 1) / p.stride_rows) * ((p.in_cols + p.stride_cols - 1) / p.stride_cols);
    return choose(m, m, p.channels, p.features, (taps + phases - 1) / phases, phases, false, sms);
  }
  return choose(taps * p.channels, taps * p.channels, p.features, p.batch * px_out, 1, 1, true, sms);
}

size_t slices_bytes(const Tiling& t, const PdnnConv2DParams& p) {
  return (size_t)t.slices * p.window_rows * p.window_cols * p.channels * p.features * sizeof(float);
}

// Where a thread to an output is still the better one (direct_conv.cu): its time is the length of a sum until the work fills the
// device, that of the tiles the latency of their loads.  Measured on 22861 random layers, tiles / thread to an output, means:
//   terms of a sum                 |   f32, multiply-adds of the layer      |   16 bits
//                                  | 1e5    1e6..3e6   3e6..1e7   1e7..3e7  | 1e5    1e6..3e6   3e6..1e7   1e7..3e7
//   forward, taps * channels    16 | 1.94   1.10       0.77       0.52      | 2.21   1.56       0.76       0.49
//                               64 | 0.96   1.00       0.89       0.55      | 1.83   1.80       1.35       0.67
//                              160 | 0.52   0.48       0.47       0.45      | 1.19   1.03       1.02       0.75
//                              700 | 0.18   0.17       0.17       0.23      | 0.45   0.42       0.41       0.46
//   input gradient, taps *      16 | 1.77   0.95       0.56       0.41      | 2.24   1.14       0.72       0.56
//   features / strides          64 | 0.91   0.97       0.74       0.48      | 1.57   1.27       1.02       0.56
//                              160 | 0.51   0.56       0.50       0.40      | 0.82   0.92       0.84       0.59
//     (fp32 at stride 1, up to 3e6: 1.13 at 64 to 100; a thread looks at every tap, at stride 2 too, whose terms are a quarter)
//   filter gradient, pixels     32 | 1.70   0.69                            | 1.93   0.62       0.43
//                              100 | 0.89   0.47       0.25       0.20      | 1.01   0.53       0.28       0.19
// On average the choice is 3.2, 2.7 and 0.6 % (16 bits 3.9, 2.3 and 0.5 %) behind the faster of the two.  Fewer than four columns leave most
// of a tile idle: 1.8 to 4.4 (sums of up to 64 terms, 1e6 multiply-adds and more), whatever the work.  The forward pass moves over by the terms of a
// sum or by the work of one image: an image has the same result alone and in any batch.
bool thread_to_an_output(int pass, int dtype, const PdnnConv2DParams& p) {
  const double taps = (double)p.window_rows * p.window_cols, pixels = (double)p.out_rows * p.out_cols;
  const double per_image = pixels * taps * p.channels * p.features, macs = per_image * p.batch;
  const bool half = dtype != PDNN_F32;
  if (pass != PDNN_FILTER_BACKPROP) {
    const bool forward = pass == PDNN_FORWARD;
    const double terms = taps * (forward ? p.channels : p.features);
    if ((forward ? p.features : p.channels) < 4 && terms < (half ? 128 : 64)) return true;
    if (forward) return terms < (half ? 128 : 48) && per_image < (half ? 1e6 : 5e5);
    return half ? terms * 2 < 115.0 * (p.stride_rows + p.stride_cols) && macs < 5e6 : terms < 90 && macs < 3e6;
  }
  return pixels * p.batch < 80 && macs < 5e5;
}

// Whether a tap of an output (of a pixel of the input, in an input gradient) can lie outside along one axis.
bool taps_miss(int pass, int in, int out, int window, int stride, int pad) {
  if (pass == PDNN_INPUT_BACKPROP) return pad < window - 1 || ((long long)in - 1 + pad) / stride > out - 1;
  return pad > 0 || ((long long)out - 1) * stride - pad + window > in;
}

int sm_count() {
  const int sms = device_sm_count();
  return sms > 0 ? sms : 148;
}

}  // namespace

bool simt_conv_applicable(int pass, int dtype, const PdnnConv2DParams& p) {
  if (p.groups != 1 || p.input_format != 0 || (p.filter_format != 0 && p.filter_format != 2)) return false;
  const long long taps = (long long)p.window_rows * p.window_cols;
  const long long x = (long long)p.batch * p.in_rows * p.in_cols * p.channels, y = (long long)p.batch * p.out_rows * p.out_cols * p.features;
  const long long w = taps * p.channels * p.features;
  if (x > kMostElements || y > kMostElements || w > kMostElements) return false;
  // positions of taps outside the image are formed before they are found to be outside
  const long long reach = ((long long)p.pad_rows + p.window_rows + 1) * p.in_cols + p.pad_cols + p.window_cols + 1;
  const long long back = ((long long)p.window_rows + p.pad_rows + 1) * p.out_cols + p.window_cols + p.pad_cols + 1;
  if (x + reach * p.channels > kMostElements || y + back * p.features > kMostElements) return false;
  if (p.stride_rows > 64 || p.stride_cols > 64) return false;
  const Tiling t = conv_tiling(pass, p, true, sm_count());
  const double blocks = (double)t.m_tiles * t.n_tiles * t.slices * kMaxSplits * (pass == PDNN_INPUT_BACKPROP ? p.stride_rows * p.stride_cols : 1);
  return blocks < 2147483632.0 && !thread_to_an_output(pass, dtype, p);
}

size_t simt_conv_workspace_elems(int pass, int dtype, const PdnnConv2DParams& p) {
  if (pass != PDNN_FILTER_BACKPROP || !simt_conv_applicable(pass, dtype, p)) return 0;
  const Tiling t = conv_tiling(pass, p, true, sm_count());
  if (t.slices == 1) return 0;
  return slices_bytes(t, p) / dtype_size(dtype);
}

int simt_conv(int pass, int dtype, const void* in, const void* fil, void* out, const PdnnConv2DParams& p,
              const PdnnConvEpilogue* epi, void* ws, size_t ws_elems, cudaStream_t s) {
  const int sms = sm_count(), taps = p.window_rows * p.window_cols;
  Tiling t = conv_tiling(pass, p, pass != PDNN_FORWARD || (epi != nullptr && epi->any_order), sms);
  const bool fhwc = p.filter_format == 2;
  SimtArgs g = {};
  g.a = in, g.b = fil, g.out = out;
  g.conv = 1, g.alpha = 1.f, g.act = PDNN_ACT_NONE, g.on = 1;
  g.batch = p.batch, g.step_rows = p.stride_rows, g.step_cols = p.stride_cols, g.pad_rows = p.pad_rows, g.pad_cols = p.pad_cols;
  g.window_rows = p.window_rows, g.window_cols = p.window_cols, g.dir = 1;
  g.rows = p.out_rows, g.cols = p.out_cols;
  g.a_rows = p.in_rows, g.a_cols = p.in_cols, g.a_channels = p.channels;
  const int of_c = fhwc ? 1 : p.features, of_k = fhwc ? taps * p.channels : 1;
  g.bs = fhwc ? p.channels : p.channels * p.features;
  int outer = 1;
  if (pass == PDNN_FORWARD) {
    g.n = p.features, g.inner = p.channels, g.bk = of_c, g.bn = of_k, g.om = p.features;
    g.staged = 1;
    if (epi != nullptr) g.bias = epi->bias, g.act = epi->activation, g.alpha = epi->alpha, g.beta = epi->beta;
  } else if (pass == PDNN_INPUT_BACKPROP) {
    g.n = p.channels, g.inner = p.features, g.bk = of_k, g.bn = of_c, g.om = p.channels;
    g.dir = -1, g.rows = p.in_rows, g.cols = p.in_cols;
    g.a_rows = p.out_rows, g.a_cols = p.out_cols, g.a_channels = p.features;
    outer = p.stride_rows * p.stride_cols;
  } else {
    g.n = p.features, g.inner = p.batch * p.out_rows * p.out_cols, g.m = taps * p.channels;
    g.bs = 0, g.bk = p.features, g.bn = 1;
    g.om = fhwc ? 1 : p.features, g.on = fhwc ? taps * p.channels : 1;
  }
  g.misses = taps_miss(pass, p.in_rows, p.out_rows, p.window_rows, p.stride_rows, p.pad_rows) ||
             taps_miss(pass, p.in_cols, p.out_cols, p.window_cols, p.stride_cols, p.pad_cols);
  const size_t n_out = (size_t)taps * p.channels * p.features;
  bool own = false;
  if (t.slices > 1) {
    const size_t need = slices_bytes(t, p);
    own = ws == nullptr || !aligned16(ws) || ws_elems * dtype_size(dtype) < need;
    g.partial = static_cast<float*>(ws);
    if (own && cudaMallocAsync(reinterpret_cast<void**>(&g.partial), need, s) != cudaSuccess) {
      cudaGetLastError();
      g.partial = nullptr, own = false, t.slices = 1;
    }
  }
  g.m_tiles = t.m_tiles, g.n_tiles = t.n_tiles, g.splits = t.splits, g.slices = t.slices;
  const long long blocks = (long long)outer * t.slices * t.n_tiles * t.m_tiles * t.splits;
  int st;
  if (pass == PDNN_FILTER_BACKPROP) st = launch_typed<kPixels, false>(dtype, t.bn, g, (unsigned)blocks, s);
  else if (g.bk == 1 && g.bn != 1) st = launch_typed<kRows, true>(dtype, t.bn, g, (unsigned)blocks, s);
  else st = launch_typed<kRows, false>(dtype, t.bn, g, (unsigned)blocks, s);
  if (st == PDNN_OK && t.slices > 1) {
    if (dtype == PDNN_F32) launch_column_sums(g.partial, t.slices, n_out, sms, s, StoreSum<float>{static_cast<float*>(out), false});
    else if (dtype == PDNN_F16) launch_column_sums(g.partial, t.slices, n_out, sms, s, StoreSum<__half>{static_cast<__half*>(out), false});
    else launch_column_sums(g.partial, t.slices, n_out, sms, s, StoreSum<__nv_bfloat16>{static_cast<__nv_bfloat16*>(out), false});
    st = check_launch("conv2d filter gradient");
  }
  if (own) cudaFreeAsync(g.partial, s);
  return st;
}

bool simt_matmul_tiled(int dtype, int tl, int tr, const void* lhs, const void* rhs, void* out, int batches, int m, int k,
                       int n, float beta, cudaStream_t s, bool out_f32, int* status) {
  if ((long long)m * k > kMostElements || (long long)k * n > kMostElements || n > kMostElements - 64 || m > kMostElements - 128) return false;
  const Tiling t = choose(m, m, n, k, 1, batches, false, sm_count());
  const long long tiles = (long long)batches * t.n_tiles * t.m_tiles, blocks = tiles * t.splits;
  if (blocks > 0x7FFFFFF0ll) return false;
  // What each side takes, in us: a thread to an output walks its terms (26 ns each in fp32, 44 in 16 bits, 52 where the terms of lhs, or of
  // 32 and more rows of rhs, lie apart) or the device is full (2.5 multiply-adds per ps, 1.5 with rows of rhs apart); here a
  // step takes 0.75 us or the tiles, remainders and all, fill it (10 per ps).  Over 11417 random products the choice is 0.9 % behind the
  // faster side on average, and slower than a thread to an output by more than 11 % in one of a hundred.  Measured, thread to an output / here: f16
  // 2 x 1008 x 543 51 / 12.4, 2 x 543 x 1008 (rhs transposed) 32 / 11.2, 500 x 2000 x 1001 380 / 122, 1001 x 2000 transposed 1502 / 127;
  // f32 128 x 1024 x 333 33 / 11.8, 16 of 3000 x 37 x 51 37 / 25; and f32 2000 of 16 x 17 x 15 7.3 / 31, 16 of 400 x 13 x 13 3.6 / 7.5,
  // f16 10 x 100 x 11 7.2 / 11, f32 4000000 x 3 x 3 73 / 548.
  const double steps = (k + kTerms - 1) / kTerms, macs = (double)batches * m * n * k;
  const bool apart = tr && n >= 32;
  const double term = tl || apart ? 0.052 : tr ? 0.03 : dtype == PDNN_F32 ? 0.026 : 0.044;
  const double walk = 3 + term * k + macs / (apart ? 1.5e6 : 2.5e6), here = 5 + 0.75 * steps / t.splits + (double)tiles * kOutputs * steps * kTerms / 1e7;
  if (walk <= here) return false;
  SimtArgs g = {};
  g.a = lhs, g.b = rhs, g.out = out;
  g.a_batch = (long long)m * k, g.b_batch = (long long)k * n, g.out_batch = (long long)m * n;
  g.m = m, g.n = n, g.inner = k, g.dir = 1, g.a_rows = g.a_cols = 1;
  g.lda = tl ? m : k;
  g.bk = tr ? 1 : n, g.bn = tr ? k : 1;
  g.om = n, g.on = 1;
  g.window_cols = 1;
  g.beta = beta, g.out_f32 = out_f32;
  g.m_tiles = t.m_tiles, g.n_tiles = t.n_tiles, g.splits = t.splits, g.slices = 1;
  if (tl) *status = tr ? launch_typed<kColumns, true>(dtype, t.bn, g, (unsigned)blocks, s) : launch_typed<kColumns, false>(dtype, t.bn, g, (unsigned)blocks, s);
  else *status = tr ? launch_typed<kRows, true>(dtype, t.bn, g, (unsigned)blocks, s) : launch_typed<kRows, false>(dtype, t.bn, g, (unsigned)blocks, s);
  return true;
}

}  // namespace pdnn
