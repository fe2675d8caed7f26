// Convolutions of 16-bit tensors whose channel or feature count is not a multiple of 8 (or whose tensors
// start off a 16-byte boundary): TMA needs rows that start on 16 bytes, so the operands are copied into
// rows padded with zeros (padded_count), the tensor-core kernels run on the copies, and what they
// wrote is cut back.  The padding adds zero terms to the sums and columns that are dropped; operands that
// are in order are read, and results written, in place.
//
// Bound by the convolution itself, then by the launches around it.  7 x 45x61, 100 -> 150 channels, 3x3, bf16,
// all three passes: 15580 us on the direct kernel, 77 us here.
#include "padded_conv.cuh"
#include "tc_gemm.cuh"

#include <type_traits>

namespace pdnn {
namespace {

constexpr int kBlock = 256;
constexpr int kUnroll = 4;  // packets a thread has in flight

size_t round_up(size_t v, size_t to) { return (v + to - 1) / to * to; }

// out[a][b][c] = in[a][b][c], zero where in has no such b or c.  Extents: bo x co per matrix of out, bi x ci
// per matrix of in; larger extents in out pad, smaller ones cut.
struct RepitchJob {
  const unsigned short* in;
  unsigned short* out;
  unsigned items;  // packets of out
  int bo, bi, co, ci;
  int vw;  // elements per packet: 4, 2 or 1, a divisor of ci and co that both pointers are aligned to
  unsigned first_block;
};
constexpr int kMaxJobs = 3;
struct RepitchJobs {
  RepitchJob job[kMaxJobs];
  int count;
  unsigned blocks;
};

template <int VW>
struct Packet;
template <>
struct Packet<1> { using type = unsigned short; };
template <>
struct Packet<2> { using type = unsigned; };
template <>
struct Packet<4> { using type = uint2; };

template <int VW>
__device__ __forceinline__ void repitch(const RepitchJob& j, unsigned first, unsigned step) {
  using P = typename Packet<VW>::type;
  const unsigned cv = (unsigned)(j.co / VW), civ = (unsigned)(j.ci / VW), bo = (unsigned)j.bo, bi = (unsigned)j.bi;
  const P* in = reinterpret_cast<const P*>(j.in);
  P* out = reinterpret_cast<P*>(j.out);
  for (unsigned i0 = first; i0 < j.items; i0 += step * kUnroll) {
    P v[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const unsigned i = i0 + u * step;
      v[u] = P{};
      if (i < j.items) {
        const unsigned row = i / cv, c = i - row * cv;
        const unsigned a = row / bo, b = row - a * bo;
        if (c < civ && b < bi) v[u] = in[((size_t)a * bi + b) * civ + c];
      }
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
      if (i0 + u * step < j.items) out[i0 + u * step] = v[u];
  }
}

// Up to three copies (activations, filter, bias) side by side in one launch.
__global__ void __launch_bounds__(kBlock) repitch_kernel(const RepitchJobs jobs) {
  overlap_wait();
  int n = 0;
  while (n + 1 < jobs.count && blockIdx.x >= jobs.job[n + 1].first_block) ++n;
  const RepitchJob& j = jobs.job[n];
  const unsigned last = n + 1 < jobs.count ? jobs.job[n + 1].first_block : jobs.blocks;
  const unsigned first = (blockIdx.x - j.first_block) * kBlock + threadIdx.x, step = (last - j.first_block) * kBlock;
  if (j.vw == 4) repitch<4>(j, first, step);
  else if (j.vw == 2) repitch<2>(j, first, step);
  else repitch<1>(j, first, step);
}

void add_job(RepitchJobs& jobs, const void* in, void* out, size_t matrices, int bi, int bo, int ci, int co, int sms) {
  RepitchJob& j = jobs.job[jobs.count++];
  j.in = static_cast<const unsigned short*>(in);
  j.out = static_cast<unsigned short*>(out);
  j.bi = bi, j.bo = bo, j.ci = ci, j.co = co;
  j.vw = 4;
  const uintptr_t at = reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out);
  while (j.vw > 1 && (ci % j.vw != 0 || co % j.vw != 0 || at % (2u * j.vw) != 0)) j.vw /= 2;
  j.items = (unsigned)(matrices * bo * (co / j.vw));
  j.first_block = jobs.blocks;
  jobs.blocks += grid_for(round_up(j.items, kUnroll) / kUnroll, kBlock, sms);
}

int run_jobs(const RepitchJobs& jobs, cudaStream_t s) {
  if (jobs.count == 0) return PDNN_OK;
  launch_overlapped(repitch_kernel, jobs.blocks, kBlock, s, jobs);
  return check_launch("conv2d padding");
}

// out[a][b][c] (+)= in[a][b][c] with another element type; in has bi x ci elements per matrix, out bo x co.
template <typename InT, typename OutT>
__global__ void __launch_bounds__(kBlock)
    cut_kernel(const InT* in, OutT* __restrict__ out, unsigned n, int bo, int bi, int co, int ci, bool accumulate) {
  overlap_wait();
  const unsigned step = gridDim.x * kBlock;
  for (unsigned i0 = blockIdx.x * kBlock + threadIdx.x; i0 < n; i0 += kUnroll * step) {
    float v[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const unsigned i = i0 + u * step;
      if (i >= n) break;
      const unsigned row = i / (unsigned)co, c = i - row * (unsigned)co, a = row / (unsigned)bo, b = row - a * (unsigned)bo;
      v[u] = to_f32(in[((size_t)a * bi + b) * ci + c]);
      if (accumulate) v[u] += to_f32(out[i]);
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
      if (i0 + u * step < n) out[i0 + u * step] = from_f32<OutT>(v[u]);
  }
}

// A count off a multiple of 8, padded.  A multiple of 8 would do, but rows that start inside a 32-byte sector cost the tiles' loads
// one more sector and often a second line each (bf16, us, 7x45x61 3x3, input gradient: 128 -> 152 features 27.0, 160 16.5,
// 192 13.1; forward pass, 104 -> 128 channels 14.5, 112 11.7, 128 10.1).  So whole lines of 64 where they
// are hardly more to copy, else whole sectors of 16; `narrow`: the multiple of 8.  A window of one pixel reads each row once, so that
// what is copied counts for more (lines / multiples of 8, means over 8535 random layers, tensors 12 to 20 % wider: 1x1 forward
// 1.02, filter gradient 1.04, a third wider 1.04 and 1.06; 3x3 0.82).
int padded_count(int n, bool narrow, bool one_pixel) {
  if (n % 8 == 0) return n;
  if (narrow) return (int)round_up((size_t)n, 8);
  const int lines = (int)round_up((size_t)n, 64);
  return 10ll * lines <= (one_pixel ? 11ll : 13ll) * n ? lines : (int)round_up((size_t)n, 16);
}

struct Plan {
  PdnnConv2DParams q;          // the convolution the tensor-core kernels run
  size_t x, w, y;              // elements of the padded tensors
  size_t real_x, real_w, real_y;
  bool same_c, same_k;
};

// The tensor-core kernels have to take the padded layer; `plan.q` keeps the channels of a few-channel
// layer, which is packed on its own there.
bool plan_with(int pass, int dtype, const PdnnConv2DParams& p, bool narrow, Plan* plan) {
  if (dtype == PDNN_F32 || p.groups != 1 || p.input_format != 0) return false;
  if (p.filter_format != 0 && p.filter_format != 2) return false;
  PdnnConv2DParams q = p;
  const void* aligned = reinterpret_cast<const void*>(uintptr_t(256));
  const bool one_pixel = p.window_rows * p.window_cols == 1;
  q.features = padded_count(p.features, narrow, one_pixel);
  if (!tc_conv_supported(pass, dtype, aligned, aligned, aligned, q)) {
    q.channels = padded_count(p.channels, narrow, one_pixel);
    if (!tc_conv_supported(pass, dtype, aligned, aligned, aligned, q)) return false;
  }
  const size_t px_in = (size_t)p.batch * p.in_rows * p.in_cols, px_out = (size_t)p.batch * p.out_rows * p.out_cols;
  const size_t taps = (size_t)p.window_rows * p.window_cols;
  plan->q = q;
  plan->x = px_in * q.channels, plan->w = taps * q.channels * q.features, plan->y = px_out * q.features;
  plan->real_x = px_in * p.channels, plan->real_w = taps * p.channels * p.features, plan->real_y = px_out * p.features;
  plan->same_c = q.channels == p.channels, plan->same_k = q.features == p.features;
  const size_t most = 0xF0000000u;  // packet indices are 32 bits wide
  return plan->x < most && plan->w < most && plan->y < most;
}

// Multiples of 8 where wider copies have too many elements.
bool make_plan(int pass, int dtype, const PdnnConv2DParams& p, Plan* plan) {
  return plan_with(pass, dtype, p, false, plan) || plan_with(pass, dtype, p, true, plan);
}

// The copies, the kernels' own workspace and the padded result, each on a boundary of 256 bytes.
size_t scratch_bytes(int pass, int dtype, const Plan& plan) {
  const size_t inner = tc_conv_workspace_elems(pass, dtype, plan.q);
  return round_up(plan.x * 2, 256) + round_up(plan.y * 2, 256) + round_up(plan.w * (pass == PDNN_FILTER_BACKPROP ? 4 : 2), 256) +
         round_up((size_t)plan.q.features * 2, 256) + round_up(inner * 2, 256) + 256;
}

// Where the general kernels, one launch that needs no copies, are still the better ones (a thread to an output or fp32 tiles, as
// simt_gemm.cu chooses).  Measured on 14652 random layers, copies and tensor cores / general, means:
//   terms of a sum                  |  multiply-adds of the layer
//                                   | 1e5    1e5..3e5   3e5..1e6   1e6..3e6   3e6..1e7   1e7..3e7
//   forward, taps * channels     32 | 2.02   2.08       2.00       1.53       1.07       0.93
//                                64 | 1.33   1.35       1.35       1.19       1.06       0.86
//                               128 | 0.69   0.69       0.68       0.75       0.78       0.82
//   input gradient, taps *       32 | 2.73   2.24       1.95       1.44       0.83       0.81
//   features / strides           64 | 1.20   1.08       1.11       1.08       0.92       0.88
//                               128 | 0.77   0.87       0.84       0.80       0.80       0.80
//   filter gradient, pixels      32 | 2.37   1.79       1.17       0.64       0.59
//                                64 | 1.40   1.23       0.70       0.70       0.83
//                               128 | 0.91   0.76       0.77       0.71       1.00
// On average the choice is 2.7, 3.2 and 0.8 % behind the faster of the two.  The forward pass moves over by the terms of a
// sum or by the work of one image, not of the batch: the kernels add up in different orders, and an image has the same result
// alone and in any batch.  (With 3e5 for an image 1.4 %, but 35 images of 13x18, 27 -> 192 1x1/2, 11.4 us for 6.4.)
bool general_is_better(int pass, const PdnnConv2DParams& p) {
  const double taps = (double)p.window_rows * p.window_cols, pixels = (double)p.out_rows * p.out_cols;
  const double per_image = pixels * taps * p.channels * p.features, macs = per_image * p.batch;
  if (pass == PDNN_FORWARD) return taps * p.channels < 64 && per_image < 1e5;
  if (pass == PDNN_FILTER_BACKPROP) return pixels * p.batch < 64 && macs < 5e5;
  return taps * p.features < 64.0 * p.stride_rows * p.stride_cols && macs < 5e6;
}

}  // namespace

bool padded_conv_applicable(int pass, int dtype, const PdnnConv2DParams& p, const PdnnConvEpilogue* epi) {
  if (pass == PDNN_FORWARD && epi != nullptr && epi->beta != 0.f) return false;  // (reads what the output holds)
  Plan plan;
  return !general_is_better(pass, p) && make_plan(pass, dtype, p, &plan);
}

size_t padded_conv_workspace_elems(int pass, int dtype, const PdnnConv2DParams& p) {
  Plan plan;
  if (!padded_conv_applicable(pass, dtype, p, nullptr) || !make_plan(pass, dtype, p, &plan)) return 0;
  if (plan.same_c && plan.same_k) return 0;  // only off-boundary tensors would be copied
  return scratch_bytes(pass, dtype, plan) / 2;
}

int padded_conv(int pass, int dtype, const void* in, const void* fil, void* out, const PdnnConv2DParams& p,
                const PdnnConvEpilogue* epi, const PdnnBackpropFusion* fusion, void* ws, size_t ws_elems, cudaStream_t s) {
  Plan plan;
  if (!make_plan(pass, dtype, p, &plan)) return kNeedsDirect;
  const int sms = device_sm_count();
  size_t need = scratch_bytes(pass, dtype, plan);
  // Scratch that holds copies to multiples of 8 only is used for those, whether the caller brought it or no more is to be had.
  auto make_do = [&](size_t at_most) {
    Plan less;
    const size_t need_less = plan_with(pass, dtype, p, true, &less) ? scratch_bytes(pass, dtype, less) : need;
    if (need_less >= need || need_less > at_most) return false;
    plan = less, need = need_less;
    return true;
  };
  char* base = static_cast<char*>(ws);
  if (base != nullptr && ws_elems * 2 < need) make_do(ws_elems * 2);
  const bool own = base == nullptr || ws_elems * 2 < need;
  auto allocate = [&] {
    if (cudaMallocAsync(reinterpret_cast<void**>(&base), need, s) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
  };
  if (own && !allocate() && !(make_do(need) && allocate())) return kNeedsDirect;  // (the direct kernel reads the tensors where they are)
  const PdnnConv2DParams& q = plan.q;
  char* at = reinterpret_cast<char*>(round_up(reinterpret_cast<uintptr_t>(base), 256));
  auto take = [&](size_t bytes) {
    char* r = at;
    at += round_up(bytes, 256);
    return r;
  };
  const int taps = p.window_rows * p.window_cols;
  const bool fhwc = p.filter_format == 2;
  RepitchJobs jobs = {};
  // a tensor of pixels x (real -> padded) elements, copied unless it is in order
  auto pixels = [&](const void* t, size_t n_px, int real, int padded) -> const void* {
    if (real == padded && aligned16(t)) return t;
    void* to = take(n_px * padded * 2);
    add_job(jobs, t, to, 1, (int)n_px, (int)n_px, real, padded, sms);
    return to;
  };
  auto filter = [&]() -> const void* {
    if (plan.same_c && plan.same_k && aligned16(fil)) return fil;
    void* to = take(plan.w * 2);
    if (fhwc) add_job(jobs, fil, to, 1, p.features * taps, q.features * taps, p.channels, q.channels, sms);
    else add_job(jobs, fil, to, taps, p.channels, q.channels, p.features, q.features, sms);
    return to;
  };
  const int px_in = p.batch * p.in_rows * p.in_cols, px_out = p.batch * p.out_rows * p.out_cols;
  int st = PDNN_OK;
  auto rest = [&](size_t* elems) {  // what is left of the scratch, for the kernels' own use
    *elems = (size_t)(base + need - at) / 2;
    return static_cast<void*>(at);
  };
  size_t inner_elems = 0;
  if (pass == PDNN_FORWARD) {
    const void* x = pixels(in, px_in, p.channels, q.channels);
    const void* w = filter();
    PdnnConvEpilogue e;
    if (epi != nullptr) {
      e = *epi;
      if (w != fil) e.constant_filter = 0;  // the copy is made by the preceding kernel
      if (e.bias != nullptr && !(plan.same_k && aligned16(e.bias))) {
        void* b = take((size_t)q.features * 2);
        add_job(jobs, e.bias, b, 1, 1, 1, p.features, q.features, sms);
        e.bias = b;
        e.constant_filter = 0;
      }
      if (!plan.same_k) e.relu_bitmask = nullptr;  // (asked for with multiples of 8 features only)
    }
    const bool direct_out = plan.same_k && aligned16(out);
    void* y = direct_out ? out : take(plan.y * 2);
    st = run_jobs(jobs, s);
    void* inner = rest(&inner_elems);
    if (st == PDNN_OK) st = tc_conv2d(pass, dtype, x, w, y, q, epi != nullptr ? &e : nullptr, nullptr, inner, inner_elems, s);
    if (st == PDNN_OK && !direct_out) {
      RepitchJobs back = {};
      add_job(back, y, out, 1, px_out, px_out, q.features, p.features, sms);
      st = run_jobs(back, s);
    }
  } else if (pass == PDNN_INPUT_BACKPROP) {
    const void* dy = pixels(in, px_out, p.features, q.features);
    const void* w = filter();
    const bool direct_out = plan.same_c && aligned16(out);
    PdnnBackpropFusion f = {};
    if (fusion != nullptr && direct_out) {  // dx is laid out as the caller's masks are
      f = *fusion;
      if (w != fil) f.constant_filter = 0;
    }
    void* dx = direct_out ? out : take(plan.x * 2);
    st = run_jobs(jobs, s);
    void* inner = rest(&inner_elems);
    if (st == PDNN_OK) st = tc_conv2d(pass, dtype, dy, w, dx, q, nullptr, &f, inner, inner_elems, s);
    if (st == PDNN_OK && !direct_out) {
      const unsigned n = (unsigned)plan.real_x;
      if (fusion != nullptr && fusion->accumulate) {
        if (dtype == PDNN_F16)
          launch_overlapped(cut_kernel<__half, __half>, grid_for(n, kBlock, sms), kBlock, s, static_cast<const __half*>(dx),
                            static_cast<__half*>(out), n, px_in, px_in, p.channels, q.channels, true);
        else
          launch_overlapped(cut_kernel<__nv_bfloat16, __nv_bfloat16>, grid_for(n, kBlock, sms), kBlock, s,
                            static_cast<const __nv_bfloat16*>(dx), static_cast<__nv_bfloat16*>(out), n, px_in, px_in,
                            p.channels, q.channels, true);
        st = check_launch("conv2d input gradient");
      } else {
        RepitchJobs back = {};
        add_job(back, dx, out, 1, px_in, px_in, q.channels, p.channels, sms);
        st = run_jobs(back, s);
      }
      if (st == PDNN_OK && fusion != nullptr && fusion->relu_bitmask != nullptr)
        st = launch_relu_grad_bits(dtype, fusion->relu_bitmask, out, n, s);
      else if (st == PDNN_OK && fusion != nullptr && fusion->relu_forward_output != nullptr)
        st = launch_pointwise_grad(PDNN_ACT_RELU, dtype, fusion->relu_forward_output, out, out, n, s);
    }
  } else {
    const void* x = pixels(in, px_in, p.channels, q.channels);
    const void* dy = pixels(fil, px_out, p.features, q.features);
    float* dw = reinterpret_cast<float*>(take(plan.w * 4));
    PdnnBackpropFusion f = {};
    f.output_f32 = 1;
    st = run_jobs(jobs, s);
    void* inner = rest(&inner_elems);
    if (st == PDNN_OK) st = tc_conv2d(pass, dtype, x, dy, dw, q, nullptr, &f, inner, inner_elems, s);
    if (st == PDNN_OK) {
      const unsigned n = (unsigned)plan.real_w, grid = grid_for(n, kBlock, sms);
      const bool add = fusion != nullptr && fusion->accumulate;
      auto cut = [&](auto* to) {
        launch_overlapped(cut_kernel<float, std::remove_pointer_t<decltype(to)>>, grid, kBlock, s, dw, to, n, p.channels,
                          q.channels, p.features, q.features, add);
      };
      if (fusion != nullptr && fusion->output_f32) cut(static_cast<float*>(out));
      else if (dtype == PDNN_F16) cut(static_cast<__half*>(out));
      else cut(static_cast<__nv_bfloat16*>(out));
      st = check_launch("conv2d filter gradient");
    }
  }
  if (own) cudaFreeAsync(base, s);
  return st;
}

}  // namespace pdnn
