// Matrix products and convolutions in fp32 arithmetic on the CUDA cores (simt_gemm.cu): what the tensor-core
// kernels cannot tile.
#pragma once

#include "common.cuh"

namespace pdnn {

// Whether simt_conv takes the layer: NHWC tensors, one group, element indices of 32 bits, and a layer that gains by it.
bool simt_conv_applicable(int pass, int dtype, const PdnnConv2DParams& p);

// Scratch elements (of dtype) that the pass can use: the slices of a long filter gradient.
size_t simt_conv_workspace_elems(int pass, int dtype, const PdnnConv2DParams& p);

// The result is what launch_direct_conv() gives up to the order of the sums.  Without scratch for its slices a filter gradient
// allocates it, and runs in one slice where there is no memory.
int simt_conv(int pass, int dtype, const void* in, const void* fil, void* out, const PdnnConv2DParams& p,
              const PdnnConvEpilogue* epi, void* ws, size_t ws_elems, cudaStream_t s);

// As simt_matmul() in tc_gemm.cuh; false where that one is to run.
bool simt_matmul_tiled(int dtype, int tl, int tr, const void* lhs, const void* rhs, void* out, int batches, int m, int k,
                       int n, float beta, cudaStream_t s, bool out_f32, int* status);

}  // namespace pdnn
