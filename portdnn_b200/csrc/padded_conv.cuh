// Convolutions the tensor-core engine takes only on copies padded to whole 16-byte rows (padded_conv.cu).
#pragma once

#include "common.cuh"

namespace pdnn {

// True if the pass runs on padded copies: 16-bit NHWC tensors, groups == 1, everything else as
// tc_conv_supported asks, and enough work to pay for the copies.
bool padded_conv_applicable(int pass, int dtype, const PdnnConv2DParams& p, const PdnnConvEpilogue* epi);

// Scratch elements (of dtype) of the copies; without them the call allocates, and where there is no memory
// either padded_conv asks for the direct kernel.  (Tensors off a 16-byte boundary are not known to the query:
// their copies are not counted for a layer whose channel and feature counts need none.)
size_t padded_conv_workspace_elems(int pass, int dtype, const PdnnConv2DParams& p);

// May return kNeedsDirect (tc_gemm.cuh).
int padded_conv(int pass, int dtype, const void* in, const void* fil, void* out, const PdnnConv2DParams& p,
                const PdnnConvEpilogue* epi, const PdnnBackpropFusion* fusion, void* ws, size_t ws_elems, cudaStream_t s);

}  // namespace pdnn
