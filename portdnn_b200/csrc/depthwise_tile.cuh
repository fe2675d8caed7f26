// Depthwise 3x3 operators on tiles that TMA brings into shared memory (depthwise_tile.cu).
#pragma once

#include "common.cuh"

namespace pdnn {

// First stage of the filter gradient: partial[slice][tap][channel] for at most max_slices slices.  Returns the
// number of slices written (a launch error is left to check_launch()), or 0 where the layer is not for this
// kernel: windows other than 3x3, strides other than 1 and 2, channels that are not whole 16-byte packets.
int launch_depthwise_filter_tiles(int dtype, const void* x, const void* dy, float* partial, const PdnnDepthwiseConv2DParams& p,
                                  int max_slices, cudaStream_t s);

// Forward pass of 16-bit tensors; mirrored: with the filter's taps in reverse order, which with the tensors' and paddings' roles exchanged
// in p is the input gradient of stride 1.  False where the layer is not for this kernel.
bool launch_depthwise_forward_tiles(int dtype, const void* x, const void* filter, void* out, const PdnnDepthwiseConv2DParams& p,
                                    bool mirrored, cudaStream_t s);

}  // namespace pdnn
