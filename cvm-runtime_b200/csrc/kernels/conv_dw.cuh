// Interface between cvmk_conv2d_direct and the tensor-core kernel for depthwise 3 x 3 layers (conv_dw.cu).
#pragma once
#include <stdint.h>
#include "common.cuh"

namespace cvmk {

// Launches the layer with its chain, or returns -1 when it is not one for this kernel.
int launch_conv_dw(const cvmk_conv_direct_desc& d, const DevChain& chain, cudaStream_t stream);
// Whether it would launch it.
bool conv_dw_takes(const cvmk_conv_direct_desc& d);

}  // namespace cvmk
