// Interface between cvmk_conv2d_direct and the tensor-core kernel for depthwise 3 x 3 layers (conv_dw.cu).
#pragma once
#include <stdint.h>
#include "common.cuh"

namespace cvmk {

// The chain of a depthwise layer in the packed form: [bias,] then ((sum + bias + add) * mul) >> 16 clamped to [lo, hi].
struct DwRequant {
  const int32_t* bias;
  int mul, add;
  int lo, hi;
};

// Launches the layer, or returns -1 when it is not one for this kernel.
int launch_conv_dw(const cvmk_conv_direct_desc& d, const DwRequant& rq, cudaStream_t stream);

}  // namespace cvmk
