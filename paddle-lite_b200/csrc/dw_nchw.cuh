// Depthwise convolution on NCHW tensors as they are (dw_nchw.cu).
#pragma once
#include "common.cuh"
#include "kernels_simple.cuh"

namespace plb {

// 3x3 and 5x5 filters, strides 1 and 2 (equal in both directions), no dilation, planes that fit in shared memory.
bool dw_nchw_supported(const ConvGeom& g, int mode);
// x [batch, c, h, w]; w_tc [kh * kw][cg_pad]; out.y [batch, c, ho, wo]
int dw_nchw_launch(plb_ctx* ctx, const ConvGeom& g, const int8_t* x, const int8_t* w_tc, const OutSpec& out);

}  // namespace plb
