// Convolutions whose operands are split into 16-bit parts once, before the matrix kernel; see conv_split.cu.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace cunn {
namespace split {

// A convolution: x [N][C][H][W], weight [K][C][kH][kW], y [N][K][oH][oW].
struct Geometry {
    int N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW, oH, oW;
};

// Bytes of scratch memory, 16-byte aligned, that the pass takes; 0: it is better off, or only possible, on the other kernels.
size_t forward_scratch(const Geometry &g);
size_t grad_input_scratch(const Geometry &g);
size_t grad_weight_scratch(const Geometry &g);

// The passes, for geometries whose scratch size is not 0.  bias may be null (the input gradient adds it to every plane of gx: the forward
// pass of a transposed convolution); grad_weight and grad_bias (may be null) are accumulated into.
int forward(const Geometry &g, const float *x, const float *weight, const float *bias, float *y, void *scratch, cudaStream_t stream);
int grad_input(const Geometry &g, const float *gy, const float *weight, const float *bias, float *gx, void *scratch, cudaStream_t stream);
int grad_weight(const Geometry &g, const float *x, const float *gy, float *grad_weight, float *grad_bias, float scale, void *scratch,
                cudaStream_t stream);

}  // namespace split
}  // namespace cunn
