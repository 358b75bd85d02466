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

// What queues the same pass over images [first, first + n) on kernels that do nothing where *gate is 0 when they run: those for values that
// are too different in size to share exponents.
struct Fallback {
    int (*call)(const void *self, int first, int n, const int *gate);
    const void *self;
    int operator()(int first, int n, const int *gate) const { return call(self, first, n, gate); }
};
template <class F>
Fallback fallback_of(const F &f)
{
    return {[](const void *self, int first, int n, const int *gate) { return (*static_cast<const F *>(self))(first, n, gate); }, &f};
}
// The head of a parameter gradient's scratch memory: the gate, the channels' ranges and the sums.  The fallback has the rest to itself; it adds
// scale * its own sums to the gradient or, where *gate is 0, scale * these.
constexpr size_t GATE_BYTES = 256;
inline size_t max_bytes(const Geometry &g) { return ((size_t)(g.C + g.K) * 8 + 255) & ~(size_t)255; }
inline size_t grad_weight_head(const Geometry &g) { return GATE_BYTES + max_bytes(g) + (((size_t)g.K * g.C * g.kH * g.kW * 4 + 255) & ~(size_t)255); }
inline float *grad_weight_sums(const Geometry &g, void *scratch) { return (float *)((char *)scratch + GATE_BYTES + max_bytes(g)); }

// Bytes of scratch memory, 16-byte aligned, that the pass takes; 0: it is better off, or only possible, on the other kernels.
// again_bytes: workspace of a round on the fallback's kernels.
size_t forward_scratch(const Geometry &g);
size_t grad_input_scratch(const Geometry &g);
size_t grad_weight_scratch(const Geometry &g, size_t (*again_bytes)(const Geometry &));

// The passes, for geometries whose scratch size is not 0.  bias may be null (the input gradient adds it to every plane of gx: the forward
// pass of a transposed convolution); grad_bias (may be null) is accumulated into.
int forward(const Geometry &g, const float *x, const float *weight, const float *bias, float *y, const Fallback &again, void *scratch,
            cudaStream_t stream);
int grad_input(const Geometry &g, const float *gy, const float *weight, const float *bias, float *gx, const Fallback &again, void *scratch,
               cudaStream_t stream);
int grad_weight(const Geometry &g, const float *x, const float *gy, float *grad_bias, float scale, const Fallback &again, void *scratch,
                cudaStream_t stream);

}  // namespace split
}  // namespace cunn
