// Batch normalisation over [N, C, S] (S = H*W) for sm_100a: forward (training and inference) and backward.
//
// The reference runs one 512-thread CTA per channel, which leaves most of a 148-SM GPU idle when C is
// small and reads the input three times.  Here every pass is spread over (channel x chunk) warps or CTAs:
//   * statistics: each warp reduces an equal run of one channel with 16-byte loads.  Sums
//     are taken of (x - K) and (x - K)^2 with K the mean of the chunk's first elements, which keeps fp32
//     accumulation accurate even when |mean| >> std; chunks are merged in fp64 by the channel's last warp,
//     which also writes save_mean / save_std and updates the running statistics;
//   * normalisation / gradient: one grid-stride pass with 16-byte loads and stores.
// Formulas (lib/THCUNN/BatchNormalization.cu:141-283): save_std holds 1/sqrt(biased var + eps) (0 when
// var == 0 and eps == 0), running_var is updated with the unbiased variance n/(n-1).
#include "common.cuh"

#include <algorithm>
#include <stdlib.h>

namespace cunn {
namespace bn {

struct ChunkStat {
    float k;      // shift
    float s1;     // sum (x - k)
    float s2;     // sum (x - k)^2
    float n;      // element count
};

// Merges the chunk statistics of channel c in fp64, publishes mean / inverse std and updates the running statistics; by one warp, without
// a division per partial (they cost 0.3 us each): the mean first, then the squares about it, sum (x - mean)^2 = s2 - 2 d s1 + n d^2
// with d = mean - k, in a fixed order.  `part` points at the channel's first partial.
__device__ __forceinline__ void finish_stats_channel_warp(const ChunkStat *part, int c, int chunks, float *running_mean,
                                                          float *running_var, float *save_mean, float *save_std,
                                                          double momentum, double eps)
{
    const int lane = threadIdx.x & 31;
    const float4 *raw = reinterpret_cast<const float4 *>(part);                 // k, s1, s2, n
    double n = 0.0, sum = 0.0, m2 = 0.0;
#pragma unroll 4
    for (int j = lane; j < chunks; j += 32) {
        const float4 p = __ldcg(raw + j);
        n += (double)p.w;
        sum += (double)p.w * (double)p.x + (double)p.y;
    }
    n = warp_sum(n);
    const double mean = warp_sum(sum) / n;
#pragma unroll 4
    for (int j = lane; j < chunks; j += 32) {
        const float4 p = __ldcg(raw + j);
        const double d = mean - (double)p.x;
        m2 += (double)p.z - 2.0 * d * (double)p.y + (double)p.w * d * d;
    }
    m2 = warp_sum(m2);
    if (lane != 0) return;
    if (m2 < 0.0) m2 = 0.0;
    // The reference computes in float for float tensors; follow its formulas on the float-rounded mean.
    const float meanf = (float)mean;
    const float varN = (float)m2;
    float invstd = 0.f;
    if (varN != 0.f || (float)eps != 0.f) invstd = 1.f / sqrtf((float)(m2 / n) + (float)eps);
    const float unbiased = (float)(m2 / (n - 1.0));
    save_mean[c] = meanf;
    save_std[c] = invstd;
    running_mean[c] = (float)((1.0 - momentum) * (double)running_mean[c] + momentum * (double)meanf);
    running_var[c] = (float)((1.0 - momentum) * (double)running_var[c] + momentum * (double)unbiased);
}

// The sums of both passes are taken by single warps: chunk j of channel c is the j-th of `chunks` equal runs of the channel's items
// (16-byte pieces where planes allow it, else elements) in (image, plane) order, and a warp walks it 32 items at a time, U loads in flight
// and U independent sums per lane.  Nothing waits for another warp, so chunks can be short and the GPU evenly full whatever N, C and
// S are.  CTAs that reduced whole images of a channel spent more on probing the shift, two block reductions and their ticket than on
// data: 128 x 512 x 14 x 14, cold cache: forward sums (51 MB) 25.8 us with them, 20.4 us with warps; gradient sums (103 MB) 34.6 and 27.9 us.
template <typename T>
struct ChunkWalk {
    int i, L, rstep, left;            // item in the plane, items per plane, 32 mod L, items of this lane still to come
    unsigned off, step, wrap;         // element offset; what 32 items and the end of a plane add to it
    __device__ __forceinline__ int init(int N, int C, int S, int c, int chunks, int j)
    {
        constexpr int V = (int)(sizeof(T) / sizeof(float));
        const int lane = threadIdx.x & 31;
        L = S / V;
        const int total = N * L, each = total / chunks, more = total - each * chunks;      // the first `more` chunks have one item more
        const int q = j * each + min(j, more) + lane, items = each + (j < more ? 1 : 0);
        const int n = q / L;
        i = q - n * L;
        left = items > lane ? (items - lane + 31) / 32 : 0;
        off = ((unsigned)n * (unsigned)C + (unsigned)c) * (unsigned)S + (unsigned)i * V;
        rstep = 32 % L;
        step = (unsigned)(32 / L) * (unsigned)C * (unsigned)S + (unsigned)rstep * V;
        wrap = (unsigned)(C - 1) * (unsigned)S;
        return items * V;             // elements of the chunk
    }
    // The next U items of x (and of y); returns how many this lane has.
    template <int U, bool TWO>
    __device__ __forceinline__ int load(const float *x, const float *y, T (&v)[U], T (&w)[U])
    {
        const int m = min(left, U);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (u < m) {
                v[u] = __ldg(reinterpret_cast<const T *>(x + off));
                if (TWO) w[u] = __ldg(reinterpret_cast<const T *>(y + off));
                off += step;
                i += rstep;
                if (i >= L) { i -= L; off += wrap; }
            }
        }
        left -= m;
        return m;
    }
};
__device__ __forceinline__ void each_of(const float4 &v, float (&o)[4]) { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
__device__ __forceinline__ void each_of(const float &v, float (&o)[1]) { o[0] = v; }

// The warp that hands in a channel's last partial finishes the channel: ticket counter per channel, zero before the launch and zero
// again after it.  Same answer in every lane.
__device__ __forceinline__ bool last_warp_of_channel(unsigned int *counters, int c, int chunks)
{
    int last = 0;
    if ((threadIdx.x & 31) == 0) {
        __threadfence();                                   // this warp's partial is visible before its ticket
        last = atomicAdd(counters + c, 1u) == (unsigned int)(chunks - 1);
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    __syncwarp();                                          // a shuffle orders no memory: the other lanes read after lane 0's ticket
    if (last) __threadfence();                            // the other warps' partials are visible after their tickets
    return last != 0;
}

// Shifted sums of one chunk: s1 = sum (x - k), s2 = sum (x - k)^2, with k the mean of the chunk's first (up to 32) items: close to the
// channel mean, so the sums of (x - k) stay small and keep their fp32 accuracy even when a single element is an outlier.
template <typename T, int U>
__device__ __forceinline__ ChunkStat chunk_stats(const float *x, int N, int C, int S, int c, int chunks, int j)
{
    constexpr int V = (int)(sizeof(T) / sizeof(float));
    ChunkWalk<T> w;
    const int elements = w.init(N, C, S, c, chunks, j);
    T v[U];
    int m = w.template load<U, false>(x, nullptr, v, v);
    // a power of two of equal values adds up without rounding: a constant channel has a variance of exactly zero
    const int probe = min(32, 1 << (31 - __clz(elements / V)));
    float first = 0.f, e[V];
    if ((int)(threadIdx.x & 31) < probe) {
        each_of(v[0], e);
        if constexpr (V == 4) first = ((e[0] + e[1]) + (e[2] + e[3])) * 0.25f;
        else first = e[0];
    }
    // no shift where the items hold an infinity or a NaN, or add up to one: x - k would be NaN for items that are neither
    float k = warp_sum(first) / (float)probe;
    if (!(fabsf(k) < INFINITY)) k = 0.f;
    float s1[U], s2[U];
#pragma unroll
    for (int u = 0; u < U; ++u) s1[u] = s2[u] = 0.f;
    while (m > 0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (u >= m) continue;
            each_of(v[u], e);
#pragma unroll
            for (int q = 0; q < V; ++q) {
                const float t = e[q] - k;
                s1[u] += t;
                s2[u] = fmaf(t, t, s2[u]);
            }
        }
        m = w.template load<U, false>(x, nullptr, v, v);
    }
#pragma unroll
    for (int h = U / 2; h > 0; h /= 2)
#pragma unroll
        for (int u = 0; u < h; ++u) { s1[u] += s1[u + h]; s2[u] += s2[u + h]; }
    return ChunkStat{k, warp_sum(s1[0]), warp_sum(s2[0]), (float)elements};
}

// One warp per (channel, chunk), eight to a CTA; with `counters` the last warp of a channel also merges the partials (no second
// launch).
__global__ void __launch_bounds__(256)
stats_kernel(const float *__restrict__ x, ChunkStat *__restrict__ part, int N, int C, int S, int chunks,
             unsigned int *__restrict__ counters, float *__restrict__ running_mean, float *__restrict__ running_var,
             float *__restrict__ save_mean, float *__restrict__ save_std, double momentum, double eps)
{
    const int id = (int)blockIdx.x * 8 + ((int)threadIdx.x >> 5);
    if (id >= C * chunks) return;
    const int j = id / C, c = id - j * C;                 // images in ascending order: see launch_apply
    const bool vec = (S % 4 == 0) && (((uintptr_t)x & 15) == 0);
    const ChunkStat s = vec ? chunk_stats<float4, 4>(x, N, C, S, c, chunks, j) : chunk_stats<float, 8>(x, N, C, S, c, chunks, j);
    if ((threadIdx.x & 31) == 0) part[(size_t)c * chunks + j] = s;
    if (counters && last_warp_of_channel(counters, c, chunks)) {
        finish_stats_channel_warp(part + (size_t)c * chunks, c, chunks, running_mean, running_var, save_mean, save_std, momentum, eps);
        if ((threadIdx.x & 31) == 0) counters[c] = 0u;
    }
}

// One thread per channel: the merge as a separate launch (more channels than ticket counters).
__global__ void __launch_bounds__(128)
stats_finish_kernel(const ChunkStat *__restrict__ part, int C, int chunks, float *__restrict__ running_mean,
                    float *__restrict__ running_var, float *__restrict__ save_mean, float *__restrict__ save_std,
                    double momentum, double eps)
{
    const int c = (int)blockIdx.x * 4 + ((int)threadIdx.x >> 5);
    if (c < C) finish_stats_channel_warp(part + (size_t)c * chunks, c, chunks, running_mean, running_var, save_mean, save_std, momentum, eps);
}

// gamma * (x - mean) * invstd + beta with every rounding pinned (no fused multiply-add), so that the backward
// kernels can recompute the sign of the forward value bit for bit.
__device__ __forceinline__ float bn_value(float v, float mean, float invstd, float g, float b)
{
    return __fadd_rn(__fmul_rn(__fmul_rn(g, __fsub_rn(v, mean)), invstd), b);
}

// y = gamma * (x - mean) * invstd + beta, per plane.  Training reads mean / invstd from save_*, inference
// derives them from the running statistics.
// GROUP threads (a warp for small planes, the whole CTA for large ones) share a plane.
template <bool RELU, int GROUP>
__global__ void __launch_bounds__(256)
apply_kernel(const float *__restrict__ x, float *__restrict__ y, const float *__restrict__ weight,
             const float *__restrict__ bias, const float *__restrict__ mean_v, const float *__restrict__ std_or_var,
             int train, float eps, int C, int S, long long planes)
{
    auto act = [](float v) { return RELU ? (v > 0.f ? v : 0.f) : v; };
    const bool vec = (S % 4 == 0) && ((((uintptr_t)x | (uintptr_t)y) & 15) == 0);
    constexpr int PER_CTA = 256 / GROUP;
    const int sub = (int)threadIdx.x / GROUP, t = (int)threadIdx.x % GROUP;
    for (long long rev = (long long)blockIdx.x * PER_CTA + sub; rev < planes; rev += (long long)gridDim.x * PER_CTA) {
        const long long pl = planes - 1 - rev;                   // last image first
        const int c = (int)(pl % C);
        const float mean = __ldg(mean_v + c);
        const float invstd = train ? __ldg(std_or_var + c) : 1.f / sqrtf(__ldg(std_or_var + c) + eps);
        const float g = weight ? __ldg(weight + c) : 1.f;
        const float b = bias ? __ldg(bias + c) : 0.f;
        const float *xp = x + pl * S;
        float *yp = y + pl * S;
        if (vec) {
            const float4 *x4 = reinterpret_cast<const float4 *>(xp);
            float4 *y4 = reinterpret_cast<float4 *>(yp);
#pragma unroll 4
            for (int i = t; i < S / 4; i += GROUP) {
                const float4 v = __ldg(x4 + i);
                float4 o;
                o.x = act(bn_value(v.x, mean, invstd, g, b));
                o.y = act(bn_value(v.y, mean, invstd, g, b));
                o.z = act(bn_value(v.z, mean, invstd, g, b));
                o.w = act(bn_value(v.w, mean, invstd, g, b));
                y4[i] = o;
            }
        } else {
            for (int i = t; i < S; i += GROUP) yp[i] = act(bn_value(__ldg(xp + i), mean, invstd, g, b));
        }
    }
}

// Planes whose size is not a multiple of 4 (7x7 = 49 elements): the tensor is walked as one flat array of 16-byte
// items, four per thread and iteration; an item may straddle planes, so the channel is tracked element by element.
template <bool RELU>
__global__ void __launch_bounds__(256)
apply_flat_kernel(const float *__restrict__ x, float *__restrict__ y, const float *__restrict__ weight,
                  const float *__restrict__ bias, const float *__restrict__ mean_v, const float *__restrict__ std_or_var,
                  int train, float eps, unsigned C, unsigned S, unsigned total)
{
    auto act = [](float v) { return RELU ? (v > 0.f ? v : 0.f) : v; };
    float mean = 0.f, invstd = 0.f, g = 1.f, b = 0.f;
    auto fetch = [&](unsigned c) {
        mean = __ldg(mean_v + c);
        invstd = train ? __ldg(std_or_var + c) : 1.f / sqrtf(__ldg(std_or_var + c) + eps);
        g = weight ? __ldg(weight + c) : 1.f;
        b = bias ? __ldg(bias + c) : 0.f;
    };
    auto item = [&](unsigned q, const float4 v) {
        const unsigned e = q * 4u, pl = e / S;
        unsigned r = e - pl * S, c = pl % C;
        fetch(c);
        const float in[4] = {v.x, v.y, v.z, v.w};
        float out[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            out[j] = act(bn_value(in[j], mean, invstd, g, b));
            if (j < 3 && ++r == S) {
                r = 0;
                if (++c == C) c = 0;
                fetch(c);
            }
        }
        reinterpret_cast<float4 *>(y)[q] = make_float4(out[0], out[1], out[2], out[3]);
    };
    const unsigned items = total / 4u, stride = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    constexpr unsigned U = 4;
    for (unsigned q = tid; q < items; q += U * stride) {
        float4 v[U];
#pragma unroll
        for (unsigned u = 0; u < U; ++u)
            if (q + u * stride < items) v[u] = __ldg(x4 + (items - 1 - (q + u * stride)));       // last image first
#pragma unroll
        for (unsigned u = 0; u < U; ++u)
            if (q + u * stride < items) item(items - 1 - (q + u * stride), v[u]);
    }
    if (tid < total - items * 4u) {
        const unsigned e = items * 4u + tid;
        fetch((e / S) % C);
        y[e] = act(bn_value(__ldg(x + e), mean, invstd, g, b));
    }
}

// Per-channel coefficients of the input gradient:
//   gx = (gy - (x - mean) * proj - gmean) * gscale      (training)
//   gx = gy * gscale                                     (inference)
struct GradCoef {
    float mean, proj, gmean, gscale;
    float invstd, gamma, beta, pad;     // forward coefficients, for the sign of the fused ReLU's input
};

// Backward, pass 2 for channel c: totals the chunk sums in fp64, accumulates gradWeight / gradBias and publishes
// the coefficients of the input gradient.
// By one warp: lanes add strided subsets and are then folded in a fixed order, so the result does not depend on timing.
// Lane 0 publishes.
__device__ __forceinline__ void finish_grad_channel_warp(const float2 *part, int c, int chunks, long long count, const float *weight,
                                                         const float *bias, const float *mean_v, const float *std_or_var,
                                                         int train, double eps, double scale, float *grad_weight,
                                                         float *grad_bias, GradCoef *coef)
{
    const int lane = threadIdx.x & 31;
    double s = 0.0, d = 0.0;
#pragma unroll 4
    for (int j = lane; j < chunks; j += 32) {
        const float2 p = __ldcg(part + j);
        s += (double)p.x;
        d += (double)p.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        d += __shfl_down_sync(0xffffffffu, d, o);
    }
    if (lane != 0) return;
    const float mean = mean_v[c];
    const float stdv = train ? std_or_var[c] : (float)(1.0 / sqrt((double)std_or_var[c] + eps));
    const float w = weight ? weight[c] : 1.f;
    const double norm = 1.0 / (double)count;
    GradCoef k;
    k.mean = mean;
    k.gmean = (float)(s * norm);
    k.proj = (float)(d * norm * (double)stdv * (double)stdv);
    k.gscale = stdv * w;
    k.invstd = train ? std_or_var[c] : 1.f / sqrtf(std_or_var[c] + (float)eps);   // as the forward kernel computes it
    k.gamma = w;
    k.beta = bias ? bias[c] : 0.f;
    k.pad = 0.f;
    coef[c] = k;
    if (grad_weight) grad_weight[c] = (float)((double)grad_weight[c] + scale * d * (double)stdv);
    if (grad_bias) grad_bias[c] = (float)((double)grad_bias[c] + scale * s);
}

__global__ void __launch_bounds__(128)
grad_finish_kernel(const float2 *__restrict__ part, int C, int chunks, long long count,
                   const float *__restrict__ weight, const float *__restrict__ bias, const float *__restrict__ mean_v,
                   const float *__restrict__ std_or_var, int train, double eps, double scale,
                   float *__restrict__ grad_weight, float *__restrict__ grad_bias, GradCoef *__restrict__ coef)
{
    const int c = (int)blockIdx.x * 4 + ((int)threadIdx.x >> 5);
    if (c < C) finish_grad_channel_warp(part + (size_t)c * chunks, c, chunks, count, weight, bias, mean_v, std_or_var, train, eps, scale, grad_weight, grad_bias, coef);
}

// Sums of gy and gy * (x - mean) over one chunk.
template <typename T, int U, bool RELU>
__device__ __forceinline__ float2 chunk_grad_sums(const float *x, const float *gy, int N, int C, int S, int c, int chunks, int j, float mean,
                                                  float invstd, float gam, float bet)
{
    constexpr int V = (int)(sizeof(T) / sizeof(float));
    ChunkWalk<T> w;
    w.init(N, C, S, c, chunks, j);
    T xv[U], gv[U];
    float s[U], d[U], e[V], f[V];
#pragma unroll
    for (int u = 0; u < U; ++u) s[u] = d[u] = 0.f;
    for (;;) {
        const int m = w.template load<U, true>(x, gy, xv, gv);
        if (m <= 0) break;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (u >= m) continue;
            each_of(xv[u], e);
            each_of(gv[u], f);
#pragma unroll
            for (int q = 0; q < V; ++q) {
                // fused ReLU: the gradient passes only where the forward value was positive; its sign is recomputed from x
                const float g = RELU ? (bn_value(e[q], mean, invstd, gam, bet) > 0.f ? f[q] : 0.f) : f[q];
                s[u] += g;
                d[u] = fmaf(g, e[q] - mean, d[u]);
            }
        }
    }
#pragma unroll
    for (int h = U / 2; h > 0; h /= 2)
#pragma unroll
        for (int u = 0; u < h; ++u) { s[u] += s[u + h]; d[u] += d[u + h]; }
    return make_float2(warp_sum(s[0]), warp_sum(d[0]));
}

// Backward, pass 1: the sums of every (channel, chunk), one warp each.
template <bool RELU>
__global__ void __launch_bounds__(256)
grad_stats_kernel(const float *__restrict__ x, const float *__restrict__ gy, float2 *__restrict__ part,
                  const float *__restrict__ mean_v, const float *__restrict__ std_or_var, const float *__restrict__ weight,
                  const float *__restrict__ bias, int train, float eps, int N, int C, int S, int chunks,
                  unsigned int *__restrict__ counters, double eps_d, double scale, float *__restrict__ grad_weight,
                  float *__restrict__ grad_bias, GradCoef *__restrict__ coef)
{
    const int id = (int)blockIdx.x * 8 + ((int)threadIdx.x >> 5);
    if (id >= C * chunks) return;
    const int j = id / C, c = id - j * C;                 // images in ascending order: see launch_apply
    const float mean = __ldg(mean_v + c);
    float invstd = 0.f, gam = 1.f, bet = 0.f;
    if (RELU) {
        invstd = train ? __ldg(std_or_var + c) : 1.f / sqrtf(__ldg(std_or_var + c) + eps);
        gam = weight ? __ldg(weight + c) : 1.f;
        bet = bias ? __ldg(bias + c) : 0.f;
    }
    const bool vec = (S % 4 == 0) && ((((uintptr_t)x | (uintptr_t)gy) & 15) == 0);
    const float2 p = vec ? chunk_grad_sums<float4, 4, RELU>(x, gy, N, C, S, c, chunks, j, mean, invstd, gam, bet)
                         : chunk_grad_sums<float, 8, RELU>(x, gy, N, C, S, c, chunks, j, mean, invstd, gam, bet);
    if ((threadIdx.x & 31) == 0) part[(size_t)c * chunks + j] = p;
    if (counters && last_warp_of_channel(counters, c, chunks)) {
        finish_grad_channel_warp(part + (size_t)c * chunks, c, chunks, (long long)N * S, weight, bias, mean_v, std_or_var, train, eps_d, scale, grad_weight,
                                 grad_bias, coef);
        if ((threadIdx.x & 31) == 0) counters[c] = 0u;
    }
}

// Backward, pass 3: the input gradient.
template <bool RELU, int GROUP>
__global__ void __launch_bounds__(256)
grad_apply_kernel(const float *__restrict__ x, const float *__restrict__ gy, float *__restrict__ gx,
                  const GradCoef *__restrict__ coef, int train, int C, int S, long long planes)
{
    const bool vec = (S % 4 == 0) && ((((uintptr_t)x | (uintptr_t)gy | (uintptr_t)gx) & 15) == 0);
    constexpr int PER_CTA = 256 / GROUP;
    const int sub = (int)threadIdx.x / GROUP, t = (int)threadIdx.x % GROUP;
    for (long long rev = (long long)blockIdx.x * PER_CTA + sub; rev < planes; rev += (long long)gridDim.x * PER_CTA) {
        const long long pl = planes - 1 - rev;                   // last image first
        const GradCoef k = coef[pl % C];
        const float *xp = x + pl * S;
        const float *gp = gy + pl * S;
        float *op = gx + pl * S;
        if (vec) {
            const float4 *x4 = reinterpret_cast<const float4 *>(xp);
            const float4 *g4 = reinterpret_cast<const float4 *>(gp);
            float4 *o4 = reinterpret_cast<float4 *>(op);
#pragma unroll 4
            for (int i = t; i < S / 4; i += GROUP) {
                float4 g = __ldg(g4 + i);
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (RELU || train) v = __ldg(x4 + i);
                if (RELU) {
                    g.x = bn_value(v.x, k.mean, k.invstd, k.gamma, k.beta) > 0.f ? g.x : 0.f;
                    g.y = bn_value(v.y, k.mean, k.invstd, k.gamma, k.beta) > 0.f ? g.y : 0.f;
                    g.z = bn_value(v.z, k.mean, k.invstd, k.gamma, k.beta) > 0.f ? g.z : 0.f;
                    g.w = bn_value(v.w, k.mean, k.invstd, k.gamma, k.beta) > 0.f ? g.w : 0.f;
                }
                float4 o;
                if (train) {
                    o.x = (g.x - (v.x - k.mean) * k.proj - k.gmean) * k.gscale;
                    o.y = (g.y - (v.y - k.mean) * k.proj - k.gmean) * k.gscale;
                    o.z = (g.z - (v.z - k.mean) * k.proj - k.gmean) * k.gscale;
                    o.w = (g.w - (v.w - k.mean) * k.proj - k.gmean) * k.gscale;
                } else {
                    o.x = g.x * k.gscale; o.y = g.y * k.gscale; o.z = g.z * k.gscale; o.w = g.w * k.gscale;
                }
                o4[i] = o;
            }
        } else {
            for (int i = t; i < S; i += GROUP) {
                float g = __ldg(gp + i);
                const float v = (RELU || train) ? __ldg(xp + i) : 0.f;
                if (RELU) g = bn_value(v, k.mean, k.invstd, k.gamma, k.beta) > 0.f ? g : 0.f;
                op[i] = train ? (g - (v - k.mean) * k.proj - k.gmean) * k.gscale : g * k.gscale;
            }
        }
    }
}

// The flat walk of apply_flat_kernel for the input gradient.
template <bool RELU>
__global__ void __launch_bounds__(256)
grad_apply_flat_kernel(const float *__restrict__ x, const float *__restrict__ gy, float *__restrict__ gx,
                       const GradCoef *__restrict__ coef, int train, unsigned C, unsigned S, unsigned total)
{
    GradCoef k;
    auto fetch = [&](unsigned c) {
        const float4 *p = reinterpret_cast<const float4 *>(coef + c);
        const float4 a = __ldg(p), b = __ldg(p + 1);
        k.mean = a.x; k.proj = a.y; k.gmean = a.z; k.gscale = a.w;
        k.invstd = b.x; k.gamma = b.y; k.beta = b.z; k.pad = b.w;
    };
    auto one = [&](float v, float g) {
        if (RELU) g = bn_value(v, k.mean, k.invstd, k.gamma, k.beta) > 0.f ? g : 0.f;
        return train ? (g - (v - k.mean) * k.proj - k.gmean) * k.gscale : g * k.gscale;
    };
    auto item = [&](unsigned q, const float4 v, const float4 g) {
        const unsigned e = q * 4u, pl = e / S;
        unsigned r = e - pl * S, c = pl % C;
        fetch(c);
        const float vin[4] = {v.x, v.y, v.z, v.w}, gin[4] = {g.x, g.y, g.z, g.w};
        float out[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            out[j] = one(vin[j], gin[j]);
            if (j < 3 && ++r == S) {
                r = 0;
                if (++c == C) c = 0;
                fetch(c);
            }
        }
        reinterpret_cast<float4 *>(gx)[q] = make_float4(out[0], out[1], out[2], out[3]);
    };
    const unsigned items = total / 4u, stride = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
    const float4 *x4 = reinterpret_cast<const float4 *>(x), *g4 = reinterpret_cast<const float4 *>(gy);
    const bool need_x = RELU || train;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    constexpr unsigned U = 4;
    for (unsigned q = tid; q < items; q += U * stride) {
        float4 v[U], g[U];
#pragma unroll
        for (unsigned u = 0; u < U; ++u) {
            v[u] = zero;
            if (q + u * stride < items) {
                const unsigned at = items - 1 - (q + u * stride);             // last image first
                g[u] = __ldg(g4 + at);
                if (need_x) v[u] = __ldg(x4 + at);
            }
        }
#pragma unroll
        for (unsigned u = 0; u < U; ++u)
            if (q + u * stride < items) item(items - 1 - (q + u * stride), v[u], g[u]);
    }
    if (tid < total - items * 4u) {
        const unsigned e = items * 4u + tid;
        fetch((e / S) % C);
        gx[e] = one(need_x ? __ldg(x + e) : 0.f, __ldg(gy + e));
    }
}


// ---------------------------------------------------------------------------------------------------------------
// Grouped passes: statistics and normalisation in ONE launch, ordered so that the second read of x finds it in L2.
//
// The two-launch path above streams the whole tensor twice through HBM (3 tensor passes forward, 5 backward, for
// 2 and 3 algorithmic ones): by the time the normalise kernel starts, the statistics kernel has pushed the start
// of the tensor out of the 126 MB L2.  Here the channels are taken in groups whose slabs (N planes per channel)
// fit in a fraction of L2, and a persistent grid of co-resident CTAs (cooperative launch) walks the groups.
//
// Every CTA is two halves — eight consumer warps and one copy-issuing warp each — with a stream of their own (with four consumer warps the
// forward pass of 256 x 64 x 112 x 112 took 416 us, the backward pass 13 % more than two launches; now 382 and 6 %.  Less than 128 MB, where
// a group's sums and flags weigh more, has four: 64 x 8 x 224 x 224 62 us with eight, 56 with four):
//   * the statistics half reduces group after group (reads carry an L2 evict_last policy), hands in one partial
//     per (CTA, channel) and takes a ticket; the CTA that draws a channel's last ticket merges the partials in fp64
//     (in CTA order: results do not depend on timing), publishes mean / inverse std (or the gradient coefficients)
//     and raises the channel's ready flag.  It never waits for another CTA, so it keeps HBM busy;
//   * the apply half follows: per channel it waits for the ready flag — with a cycle limit, after which it records
//     STATUS_FLAG_TIMEOUT and the CTA leaves — re-reads the group (evict_first: finished data leaves L2 first) and
//     writes the result with 16-byte stores.  The last reader of a flag lowers it again.
// The statistics half stays at most two groups ahead of its own CTA's apply half, which bounds what must stay
// resident in L2.  All counters and flags are zero before the launch and zero after it.
//
// Data movement: each half sees its launch as ONE stream of stages (a stage = up to P consecutive float4 items of
// one channel's sequence, i.e. a few runs of whole or partial planes).  The half's producer warp keeps kStages stages
// in flight with 1-D TMA bulk copies into a shared-memory ring (a full and an empty mbarrier per slot, bounded
// waits), across group boundaries: bytes in flight do not depend on registers or on the occupancy of the arithmetic,
// and issuing copies is off the consumers' critical path.
//
// Work split: inside a group, the float4 items of its channels form one sequence (channel-major, N*L items per
// channel); CTA b takes the b-th of `grid` equal shares, which may span channel boundaries ("segments").
//
// Forward statistics are shifted, share by share, by the mean of the share's first stage (which takes 1 % of the time): sums of (x - K) and (x - K)^2 keep their fp32 accuracy
// when |mean| >> std and when an image has a border.  (With one shift per channel, from the first 32 elements of its first image, channels
// of mean / std 100 whose first 32 were zero had variances off by 6e-4.)  The partials merge in fp64 as those of the two-launch path.
struct GroupPlan {
    int N, C, S, L;         // L = S / 4: float4 items per plane
    int G, groups;          // channels per group (the last group may be smaller), number of groups
    int pstride;            // partial slots per channel
    int lookahead;          // groups the statistics half may run ahead of its CTA's apply half
    long long NL;           // items per channel
};

constexpr int kStages = 3;              // per half
constexpr int kStageBytes = 16384;      // per slot: 1024 items of one tensor (forward) or 512 items of two (backward)
// HW: warps of a half that consume; each half has one more that only issues copies.
constexpr int grouped_threads(int hw) { return 2 * 32 * (hw + 1); }

__device__ __forceinline__ unsigned long long l2_policy_evict_last()
{
    unsigned long long p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ unsigned long long l2_policy_evict_first()
{
    unsigned long long p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void st_hint(float4 *p, const float4 v, unsigned long long pol)
{
    asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;"
                 ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "l"(pol) : "memory");
}
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u32(unsigned *p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Barrier among the consumer threads of one half (barrier 0 is __syncthreads).
template <int HW>
__device__ __forceinline__ void half_sync(int half)
{
    if (half == 0) asm volatile("bar.sync 1, %0;" ::"n"(32 * HW) : "memory");
    else asm volatile("bar.sync 2, %0;" ::"n"(32 * HW) : "memory");
}

// Sum over one half, in fp64; sh: a double per warp of that half.
template <int HW>
__device__ __forceinline__ float half_sum(float v, double *sh, int half)
{
    const double d = warp_sum((double)v);
    const int lane = threadIdx.x & 31, w = (int)(threadIdx.x >> 5) % (HW + 1);
    half_sync<HW>(half);
    if (lane == 0) sh[w] = d;
    half_sync<HW>(half);
    double t = 0.0;
#pragma unroll
    for (int i = 0; i < HW; ++i) t += sh[i];
    return (float)t;
}

// The shift of a segment, by all consumers of the half: the mean of as many of the `len` items that begin it as are a power of two.  Equal values
// add up without rounding, so that a constant channel has a variance of exactly zero.  No shift where they hold an infinity or a NaN, or
// add up to one: x - K would be NaN for values that are neither.
template <int HW>
__device__ __forceinline__ float segment_shift(const float4 *items, int len, int ht, double *sh)
{
    constexpr int kHalf = 32 * HW;
    const int n = 1 << (31 - __clz(len));
    auto at = [&](int j) {
        if (j >= n) return 0.f;
        const float4 q = items[j];
        return ((q.x + q.y) + (q.z + q.w)) * 0.25f;
    };
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < kStageBytes / 16; j += 4 * kHalf) v += (at(ht + j) + at(ht + j + kHalf)) + (at(ht + j + 2 * kHalf) + at(ht + j + 3 * kHalf));
    v = warp_sum(v);
    half_sync<HW>(0);
    if ((ht & 31) == 0) sh[ht >> 5] = (double)v;
    half_sync<HW>(0);
    double t[HW];
#pragma unroll
    for (int i = 0; i < HW; ++i) t[i] = sh[i];
#pragma unroll
    for (int h = HW / 2; h > 0; h /= 2)
#pragma unroll
        for (int i = 0; i < h; ++i) t[i] += t[i + h];
    const float k = (float)t[0] / (float)n;
    return fabsf(k) < INFINITY ? k : 0.f;
}

// The CTAs whose shares touch channel cl (local index in the group) of a group of W items: first and last.
__device__ __forceinline__ void channel_ctas(long long W, long long NL, int cl, int grid, int *b_first, int *b_last)
{
    *b_first = (int)((((long long)cl * NL + 1) * grid + W - 1) / W) - 1;
    *b_last = (int)((((long long)(cl + 1) * NL) * grid + W - 1) / W) - 1;
}

struct GroupCounters {
    unsigned *tick, *ready, *done;
};

// One stage of a half's stream.
struct Stage {
    int g, cl, c;           // group, channel inside the group, channel
    int q, len;             // first item (in the channel's sequence) and item count
    bool seg_first, seg_last, group_last;
    int seg_items;          // items of the whole segment
};

// Enumerates the stages of CTA b, group after group.  Pure integer arithmetic on uniform values: the producer warp
// and the consumers each step a copy of their own.
struct StageIter {
    GroupPlan gp;
    int grid, b, P;
    int g, Gg, cl;
    long long W, lo, hi, pos, seg_end;   // the CTA's share [lo, hi) of the group sequence; position; end of the segment
    bool in_group;

    __device__ __forceinline__ void init(const GroupPlan &gp_, int grid_, int b_, int P_)
    {
        gp = gp_; grid = grid_; b = b_; P = P_;
        g = -1; in_group = false;
    }
    __device__ __forceinline__ void enter_group()
    {
        Gg = min(gp.G, gp.C - g * gp.G);
        W = (long long)Gg * gp.NL;
        lo = W * b / grid; hi = W * (b + 1) / grid;
        pos = lo;
        cl = (int)(lo / gp.NL);
        seg_end = min(hi, (long long)(cl + 1) * gp.NL);
        in_group = pos < hi;
    }
    __device__ __forceinline__ bool next(Stage &st)
    {
        while (!in_group) {
            if (++g >= gp.groups) return false;
            enter_group();
        }
        const long long cbeg = (long long)cl * gp.NL;
        const long long seg_beg = max(lo, cbeg);
        st.g = g; st.cl = cl; st.c = g * gp.G + cl;
        st.q = (int)(pos - cbeg);
        st.len = (int)min((long long)P, seg_end - pos);
        st.seg_first = pos == seg_beg;
        st.seg_items = (int)(seg_end - seg_beg);
        pos += st.len;
        st.seg_last = pos == seg_end;
        st.group_last = false;
        if (st.seg_last) {
            if (pos >= hi) { in_group = false; st.group_last = true; }
            else { ++cl; seg_end = min(hi, (long long)(cl + 1) * gp.NL); }
        }
        return true;
    }
};

// One warp: copies stage st of `tensors` tensors into a ring slot (runs of whole or partial planes, one bulk copy
// each, all counted on the slot's barrier).
template <int TENSORS>
__device__ __forceinline__ void issue_stage(const Stage &st, const GroupPlan &gp, const float4 *t0, const float4 *t1,
                                            float4 *slot_mem, int P, uint32_t bar, unsigned long long pol)
{
    const int lane = threadIdx.x & 31;
    if (lane == 0) mbar_arrive_expect_tx(bar, (uint32_t)st.len * 16u * TENSORS);
    __syncwarp();
    const int L = gp.L;
    const int n0 = st.q / L, i0 = st.q - n0 * L, end = st.q + st.len;
    const int runs = (end - 1) / L - n0 + 1;
    const long long CL = (long long)gp.C * L, cbase = (long long)st.c * L;
    for (int r = lane; r < runs; r += 32) {
        const int start = r == 0 ? st.q : (n0 + r) * L;
        const int rlen = min(r == 0 ? L - i0 : L, end - start);
        const long long goff = cbase + (long long)(n0 + r) * CL + (r == 0 ? i0 : 0);
        bulk_g2s_hint(smem_u32(slot_mem + (start - st.q)), t0 + goff, (uint32_t)rlen * 16u, bar, pol);
        if (TENSORS == 2) bulk_g2s_hint(smem_u32(slot_mem + P + (start - st.q)), t1 + goff, (uint32_t)rlen * 16u, bar, pol);
    }
}

struct GroupedArgs {
    const float *x, *gy;             // gy: backward only
    float *out;                      // y (forward) or gx (backward)
    const float *weight, *bias;
    void *part;                      // ChunkStat (forward) or float2 partials, pstride per channel
    GroupCounters cn;
    float *running_mean, *running_var, *save_mean, *save_std;     // forward: written
    const float *mean_v, *std_or_var;                              // backward: saved or running statistics
    float *grad_weight, *grad_bias;
    GradCoef *coef;
    double momentum, eps, scale;
    int train;
    GroupPlan gp;
    int *status;
};

template <bool BWD, bool RELU, int HW>
__global__ void __launch_bounds__(grouped_threads(HW), 2)
grouped_kernel(const GroupedArgs a)
{
    constexpr int T = BWD ? 2 : 1;
    constexpr int P = kStageBytes / 16 / T, kHalf = 32 * HW;
    extern __shared__ __align__(128) unsigned char ring_raw[];
    __shared__ __align__(8) unsigned long long full_s[2][kStages];      // slot filled (transaction bytes)
    __shared__ __align__(8) unsigned long long empty_s[2][kStages];     // slot read by the half's consumer warps
    __shared__ double sums_s[2][HW];
    __shared__ int flag_s[2];
    __shared__ volatile int applied_s;       // groups this CTA's apply half has finished
    __shared__ volatile int abort_s;         // a wait ran out somewhere in the CTA: everybody leaves

    const GroupPlan gp = a.gp;
    const int grid = (int)gridDim.x, b = (int)blockIdx.x;
    const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
    const int half = warp / (HW + 1), wi = warp % (HW + 1);                           // wi == HW: the half's producer warp
    const int ht = wi * 32 + lane;                                      // consumer index inside the half
    float4 *ring = reinterpret_cast<float4 *>(ring_raw) + (size_t)half * kStages * T * P;     // [kStages][T][P] of this half
    unsigned long long *bars = full_s[half], *empties = empty_s[half];
    double *sh = sums_s[half];
    const float4 *x4 = reinterpret_cast<const float4 *>(a.x), *g4 = reinterpret_cast<const float4 *>(a.gy);
    const unsigned long long pol = half == 0 ? l2_policy_evict_last() : l2_policy_evict_first();

    if (threadIdx.x == 0) {
        for (int h = 0; h < 2; ++h)
            for (int s = 0; s < kStages; ++s) {
                mbar_init(smem_u32(&full_s[h][s]), 1);
                mbar_init(smem_u32(&empty_s[h][s]), HW);
            }
        mbar_fence_init();
        applied_s = 0;
        abort_s = 0;
    }
    __syncthreads();

    // A bounded wait on a barrier phase that also gives up when another part of the CTA has.
    auto wait_phase = [&](unsigned long long *bar, uint32_t parity) -> bool {
        const uint32_t addr = smem_u32(bar);
        if (mbar_try_wait(addr, parity)) return true;
        const long long t0 = clock64();
        while (!mbar_try_wait(addr, parity)) {
            if (abort_s) return false;
            if (clock64() - t0 > 2000000000LL) {
                if (a.status) atomicExch(a.status, (int)STATUS_MBARRIER_TIMEOUT);
                abort_s = 1;
                return false;
            }
        }
        return true;
    };

    if (wi == HW) {
        // ------------------------------------------------ producer warp of this half -----------------------------------
        // Issues every stage of the half's stream, kStages ahead of the consumers: a slot is refilled as soon as the
        // consumer warps have released it.  Before leaving it lets its last copies land (shared memory stays valid until
        // the whole CTA has exited, but nothing may still be in flight when it does).
        StageIter prod;
        prod.init(gp, grid, b, P);
        Stage ps;
        int i = 0;
        for (; prod.next(ps); ++i) {
            const int slot = i % kStages;
            if (i >= kStages && !wait_phase(empties + slot, (uint32_t)(((i / kStages) - 1) & 1))) break;
            issue_stage<T>(ps, gp, x4, g4, ring + (size_t)slot * T * P, P, smem_u32(bars + slot), pol);
        }
        for (int j = max(0, i - kStages); j < i; ++j)
            if (!wait_phase(bars + j % kStages, (uint32_t)((j / kStages) & 1))) break;
        return;
    }

    StageIter cons;
    cons.init(gp, grid, b, P);
    Stage st;
    // The consumers of a half are done with a slot: one arrival per warp.
    auto release_slot = [&](int slot) {
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(empties + slot));
    };
    // Thread 0 of the half polls cond() with a cycle limit; the whole half learns the outcome.
    auto bounded = [&](auto cond) -> bool {
        if (ht == 0) {
            int ok = 1;
            if (!cond()) {
                const long long t0 = clock64();
                while (!cond()) {
                    if (abort_s || clock64() - t0 > 2000000000LL) {
                        if (!abort_s && a.status) atomicExch(a.status, (int)STATUS_FLAG_TIMEOUT);
                        abort_s = 1;
                        ok = 0;
                        break;
                    }
                    __nanosleep(64);
                }
            }
            flag_s[half] = ok;
        }
        half_sync<HW>(half);
        const bool ok = flag_s[half] != 0;
        half_sync<HW>(half);
        return ok;
    };
    const int qstep = kHalf / gp.L, rstep = kHalf % gp.L;
    const long long CL = (long long)gp.C * gp.L;

    if (half == 0) {
        // ------------------------------------------------ statistics half ------------------------------------------------
        // forward: shift, sum (x - K), sum (x - K)^2; backward: a1 = sum gy, a2 + b2 = sum gy (x - mean), in two halves, so that a thread's chains are
        // as short as those of the two-launch path (one chain had up to twice its error)
        float K = 0.f, a1 = 0.f, a2 = 0.f, b2 = 0.f;
        float mean = 0.f, invstd = 0.f, gam = 1.f, bet = 0.f;
        for (int it = 0; cons.next(st); ++it) {
            const int slot = it % kStages;
            const float4 *sx = ring + (size_t)slot * T * P, *sg = sx + P;
            const int c = st.c;
            if (st.seg_first) {
                // stay at most `lookahead` groups ahead of this CTA's apply half
                if (st.g >= gp.lookahead && !bounded([&] { return applied_s >= st.g - gp.lookahead + 1; })) return;
                a1 = 0.f; a2 = 0.f; b2 = 0.f;
                if (BWD) {
                    mean = __ldg(a.mean_v + c);
                    if (RELU) {
                        invstd = a.train ? __ldg(a.std_or_var + c) : 1.f / sqrtf(__ldg(a.std_or_var + c) + (float)a.eps);
                        gam = a.weight ? __ldg(a.weight + c) : 1.f;
                        bet = a.bias ? __ldg(a.bias + c) : 0.f;
                    }
                }
            }
            if (!wait_phase(bars + slot, (uint32_t)((it / kStages) & 1))) return;
            if (!BWD) {
                if (st.seg_first) K = segment_shift<HW>(sx, st.len, ht, sh);
#pragma unroll 4
                for (int j = ht; j < st.len; j += kHalf) {
                    const float4 q = sx[j];
                    const float e = q.x - K, f = q.y - K, gg = q.z - K, h = q.w - K;
                    a1 += (e + f) + (gg + h);
                    a2 = fmaf(e, e, a2); a2 = fmaf(f, f, a2); a2 = fmaf(gg, gg, a2); a2 = fmaf(h, h, a2);
                }
            } else {
                auto one = [&](float v, float g_) { return RELU ? (bn_value(v, mean, invstd, gam, bet) > 0.f ? g_ : 0.f) : g_; };
#pragma unroll 2
                for (int j = ht; j < st.len; j += kHalf) {
                    const float4 xv = sx[j];
                    float4 gv = sg[j];
                    gv.x = one(xv.x, gv.x); gv.y = one(xv.y, gv.y); gv.z = one(xv.z, gv.z); gv.w = one(xv.w, gv.w);
                    a1 += (gv.x + gv.y) + (gv.z + gv.w);
                    a2 = fmaf(gv.x, xv.x - mean, a2); b2 = fmaf(gv.y, xv.y - mean, b2);
                    a2 = fmaf(gv.z, xv.z - mean, a2); b2 = fmaf(gv.w, xv.w - mean, b2);
                }
            }
            release_slot(slot);
            if (st.seg_last) {
                // hand in this segment's partial; the CTA with the channel's last ticket merges and raises the flag
                a1 = half_sum<HW>(a1, sh, 0);
                a2 = half_sum<HW>(a2 + b2, sh, 0);
                int bf, bl;
                channel_ctas((long long)min(gp.G, gp.C - st.g * gp.G) * gp.NL, gp.NL, st.cl, grid, &bf, &bl);
                const int cnt = bl - bf + 1;
                ChunkStat *stats = reinterpret_cast<ChunkStat *>(a.part) + (size_t)c * gp.pstride;
                float2 *sums = reinterpret_cast<float2 *>(a.part) + (size_t)c * gp.pstride;
                if (ht == 0) {
                    if (BWD) sums[b - bf] = make_float2(a1, a2);
                    else stats[b - bf] = ChunkStat{K, a1, a2, (float)(st.seg_items * 4)};
                    __threadfence();                                  // the partial is visible before the ticket
                    flag_s[0] = atomicAdd(a.cn.tick + c, 1u) == (unsigned)(cnt - 1);
                }
                half_sync<HW>(0);
                const bool last = flag_s[0] != 0;
                half_sync<HW>(0);
                if (last) {
                    __threadfence();                                  // the other CTAs' partials are visible after their tickets
                    if (ht < 32) {
                        if (!BWD)
                            finish_stats_channel_warp(stats, c, cnt, a.running_mean, a.running_var, a.save_mean, a.save_std, a.momentum, a.eps);
                        else
                            finish_grad_channel_warp(sums, c, cnt, (long long)gp.N * gp.S, a.weight, a.bias, a.mean_v, a.std_or_var, a.train,
                                                     a.eps, a.scale, a.grad_weight, a.grad_bias, a.coef);
                        if (ht == 0) {
                            a.cn.tick[c] = 0u;
                            __threadfence();
                            st_release_u32(a.cn.ready + c, 1u);
                        }
                    }
                }
            }
        }
    } else {
        // -------------------------------------------------- apply half --------------------------------------------------
        float4 *o4 = reinterpret_cast<float4 *>(a.out);
        float mean = 0.f, invstd = 0.f, gam = 1.f, bet = 0.f;
        GradCoef kf{};
        const unsigned long long drop = pol;
        for (int it = 0; cons.next(st); ++it) {
            const int slot = it % kStages;
            const float4 *sx = ring + (size_t)slot * T * P, *sg = sx + P;
            const int c = st.c;
            if (st.seg_first) {
                // the statistics (or gradient coefficients) of this channel must have been merged
                const unsigned *rf = a.cn.ready + c;
                if (!bounded([&] { return ld_acquire_u32(rf) != 0u; })) return;
                if (!BWD) {
                    mean = __ldcg(a.save_mean + c); invstd = __ldcg(a.save_std + c);
                    gam = a.weight ? __ldg(a.weight + c) : 1.f; bet = a.bias ? __ldg(a.bias + c) : 0.f;
                } else {
                    const float4 ca = __ldcg(reinterpret_cast<const float4 *>(a.coef + c)), cb = __ldcg(reinterpret_cast<const float4 *>(a.coef + c) + 1);
                    kf.mean = ca.x; kf.proj = ca.y; kf.gmean = ca.z; kf.gscale = ca.w;
                    kf.invstd = cb.x; kf.gamma = cb.y; kf.beta = cb.z; kf.pad = cb.w;
                }
                if (ht == 0) {
                    // the last of the channel's readers lowers the flag again
                    int bf, bl;
                    channel_ctas((long long)min(gp.G, gp.C - st.g * gp.G) * gp.NL, gp.NL, st.cl, grid, &bf, &bl);
                    if (atomicAdd(a.cn.done + c, 1u) == (unsigned)(bl - bf)) {
                        a.cn.done[c] = 0u;
                        st_release_u32(a.cn.ready + c, 0u);
                    }
                }
            }
            if (!wait_phase(bars + slot, (uint32_t)((it / kStages) & 1))) return;
            // item j of the slot is item st.q + j of the channel's sequence: image (st.q + j) / L, offset (st.q + j) % L
            int n = (st.q + ht) / gp.L, i = (st.q + ht) - n * gp.L;
            float4 *obase = o4 + (long long)c * gp.L;
            auto act = [](float t) { return RELU ? (t > 0.f ? t : 0.f) : t; };
#pragma unroll 2
            for (int j = ht; j < st.len; j += kHalf) {
                const float4 v = sx[j];
                float4 o;
                if (!BWD) {
                    o.x = act(bn_value(v.x, mean, invstd, gam, bet));
                    o.y = act(bn_value(v.y, mean, invstd, gam, bet));
                    o.z = act(bn_value(v.z, mean, invstd, gam, bet));
                    o.w = act(bn_value(v.w, mean, invstd, gam, bet));
                } else {
                    const float4 q = sg[j];
                    auto one = [&](float xv, float g_) {
                        if (RELU) g_ = bn_value(xv, kf.mean, kf.invstd, kf.gamma, kf.beta) > 0.f ? g_ : 0.f;
                        return a.train ? (g_ - (xv - kf.mean) * kf.proj - kf.gmean) * kf.gscale : g_ * kf.gscale;
                    };
                    o.x = one(v.x, q.x); o.y = one(v.y, q.y); o.z = one(v.z, q.z); o.w = one(v.w, q.w);
                }
                st_hint(obase + (long long)n * CL + i, o, drop);
                n += qstep; i += rstep;
                if (i >= gp.L) { i -= gp.L; ++n; }
            }
            release_slot(slot);
            if (st.group_last && ht == 0) applied_s = st.g + 1;
        }
    }
}

// Counters at the start of the workspace, kMaxCounterChannels entries each: ticket counters of the forward
// statistics and of the gradient sums, and for the grouped kernels a ready flag and a reader counter per channel,
// forward and backward.  All zero when a call is enqueued, all zero again when its kernels have run (a kernel
// that recorded STATUS_FLAG_TIMEOUT may leave them set: clear the workspace after a non-zero device status).
constexpr int kMaxCounterChannels = 4096;
constexpr int kCounterArrays = 6;
constexpr size_t kCounterBytes = (size_t)kCounterArrays * kMaxCounterChannels * sizeof(unsigned int);

// Chunks per channel: 48 warps per SM at most, and chunks of at least kMinChunk elements.  One batch of loads per lane: small tensors are
// over soonest when every load is in flight at once (forward / backward of 12 x 144 x 37 x 29: 22.2 / 24.5 us with chunks of 2048, 17.3
// / 18.5 with 512; 128 x 1024 x 7 x 7 prefers the longer ones, 32.8 / 35.0 and 35.1 / 39.0).  Beyond kFewChunks of them chunks are
// longer, since the channel's last warp reads them all: 19 x 22 x 94 x 94 17.7 / 17.0 us with 322 chunks, 12.9 / 12.7 with 128 (13.8 / 13.0
// with CTAs per image, as before the warps); 189 x 8 x 109 x 183 87 / 109 us with 888 chunks, 142 / 171 with 128.
constexpr int kMinChunk = 512, kFewChunks = 128, kLongChunk = 2048;
static int most_chunks(int C) { return std::max(1, ceil_div(sm_count() * 48, C)); }
static int pick_chunks(int N, int C, int S)
{
    const long long count = (long long)N * S;
    const int least = S % 4 != 0 && C * count <= (1 << 19) ? kMinChunk / 2 : kMinChunk;          // a lane's batch is eight floats, or four float4
    const long long wanted = std::max(std::min<long long>(count / least, kFewChunks), count / kLongChunk);
    return (int)std::max(1LL, std::min<long long>(most_chunks(C), wanted));
}

// Planes of up to 1024 elements are handled by one warp each, larger ones by a whole CTA.
static bool small_planes(int S) { return S <= 1024; }
static int plane_grid(long long planes, int S)
{
    const long long cap = (long long)sm_count() * 16;
    const long long per_cta = small_planes(S) ? 8 : 1;
    return (int)std::max(1LL, std::min((planes + per_cta - 1) / per_cta, cap));
}

// Planes that are not a multiple of 16 bytes take the flat kernels (32-bit element indices, 16-byte aligned tensors).
static bool flat_applies(int S, long long planes, const void *a, const void *b, const void *c)
{
    // ... and so do planes of up to 256 elements (14 x 14): a warp per plane leaves 15 of 64 lane-slots idle there (input
    // gradient of 1024 x 512 x 14 x 14: 381 -> 343 us); at 784 elements the flat walk is no faster
    return (S % 4 != 0 || S <= 256) && planes * S >= 4 && planes * S < (1LL << 32) && ((((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) == 0);
}
static int flat_grid(unsigned total)
{
    return (int)std::max(1LL, std::min(ceil_div_ll((long long)(total / 4u), 1024), (long long)sm_count() * 8));
}

// The sums walk the images in ascending order, so what they read last — up to the 126 MB of L2 — is the end of the tensors: the
// elementwise passes start there and go backwards (backward pass of 128 x 128 x 56 x 56: 198 -> 187 us, forward 121 -> 118; 128 x 1024 x
// 7 x 7: 39.0 -> 36.6 us and 35.1 -> 33.3).
template <bool RELU>
static void launch_apply(const float *x, float *y, const float *weight, const float *bias, const float *mean_v,
                         const float *std_or_var, int train, float eps, int C, int S, long long planes, cudaStream_t stream)
{
    if (flat_applies(S, planes, x, y, y)) {
        const unsigned total = (unsigned)(planes * S);
        apply_flat_kernel<RELU><<<flat_grid(total), 256, 0, stream>>>(x, y, weight, bias, mean_v, std_or_var, train, eps, (unsigned)C, (unsigned)S, total);
        return;
    }
    if (small_planes(S)) apply_kernel<RELU, 32><<<plane_grid(planes, S), 256, 0, stream>>>(x, y, weight, bias, mean_v, std_or_var, train, eps, C, S, planes);
    else apply_kernel<RELU, 256><<<plane_grid(planes, S), 256, 0, stream>>>(x, y, weight, bias, mean_v, std_or_var, train, eps, C, S, planes);
}
template <bool RELU>
static void launch_grad_apply(const float *x, const float *gy, float *gx, const GradCoef *coef, int train, int C, int S,
                              long long planes, cudaStream_t stream)
{
    if (flat_applies(S, planes, x, gy, gx)) {
        const unsigned total = (unsigned)(planes * S);
        grad_apply_flat_kernel<RELU><<<flat_grid(total), 256, 0, stream>>>(x, gy, gx, coef, train, (unsigned)C, (unsigned)S, total);
        return;
    }
    if (small_planes(S)) grad_apply_kernel<RELU, 32><<<plane_grid(planes, S), 256, 0, stream>>>(x, gy, gx, coef, train, C, S, planes);
    else grad_apply_kernel<RELU, 256><<<plane_grid(planes, S), 256, 0, stream>>>(x, gy, gx, coef, train, C, S, planes);
}

}  // namespace bn
}  // namespace cunn

using namespace cunn;
using namespace cunn::bn;

// ---- grouped path: planning and launch ---------------------------------------------------------------------
// Bytes of one group's slabs, and of the two groups that are in flight at most (one waiting to be normalised, one being reduced).  Whatever
// the 126 MB of L2 keep of them is not read again; the ends of a group cost about 5 us, so that groups that fit with room to spare were
// slower.  Forward / backward of 256 x 64 x 112 x 112, group and window in MB: 28 and 56 436 / 827 us, 40 and 80 404 / 862, 52 and 104
// 384 / 641, 64 and 128 378 / 649, 78 and 156 374 / 613, 104 and 208 377 / 616; but 512 x 512 x 14 x 14: 131 / 198 with 64, 175 / 210 with 78.
// Tensors of less than 128 MB take groups of 28 MB, to have a second one at all.
static size_t g_group_bytes = (size_t)64 << 20;
static size_t g_window_bytes = (size_t)128 << 20;
#ifdef CUNN_B200_DEV_HOOKS
// sweeps only: CUNN_B200_BN_GROUP_MB / CUNN_B200_BN_WINDOW_MB override the budgets (group 0 disables the grouped kernels)
static const bool g_group_bytes_from_env = [] {
    if (const char *e = getenv("CUNN_B200_BN_GROUP_MB")) g_group_bytes = (size_t)atol(e) << 20;
    if (const char *e = getenv("CUNN_B200_BN_WINDOW_MB")) g_window_bytes = (size_t)atol(e) << 20;
    return true;
}();
#endif

// 0: never use the grouped kernels; 1 (default): where they are faster; 2: wherever they apply.
static int g_grouped_mode = 1;
// Tensors of 128 MB or more with channel slabs of at least 1 MB, two launches / grouped in us.
// Forward: 128 x 96 x 56 x 56 (154 MB) 94 / 82, 128 x 32 x 112 x 112 111 / 103, 256 x 64 x 112 x 112 420 / 382, 1024 x 64 x 56 x 56
// 454 / 387, 512 x 32 x 112 x 112 (slabs of 26 MB) 424 / 391, 2 x 16 x 1024 x 1024 315 / 69; but 128 x 256 x 28 x 28 (103 MB) 58 / 62,
// 256 x 256 x 28 x 28 (slabs of 0.8 MB) 112 / 113.
// Backward, which is instruction-bound: planes of 1025 to 4000 elements, of which the other kernels' CTAs of 256 threads make poor use
// (128 x 128 x 56 x 56 176 / 166, 1024 x 64 x 56 x 56 680 / 656, 1000 x 40 x 40 x 32 181 / 166), and few planes (16 x 64 x 256 x 256 224 / 205,
// 2 x 16 x 1024 x 1024 393 / 108); but 256 x 64 x 112 x 112 612 / 649, 256 x 128 x 32 x 32 106 / 116.
// Smaller tensors, forward, with slabs of at least 6 MB (few channels, to which the other kernels give few CTAs): 128 x 8 x 112 x 112 35 / 29,
// 64 x 8 x 224 x 224 66 / 56, 16 x 3 x 500 x 500 91 / 35.
constexpr size_t kGroupedMinBytes = (size_t)128 << 20;
static bool grouped_large(int N, int C, int S) { return (size_t)N * S * sizeof(float) * C >= kGroupedMinBytes; }
static bool grouped_is_faster(int N, int C, int S, bool backward)
{
    const size_t slab = (size_t)N * S * sizeof(float);
    if (slab < ((size_t)1 << 20)) return false;
    if (!grouped_large(N, C, S)) return !backward && slab >= ((size_t)6 << 20);
    return !backward || (S > 1024 && S <= 4000) || (long long)N * C <= 1024;
}

static int grouped_grid_cap() { return sm_count() * 2; }

// Size of the partials region: the per-(channel, chunk) partials of the two-launch path, or the per-(channel, CTA)
// partials of the grouped path (capped; shapes that would need more take the two-launch path).
static size_t part_region_bytes(int N, int C)
{
    const size_t two_launch = ((size_t)C * most_chunks(C) * sizeof(ChunkStat) + 255) & ~(size_t)255;
    const size_t grouped = std::min((size_t)C * (grouped_grid_cap() + 2) * sizeof(ChunkStat), (size_t)8 << 20);
    return std::max(two_launch, (grouped + 255) & ~(size_t)255);
}

// Fills gp and returns true when the grouped kernels apply: 16-byte rows, channel slabs (tensors_per_item tensors
// of N planes) that fit the group budget, enough items for every CTA in every group, partials that fit.
static bool plan_groups(int N, int C, int S, int tensors, const void *a, const void *b, const void *c, int *grid_, GroupPlan *gp)
{
    int grid = *grid_;
    if (g_grouped_mode == 0) return false;
    if (g_grouped_mode == 1 && !grouped_is_faster(N, C, S, tensors == 2)) return false;
    if (S % 4 != 0 || ((((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) != 0) || C > kMaxCounterChannels || grid < 1) return false;
    const size_t slab = (size_t)N * S * sizeof(float) * tensors;
    const bool large = grouped_large(N, C, S);
    const size_t group = large ? g_group_bytes : std::min(g_group_bytes, (size_t)28 << 20), window = large ? g_window_bytes : 2 * group;
    if (slab * 2 > window) return false;                         // two groups of one channel must fit the window
    const int gmax = (int)std::min<size_t>(std::max<size_t>(group / slab, 1), (size_t)C);
    const int groups = ceil_div(C, gmax);
    const int G = ceil_div(C, groups);
    if (G <= grid) grid = grid / G * G;                          // CTAs take whole shares of a channel
    const int glast = C - (ceil_div(C, G) - 1) * G;
    gp->N = N; gp->C = C; gp->S = S; gp->L = S / 4;
    gp->G = G; gp->groups = ceil_div(C, G);
    gp->NL = (long long)N * gp->L;
    gp->pstride = grid / glast + 2;
    gp->lookahead = (int)std::max<size_t>(2, window / ((size_t)G * slab));
    if ((long long)glast * gp->NL < 8LL * grid) return false;                      // too little work per CTA and group
    if ((size_t)C * gp->pstride * sizeof(ChunkStat) > part_region_bytes(N, C)) return false;
    *grid_ = grid;
    return true;
}

// CTAs of a grouped launch: as many as are co-resident (the kernels wait on one another), two per SM at most.
static int grouped_grid(const void *kernel, int threads)
{
    const int smem = 2 * kStages * kStageBytes;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return 0;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem) != cudaSuccess || occ < 1) return 0;
    return sm_count() * std::min(occ, 2);
}

extern "C" CUNN_API size_t cunn_b200_batchnorm_counter_bytes(void) { return kCounterBytes; }
extern "C" CUNN_API void cunn_b200_batchnorm_set_grouped(int mode) { g_grouped_mode = mode < 0 ? 0 : (mode > 2 ? 2 : mode); }
extern "C" CUNN_API int cunn_b200_batchnorm_get_grouped(void) { return g_grouped_mode; }

// Workspace layout: [counters, kCounterBytes] [partials, part_region_bytes] [gradient coefficients].
extern "C" CUNN_API size_t cunn_b200_batchnorm_workspace(int N, int C)
{
    if (N <= 0 || C <= 0) return 0;
    return kCounterBytes + part_region_bytes(N, C) + (size_t)C * sizeof(GradCoef) + 256;
}

static int bn_forward_impl(const float *x, float *y, const float *weight, const float *bias, float *running_mean,
                           float *running_var, float *save_mean, float *save_std, int N, int C, int S, int train,
                           double momentum, double eps, void *workspace, size_t workspace_bytes, cunn_stream_t stream_,
                           bool relu)
{
    clear_error();
    cudaStream_t stream = (cudaStream_t)stream_;
    CUNN_CHECK_ARG(N >= 0 && C > 0 && S > 0, "bad batch-norm sizes N=%d C=%d S=%d", N, C, S);
    CUNN_CHECK_ARG((long long)N * C * (long long)S < (1LL << 31), "tensors of 2^31 or more elements are not supported");
    if (N == 0) return 0;
    CUNN_CHECK_ARG(x && y && running_mean && running_var, "null tensor pointer");
    const long long planes = (long long)N * C;
    if (train) {
        CUNN_CHECK_ARG(save_mean && save_std, "training-mode batch norm needs save_mean and save_std");
        const int chunks = pick_chunks(N, C, S);
        const size_t need = kCounterBytes + part_region_bytes(N, C);
        CUNN_CHECK_ARG(workspace && workspace_bytes >= need && ((uintptr_t)workspace & 15) == 0,
                       "batch norm needs %zu bytes of 16-byte aligned workspace, got %zu", need,
                       workspace ? workspace_bytes : (size_t)0);
        unsigned int *counters = C <= kMaxCounterChannels ? (unsigned int *)workspace : nullptr;
        ChunkStat *part = (ChunkStat *)((char *)workspace + kCounterBytes);
        {
            GroupedArgs ga{};
            const bool large = grouped_large(N, C, S);
            const void *fn = large ? (relu ? (const void *)grouped_kernel<false, true, 8> : (const void *)grouped_kernel<false, false, 8>)
                                   : (relu ? (const void *)grouped_kernel<false, true, 4> : (const void *)grouped_kernel<false, false, 4>);
            const int threads = grouped_threads(large ? 8 : 4);
            int grid = grouped_grid(fn, threads);
            if (plan_groups(N, C, S, 1, x, y, y, &grid, &ga.gp)) {
                unsigned int *cw = (unsigned int *)workspace;
                ga.x = x; ga.out = y; ga.weight = weight; ga.bias = bias; ga.part = part;
                ga.cn = GroupCounters{cw, cw + 2 * kMaxCounterChannels, cw + 3 * kMaxCounterChannels};
                ga.running_mean = running_mean; ga.running_var = running_var; ga.save_mean = save_mean; ga.save_std = save_std;
                ga.momentum = momentum; ga.eps = eps; ga.train = 1; ga.status = device_status_ptr();
                void *args[] = {(void *)&ga};
                CUNN_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(threads), args, (size_t)2 * kStages * kStageBytes, stream));
                return 0;
            }
        }
        stats_kernel<<<ceil_div(C * chunks, 8), 256, 0, stream>>>(x, part, N, C, S, chunks, counters, running_mean, running_var, save_mean,
                                                     save_std, momentum, eps);
        CUNN_LAUNCH_CHECK("batch norm statistics");
        if (!counters) {
            stats_finish_kernel<<<ceil_div(C, 4), 128, 0, stream>>>(part, C, chunks, running_mean, running_var, save_mean,
                                                                     save_std, momentum, eps);
            CUNN_LAUNCH_CHECK("batch norm statistics finish");
        }
        if (relu) launch_apply<true>(x, y, weight, bias, save_mean, save_std, 1, (float)eps, C, S, planes, stream);
        else launch_apply<false>(x, y, weight, bias, save_mean, save_std, 1, (float)eps, C, S, planes, stream);
    } else {
        if (relu) launch_apply<true>(x, y, weight, bias, running_mean, running_var, 0, (float)eps, C, S, planes, stream);
        else launch_apply<false>(x, y, weight, bias, running_mean, running_var, 0, (float)eps, C, S, planes, stream);
    }
    CUNN_LAUNCH_CHECK("batch norm apply");
    return 0;
}

extern "C" CUNN_API int cunn_b200_batchnorm_forward(const float *x, float *y, const float *weight, const float *bias,
                                                    float *running_mean, float *running_var, float *save_mean,
                                                    float *save_std, int N, int C, int S, int train, double momentum,
                                                    double eps, void *workspace, size_t workspace_bytes,
                                                    cunn_stream_t stream)
{
    return bn_forward_impl(x, y, weight, bias, running_mean, running_var, save_mean, save_std, N, C, S, train, momentum, eps,
                           workspace, workspace_bytes, stream, false);
}

extern "C" CUNN_API int cunn_b200_batchnorm_relu_forward(const float *x, float *y, const float *weight, const float *bias,
                                                         float *running_mean, float *running_var, float *save_mean,
                                                         float *save_std, int N, int C, int S, int train, double momentum,
                                                         double eps, void *workspace, size_t workspace_bytes,
                                                         cunn_stream_t stream)
{
    return bn_forward_impl(x, y, weight, bias, running_mean, running_var, save_mean, save_std, N, C, S, train, momentum, eps,
                           workspace, workspace_bytes, stream, true);
}

static int bn_backward_impl(const float *x, const float *gy, bool relu, const float *bias, float *gx, float *grad_weight,
                            float *grad_bias, const float *weight, const float *running_mean, const float *running_var,
                            const float *save_mean, const float *save_std, int N, int C, int S, int train, double scale,
                            double eps, void *workspace, size_t workspace_bytes, cunn_stream_t stream_)
{
    clear_error();
    cudaStream_t stream = (cudaStream_t)stream_;
    CUNN_CHECK_ARG(N >= 0 && C > 0 && S > 0, "bad batch-norm sizes N=%d C=%d S=%d", N, C, S);
    CUNN_CHECK_ARG((long long)N * C * (long long)S < (1LL << 31), "tensors of 2^31 or more elements are not supported");
    if (N == 0) return 0;
    CUNN_CHECK_ARG(x && gy, "null tensor pointer");
    CUNN_CHECK_ARG(train ? (save_mean && save_std) : (running_mean && running_var),
                   "batch norm backward needs %s", train ? "save_mean and save_std" : "running_mean and running_var");
    const int chunks = pick_chunks(N, C, S);
    const size_t part_bytes = part_region_bytes(N, C);
    const size_t need = kCounterBytes + part_bytes + (size_t)C * sizeof(GradCoef);
    CUNN_CHECK_ARG(workspace && workspace_bytes >= need && ((uintptr_t)workspace & 15) == 0,
                   "batch norm backward needs %zu bytes of 16-byte aligned workspace, got %zu", need,
                   workspace ? workspace_bytes : (size_t)0);
    unsigned int *counters = C <= kMaxCounterChannels ? (unsigned int *)workspace + kMaxCounterChannels : nullptr;
    float2 *part = (float2 *)((char *)workspace + kCounterBytes);
    GradCoef *coef = (GradCoef *)((char *)workspace + kCounterBytes + part_bytes);
    const float *mean_v = train ? save_mean : running_mean;
    const float *sv = train ? save_std : running_var;
    const long long planes = (long long)N * C;
    // inference-mode input gradient needs no sums; they are still required for gradWeight / gradBias
    const bool need_sums = train || grad_weight || grad_bias;
    if (gx && need_sums) {
        GroupedArgs ga{};
        const void *fn = relu ? (const void *)grouped_kernel<true, true, 8> : (const void *)grouped_kernel<true, false, 8>;
        const int threads = grouped_threads(8);
        int grid = grouped_grid(fn, threads);
        if (plan_groups(N, C, S, 2, x, gy, gx, &grid, &ga.gp)) {
            unsigned int *cw = (unsigned int *)workspace;
            ga.x = x; ga.gy = gy; ga.out = gx; ga.weight = weight; ga.bias = bias; ga.part = part;
            ga.cn = GroupCounters{cw + kMaxCounterChannels, cw + 4 * kMaxCounterChannels, cw + 5 * kMaxCounterChannels};
            ga.mean_v = mean_v; ga.std_or_var = sv; ga.grad_weight = grad_weight; ga.grad_bias = grad_bias; ga.coef = coef;
            ga.eps = eps; ga.scale = scale; ga.train = train; ga.status = device_status_ptr();
            void *args[] = {(void *)&ga};
            CUNN_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(threads), args, (size_t)2 * kStages * kStageBytes, stream));
            return 0;
        }
    }
    if (need_sums) {
        if (relu) grad_stats_kernel<true><<<ceil_div(C * chunks, 8), 256, 0, stream>>>(x, gy, part, mean_v, sv, weight, bias, train, (float)eps, N, C, S, chunks,
                                                                          counters, eps, scale, grad_weight, grad_bias, coef);
        else grad_stats_kernel<false><<<ceil_div(C * chunks, 8), 256, 0, stream>>>(x, gy, part, mean_v, sv, weight, bias, train, (float)eps, N, C, S, chunks,
                                                                       counters, eps, scale, grad_weight, grad_bias, coef);
        CUNN_LAUNCH_CHECK("batch norm gradient sums");
    } else {
        CUNN_CUDA(cudaMemsetAsync(part, 0, (size_t)C * chunks * sizeof(float2), stream));
    }
    if (!need_sums || !counters) {
        grad_finish_kernel<<<ceil_div(C, 4), 128, 0, stream>>>(part, C, chunks, (long long)N * S, weight, bias, mean_v, sv, train,
                                                                eps, scale, grad_weight, grad_bias, coef);
        CUNN_LAUNCH_CHECK("batch norm gradient finish");
    }
    if (gx) {
        if (relu) launch_grad_apply<true>(x, gy, gx, coef, train, C, S, planes, stream);
        else launch_grad_apply<false>(x, gy, gx, coef, train, C, S, planes, stream);
        CUNN_LAUNCH_CHECK("batch norm input gradient");
    }
    return 0;
}

extern "C" CUNN_API int cunn_b200_batchnorm_backward(const float *x, const float *gy, float *gx, float *grad_weight,
                                                     float *grad_bias, const float *weight, const float *running_mean,
                                                     const float *running_var, const float *save_mean,
                                                     const float *save_std, int N, int C, int S, int train, double scale,
                                                     double eps, void *workspace, size_t workspace_bytes,
                                                     cunn_stream_t stream)
{
    return bn_backward_impl(x, gy, false, nullptr, gx, grad_weight, grad_bias, weight, running_mean, running_var, save_mean, save_std,
                            N, C, S, train, scale, eps, workspace, workspace_bytes, stream);
}

extern "C" CUNN_API int cunn_b200_batchnorm_relu_backward(const float *x, const float *gy, float *gx, float *grad_weight,
                                                          float *grad_bias, const float *weight, const float *bias,
                                                          const float *running_mean, const float *running_var,
                                                          const float *save_mean, const float *save_std, int N, int C,
                                                          int S, int train, double scale, double eps, void *workspace,
                                                          size_t workspace_bytes, cunn_stream_t stream)
{
    return bn_backward_impl(x, gy, true, bias, gx, grad_weight, grad_bias, weight, running_mean, running_var, save_mean, save_std, N, C,
                            S, train, scale, eps, workspace, workspace_bytes, stream);
}
