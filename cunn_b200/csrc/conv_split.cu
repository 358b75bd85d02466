// Convolutions on operands that are split once.
//
// The kernels of convmm.cu gather every operand value for every tap and split it on the way: for a 3x3 layer each input value is
// copied with 4-byte copies, and split, nine times per column tile, and the warps that do so are what the layer waits for.  Here a
// first pass over the tensors writes every value once, as two fp16 parts in pixel-major order (channels contiguous), and the matrix
// kernel fetches its tiles with im2col tensor-map copies: 128 consecutive output pixels x 32 channels of one tap are one copy, zeros
// outside the image included, in the layout that the tensor core reads.  No thread touches an operand again.
//
// Split.  v = (hi + lo) * 2^e with hi, lo of 11 bits each, products hi*hi + hi*lo + lo*hi: as the 3xTF32 split with rounding (tf32 and
// fp16 have 11-bit significands), at twice the rate of tf32 and half its bytes.  fp16 has five exponent bits, so values share exponents,
// powers of two that scale them exactly:
//   * activations of the forward pass and of input gradients: one exponent per pixel and group of 64 channels, that of its largest
//     finite value.  It varies along the reduction, so the tensor core sums one block of 64 channels at a time and the block's sum
//     is scaled when it is added to fp32 registers.
//   * weights: one exponent per filter (input gradient: per input channel), applied when the result is written.
//   * weight gradients reduce over pixels: one exponent per channel of x and of gy, found by a pass over both.
// A value is kept to max(2^-23 |v|, 2^-40 of the largest in its group).  Infinities and NaN stay what they are (lo = 0) and do not
// count for the exponent.
//
// Range.  Values below 2^-17 of their group's largest lose bits.  The sums do not show it where the largest is part of them, and it mostly is:
// behind a batch normalisation whole channels are 1e-5 or 1e-7 of others.  But where it meets zeros the error is the sum's: a channel of 1e9
// without weights among ordinary ones left 3 digits, one of 1e13 none.  So the sums are compared with what the exponents of their operands
// allow for: SMALL_SUM and SMALL_GRAD say when they are too small for that, by more than chance, and the images of the round are done again by the
// kernels of convmm.cu, whose tf32 operands have an exponent each.  Those are launched every time and leave at once if *gate says that
// nothing was lost, which costs a pass 2 to 8 us with looking at the sums.  (Looking at the operands instead cost the split as much, and sent the gradients of half of
// MobileNetV1's pointwise layers there.)
//
// Accumulation: the tensor core truncates when it adds, so a chain is one block, 64 channels (or pixels) of 12 additions, the eight of
// the cross terms first, while the accumulator is small; blocks are added in registers with rounding (two TMEM buffers in turn).
//
// Forward / input gradient / parameter gradient in us, gathering kernels and here: 3x3 256 -> 256 on 128 x 14 x 14 270 / 313 / 354 and
// 106 / 106 / 129; 3x3 stride 2 128 -> 256 on 64 x 56 x 56 312 / 427 / 360 and 139 / 174 / 185; 4x4 stride 2 transposed 256 -> 128 on
// 64 x 14 x 14 240 / 193 / 172 and 69 / 61 / 84; 7x7 stride 2, 3 -> 64 on 32 x 224 x 224 234 / - / 316 and 131 / - / 189.  2-norm errors of the
// first 9.7e-7 / 2.1e-6 / 2.7e-6 and 0.8e-7 / 1.6e-7 / 1.9e-7.  The split takes 14 of the 106 us, looking at the sums 3, the idle launch after the
// kernel 5; in a parameter gradient the maxima take 19 and the split 20 of 130.  The matrix kernel needs 1,100 to 1,200 clocks per 128 x 256 x 32 values, where the tensor pipe needs 768 and reading
// its operands from shared memory, and filling them, 940.
//
// Work: 128 x BN tiles of the persistent grid; the tiles of a last wave that would leave SMs idle are cut along the reduction, and the
// CTA that finishes a tile last adds its parts in their order (a counter per tile; nobody waits).
#include "axis_phases.h"
#include "conv_split.h"
#include "umma.cuh"

#include <algorithm>
#include <cmath>
#include <cuda.h>
#include <cuda_fp16.h>
#include <new>

namespace cunn {
namespace split {

using namespace mm;

constexpr int BM = 128;                  // tile rows (TMEM lanes)
constexpr int BK = 32;                   // reduction values per stage
constexpr int GROUP = 64;                // channels that share an exponent; M/N-major operands: values per 128-byte row
constexpr int EPI_WARPS = 8;
constexpr int MMA_WARP = EPI_WARPS + 3;            // two warpgroups that sum, then three warps that issue copies and one for the MMAs
constexpr int THREADS = (MMA_WARP + 1) * 32;
// Registers: the block is launched with 168 a thread (65,536 / 384); 2 x 224 + 56 = 3 x 168.
constexpr int SUM_REGS = 224, ISSUE_REGS = 56;
constexpr int MAX_PHASES = 4;            // stride 2
constexpr size_t RING_BYTES = 192 * 1024;
constexpr int STORE_COLS = 16, STORE_BYTES = STORE_COLS * (128 + 16);     // columns that a summing warp stores at a time, and its room for them
constexpr size_t SMEM = RING_BYTES + EPI_WARPS * STORE_BYTES;
constexpr int SCALED_MAX = 14;           // the largest value of a group lies in [2^14, 2^15) after scaling
// Values below 2^-2 after scaling are off by 2^-26.8 on average, 2^-25 at most.  A block's sum of 64 products is off by 2^-9.3 on average and 2^-3
// at most if all its values are lost on both sides; a sum of less than 2^12 per block (2^(exponent of the block), ordinary ones are 2^26) can be
// off by more than 5e-7 on average, which is what the gathering kernels' sums are off by.  Ordinary sums are that small one in 30,000 times.
constexpr float SMALL_SUM = 4096.f;
constexpr int MOST_SMALL = 8;            // ... of the 32 x 16 sums that a warp writes at a time; a lost row makes 16, a lost column 32
// The same of a parameter gradient's sum of n products, beside sqrt(n): 2^25 ordinary, off by 2^-12 on average if all values are lost.  Sums of
// mostly zeros are small without that: only those count one of whose channels has a WIDE range, pieces of it (channel_max_kernel's, planes of up to 2048
// values) being below 2^-16 of its largest.
constexpr float SMALL_GRAD = 512.f;
constexpr int WIDE = 16, MOST_SMALL_GRADS = 2;             // threads of a block of 32 x 4 to 32 gradients


// A pass is a few kernels, each launched while the one before still runs; it waits for it (pdl_wait) before it reads or writes.  What an
// earlier kernel of the pass wrote is read by plain loads: the read-only path (__ldg) is for memory that nobody writes while a kernel exists.

// ---- exponents ----------------------------------------------------------------------------------------------------------------
// Exponent of a group from the bits of its largest finite magnitude; 2^(SCALED_MAX - e) is a normal number.
constexpr int ZERO_EXP = -112;           // of zeros, or the next thing to them
__device__ __forceinline__ int group_exp(uint32_t max_bits) { return max((int)(max_bits >> 23) - 127, ZERO_EXP); }
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }      // -126 <= e <= 127
// s * 2^e, |e| <= 252, in two steps that neither overflow nor lose bits unless the result does
__device__ __forceinline__ float scale_by(float s, int e)
{
    const int h = e / 2;
    return s * pow2(h) * pow2(e - h);
}
__device__ __forceinline__ bool finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ float finite_abs(float v) { return finite(v) ? fabsf(v) : 0.f; }
// The two parts of v * s; lo of what is not finite is zero.
__device__ __forceinline__ void parts(float v, float s, __half &hi, __half &lo)
{
    const float t = v * s;
    hi = __float2half_rn(t);
    lo = finite(v) ? __float2half_rn(t - __half2float(hi)) : __float2half_rn(0.f);
}

// Row windows: an image has zeros around it or in it, whose sums are small without loss.  Here the values are looked at: 32 consecutive ones of a
// row and channel that are lost, fewer than 19 bits left, beside the row's largest; most of a row; a quarter of a filter.  Fewer than four of 32 are
// chance.
__device__ __forceinline__ bool is_lost(float v, float s) { return fabsf(v * s) < 0x1p-5f && v != 0.f; }
struct Lost {
    uint32_t values = 0, lost = 0;
    __device__ __forceinline__ void take(float v, float s)
    {
        values += v != 0.f;
        lost += is_lost(v, s);
    }
    // One in `share` of all threads' values of a block of 256, by all of them.
    __device__ __forceinline__ bool too_many(uint32_t share) const
    {
        __shared__ uint32_t sums[2][8];
        const uint32_t v = __reduce_add_sync(0xffffffffu, values), l = __reduce_add_sync(0xffffffffu, lost);
        if ((threadIdx.x & 31) == 0) { sums[0][threadIdx.x >> 5] = v; sums[1][threadIdx.x >> 5] = l; }
        __syncthreads();
        uint32_t all = 0, n = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) { all += sums[0][i]; n += sums[1][i]; }
        return n > 1 && n * share > all;
    }
};

// ---- splitting --------------------------------------------------------------------------------------------------------------------
constexpr int TILE_PITCH = 65, TILE_VALUES = GROUP * TILE_PITCH;          // shared memory of a splitting block, in fp32 values

// Few input channels: a convolution of kH x kW taps and C channels is one of kH x 1 taps and kW * C channels on the tensor of row windows
// x'[n][h][ow][kw * C + c] = x[n][c][h][ow * dW - padW + kw].  C = 0: the tensor as it is.
struct Window {
    int C, kW, dW, padW, W, oW;
    // values of one row of the image, in pixel-major order with its padding, that the windows of the row cut out
    __host__ __device__ int row_values() const { return ((oW - 1) * dW + kW) * C; }
    __host__ __device__ int block_rows() const { return row_values() <= TILE_VALUES / 4 ? 4 : row_values() <= TILE_VALUES / 2 ? 2 : 1; }
};
struct Act {                     // [images][C][HW] fp32 -> hi, lo: [2][images * HW][Cp] fp16
    const float *src;
    __half *dst;
    int8_t *exps;                // per pixel and group: exponent; null: exponents come from chmax
    const uint32_t *chmax;       // per channel: bits of the largest finite magnitude
    int C, Cp, HW, groups, blocks, ctas;      // tiles (row windows: rows), and the blocks that take them
    int vec;                     // planes of a multiple of four values, 16-byte aligned
    Window win;
    uint32_t pixels;
};
struct PrepParams {
    Act act[2];
    // weights, a block per row (filter, or input channel of an input gradient): value (row, c, tap) at row * w_row + c * w_c + tap
    const float *w;
    __half *w_dst;               // [2][taps][rows][Cp]
    int *w_exp;                  // [rows]: exponent
    int rows, w_C, w_Cp, taps;
    long long w_row, w_c;
    int win_C, win_kW;           // Window's: value (row, kw * C + c, th) at row * w_row + c * w_c + th * kW + kw; 0: none
    int *tickets;
    int n_tickets;
    int *gate;                   // zero for the matrix kernel to set; weight gradient: it is zero already
    uint8_t *wide;               // row windows: per block, whether values were lost
};

// COUNT: returns whether values were lost.
template <bool COUNT>
__device__ __forceinline__ bool prep_weights(const PrepParams &p, int row, float *tile)
{
    __shared__ uint32_t red[8];
    const float *w = p.w + (long long)row * p.w_row;
    const int C = p.win_C ? p.win_C : p.w_C, per = p.win_C ? p.taps * p.win_kW : p.taps, n = p.w_C * p.taps;      // channels, taps of each, values
    float m = 0.f;
#pragma unroll 8
    for (int i = threadIdx.x; i < n; i += 256) {
        const int c = i / per;
        const float v = __ldg(w + c * p.w_c + (i - c * per));
        if (i < TILE_VALUES) tile[i] = v;
        m = fmaxf(m, finite_abs(v));
    }
    uint32_t b = __float_as_uint(m);
    b = __reduce_max_sync(0xffffffffu, b);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = b;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) b = max(b, red[i]);
    const int e = group_exp(b);
    if (threadIdx.x == 0) p.w_exp[row] = e;
    const float s = pow2(SCALED_MAX - e);
    const size_t part = (size_t)p.taps * p.rows * p.w_Cp;
    Lost filter;
#pragma unroll 4
    for (int i = threadIdx.x; i < p.w_Cp * p.taps; i += 256) {
        const int t = i / p.w_Cp, c = i - t * p.w_Cp;
        float v = 0.f;
        if (c < p.w_C) {
            const int kw = p.win_C ? c / C : 0, ch = c - kw * C, at = p.win_C ? t * p.win_kW + kw : t, flat = ch * per + at;
            v = flat < TILE_VALUES ? tile[flat] : __ldg(w + ch * p.w_c + at);
        }
        __half hi, lo;
        parts(v, s, hi, lo);
        __half *d = p.w_dst + ((size_t)t * p.rows + row) * p.w_Cp + c;
        d[0] = hi;
        d[part] = lo;
        if (COUNT) filter.take(v, s);
    }
    return COUNT && filter.too_many(4);
}

// One block: 64 pixels (of the flat pixel sequence) x 64 channels, through shared memory: read along the pixels, written along the
// channels, a warp four pixels of 128 bytes at a time (16 bytes of each of 32 pixels per instruction took twice as long).
template <bool PER_CHANNEL>
__device__ __forceinline__ void prep_act(const Act &a, int block, float *tile_)
{
    float(*tile)[TILE_PITCH] = reinterpret_cast<float(*)[TILE_PITCH]>(tile_);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pb = block / a.groups, g = block - pb * a.groups;
    const uint32_t p0 = (uint32_t)pb * 64u;
    if (a.vec) {
        // four consecutive pixels of a channel: lanes 0-15 of one, 16-31 of the next
        const uint32_t px = p0 + (lane & 15) * 4, im = px / (uint32_t)a.HW;
        const bool ok = px < a.pixels;                                    // pixels is a multiple of four
        const float *src = a.src + (ok ? (size_t)im * a.C * a.HW + (px - im * a.HW) : 0);
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c = g * GROUP + warp * 8 + i * 2 + (lane >> 4);
            v[i] = ok && c < a.C ? __ldg(reinterpret_cast<const float4 *>(src + (size_t)c * a.HW)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float *t = &tile[warp * 8 + i * 2 + (lane >> 4)][(lane & 15) * 4];
            t[0] = v[i].x; t[1] = v[i].y; t[2] = v[i].z; t[3] = v[i].w;
        }
    } else {
        const float *src[2];
        bool ok[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t px = p0 + h * 32 + lane, im = px / (uint32_t)a.HW;
            ok[h] = px < a.pixels;
            src[h] = a.src + (ok[h] ? (size_t)im * a.C * a.HW + (px - im * a.HW) : 0);
        }
        float v[8][2];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int c = g * GROUP + warp * 8 + i;
#pragma unroll
            for (int h = 0; h < 2; ++h) v[i][h] = ok[h] && c < a.C ? __ldg(src[h] + (size_t)c * a.HW) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
#pragma unroll
            for (int h = 0; h < 2; ++h) tile[warp * 8 + i][h * 32 + lane] = v[i][h];
        }
    }
    const int piece = lane & 7, c0 = g * GROUP + piece * 8;               // eight channels of a pixel
    float f[8];
    if (PER_CHANNEL) {
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = pow2(SCALED_MAX - group_exp(c0 + i < a.C ? a.chmax[c0 + i] : 0u));
    }
    __syncthreads();
    const size_t part = (size_t)a.pixels * a.Cp;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int col = warp * 8 + h * 4 + (lane >> 3);
        const uint32_t px = p0 + col;
        float r[8], m = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = tile[piece * 8 + i][col];
        if (!PER_CHANNEL) {
#pragma unroll
            for (int i = 0; i < 8; ++i) m = fmaxf(m, finite_abs(r[i]));
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            const int e = group_exp(__float_as_uint(m));
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = pow2(SCALED_MAX - e);
            if (piece == 0 && px < a.pixels) a.exps[(size_t)px * a.groups + g] = (int8_t)e;
        }
        if (px < a.pixels && c0 < a.Cp) {
            __align__(16) __half hi[8];
            __align__(16) __half lo[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) parts(r[i], f[i], hi[i], lo[i]);
            __half *d = a.dst + (size_t)px * a.Cp + c0;
            *reinterpret_cast<uint4 *>(d) = *reinterpret_cast<const uint4 *>(hi);
            *reinterpret_cast<uint4 *>(d + part) = *reinterpret_cast<const uint4 *>(lo);
        }
    }
}

// Row windows: a block takes up to four rows of the images.  A row's values are split once, into shared memory in pixel-major order; a
// window is a run of them.  Returns whether values were lost (PER_CHANNEL: false).  (Split where they are written, 3.5 times each for 7x7 stride 2, 32 x 3 x 224 x 224 took 59 us; with a block
// per row 45.)  One exponent per row.
template <bool PER_CHANNEL>
__device__ __forceinline__ bool prep_window(const Act &a, int block, float *tile)
{
    __shared__ uint32_t red[8];
    const Window &w = a.win;
    const int n = w.row_values(), R = w.block_rows(), T = 256 / R, slot = threadIdx.x / T, tid = threadIdx.x - slot * T;
    const int rows = a.HW / w.oW, row = block * R + slot, cols = n / w.C;
    const bool ok = row < a.blocks;
    const int im = ok ? row / rows : 0, h = ok ? row - im * rows : 0;
    const size_t plane = (size_t)rows * w.W;
    const float *src = a.src + (size_t)im * w.C * plane + (size_t)h * w.W;
    __half *hi = reinterpret_cast<__half *>(tile) + slot * (2 * TILE_VALUES / R), *lo = hi + n;
    float s = 0.f;
    if (!PER_CHANNEL) {
        float m = 0.f;
        for (int c = 0; c < w.C; ++c) {
#pragma unroll 4
            for (int i = tid; i < w.W; i += T) m = fmaxf(m, finite_abs(__ldg(src + c * plane + i)));
        }
        uint32_t b = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = b;
        __syncthreads();
        for (int i = 0; i < 8 / R; ++i) b = max(b, red[slot * (8 / R) + i]);
        const int e = group_exp(b);
        s = pow2(SCALED_MAX - e);
        if (ok)
            for (int i = tid; i < w.oW; i += T) a.exps[(size_t)row * w.oW + i] = (int8_t)e;
    }
    bool some = false, wide = false;
    for (int c = 0; c < w.C; ++c) {
        if (PER_CHANNEL) s = pow2(SCALED_MAX - group_exp(a.chmax[c]));
#pragma unroll 4
        for (int i = tid; i < cols; i += T) {
            const int at = i - w.padW;
            const float v = (unsigned)at < (unsigned)w.W ? __ldg(src + c * plane + at) : 0.f;
            parts(v, s, hi[i * w.C + c], lo[i * w.C + c]);
            if (!PER_CHANNEL) some |= is_lost(v, s);
        }
    }
    if (PER_CHANNEL) {
        __syncthreads();
    } else if (__syncthreads_or(some)) {
        Lost rows;
#pragma unroll 1
        for (int c = 0; ok && c < w.C; ++c) {
#pragma unroll 1
            for (int i0 = tid & ~31; i0 < w.W; i0 += T) {                  // T is a multiple of 32
                const int i = i0 + (tid & 31);
                const float v = i < w.W ? __ldg(src + c * plane + i) : 0.f;
                const uint32_t values = __ballot_sync(0xffffffffu, v != 0.f), kept = __ballot_sync(0xffffffffu, v != 0.f && !is_lost(v, s));
                wide |= __popc(values) >= 4 && !kept;
                rows.take(v, s);
            }
        }
        wide = __syncthreads_or(wide);
        wide |= rows.too_many(8);                                          // most of one row of four
    }
    if (!ok) return wide;
    // 16-byte pieces of the windows; those past a window's last value are zeros
    const int pieces = a.Cp / 8, step = w.dW * w.C;
    const size_t part = (size_t)a.pixels * a.Cp;
    __half *dst = a.dst + (size_t)row * w.oW * a.Cp;
    for (int i = tid; i < w.oW * pieces; i += T) {
        const int ow = i / pieces, c0 = (i - ow * pieces) * 8, at = ow * step + c0, left = a.C - c0;
        __align__(16) __half ph[8];
        __align__(16) __half pl[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            ph[k] = k < left ? hi[at + k] : __ushort_as_half(0);
            pl[k] = k < left ? lo[at + k] : __ushort_as_half(0);
        }
        *reinterpret_cast<uint4 *>(dst + (size_t)i * 8) = *reinterpret_cast<const uint4 *>(ph);
        *reinterpret_cast<uint4 *>(dst + part + (size_t)i * 8) = *reinterpret_cast<const uint4 *>(pl);
    }
    return wide;
}

// WINDOW: the last tensor is one of row windows.
template <bool PER_CHANNEL, bool WINDOW>
__global__ void __launch_bounds__(256)
prep_kernel(const __grid_constant__ PrepParams p)
{
    __shared__ float tile[TILE_VALUES];
    pdl_wait();
    pdl_launch_dependents();
    int b = (int)blockIdx.x;
    if (!PER_CHANNEL && b == 0) {
        for (int i = threadIdx.x; i < p.n_tickets; i += 256) p.tickets[i] = 0;
        if (threadIdx.x == 0) *p.gate = 0;
    }
    bool wide = false;
    if (b < p.rows) {
        wide = prep_weights<WINDOW>(p, b, tile);
    } else {
        b -= p.rows;
        const Act &act = p.act[PER_CHANNEL && b >= p.act[0].ctas ? 1 : 0];
        if (PER_CHANNEL && b >= p.act[0].ctas) b -= p.act[0].ctas;
        if (WINDOW && act.win.C) wide = prep_window<PER_CHANNEL>(act, b, tile);
        else prep_act<PER_CHANNEL>(act, b, tile);
    }
    if (WINDOW && !PER_CHANNEL && threadIdx.x == 0) p.wide[blockIdx.x] = wide;
}

// Largest finite magnitude of every channel and the smallest of its pieces' largest, and the sums of the first tensor's channels (the bias
// gradient): block = (channel, chunk of the channel's pieces), a warp per piece of a plane.
constexpr int PIECE = 2048;              // values of a plane that a warp takes, at most
struct MaxParams {
    const float *src[2];
    uint32_t *chmax[2], *chlow[2];                               // chlow: the complement of the smallest piece's largest, 0: no piece has values
    double *sums;                                                // [chunks][C] of the first tensor, or null
    int C[2], HW[2], pieces[2], chunks[2], vec[2], images;       // pieces of a plane; vec: planes of a multiple of four values, 16-byte aligned
};
__global__ void __launch_bounds__(256, 5)
channel_max_kernel(const __grid_constant__ MaxParams p)
{
    pdl_launch_dependents();
    __shared__ double part[8];
    __shared__ uint32_t red[8], red_low[8];
    int b = (int)blockIdx.x, t = 0;
    if (b >= p.C[0] * p.chunks[0]) { b -= p.C[0] * p.chunks[0]; t = 1; }
    const int chunk = b / p.C[t], c = b - chunk * p.C[t], HW = p.HW[t], per = p.pieces[t], warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long total = (long long)p.images * per;
    const int n0 = (int)(total * chunk / p.chunks[t]), n1 = (int)(total * (chunk + 1) / p.chunks[t]);
    const int unit = p.vec[t] ? HW / 4 : HW, len = (unit + per - 1) / per;           // (per - 1) * len < unit
    const float *src = p.src[t] + (size_t)c * HW;
    const bool add = p.sums && t == 0;
    uint32_t bits = 0, low = 0;
    double sum = 0.0;
    for (int n = n0 + warp; n < n1; n += 32) {                             // four pieces at a time
        float m[4] = {0.f, 0.f, 0.f, 0.f};
        const float *s[4];
        int left[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            // a piece past the last, or a value past a piece's last, repeats another one: loads without conditions
            const int k = n + 8 * j < n1 ? n + 8 * j : n, im = per == 1 ? k : k / per, from = (k - im * per) * len;
            s[j] = src + (size_t)im * p.C[t] * HW + (size_t)from * (p.vec[t] ? 4 : 1);
            left[j] = min(len, unit - from) - 1;
        }
        if (p.vec[t]) {
#pragma unroll 2
            for (int i = lane; i < len; i += 32) {
                float4 v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = __ldg(reinterpret_cast<const float4 *>(s[j]) + min(i, left[j]));
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    m[j] = fmaxf(m[j], fmaxf(fmaxf(finite_abs(v[j].x), finite_abs(v[j].y)), fmaxf(finite_abs(v[j].z), finite_abs(v[j].w))));
                if (add) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (i <= left[j] && n + 8 * j < n1) sum += ((double)v[j].x + (double)v[j].y) + ((double)v[j].z + (double)v[j].w);
                }
            }
        } else {
#pragma unroll 2
            for (int i = lane; i < len; i += 32) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float v = __ldg(s[j] + min(i, left[j]));
                    m[j] = fmaxf(m[j], finite_abs(v));
                    if (add && i <= left[j] && n + 8 * j < n1) sum += (double)v;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t piece = __reduce_max_sync(0xffffffffu, __float_as_uint(m[j]));
            bits = max(bits, piece);
            low = max(low, piece ? ~piece : 0u);
        }
    }
    if (lane == 0) { red[warp] = bits; red_low[warp] = low; }
    if (add) {
        sum = warp_sum(sum);
        if (lane == 0) part[warp] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 1; i < 8; ++i) {
            bits = max(bits, red[i]);
            low = max(low, red_low[i]);
        }
        atomicMax(p.chmax[t] + c, bits);
        atomicMax(p.chlow[t] + c, low);
        if (add) {
#pragma unroll
            for (int i = 1; i < 8; ++i) sum += part[i];
            p.sums[(size_t)chunk * p.C[0] + c] = sum;
        }
    }
}

// ---- matrix kernel ------------------------------------------------------------------------------------------------------------------
// One sub-problem of the forward pass or an input gradient (a stride residue): output pixels (r / pix_W, r % pix_W) read the gathered
// tensor at (row * stH + lH + th * dlH, col * stW + lW + tw * dlW) with the weight of tap w_base + th * w_sH + tw * w_sW, and are written
// at o_off + row * o_sH + col * o_sW of an output plane.
struct Phase {
    int tile0, HW, pix_W, M_total;
    int taps, kW, blocks;                    // blocks of the reduction: taps * Params::groups
    int lH, lW, stH, stW, dlH, dlW;
    int w_base, w_sH, w_sW;
    int o_off, o_sH, o_sW;
};
struct Params {
    const int8_t *exps;                      // exponent per (pixel, group) of the gathered tensor
    const int *w_exp;                        // ... per column
    const float *bias;                       // or null
    float *out, *partial;
    int *tickets, *status, *gate;
    const uint8_t *wide;                     // row windows: the splitting blocks' verdicts
    int n_wide;                              // ... and their number; otherwise the sums are looked at
    const float *raw_a, *raw_w;              // the operands in fp32, for sums that came out as NaN; null: left as they are
    int images, g_C, g_H, g_W, groups;
    int w_kk, o_HW, N_total, n_tiles, width; // columns in all, column tiles and a tile's columns
    int n_phases, full, splits, items;       // items [0, full) are whole tiles, then `splits` parts of each further tile
    // weight gradient: rows = output channels, columns = (tap, group of 64 input channels) pairs, reduction over pixels
    int m_tiles, tiles, blocks, per_split, col_groups, kW, pix_HW, pix_W;
    int lH, lW, stH, stW, dlH, dlW;
    Phase ph[MAX_PHASES];
};
struct Maps {
    CUtensorMap a[MAX_PHASES];               // weight gradient: [0] gy
    CUtensorMap b;
};

__device__ __forceinline__ void load_im2col(uint32_t dst, const CUtensorMap *map, int c, int w, int h, int n, int ow, int oh, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6], {%7, %8};"
                 ::"r"(dst), "l"((uint64_t)map), "r"(c), "r"(w), "r"(h), "r"(n), "r"(bar), "h"((uint16_t)ow), "h"((uint16_t)oh) : "memory");
}
__device__ __forceinline__ void load_3d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_f16_acc(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc)
{
    asm volatile("tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, 1;" ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc) : "memory");
}

// What item i of the work list is.
struct Item {
    int phase, m_tile, n_tile, part, tail, begin, end;       // tail: index among the tiles that are cut, -1: a whole tile
};
template <bool WG>
__device__ __forceinline__ Item item_of(const Params &p, int i)
{
    Item it;
    it.phase = 0;
    if (WG) {
        it.part = i / p.tiles;
        const int t = i - it.part * p.tiles;
        it.m_tile = t / p.n_tiles;
        it.n_tile = t - it.m_tile * p.n_tiles;
        it.tail = 0;
        it.begin = it.part * p.per_split;
        it.end = min(it.begin + p.per_split, p.blocks);
        return it;
    }
    int t = i;
    it.part = 0;
    it.tail = -1;
    if (i >= p.full) {
        const int j = i - p.full;
        it.tail = j / p.splits;
        it.part = j - it.tail * p.splits;
        t = p.full + it.tail;
        if (p.splits == 1) it.tail = -1;
    }
    while (it.phase + 1 < p.n_phases && t >= p.ph[it.phase + 1].tile0) ++it.phase;
    const Phase &f = p.ph[it.phase];
    const int r = t - f.tile0;
    it.m_tile = r / p.n_tiles;
    it.n_tile = r - it.m_tile * p.n_tiles;
    it.begin = 0;
    it.end = f.blocks;
    if (it.tail >= 0) {
        it.begin = (int)((long long)f.blocks * it.part / p.splits);
        it.end = (int)((long long)f.blocks * (it.part + 1) / p.splits);
    }
    return it;
}

__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// The wait names the registers, so that nothing reads them before it.
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[32])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]),
                   "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
                   "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}
// Barrier of the warps that share a tile.
template <int SETS>
__device__ __forceinline__ void sums_sync(int set)
{
    if (SETS == 1) asm volatile("bar.sync 1, 256;" ::: "memory");
    else if (set == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
    else asm volatile("bar.sync 2, 128;" ::: "memory");
}

// One input-gradient value in plain fp32: products with the zeros in place of taps outside gy, or of an infinity's parts, can make a
// NaN that the definition does not have.
__device__ float plain_sum(const Params &p, const Phase &f, int im, int row, int col, int n)
{
    const float *src = p.raw_a + (size_t)im * p.g_C * p.g_H * p.g_W;
    float s = 0.f;
#pragma unroll 1
    for (int th = 0; th < f.taps / f.kW; ++th) {
        const int ih = row * f.stH + f.lH + th * f.dlH;
        if ((unsigned)ih >= (unsigned)p.g_H) continue;
#pragma unroll 1
        for (int tw = 0; tw < f.kW; ++tw) {
            const int iw = col * f.stW + f.lW + tw * f.dlW;
            if ((unsigned)iw >= (unsigned)p.g_W) continue;
#pragma unroll 8
            for (int c = 0; c < p.g_C; ++c)
                s = fmaf(__ldg(p.raw_w + ((size_t)c * p.N_total + n) * p.w_kk + f.w_base + th * f.w_sH + tw * f.w_sW),
                         __ldg(src + ((size_t)c * p.g_H + ih) * p.g_W + iw), s);
        }
    }
    return s;
}

// Exponents below every group's: of pixels outside the tensor, and of a row before its first block.
constexpr int NO_EXP = -120;
// 2^(e - top) for e <= top; what lies 2^126 below the row's largest block is nothing.
__device__ __forceinline__ float step(int e, int top) { return top - e > 126 ? 0.f : pow2(e - top); }
__device__ __forceinline__ uint64_t pack2(float lo, float hi) { return (uint64_t)__float_as_uint(hi) << 32 | __float_as_uint(lo); }
// two fp32 operations, each rounded as the scalar one
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
template <int N>
__device__ __forceinline__ void raise(uint64_t (&acc2)[N], float &blocks, int &top, int to)
{
    const float f = step(top, to);
    blocks *= f;
    const uint64_t f2 = pack2(f, f);
#pragma unroll
    for (int j = 0; j < N; ++j) acc2[j] = mul2(acc2[j], f2);
    top = to;
}

// Warps 0-7: sums (TMEM -> registers -> memory), two per TMEM lane quarter, each half of the columns; warps 8-10: copies; warp 11: MMAs.
// BG (weight gradient): values per row of the gathered operand, 64 or, for tensors of up to 32 channels, 32.
template <int BN, bool WG, int BG = GROUP>
__global__ void __launch_bounds__(THREADS, 1)
split_gemm_kernel(const __grid_constant__ Params p, const __grid_constant__ Maps maps)
{
    constexpr int STAGE = 2 * BK * 2 * (BM + BN), NS = (int)(RING_BYTES / STAGE);
    constexpr int A_PART = BM * BK * 2, B_PART = BN * BK * 2, A_LO = A_PART, B_HI = 2 * A_PART, B_LO = B_HI + B_PART;
    // The two summing warpgroups take half of the columns of a tile each; or, where a thread can hold a whole row, they work on a tile
    // each, with half of the stages and of TMEM and an issuing warp of its own (ALT).  A block of 64 channels costs its issuing thread
    // 250 clocks of waits, 180 of commits and 70 per MMA, which is more than the MMAs of narrow tiles take, and one group writes its tile
    // while the other one sums (7x7 on 3 channels has seven blocks a tile).
    constexpr bool ALT = !WG && BN <= 128;
    constexpr int HALF_COLS = ALT ? BN : BN / 2, SETS = ALT ? 2 : 1, BUFS = 512 / BN / SETS;      // TMEM buffers per set
    constexpr int RING = NS / SETS;                                                                // stages per set
    constexpr size_t PART = BN * BM + 2 * BM;         // partial sums of a cut tile, their rows' exponents and sizes of blocks

    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t full[NS], empty[NS];          // stage landed; its MMAs are done
    __shared__ uint64_t ready[SETS * BUFS], drained[SETS * BUFS];         // a block's sums are in TMEM buffer b; they have been read
    __shared__ uint32_t tmem_base_s;
    __shared__ int last_s[2];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) { mbar_init(smem_u32(full + s), 1); mbar_init(smem_u32(empty + s), 1); }
        for (int b = 0; b < SETS * BUFS; ++b) { mbar_init(smem_u32(ready + b), 1); mbar_init(smem_u32(drained + b), EPI_WARPS / SETS); }
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(smem_u32(&tmem_base_s), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;
    pdl_wait();
    pdl_launch_dependents();

    if (warp >= EPI_WARPS) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ISSUE_REGS));
      const int set = ALT ? warp & 1 : 0, first_item = (int)blockIdx.x + set * (int)gridDim.x, item_step = SETS * (int)gridDim.x;
      uint64_t *const my_full = full + set * RING, *const my_empty = empty + set * RING;
      unsigned char *const my_smem = smem + (size_t)set * RING * STAGE;
      if (warp < (ALT ? MMA_WARP - 1 : MMA_WARP)) {
        // A thread's copies start about 100 clocks apart and 4 or 8 KB each take 60 to 180: three warps share them, or one has a set's.
        const int part_of = ALT ? 0 : warp - EPI_WARPS;
        if (lane == 0) {
            int rs = 0;
            uint32_t parity = 1;                      // the first round finds the stages empty
            bool ok = true;
            for (int i = first_item; ok && i < p.items; i += item_step) {
                const Item it = item_of<WG>(p, i);
                if (!WG) {
                    const Phase &f = p.ph[it.phase];
                    const int m0 = it.m_tile * BM, im = m0 / f.HW, r = m0 - im * f.HW, row = r / f.pix_W, col = r - row * f.pix_W;
                    const int h0 = row * f.stH + f.lH, w0 = col * f.stW + f.lW, n0 = it.n_tile * p.width;
                    const int tap = it.begin / p.groups;
                    int c = (it.begin - tap * p.groups) * GROUP, th = tap / f.kW, tw = tap - th * f.kW;
                    const CUtensorMap *ma = &maps.a[it.phase];
                    for (int q = it.begin; q < it.end;) {
                        if (!mbar_wait(smem_u32(my_empty + rs), parity, p.status)) { ok = false; break; }
                        const uint32_t bar = smem_u32(my_full + rs), s = smem_u32(my_smem) + (uint32_t)(rs * STAGE);
                        if (part_of == 0) mbar_arrive_expect_tx(bar, STAGE);
                        if (ALT || part_of < 2)
                            load_im2col(s + (uint32_t)(part_of * A_LO), ma, c, w0, h0, im + part_of * p.images, tw * f.dlW, th * f.dlH, bar);
                        if (ALT || part_of == 2) {
                            const int wt = f.w_base + th * f.w_sH + tw * f.w_sW;
                            load_3d(s + B_HI, &maps.b, c, n0, wt, bar);
                            if (ALT) load_im2col(s + A_LO, ma, c, w0, h0, im + p.images, tw * f.dlW, th * f.dlH, bar);
                            load_3d(s + B_LO, &maps.b, c, n0, wt + p.w_kk, bar);
                        }
                        c += BK;
                        if (c >= p.g_C) { c = 0; if (++tw == f.kW) { tw = 0; ++th; } }
                        if ((c & (GROUP - 1)) == 0) ++q;                           // the group's last stage
                        if (++rs == RING) { rs = 0; parity ^= 1u; }
                    }
                } else {
                    const int g0 = it.n_tile * (BN / BG), ng = min(BN / BG, p.col_groups - g0);
                    const int mg = min(BM / GROUP, (p.N_total - it.m_tile * BM + GROUP - 1) / GROUP);      // rows past the last are left as they are
                    // this warp's copies of the gathered operand: l = part_of + 3 k -> part l & 1 of group l >> 1
                    constexpr int PER_WARP = (2 * (BN / BG) + 2) / 3;
                    int chan[PER_WARP], offs[PER_WARP];
#pragma unroll
                    for (int k = 0; k < PER_WARP; ++k) {
                        const int j = (part_of + 3 * k) >> 1, tap = (g0 + j) / p.groups, th = tap / p.kW, tw = tap - th * p.kW;
                        chan[k] = (g0 + j - tap * p.groups) * BG;
                        offs[k] = tw * p.dlW | th * p.dlH << 16;
                    }
                    for (int q = 2 * it.begin; q < 2 * it.end; ++q) {
                        if (!mbar_wait(smem_u32(empty + rs), parity, p.status)) { ok = false; break; }
                        const uint32_t bar = smem_u32(full + rs), s = smem_u32(smem) + (uint32_t)(rs * STAGE);
                        if (part_of == 0) mbar_arrive_expect_tx(bar, (uint32_t)((2 * mg * GROUP + 2 * ng * BG) * BK * 2));
                        const int p0 = q * BK, im = p0 / p.pix_HW, r = p0 - im * p.pix_HW, row = r / p.pix_W, col = r - row * p.pix_W;
                        const int h0 = row * p.stH + p.lH, w0 = col * p.stW + p.lW;
                        for (int l = part_of; l < 2 * mg; l += 3)
                            load_3d(s + (uint32_t)((l & 1) * A_PART + (l >> 1) * GROUP * BK * 2), &maps.a[0], it.m_tile * BM + (l >> 1) * GROUP, p0, l & 1, bar);
#pragma unroll
                        for (int k = 0; k < PER_WARP; ++k) {
                            const int l = part_of + 3 * k, part = l & 1, j = l >> 1;
                            if (j < ng)
                                load_im2col(s + (uint32_t)(B_HI + part * B_PART + j * BG * BK * 2), &maps.b, chan[k], w0, h0, im + part * p.images,
                                            offs[k] & 0xffff, offs[k] >> 16, bar);
                        }
                        if (++rs == NS) { rs = 0; parity ^= 1u; }
                    }
                }
            }
        }
      } else {
        if (lane == 0) {
            // descriptors: K-major tiles of 64-byte rows in the 64-byte swizzle (groups of 8 rows 512 bytes apart); M/N-major ones of
            // 128-byte rows in the 128-byte swizzle (8 k values 1024 bytes, 64 values of M or N 4096 bytes apart), or of 64-byte rows
            constexpr bool NARROW = WG && BG == 32;
            constexpr uint32_t A_LOW = WG ? (uint32_t)(GROUP * BK * 2 >> 4) << 16 : 1u << 16, B_LOW = NARROW ? (uint32_t)(BG * BK * 2 >> 4) << 16 : A_LOW;
            constexpr uint32_t A_HIGH = (uint32_t)((WG ? 1024 : 512) >> 4) | (1u << 14) | ((WG ? 2u : 4u) << 29);
            constexpr uint32_t B_HIGH = NARROW ? (uint32_t)(512 >> 4) | (1u << 14) | (4u << 29) : A_HIGH;
            constexpr uint32_t A_STEP = WG ? 2048u >> 4 : 2u, B_STEP = NARROW ? 1024u >> 4 : A_STEP;       // 16 k values
            auto da = [](uint32_t low) { return ((uint64_t)A_HIGH << 32) | low; };
            auto db = [](uint32_t low) { return ((uint64_t)B_HIGH << 32) | low; };
            const uint32_t ring = (smem_u32(my_smem) >> 4) & 0x3fffu;
            int rs = 0, buf = 0;
            uint32_t parity = 0, freed = 1;
            bool ok = true;
            for (int i = first_item; ok && i < p.items; i += item_step) {
                const Item it = item_of<WG>(p, i);
                const int cols = WG ? min(BN, (p.col_groups - it.n_tile * (BN / BG)) * BG)
                                    : min(p.width, ((p.N_total - it.n_tile * p.width) + 15) & ~15);
                const uint32_t idesc = (1u << 4) | ((WG ? 1u : 0u) << 15) | ((WG ? 1u : 0u) << 16) | ((uint32_t)(cols >> 3) << 17) |
                                       ((uint32_t)(BM >> 4) << 24);
                int c = WG ? 0 : it.begin % p.groups * GROUP;
                for (int q = it.begin; q < it.end; ++q) {
                    const int slot = set * BUFS + buf;
                    if (!mbar_wait(smem_u32(drained + slot), freed, p.status)) { ok = false; break; }
                    const uint32_t d = tmem_base + (uint32_t)(slot * BN);
                    // 16-channel steps of the group that hold channels, two per stage
                    const int steps = WG ? 4 : min(4, (p.g_C - c + 15) >> 4);
                    // the small products first, while the accumulator is small: both stages' cross terms, then their hi*hi
                    uint32_t st[2];
                    const int first = rs;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (2 * h >= steps) break;
                        if (!mbar_wait(smem_u32(my_full + rs), parity, p.status)) { ok = false; break; }
                        tc_fence_after();
                        st[h] = ring + (uint32_t)(rs * STAGE >> 4);
                        const uint32_t ah = st[h] | A_LOW, al = (st[h] + (A_LO >> 4)) | A_LOW;
                        const uint32_t bh = (st[h] + (B_HI >> 4)) | B_LOW, bl = (st[h] + (B_LO >> 4)) | B_LOW;
                        umma_f16(d, da(al), db(bh), idesc, h ? 1u : 0u);           // a block's first one overwrites the buffer
                        umma_f16_acc(d, da(ah), db(bl), idesc);
                        if (2 * h + 1 < steps) {
                            umma_f16_acc(d, da(al + A_STEP), db(bh + B_STEP), idesc);
                            umma_f16_acc(d, da(ah + A_STEP), db(bl + B_STEP), idesc);
                        }
                        if (++rs == RING) { rs = 0; parity ^= 1u; }
                    }
                    if (!ok) break;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (2 * h >= steps) break;
                        const uint32_t ah = st[h] | A_LOW, bh = (st[h] + (B_HI >> 4)) | B_LOW;
                        umma_f16_acc(d, da(ah), db(bh), idesc);
                        if (2 * h + 1 < steps) umma_f16_acc(d, da(ah + A_STEP), db(bh + B_STEP), idesc);
                        umma_commit(smem_u32(my_empty + (h == 0 ? first : first + 1 == RING ? 0 : first + 1)));
                    }
                    umma_commit(smem_u32(ready + slot));
                    c += GROUP;
                    if (c >= p.g_C) c = 0;
                    if (++buf == BUFS) { buf = 0; freed ^= 1u; }
                }
            }
        }
      }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SUM_REGS));
        const int quarter = warp & 3, half = warp >> 2, col0 = ALT ? 0 : half * HALF_COLS, row_in = quarter * 32 + lane;
        const uint32_t tsrc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ALT ? half * BUFS * BN : col0);
        const int first_item = (int)blockIdx.x + (ALT ? half * (int)gridDim.x : 0), item_step = SETS * (int)gridDim.x;
        uint64_t *const my_ready = ready + (ALT ? half * BUFS : 0), *const my_drained = drained + (ALT ? half * BUFS : 0);
        int buf = 0;
        uint32_t parity = 0;
        bool ok = true, nan_seen = false, tail_done = false;
        if (!WG && p.n_wide) {
            // this CTA's share of the verdicts, while the first block is on its way
            bool wide = false;
            for (int i = (int)blockIdx.x * (EPI_WARPS * 32) + tid; i < p.n_wide; i += (int)gridDim.x * (EPI_WARPS * 32)) wide |= p.wide[i] != 0;
            if (wide) *p.gate = 1;
        }
        // this lane's pixel of a tile
        auto locate = [&](const Item &it, const Phase &f, int &im, int &row, int &col) {
            const int m = it.m_tile * BM + row_in;
            im = m / f.HW;
            const int r = m - im * f.HW;
            row = r / f.pix_W;
            col = r - row * f.pix_W;
            return m < f.M_total;
        };
        for (int i = first_item; ok && i < p.items; i += item_step) {
            const Item it = item_of<WG>(p, i);
            const Phase &f = p.ph[it.phase];
            uint64_t acc2[HALF_COLS / 2];                                          // columns 2 j and 2 j + 1
#pragma unroll
            for (int j = 0; j < HALF_COLS / 2; ++j) acc2[j] = 0;
            const int cols = WG ? min(BN, (p.col_groups - it.n_tile * (BN / BG)) * BG) : min(p.width, p.N_total - it.n_tile * p.width);
            const int my_cols = cols - col0;                                       // may be zero or negative
            int im = 0, row = 0, col = 0;
            bool row_ok = true;
            if (!WG) row_ok = locate(it, f, im, row, col);
            // exponents of the blocks, one ahead; the registers hold the row's sums / 2^top, which is raised before a block would exceed it
            int g = 0, th = 0, tw = 0;
            if (!WG) { const int tap = it.begin / p.groups; g = it.begin - tap * p.groups; th = tap / f.kW; tw = tap - th * f.kW; }
            const int ih0 = row * f.stH + f.lH, iw0 = col * f.stW + f.lW;
            auto exp_at = [&]() -> int {
                const int ih = ih0 + th * f.dlH, iw = iw0 + tw * f.dlW;
                return row_ok && (unsigned)ih < (unsigned)p.g_H && (unsigned)iw < (unsigned)p.g_W
                           ? (int)p.exps[(((size_t)im * p.g_H + ih) * p.g_W + iw) * p.groups + g] : NO_EXP;
            };
            int next = WG ? 0 : exp_at(), top = NO_EXP;
            float blocks = 0.f;                                                    // the sum of the blocks' 2^(e - top)
            for (int q = it.begin; q < it.end; ++q) {
                const int e = next;
                if (!WG && q + 1 < it.end) {
                    if (++g == p.groups) { g = 0; if (++tw == f.kW) { tw = 0; ++th; } }
                    next = exp_at();
                }
                float s = 1.f;
                if (!WG) {
                    if (__any_sync(0xffffffffu, e > top)) raise(acc2, blocks, top, max(e + 4, top));
                    s = step(e, top);
                    if (e > ZERO_EXP) blocks += s;
                }
                if (!mbar_wait(smem_u32(my_ready + buf), parity, p.status)) { ok = false; break; }
                tc_fence_after();
                const uint32_t t0 = tsrc + (uint32_t)(buf * BN);
                const uint64_t s2 = pack2(s, s);
                uint32_t r[2][32];
                tmem_ld32_issue(t0, r[0]);
#pragma unroll
                for (int c = 0; c < HALF_COLS; c += 32) {                          // columns past the tile's hold anything and are not used
                    tmem_wait_ld(r[(c / 32) & 1]);
                    if (c + 32 < HALF_COLS) tmem_ld32_issue(t0 + (uint32_t)(c + 32), r[(c / 32 + 1) & 1]);
#pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        const uint64_t v = (uint64_t)r[(c / 32) & 1][j + 1] << 32 | r[(c / 32) & 1][j];
                        uint64_t &a = acc2[(c + j) / 2];
                        a = WG ? add2(a, v) : fma2(v, s2, a);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(my_drained + buf));
                if (++buf == BUFS) { buf = 0; parity ^= 1u; }
            }
            if (!ok) break;
            float acc[HALF_COLS];
#pragma unroll
            for (int j = 0; j < HALF_COLS; j += 2) {
                acc[j] = __uint_as_float((uint32_t)acc2[j / 2]);
                acc[j + 1] = __uint_as_float((uint32_t)(acc2[j / 2] >> 32));
            }
            if (WG) {
                // [split][column][row]: a warp writes 128 consecutive bytes of a column
                float *dst = p.partial + ((size_t)it.part * p.n_tiles * BN + (size_t)it.n_tile * BN + col0) * (p.m_tiles * BM) + it.m_tile * BM + row_in;
                const int stride = p.m_tiles * BM;
#pragma unroll
                for (int j = 0; j < HALF_COLS; ++j, dst += stride) *dst = acc[j];
                continue;
            }
            if (it.tail >= 0) {
                float *mine = p.partial + (size_t)(it.tail * p.splits + it.part) * PART + (size_t)col0 * BM + row_in;
                int *my_top = reinterpret_cast<int *>(p.partial + (size_t)(it.tail * p.splits + it.part) * PART + BN * BM) + row_in;
                if (ALT || half == 0) {
                    __stcg(my_top, top);
                    __stcg(reinterpret_cast<float *>(my_top + BM), blocks);
                }
#pragma unroll
                for (int j = 0; j < HALF_COLS; ++j) __stcg(mine + j * BM, acc[j]);
                __threadfence();
                sums_sync<SETS>(half);
                if ((tid & (ALT ? 127 : 255)) == 0) last_s[half] = atomicAdd(p.tickets + it.tail, 1) == p.splits - 1;
                sums_sync<SETS>(half);
                if (!last_s[ALT ? half : 0]) continue;
                __threadfence();
                const float *first = p.partial + (size_t)it.tail * p.splits * PART + row_in;
                auto top_of = [&](int s) { return __ldcg(reinterpret_cast<const int *>(first + (size_t)s * PART + BN * BM)); };
                top = NO_EXP;
                blocks = 0.f;
                for (int s = 0; s < p.splits; ++s) top = max(top, top_of(s));
#pragma unroll
                for (int j = 0; j < HALF_COLS; ++j) acc[j] = 0.f;
#pragma unroll 1
                for (int s = 0; s < p.splits; ++s) {
                    const float w = step(top_of(s), top);
                    blocks = fmaf(__ldcg(first + (size_t)s * PART + BN * BM + BM), w, blocks);
                    const float *src = first + (size_t)s * PART + (size_t)col0 * BM;
#pragma unroll
                    for (int j = 0; j < HALF_COLS; ++j) acc[j] = fmaf(__ldcg(src + j * BM), w, acc[j]);
                }
                tail_done = true;
            }
            // Through shared memory, 16 columns at a time, so that the columns can be a loop: as straight code over registers, run once a
            // tile, it is fetched from memory and took 20 us of a layer.  2^(row + column exponent) goes on in two halves, see scale_by;
            // a lane fetches a column's halves and bias for all (from memory in the loop: 160 clocks a column; by shuffles 90).
            const int n0 = it.n_tile * p.width + col0, he = (top - 2 * SCALED_MAX) / 2;
            const float ra = pow2(he), rb = pow2(top - 2 * SCALED_MAX - he), small_sum = p.n_wide ? 0.f : blocks * SMALL_SUM;
            float *dst = p.out + ((size_t)im * p.N_total + n0) * p.o_HW + (f.o_off + row * f.o_sH + col * f.o_sW);
            float *stage = reinterpret_cast<float *>(smem + RING_BYTES + warp * STORE_BYTES) + lane;        // a lane reads what it wrote itself
            float4 *column = reinterpret_cast<float4 *>(smem + RING_BYTES + warp * STORE_BYTES + STORE_COLS * 128);
#pragma unroll
            for (int c = 0; c < HALF_COLS; c += STORE_COLS) {
                if (c >= my_cols) break;
                const int last = min(STORE_COLS, my_cols - c);
                __syncwarp();
                if (lane < STORE_COLS) {
                    const int ec = lane < last ? p.w_exp[n0 + c + lane] : 0, hc = ec / 2;
                    // a filter of zeros loses nothing
                    column[lane] = make_float4(pow2(hc), pow2(ec - hc), p.bias && lane < last ? __ldg(p.bias + n0 + c + lane) : 0.f, ec > ZERO_EXP ? 1.f : 0.f);
                }
#pragma unroll
                for (int j = 0; j < STORE_COLS; ++j) stage[j * 32] = acc[c + j];
                __syncwarp();
                const int count = row_ok ? last : 0;
                int small = 0;
                float *to = dst + (size_t)c * p.o_HW;
#pragma unroll 1
                for (int j = 0; j < last; j += 8) {                // eight columns in step: one after the other they take 130 clocks each
                    float v[8];
                    float4 k[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) { v[i] = stage[(j + i) * 32]; k[i] = column[j + i]; }
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        nan_seen |= v[i] != v[i];
                        small += fabsf(v[i]) < small_sum * k[i].w && j + i < count;
                        v[i] = v[i] * (ra * k[i].x) * (rb * k[i].y) + k[i].z;
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i, to += p.o_HW)
                        if (j + i < count) *to = v[i];
                }
                if (__reduce_add_sync(0xffffffffu, (unsigned)small) > MOST_SMALL && lane == 0) *p.gate = 1;
            }
        }
        if (!WG && p.raw_a && __any_sync(0xffffffffu, ok && nan_seen)) {          // rows past the last may have seen some: they write nothing
            // outside the pipeline: no wait with a limit depends on how long this takes
#pragma unroll 1
            for (int i = first_item; i < p.items; i += item_step) {
                const Item it = item_of<WG>(p, i);
                if (it.tail >= 0 && !tail_done) continue;
                const Phase &f = p.ph[it.phase];
                int im, row, col;
                if (!locate(it, f, im, row, col)) continue;
                const int n0 = it.n_tile * p.width + col0, my_cols = min(p.width, p.N_total - it.n_tile * p.width) - col0;
                float *dst = p.out + ((size_t)im * p.N_total + n0) * p.o_HW + (f.o_off + row * f.o_sH + col * f.o_sW);
#pragma unroll 1
                for (int j = 0; j < HALF_COLS && j < my_cols; ++j) {
                    const float b = p.bias ? __ldg(p.bias + n0 + j) : 0.f;
                    if (isnan(dst[(size_t)j * p.o_HW]) && !isnan(b)) dst[(size_t)j * p.o_HW] = plain_sum(p, f, im, row, col, n0 + j) + b;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, 512);
}

// The sum of the splits of gw[ko][c][tap] in their order, scaled back, to `sums`; further blocks: the bias gradient from its partial sums.
// Partial sums are contiguous along the output channels, the sums along (c, tap).  They are added to the gradient by the next kernel, which
// knows all blocks' verdicts.
struct ReduceParams {
    const float *partial;
    float *sums, *gb;
    int *gate;
    const uint32_t *gy_max, *x_max, *gy_low, *x_low;
    const double *bias_part;
    int K, C, kk, groups, bg, splits, cols, rows, gw_blocks, bias_blocks;
    int shares;                              // warps that share an output's splits: 1, 2, 4 or 8
    int win_kW;                              // Window's kernel columns, or 0
    float scale, small_sum;                  // SMALL_GRAD of all products
};
__device__ __forceinline__ bool wide_range(uint32_t most, uint32_t low) { return low && (int)(most >> 23) - (int)(~low >> 23) > WIDE; }
__global__ void __launch_bounds__(256)
reduce_kernel(const __grid_constant__ ReduceParams p)
{
    pdl_wait();
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if ((int)blockIdx.x >= p.gw_blocks) {
        const int k = ((int)blockIdx.x - p.gw_blocks) * 8 + warp;
        if (k >= p.K) return;
        double s = 0.0;
        for (int i = lane; i < p.bias_blocks; i += 32) s += p.bias_part[(size_t)i * p.K + k];
        s = warp_sum(s);
        if (lane == 0) p.gb[k] = (float)((double)p.gb[k] + (double)p.scale * s);
        return;
    }
    // a warp: 32 output channels x 4 consecutive (c, tap) x every `shares`-th split
    __shared__ float tile[8][4][33];
    const int n = p.C * p.kk, per = 32 / p.shares, o_blocks = (n + per - 1) / per;
    const int kb = (int)blockIdx.x / o_blocks, ob = (int)blockIdx.x - kb * o_blocks;
    const int ko = kb * 32 + lane, share = warp & (p.shares - 1), o0 = ob * per + warp / p.shares * 4;
    const size_t split_step = (size_t)p.cols * p.rows * p.shares;
    const float *src[4];
    int c[4];
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int o = min(o0 + i, n - 1);
        c[i] = o / p.kk;
        int t = o - c[i] * p.kk, at = c[i];
        if (p.win_kW) {
            const int th = t / p.win_kW;
            at += (t - th * p.win_kW) * p.C;
            t = th;
        }
        src[i] = p.partial + ((size_t)share * p.cols + (t * p.groups + at / p.bg) * p.bg + at % p.bg) * p.rows + ko;             // ko < rows
    }
#pragma unroll 4
    for (int k = share; k < p.splits; k += p.shares)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            sum[i] += *src[i];
            src[i] += split_step;
        }
    const int eg = ko < p.K ? group_exp(p.gy_max[ko]) : 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) tile[warp][i][lane] = scale_by(sum[i], eg + group_exp(p.x_max[c[i]]) - 2 * SCALED_MAX);
    __syncthreads();
    bool small = false;
    for (int i = tid; i < 32 * per; i += 256) {
        const int k = i / per, o = i - k * per, row = kb * 32 + k, col = ob * per + o;
        if (row >= p.K || col >= n) continue;
        float s = 0.f;
        for (int j = 0; j < p.shares; ++j) s += tile[(o >> 2) * p.shares + j][o & 3][k];
        p.sums[(size_t)row * n + col] = s;
        const int ch = col / p.kk;
        const uint32_t gm = p.gy_max[row], xm = p.x_max[ch];
        if (gm && xm && (wide_range(gm, p.gy_low[row]) || wide_range(xm, p.x_low[ch])))
            small |= fabsf(s) < scale_by(p.small_sum, group_exp(gm) + group_exp(xm) - 2 * SCALED_MAX);
    }
    if (__syncthreads_count(small) > MOST_SMALL_GRADS && tid == 0) *p.gate = 1;
}

// ---- host ---------------------------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*EncodeIm2colFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                   const int *, const int *, cuuint32_t, cuuint32_t, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static void *driver_entry(const char *name)
{
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, &ptr, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) ptr = nullptr;
    return ptr;
}
static EncodeTiledFn encode_tiled()
{
    static EncodeTiledFn fn = (EncodeTiledFn)driver_entry("cuTensorMapEncodeTiled");
    return fn;
}
static EncodeIm2colFn encode_im2col()
{
    static EncodeIm2colFn fn = (EncodeIm2colFn)driver_entry("cuTensorMapEncodeIm2col");
    return fn;
}

static bool can_vec(const float *src, int HW) { return HW % 4 == 0 && ((uintptr_t)src & 15) == 0; }
// Blocks of a splitting launch.
static int prep_grid(PrepParams &q, int tensors)
{
    int grid = q.rows;
    for (int i = 0; i < tensors; ++i) {
        Act &a = q.act[i];
        a.blocks = a.win.C ? (int)(a.pixels / (uint32_t)a.win.oW) : (int)ceil_div_ll((long long)a.pixels, 64) * a.groups;
        a.ctas = a.win.C ? ceil_div(a.blocks, a.win.block_rows()) : a.blocks;
        grid += a.ctas;
    }
    return grid;
}
// Channels of a split tensor, padded with zeros: pixels start on 32 or 64 bytes.  A copy's rows of 64 bytes that begin anywhere else
// take three times as long (pixels of 48 bytes: 3.3 clocks a row).
static int padded(int c) { return c < 64 ? (c + 15) & ~15 : (c + 31) & ~31; }
static size_t round256(size_t v) { return (v + 255) & ~(size_t)255; }

// fp16 [d2][d1][d0], boxes of box0 x box1 x 1.
static int map_3d(CUtensorMap *m, const __half *base, long long d0, long long d1, long long d2, int box0, int box1, CUtensorMapSwizzle swz)
{
    cuuint64_t dims[3] = {(cuuint64_t)d0, (cuuint64_t)d1, (cuuint64_t)d2};
    cuuint64_t strides[2] = {(cuuint64_t)d0 * 2, (cuuint64_t)d0 * (cuuint64_t)d1 * 2};
    cuuint32_t box[3] = {(cuuint32_t)box0, (cuuint32_t)box1, 1}, estr[3] = {1, 1, 1};
    const CUresult r = encode_tiled()(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void *)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                      swz, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : fail("cuTensorMapEncodeTiled failed with code %d", (int)r);
}
// An axis of an im2col walk: positions low, low + step, ... (n of them) of an axis of `size`, plus a tap's offset of up to (taps - 1) * dil.
struct Walk {
    int size, low, n, step, taps, dil;
    int upper() const { return low + (n - 1) * step - (size - 1); }
    // the map's fields: corners of 8 bits with sign, offsets of 8 bits, steps of up to 8
    bool fits() const { return low >= -128 && low <= 127 && upper() >= -128 && upper() <= 127 && (taps - 1) * dil <= 255 && step <= 8; }
};
// fp16 [images2][H][W][Cp] (both parts' images), boxes of `pixels` consecutive pixels of the walk x `channels`.
static int map_im2col(CUtensorMap *m, const __half *base, int Cp, int images2, const Walk &h, const Walk &w, int channels, int pixels,
                      CUtensorMapSwizzle swz)
{
    cuuint64_t dims[4] = {(cuuint64_t)Cp, (cuuint64_t)w.size, (cuuint64_t)h.size, (cuuint64_t)images2};
    cuuint64_t strides[3] = {(cuuint64_t)Cp * 2, (cuuint64_t)Cp * 2 * w.size, (cuuint64_t)Cp * 2 * w.size * h.size};
    const int lower[2] = {w.low, h.low}, upper[2] = {w.upper(), h.upper()};
    cuuint32_t estr[4] = {1, (cuuint32_t)w.step, (cuuint32_t)h.step, 1};
    const CUresult r = encode_im2col()(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, (void *)base, dims, strides, lower, upper, (cuuint32_t)channels,
                                       (cuuint32_t)pixels, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : fail("cuTensorMapEncodeIm2col failed with code %d", (int)r);
}

template <class... Args>
static int launch(const char *name, const void *kern, int grid, int threads, size_t smem, cudaStream_t stream, bool dependent, Args &...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
    if (smem) CUNN_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    void *ptrs[] = {(void *)&args...};
    const cudaError_t e = cudaLaunchKernelExC(&cfg, kern, ptrs);
    return e == cudaSuccess ? 0 : fail("launch of %s failed: %s", name, cudaGetErrorString(e));
}

// Images per round: the parts of one round's images take about as much memory as the images and are bounded.
constexpr size_t ROUND_BYTES = (size_t)512 << 20;
static int images_per_round(int N, size_t image_bytes)
{
    const int most = (int)std::max<size_t>(1, std::min<size_t>((size_t)N, ROUND_BYTES / std::max<size_t>(1, image_bytes)));
    return ceil_div(N, ceil_div(N, most));             // rounds of one size
}
// Smaller im2col tensor maps are left alone, as a precaution: public code for them works around what drivers encode for tensors below 128 KiB.
// Not seen here, and not to be tried: a wrong walk may read out of bounds.  It keeps layers of up to 32,768 values away, of a pass's fixed
// 12 us the smallest.
constexpr size_t MIN_MAP_BYTES = 131072;

// ---- forward pass and input gradients -------------------------------------------------------------------------------------------
// Few input channels: the geometry of the same convolution on the tensor of row windows.
static bool windowed(const Geometry &g, Geometry &v, Window &win)
{
    v = g;
    win = Window{};
    if (g.C >= 16) return true;
    win = Window{g.C, g.kW, g.dW, g.padW, g.W, g.oW};
    if (g.kH * g.kW == 1 || g.C * g.kW > GROUP || g.dilW != 1 || win.row_values() > TILE_VALUES) return false;
    v.C = g.C * g.kW; v.W = g.oW; v.kW = v.dW = v.dilW = 1; v.padW = 0;
    return true;
}

struct Plan {
    Params p;
    Window win;
    Walk wh[MAX_PHASES], ww[MAX_PHASES];
    int images, Cp, bn;                    // images per round, padded() channels of the gathered tensor, column tile of the kernel
    int rows, taps;                        // weight rows (columns of the product) and taps
    size_t off_w, off_exps, off_exp, off_tickets, off_partial, off_gate, off_wide, bytes;
};

// The tiles of `images` images: their number, which of them are cut, and into how many parts.
static void plan_tiles(Params &p, int images)
{
    p.images = images;
    int tiles = 0, blocks = 1 << 30;
    for (int i = 0; i < p.n_phases; ++i) {
        Phase &f = p.ph[i];
        f.tile0 = tiles;
        f.M_total = images * f.HW;
        f.blocks = f.taps * p.groups;
        tiles += ceil_div(f.M_total, BM) * p.n_tiles;
        blocks = std::min(blocks, f.blocks);
    }
    const int grid = sm_count(), rest = tiles % grid;
    p.full = tiles - rest;
    p.splits = rest ? std::max(1, std::min(std::min(grid / rest, blocks / 4), 16)) : 1;
    p.items = p.full + rest * p.splits;
}

// `gathered`: channels, rows and columns of the tensor that is read; `columns`: channels of the tensor that is written.
static bool finish_plan(Plan &pl, int N, int gC, int gH, int gW, int columns, int kk, int oHW)
{
    Params &p = pl.p;
    p.g_C = gC; p.g_H = gH; p.g_W = gW;
    p.groups = ceil_div(gC, GROUP);
    p.w_kk = kk; p.o_HW = oHW; p.N_total = columns;
    pl.bn = columns <= 64 ? 64 : columns <= 128 ? 128 : 256;
    p.n_tiles = ceil_div(columns, pl.bn);
    p.width = (ceil_div(columns, p.n_tiles) + 15) & ~15;
    pl.Cp = padded(gC);
    pl.rows = columns; pl.taps = kk;
    const size_t image_bytes = (size_t)gH * gW * pl.Cp * 4;
    pl.images = images_per_round(N, image_bytes);
    if (pl.images * image_bytes < MIN_MAP_BYTES) return false;
    for (int i = 0; i < p.n_phases; ++i)
        if (!pl.wh[i].fits() || !pl.ww[i].fits()) return false;
    plan_tiles(p, pl.images);
    size_t at = round256(pl.images * image_bytes);
    pl.off_w = at; at += round256((size_t)2 * kk * columns * pl.Cp * 2);
    pl.off_exps = at; at += round256((size_t)pl.images * gH * gW * p.groups);
    pl.off_exp = at; at += round256((size_t)columns * 4);
    pl.off_tickets = at; at += round256((size_t)sm_count() * 4);
    pl.off_partial = at; at += round256((size_t)sm_count() * (pl.bn + 2) * BM * 4);
    pl.off_gate = at; at += 256;
    if (pl.win.C) { pl.off_wide = at; at += round256((size_t)columns + (size_t)pl.images * gH); }         // a block has a row or more
    pl.bytes = at + 256;
    return true;
}

// Column tile of the element-copy kernels: narrower ones while the wide ones leave half of the SMs without a tile.
static int element_copy_columns(int columns, long long rows)
{
    int bn = columns <= 32 ? 32 : columns <= 64 ? 64 : 128;
    while (bn > 32 && ceil_div_ll(rows, BM) * ceil_div(columns, bn) * 2 <= sm_count()) bn /= 2;
    return bn;
}
// Whether a pass is over sooner here than on the gathering kernels (convmm.cu): the split reads and writes the whole tensor, so short sums
// that read it once or twice (few channels, strides, small images) are better off there.  Both times are estimated, in us: here from
// the column tile's blocks that the busiest SM sums, the values that the split reads and writes, what is written, and whether tiles are
// cut; there from the k-blocks of the busiest SM and what is written.  The coefficients were fitted to 859 layers drawn over 16 to
// 1024 channels (few-channel layers: 3), kernels of 2x2 to 11x11 and maps of 7 to 224; nine in ten estimates lie within 0.72 to 1.24 of
// the time.  Sums of the times in ms, there / here / by the rule / with the better one each time, and the rule's losses of more than 3 %:
//   forward               53.0 / 21.9 / 21.9 / 21.7    5 of 314, the worst 1.17
//   few channels          7.08 / 5.21 / 4.68 / 4.65    0 of 110   (kernels of up to 32 taps)
//                         4.64 / 3.48 / 3.39 / 3.38    1 of 88, 1.03
//   strided gradients     22.3 / 9.06 / 9.02 / 9.00    1 of 129, 1.06   (stride 1: 29.3 / 8.0, never slower here)
//   parameter gradients   54.1 / 30.1 / 28.8 / 28.5    6 of 347, 1.40
//   ... few channels      11.5 / 13.1 / 10.5 / 10.4    1 of 198, 1.32
// and of 330 1x1 layers, on whose planes tensor maps work / do not:
//   forward               4.15 / 5.31 / 4.04 / 4.03    0 of 106        8.23 / 7.26 / 6.83 / 6.76    2 of 190, 1.27
//   input gradients       3.51 / 4.91 / 3.39 / 3.37    0 of 86         4.79 / 4.07 / 3.90 / 3.88    4 of 101, 1.09
//   parameter gradients   4.73 / 8.70 / 4.73 / 4.72    0 of 120        7.77 / 11.2 / 7.61 / 7.47    0 of 163
struct HereCost {
    double fixed, block256, block128, block64, value, out, cut, weight;            // the last five but cut per million
};
struct ThereCost {
    double fixed, wave, block128, block64, block32, out, longest, in = 0.0;
};
constexpr HereCost HERE_FORWARD{13.2, 0.97, 0.80, 0.51, 0.82, 1.25, 5.8, 12.7}, HERE_FEW{12.5, 0.30, 0.30, 0.15, 3.33, 1.67, 0.0, 137.0},
    HERE_FEW_LARGE{13.3, 0.60, 0.60, 0.30, 2.28, 0.46, 4.5, 13.5}, HERE_STRIDED{15.2, 1.37, 0.79, 0.52, 0.51, 1.65, 5.5, 8.0};
constexpr ThereCost THERE_FORWARD{9.2, 1.72, 1.35, 1.18, 1.0, 0.51, 0.0}, THERE_FEW{6.1, 0.0, 5.69, 4.20, 3.84, 0.45, 0.78},
    THERE_FEW_LARGE{6.7, 2.87, 1.80, 1.37, 1.21, 0.79, 0.0}, THERE_STRIDED{4.2, 3.97, 1.97, 1.42, 1.20, 0.45, 0.44};
// 1x1 layers of stride 1 on planes and channels that tensor maps take (multiples of four), and the others.
constexpr HereCost HERE_POINT{14.7, 1.10, 0.57, 0.06, 0.71, 1.35, 5.6, 5.0}, HERE_POINT_GRAD{13.2, 1.30, 0.77, 0.30, 0.72, 1.09, 5.0, 6.5};
constexpr ThereCost THERE_POINT{9.1, 0.26, 0.66, 0.53, 0.45, 0.76, 0.0, 0.06}, THERE_POINT_ODD{8.3, 0.71, 1.10, 0.85, 0.79, 2.19, 0.15, 0.09},
    THERE_POINT_GRAD{7.6, 0.42, 0.74, 0.61, 0.52, 0.20, 0.0, 0.04}, THERE_POINT_GRAD_ODD{7.8, 0.10, 1.26, 1.15, 1.10, 1.18, 0.0};
constexpr double MARGIN = 1.05;

// `aligned`: the other kernel works on whole groups of 32 pixels of an image.
static bool is_faster(const Plan &pl, int N, const HereCost &h, const ThereCost &t, double values, double out, double weights, bool aligned = false)
{
    const Params &p = pl.p;
    const int grid = sm_count();
    double blocks = 0, there_blocks = 0, rows = 0, longest = 0;
    int tiles = 0;
    for (int i = 0; i < p.n_phases; ++i) rows += (double)N * (aligned ? ceil_div(p.ph[i].HW, 32) * 32 : p.ph[i].HW);
    const int bn = element_copy_columns(p.N_total, (long long)rows), there_cols = ceil_div(p.N_total, bn);
    double there_tiles = 0;
    for (int i = 0; i < p.n_phases; ++i) {
        const Phase &f = p.ph[i];
        const double m = std::ceil((double)N * f.HW / BM), k = ceil_div(f.taps * p.g_C, BK);
        tiles += (int)m * p.n_tiles;
        blocks += m * p.n_tiles * f.taps * p.groups;
        const double there_m = aligned ? std::ceil(rows / BM) : m;
        there_tiles += there_m * there_cols;
        there_blocks += there_m * there_cols * k;
        longest = std::max(longest, k);
    }
    const double busiest = blocks / tiles * (tiles / grid + (tiles % grid ? 1.0 / p.splits : 0.0)), waves = std::ceil(there_tiles / grid);
    const double here = h.fixed + (pl.bn == 256 ? h.block256 : pl.bn == 128 ? h.block128 : h.block64) * busiest + (h.value * values + h.out * out + h.weight * weights) / 1e6 +
                        (p.splits > 1 ? h.cut : 0.0);
    const double there = t.fixed + waves * (t.wave + (bn == 128 ? t.block128 : bn == 64 ? t.block64 : t.block32) * there_blocks / there_tiles) + t.out * out / 1e6 +
                         t.in * rows * p.g_C / 1e6 + (waves == 1.0 ? t.longest * longest : 0.0);
    return here * MARGIN < there;
}

static bool plan_forward(Plan &pl, const Geometry &whole)
{
    pl = Plan{};
    Geometry g;
    if (whole.K < 16 || !windowed(whole, g, pl.win)) return false;
    Phase &f = pl.p.ph[0];
    f.HW = g.oH * g.oW; f.pix_W = g.oW; f.taps = g.kH * g.kW; f.kW = g.kW;
    f.lH = -g.padH; f.lW = -g.padW; f.stH = g.dH; f.stW = g.dW; f.dlH = g.dilH; f.dlW = g.dilW;
    f.w_sH = g.kW; f.w_sW = 1; f.o_sH = g.oW; f.o_sW = 1;
    pl.p.n_phases = 1;
    pl.wh[0] = Walk{g.H, f.lH, g.oH, g.dH, g.kH, g.dilH};
    pl.ww[0] = Walk{g.W, f.lW, g.oW, g.dW, g.kW, g.dilW};
    if (!finish_plan(pl, g.N, g.C, g.H, g.W, g.K, g.kH * g.kW, f.HW)) return false;
    const double in = (double)whole.N * whole.C * whole.H * whole.W, split = (double)g.N * g.H * g.W * pl.Cp, out = (double)g.N * g.K * f.HW;
    const double weights = (double)whole.K * whole.C * whole.kH * whole.kW;
    if (whole.kH * whole.kW == 1) {
        const bool aligned = whole.dH == 1 && whole.dW == 1 && whole.padH == 0 && whole.padW == 0 && f.HW % 4 == 0 && whole.C % 4 == 0;
        return is_faster(pl, g.N, HERE_POINT, aligned ? THERE_POINT : THERE_POINT_ODD, in + split, out, weights, aligned);
    }
    const bool large = whole.kH * whole.kW > 32;               // of 16 channels and more: always faster here
    if (!pl.win.C) return large || is_faster(pl, g.N, HERE_FORWARD, THERE_FORWARD, in + split, out, weights);
    return is_faster(pl, g.N, large ? HERE_FEW_LARGE : HERE_FEW, large ? THERE_FEW_LARGE : THERE_FEW, in + split, out, weights);
}

// Residues of fewer than 48 products belong to phase_fma_kernel, which loses no bits of them.
static bool plan_grad_input(Plan &pl, const Geometry &g)
{
    pl = Plan{};
    if (g.C < 16 || g.K < 64 || g.dH > 2 || g.dW > 2) return false;
    bool gaps = false;
    const std::vector<AxisPhase> ah = axis_phases(g.H, g.kH, g.dH, g.padH, g.dilH, false, &gaps), aw = axis_phases(g.W, g.kW, g.dW, g.padW, g.dilW, false, &gaps);
    if (gaps || ah.empty() || aw.empty()) return false;
    Params &p = pl.p;
    struct Pair { const AxisPhase *a, *b; } order[MAX_PHASES];
    for (const AxisPhase &a : ah)
        for (const AxisPhase &b : aw) order[p.n_phases++] = Pair{&a, &b};
    // longest reductions first: the tiles that are cut, and the last wave, are the short ones
    std::stable_sort(order, order + p.n_phases, [](const Pair &u, const Pair &v) { return u.a->taps * u.b->taps > v.a->taps * v.b->taps; });
    for (int i = 0; i < p.n_phases; ++i) {
        const AxisPhase &a = *order[i].a, &b = *order[i].b;
        Phase &f = p.ph[i];
        f.HW = a.n * b.n; f.pix_W = b.n; f.taps = a.taps * b.taps; f.kW = b.taps;
        // taps in ascending order of position: the last tap of the residue reads the first one
        f.lH = a.o0 - (a.taps - 1) * a.ostep; f.lW = b.o0 - (b.taps - 1) * b.ostep;
        f.stH = f.stW = 1; f.dlH = a.ostep; f.dlW = b.ostep;
        f.w_base = (a.k0 + (a.taps - 1) * a.kstep) * g.kW + b.k0 + (b.taps - 1) * b.kstep;
        f.w_sH = -a.kstep * g.kW; f.w_sW = -b.kstep;
        f.o_off = a.h0 * g.W + b.h0; f.o_sH = g.dH * g.W; f.o_sW = g.dW;
        pl.wh[i] = Walk{g.oH, f.lH, a.n, 1, a.taps, a.ostep};
        pl.ww[i] = Walk{g.oW, f.lW, b.n, 1, b.taps, b.ostep};
    }
    if (!finish_plan(pl, g.N, g.K, g.oH, g.oW, g.C, g.kH * g.kW, g.H * g.W)) return false;
    if (g.kH * g.kW == 1 && g.dH == 1 && g.dW == 1) {
        const bool aligned = g.padH == 0 && g.padW == 0 && g.H * g.W % 4 == 0 && g.C % 4 == 0;
        return is_faster(pl, g.N, HERE_POINT_GRAD, aligned ? THERE_POINT_GRAD : THERE_POINT_GRAD_ODD, (double)g.N * g.oH * g.oW * (g.K + pl.Cp),
                         (double)g.N * g.C * g.H * g.W, (double)g.K * g.C, aligned);
    }
    if (p.n_phases == 1 || g.kH * g.kW > 32) return true;
    return is_faster(pl, g.N, HERE_STRIDED, THERE_STRIDED, (double)g.N * g.oH * g.oW * (g.K + pl.Cp), (double)g.N * g.C * g.H * g.W,
                     (double)g.K * g.C * g.kH * g.kW);
}

// src: the gathered tensor; weights of (row, channel, tap) at row * w_row + channel * w_c + tap.
static int run_plan(Plan &pl, int N, const float *src, const float *weight, long long w_row, long long w_c, const float *bias, float *out, bool redo_nan,
                    const Fallback &again, void *scratch, cudaStream_t stream)
{
    Params &p = pl.p;
    char *ws = (char *)scratch;
    __half *a = (__half *)ws, *w = (__half *)(ws + pl.off_w);
    p.exps = (const int8_t *)(ws + pl.off_exps); p.w_exp = (int *)(ws + pl.off_exp); p.tickets = (int *)(ws + pl.off_tickets);
    p.partial = (float *)(ws + pl.off_partial); p.bias = bias; p.status = device_status_ptr();
    p.gate = (int *)(ws + pl.off_gate); p.wide = (const uint8_t *)(ws + pl.off_wide);
    const int g_HW = p.g_H * p.g_W;
    alignas(64) Maps maps;
    if (map_3d(&maps.b, w, pl.Cp, pl.rows, 2 * pl.taps, BK, pl.bn, CU_TENSOR_MAP_SWIZZLE_64B)) return 1;
    for (int at = 0; at < N; at += pl.images) {
        const int n = std::min(pl.images, N - at);
        plan_tiles(p, n);
        const float *from = src + (size_t)at * (pl.win.C ? (size_t)pl.win.C * p.g_H * pl.win.W : (size_t)p.g_C * g_HW);
        p.out = out + (size_t)at * p.N_total * p.o_HW;
        p.raw_a = redo_nan ? from : nullptr;
        p.raw_w = weight;
        for (int i = 0; i < p.n_phases; ++i)
            if (map_im2col(&maps.a[i], a, pl.Cp, 2 * n, pl.wh[i], pl.ww[i], BK, BM, CU_TENSOR_MAP_SWIZZLE_64B)) return 1;
        PrepParams q{};
        Act &act = q.act[0];
        act.src = from; act.dst = a; act.exps = const_cast<int8_t *>(p.exps); act.C = p.g_C; act.Cp = pl.Cp; act.HW = g_HW;
        act.groups = p.groups; act.pixels = (uint32_t)n * g_HW; 
        act.vec = can_vec(from, g_HW);
        act.win = pl.win;
        q.w = weight; q.w_dst = w; q.w_exp = const_cast<int *>(p.w_exp); q.rows = at ? 0 : pl.rows; q.w_C = p.g_C; q.w_Cp = pl.Cp; q.taps = pl.taps;
        q.w_row = w_row; q.w_c = w_c; q.win_C = pl.win.C; q.win_kW = pl.win.kW; q.tickets = p.tickets; q.n_tickets = sm_count();
        q.gate = p.gate; q.wide = const_cast<uint8_t *>(p.wide) + (at ? pl.rows : 0);        // the weights' verdicts count for all rounds
        const int blocks = prep_grid(q, 1);
        p.n_wide = pl.win.C ? pl.rows + act.ctas : 0;
        if (launch("convolution operand split", pl.win.C ? (const void *)prep_kernel<false, true> : (const void *)prep_kernel<false, false>, blocks, 256, 0, stream, true, q)) return 1;
        const void *kern = pl.bn == 64    ? (const void *)split_gemm_kernel<64, false>
                           : pl.bn == 128 ? (const void *)split_gemm_kernel<128, false>
                                          : (const void *)split_gemm_kernel<256, false>;
        if (launch("convolution of split operands", kern, std::min(p.items, sm_count()), THREADS, SMEM, stream, true, p, maps)) return 1;
        if (again(at, n, p.gate)) return 1;
    }
    return 0;
}

size_t forward_scratch(const Geometry &g)
{
    Plan pl;
    return plan_forward(pl, g) ? pl.bytes : 0;
}
size_t grad_input_scratch(const Geometry &g)
{
    Plan pl;
    return plan_grad_input(pl, g) ? pl.bytes : 0;
}
int forward(const Geometry &g, const float *x, const float *weight, const float *bias, float *y, const Fallback &again, void *scratch,
            cudaStream_t stream)
{
    Plan pl;
    if (!plan_forward(pl, g)) return fail("convolution forward: no plan for split operands");
    const int kk = g.kH * g.kW;
    return run_plan(pl, g.N, x, weight, (long long)g.C * kk, kk, bias, y, false, again, scratch, stream);
}
int grad_input(const Geometry &g, const float *gy, const float *weight, const float *bias, float *gx, const Fallback &again, void *scratch,
               cudaStream_t stream)
{
    Plan pl;
    if (!plan_grad_input(pl, g)) return fail("convolution input gradient: no plan for split operands");
    const int kk = g.kH * g.kW;
    return run_plan(pl, g.N, gy, weight, kk, (long long)g.C * kk, bias, gx, g.dH > 1 || g.dW > 1, again, scratch, stream);
}

// ---- weight gradients ---------------------------------------------------------------------------------------------------------------
struct WgradPlan {
    Params p;
    Window win;
    Geometry v;                                // the convolution, on row windows where the channels are few
    Walk wh, ww;
    int images, Cp, Kp, bn, bg;
    size_t off_x, off_gy, off_bias, off_partial, bytes;
};
static void plan_splits(WgradPlan &pl, int images)
{
    Params &p = pl.p;
    p.images = images;
    p.blocks = (int)ceil_div_ll((long long)images * p.pix_HW, 2 * BK);
    const int grid = sm_count();
    double best = -1.0;
    for (int waves = 1; waves <= 8; ++waves) {
        const int want = std::max(1, std::min(p.blocks, waves * grid / p.tiles));
        const int per = ceil_div(p.blocks, want), splits = ceil_div(p.blocks, per);
        // a tile's partial sums cost about four blocks, and the reduction reads all of them
        const double cost = (double)ceil_div_ll((long long)p.tiles * splits, grid) * (per + 4.0) + (double)splits * p.tiles * 4.0 / grid;
        if (best < 0.0 || cost < best * 0.999) { best = cost; p.per_split = per; p.splits = splits; }
    }
    p.items = p.tiles * p.splits;
}
// As is_faster.
static bool grad_weight_is_faster(const WgradPlan &pl, const Geometry &g)
{
    if (!pl.win.C && g.kH * g.kW > 32) return true;
    const Params &p = pl.p;
    const bool few = pl.win.C != 0;
    const int grid = sm_count();
    const double weights = (double)g.K * g.C * g.kH * g.kW / 1e6, values = ((double)g.N * g.C * g.H * g.W + (double)g.N * g.K * p.pix_HW) / 1e6;
    const double split = ((double)g.N * pl.v.H * pl.v.W * pl.Cp + (double)g.N * p.pix_HW * pl.Kp) / 1e6, partial = (double)p.items * pl.bn * BM / 1e6;
    const double busiest = (double)ceil_div(p.items, grid) * p.per_split;
    if (g.kH * g.kW == 1) {
        // 1x1: against the tensor-map kernel never; planes that it does not take
        if (g.dH == 1 && g.dW == 1 && g.padH == 0 && g.padW == 0 && p.pix_HW % 4 == 0) return false;
        const double t = (double)ceil_div(g.K, BM) * ceil_div(g.C, g.C <= 32 ? 32 : g.C <= 64 ? 64 : 128), b = (double)ceil_div_ll((long long)g.N * p.pix_HW, BK);
        const double here = 17.6 + (pl.bn == 256 ? 1.27 : 1.91) * busiest + 3.98 * partial + 3.04 * split;
        return here * MARGIN < 16.9 + 1.19 * t * b / grid + 18.0 * weights + (t * b > grid ? 0.72 : 0.0) + 0.19 * std::min(b, std::ceil(t * b / grid));
    }
    const double here = few ? 19.0 + 0.68 * busiest + 3.97 * partial + 2.04 * values + 2.41 * split
                            : 17.8 + (pl.bn == 256 ? 1.38 : 1.07) * busiest + 2.60 * partial + 2.71 * split + 4.0 * weights;
    const double tiles = (double)ceil_div(g.K, BM) * ceil_div(g.C * g.kH * g.kW, BM), blocks = (double)ceil_div_ll((long long)g.N * p.pix_HW, BK);
    const double there = few ? 16.1 + 1.26 * tiles * blocks / grid + 196.0 * weights + 0.47 * std::min(blocks, std::ceil(tiles * blocks / grid))
                             : 16.3 + 1.97 * tiles * blocks / grid + 6.14 * weights;
    return here * MARGIN < there;
}
static bool plan_grad_weight(WgradPlan &pl, const Geometry &whole)
{
    pl = WgradPlan{};
    Params &p = pl.p;
    if (whole.K < 16 || !windowed(whole, pl.v, pl.win)) return false;
    const Geometry &g = pl.v;
    const int kk = g.kH * g.kW;
    pl.bg = g.C <= 32 && kk > 2 ? 32 : GROUP;
    p.groups = ceil_div(g.C, pl.bg);
    p.col_groups = kk * p.groups;
    pl.bn = p.col_groups * pl.bg <= 128 ? 128 : 256;
    p.n_tiles = ceil_div(p.col_groups, pl.bn / pl.bg);
    p.m_tiles = ceil_div(g.K, BM);
    p.N_total = g.K;
    p.tiles = p.n_tiles * p.m_tiles;
    p.kW = g.kW; p.pix_HW = g.oH * g.oW; p.pix_W = g.oW;
    p.lH = -g.padH; p.lW = -g.padW; p.stH = g.dH; p.stW = g.dW; p.dlH = g.dilH; p.dlW = g.dilW;
    pl.wh = Walk{g.H, p.lH, g.oH, g.dH, g.kH, g.dilH};
    pl.ww = Walk{g.W, p.lW, g.oW, g.dW, g.kW, g.dilW};
    if (!pl.wh.fits() || !pl.ww.fits()) return false;
    pl.Cp = padded(g.C); pl.Kp = padded(g.K);
    const size_t x_bytes = (size_t)g.H * g.W * pl.Cp * 4, gy_bytes = (size_t)p.pix_HW * pl.Kp * 4;
    pl.images = images_per_round(g.N, std::max(x_bytes, gy_bytes));
    if (pl.images * x_bytes < MIN_MAP_BYTES) return false;
    plan_splits(pl, pl.images);
    if (!grad_weight_is_faster(pl, whole)) return false;
    size_t at = grad_weight_head(whole);
    pl.off_x = at; at += round256(pl.images * x_bytes);
    pl.off_gy = at; at += round256(pl.images * gy_bytes);
    pl.off_bias = at; at += round256((size_t)ceil_div_ll((long long)pl.images * ceil_div(p.pix_HW, PIECE), 8) * g.K * 8);
    // a round of fewer images may be cut into a few more parts than a whole one
    pl.off_partial = at; at += round256((size_t)(p.splits + 1) * p.n_tiles * pl.bn * p.m_tiles * BM * 4);
    pl.bytes = at + 256;
    return true;
}
size_t grad_weight_scratch(const Geometry &g, size_t (*again_bytes)(const Geometry &))
{
    WgradPlan pl;
    if (!plan_grad_weight(pl, g)) return 0;
    size_t bytes = pl.bytes;
    Geometry round = g;
    for (int images : {pl.images, (g.N - 1) % pl.images + 1}) {
        round.N = images;
        bytes = std::max(bytes, grad_weight_head(g) + again_bytes(round));
    }
    return bytes;
}
int grad_weight(const Geometry &g, const float *x, const float *gy, float *grad_bias, float scale, const Fallback &again, void *scratch,
                cudaStream_t stream)
{
    WgradPlan pl;
    if (!plan_grad_weight(pl, g)) return fail("convolution parameter gradient: no plan for split operands");
    Params &p = pl.p;
    char *ws = (char *)scratch;
    p.gate = (int *)ws;
    __half *xs = (__half *)(ws + pl.off_x), *gs = (__half *)(ws + pl.off_gy);
    uint32_t *gy_max = (uint32_t *)(ws + GATE_BYTES), *x_max = gy_max + g.K, *gy_low = x_max + g.C, *x_low = gy_low + g.K;
    double *bias_part = (double *)(ws + pl.off_bias);
    p.partial = (float *)(ws + pl.off_partial);
    p.status = device_status_ptr();
    const int kk = g.kH * g.kW, x_HW = g.H * g.W;
    const int most = p.splits + 1;
    for (int at = 0; at < g.N; at += pl.images) {
        const int n = std::min(pl.images, g.N - at);
        plan_splits(pl, n);
        if (p.splits > most) { p.per_split = ceil_div(p.blocks, most); p.splits = ceil_div(p.blocks, p.per_split); p.items = p.tiles * p.splits; }
        const float *xr = x + (size_t)at * g.C * x_HW, *gr = gy + (size_t)at * g.K * p.pix_HW;
        alignas(64) Maps maps;
        if (map_3d(&maps.a[0], gs, pl.Kp, (long long)n * p.pix_HW, 2, GROUP, BK, CU_TENSOR_MAP_SWIZZLE_128B)) return 1;
        if (map_im2col(&maps.b, xs, pl.Cp, 2 * n, pl.wh, pl.ww, pl.bg, BK, pl.bg == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B)) return 1;
        CUNN_CUDA(cudaMemsetAsync(ws, 0, GATE_BYTES + max_bytes(g), stream));
        MaxParams m{};
        m.src[0] = gr; m.src[1] = xr; m.chmax[0] = gy_max; m.chmax[1] = x_max; m.chlow[0] = gy_low; m.chlow[1] = x_low; m.C[0] = g.K; m.C[1] = g.C; m.HW[0] = p.pix_HW; m.HW[1] = x_HW;
        m.images = n;
        m.sums = grad_bias ? bias_part : nullptr;
        for (int t = 0; t < 2; ++t) {
            // 32 pieces a block, so that a warp has four loads in flight, or 8 where that leaves SMs idle
            m.pieces[t] = ceil_div(m.HW[t], PIECE);
            const long long pieces = (long long)n * m.pieces[t];
            m.chunks[t] = (int)std::max(ceil_div_ll(pieces, 32), std::min(ceil_div_ll(pieces, 8), (long long)ceil_div(2 * sm_count(), m.C[t])));
            m.vec[t] = can_vec(m.src[t], m.HW[t]);
        }
        if (launch("convolution channel maxima", (const void *)channel_max_kernel, m.C[0] * m.chunks[0] + m.C[1] * m.chunks[1], 256, 0, stream, false, m)) return 1;
        PrepParams q{};
        for (int t = 0; t < 2; ++t) {
            Act &act = q.act[t];
            act.src = t ? xr : gr; act.dst = t ? xs : gs; act.chmax = t ? x_max : gy_max;
            act.C = t ? pl.v.C : g.K; act.Cp = t ? pl.Cp : pl.Kp; act.HW = t ? pl.v.H * pl.v.W : p.pix_HW; act.groups = ceil_div(act.C, GROUP);
            if (t) act.win = pl.win;
            act.vec = can_vec(act.src, act.HW);
            act.pixels = (uint32_t)n * act.HW;
        }
        if (launch("convolution operand split", pl.win.C ? (const void *)prep_kernel<true, true> : (const void *)prep_kernel<true, false>, prep_grid(q, 2), 256, 0, stream, true, q)) return 1;
        const void *kern = pl.bg == 32    ? pl.bn == 128 ? (const void *)split_gemm_kernel<128, true, 32> : (const void *)split_gemm_kernel<256, true, 32>
                           : pl.bn == 128 ? (const void *)split_gemm_kernel<128, true>
                                          : (const void *)split_gemm_kernel<256, true>;
        if (launch("convolution parameter gradient of split operands", kern, std::min(p.items, sm_count()), THREADS, SMEM, stream, true, p, maps)) return 1;
        ReduceParams r{};
        r.partial = p.partial; r.sums = grad_weight_sums(g, scratch); r.gate = p.gate; r.gb = grad_bias; r.gy_max = gy_max; r.x_max = x_max; r.gy_low = gy_low;
        r.x_low = x_low; r.bias_part = bias_part; r.small_sum = SMALL_GRAD * std::sqrt((float)n * (float)p.pix_HW);
        r.K = g.K; r.C = g.C; r.kk = kk; r.groups = p.groups; r.bg = pl.bg; r.win_kW = pl.win.kW; r.splits = p.splits; r.cols = p.n_tiles * pl.bn; r.rows = p.m_tiles * BM;
        // one warp per output leaves SMs idle where the outputs are few: 9,408 outputs of 146 splits took 36 us
        r.shares = 1;
        while (r.shares < 8 && r.shares * 8 <= p.splits && ceil_div(g.K, 32) * ceil_div(g.C * kk * r.shares, 32) < 4 * sm_count()) r.shares *= 2;
        r.gw_blocks = ceil_div(g.K, 32) * ceil_div(g.C * kk, 32 / r.shares);
        r.bias_blocks = m.chunks[0];
        r.scale = scale;
        if (launch("convolution parameter gradient sums", (const void *)reduce_kernel, r.gw_blocks + (grad_bias ? ceil_div(g.K, 8) : 0), 256, 0, stream,
                   true, r)) return 1;
        if (again(at, n, p.gate)) return 1;
    }
    return 0;
}

}  // namespace split
}  // namespace cunn
