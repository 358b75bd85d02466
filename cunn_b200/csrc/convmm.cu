// SpatialConvolutionMM on the 5th-generation tensor cores (tcgen05 / TMEM), fp32 in and out.
//
// The reference unfolds every image into a column buffer and calls SGEMM per image.  Here the three
// passes are implicit GEMMs — no column buffer exists — computed by tcgen05.mma.kind::tf32 with a
// 3xTF32 split: every fp32 operand value v is used as hi (its upper 19 bits) and lo = v - hi, and each
// K step issues lo*hi + hi*lo + hi*hi into fp32 TMEM accumulators.  The dropped lo*lo term and the tf32
// truncation of lo are ~2^-20 relative, i.e. fp32-class accuracy.
//
//   forward      D[pixel, k_out]        = sum_{c,kh,kw}  x(pixel; c,kh,kw)   * W[k_out][c,kh,kw]
//   input grad   D[pixel, c]            = sum_{k,kh,kw}  gy(pixel; k,kh,kw)  * W[k][c][flipped kh,kw]   (stride 1)
//   weight grad  D[k_out, (c,kh,kw)]    = sum_{img,pix}  gy[img][k_out][pix] * x(pix; c,kh,kw)          (split over pixels)
//
// Five kernel families share these roles:
//   * pwt::pw_tma_kernel<OP, BN, ...> (pw_tma.cuh) — 1x1 stride-1 convolutions on aligned tensors, and fully connected layers;
//   * pw::pw_gemm_kernel<OP, BN, KS> — the persistent, warp-specialised kernel (further down): KS = 1 for the other 1x1
//     stride-1 convolutions, whose operands are plain matrices in memory, KS = 3 / 0 for 3x3 / any other kernel gathered element
//     by element with asynchronous copies: of up to 32 taps, in the weight gradient of up to 16 rows and columns (256 taps);
//   * conv_gemm_kernel<OP, BN> (next) — one CTA per 128 x BN tile for kernels of more than 16 rows or columns: all 256
//     threads gather operand values (two k-blocks in flight in registers), split them and store 16-byte pieces
//     into K-major tiles in the 128-byte swizzle; one thread issues the MMAs of the k-block and commits them to
//     the mbarrier that frees the stage; the epilogue reads the accumulator with tcgen05.ld (lane = tile row)
//     and writes coalesced NCHW rows;
//   * stemconv.cu — fp32-pipe kernels for the 3-channel 3x3 first layer;
//   * pwg::gather_gemm_kernel<OP, BN> (conv_gather.cuh) — strided input gradients, one GEMM per stride residue, summed in registers, and
//     both passes of kernels of more than 32 taps; pwg::phase_fma_kernel for the residues that are better off in fp32.
// Every wait is bounded.
#include "common.cuh"
#include "axis_phases.h"
#include "conv_split.h"
#include "stemconv.h"
#include "umma.cuh"

#include <algorithm>
#include <cmath>
#include <new>
#include <type_traits>
#include <vector>

namespace cunn {
namespace mm {

enum Op : int { OP_FWD = 0, OP_DGRAD = 1, OP_WGRAD = 2 };

constexpr int BM = 128;       // tile rows (TMEM lanes)
constexpr int BK = 32;        // k-block: 8 chunks of 4 values (16 bytes)
constexpr int THREADS = 256;
constexpr int SBO = 1024;     // bytes between 8-row groups of a K-major tile (rows of 128 bytes = one k-block)

struct GemmParams {
    const float *a_src;   // FWD: x; DGRAD: gy; WGRAD: gy
    const float *b_src;   // FWD: W; DGRAD: W; WGRAD: x
    const float *bias;    // FWD only, may be null
    float *out;           // FWD: y; DGRAD: gx; WGRAD: partial sums [splits][M_total][N_total]
    int *status;
    const int *gate;      // null, or see gated_off
    // geometry of the gathered image operand (FWD: x; DGRAD: gy; WGRAD: x)
    int g_C, g_H, g_W;            // channels, rows, cols of that tensor
    int g_padH, g_padW, g_dH, g_dW;
    int kH, kW;
    int pix_W, pix_HW;            // row length and plane size of the pixel grid the gather is driven by
    // convolution sizes
    int C, K;                     // input / output channels
    int n_img;
    // GEMM sizes
    int M_total, N_total, Kd;
    int kblocks;                  // k-blocks per CTA
    int out_HW;                   // FWD / DGRAD: pixels per image of the output tensor
    // WGRAD
    int imgs_per_split, pix_blocks;  // images per split, k-blocks per image
};

// Shared-memory matrix descriptor: K-major tile in the 128-byte swizzle (row r holds its eight 16-byte chunks
// at positions chunk ^ (r & 7); groups of 8 rows are 1024 bytes apart).  The tensor core reads this form without
// bank conflicts; the unswizzled 8 x 16-byte core-matrix form measured about 20 % slower.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr)
{
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)(SBO >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor of kind::tf32: fp32 accumulator, tf32 A and B, both K-major, M = 128, N = BN.
__host__ __device__ constexpr uint32_t instr_desc(int n)
{
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

// hi = v rounded to tf32 (low 13 mantissa bits zero), lo = v - hi (exact in fp32).
__device__ __forceinline__ void split_tf32(float v, float &hi, float &lo)
{
    uint32_t h;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(v));
    hi = __uint_as_float(h);
    lo = v - hi;
}

// Byte offset of the 16-byte piece (row, chunk) inside an operand tile.
__device__ __forceinline__ uint32_t piece_offset(int row, int kc) { return (uint32_t)(row * 128 + ((kc ^ (row & 7)) << 4)); }

__device__ __forceinline__ void store_split(unsigned char *hi_tile, unsigned char *lo_tile, int row, int kc, const float4 &v)
{
    float4 h, l;
    split_tf32(v.x, h.x, l.x);
    split_tf32(v.y, h.y, l.y);
    split_tf32(v.z, h.z, l.z);
    split_tf32(v.w, h.w, l.w);
    const uint32_t off = piece_offset(row, kc);
    *reinterpret_cast<float4 *>(hi_tile + off) = h;
    *reinterpret_cast<float4 *>(lo_tile + off) = l;
}

// k index -> (channel, kh, kw).
__device__ __forceinline__ void split_k(const GemmParams &p, int k, int &c, int &kh, int &kw)
{
    const int kk = p.kH * p.kW;
    c = k / kk;
    const int r = k - c * kk;
    kh = r / p.kW;
    kw = r - kh * p.kW;
}

// Row of the gathered image operand: which image, and the top-left corner of its window.
struct PixRow {
    const float *img;   // channel 0 of this pixel's image in the gathered tensor (null: row outside the problem)
    int ih0, iw0;
};

// Four consecutive k values of the gathered operand for one pixel row (zero outside the image / problem).
__device__ __forceinline__ float4 gather_pix_chunk(const GemmParams &p, const PixRow &r, int k0)
{
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int k = k0 + j;
        float x = 0.f;
        if (r.img && k < p.Kd) {
            int c, kh, kw;
            split_k(p, k, c, kh, kw);
            const int ih = r.ih0 + kh, iw = r.iw0 + kw;
            if ((unsigned)ih < (unsigned)p.g_H && (unsigned)iw < (unsigned)p.g_W)
                x = __ldg(r.img + ((size_t)c * p.g_H + ih) * p.g_W + iw);
        }
        v[j] = x;
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}

// Four consecutive values of a row-major [rows][len] matrix row (zero past the end).
__device__ __forceinline__ float4 rowmajor_chunk(const float *row, int k0, int len, bool vec_ok)
{
    if (!row || k0 >= len) return make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec_ok && k0 + 3 < len) return __ldg(reinterpret_cast<const float4 *>(row + k0));
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = (k0 + j < len) ? __ldg(row + k0 + j) : 0.f;
    return make_float4(v[0], v[1], v[2], v[3]);
}

template <int OP, int BN>
__global__ void __launch_bounds__(THREADS, 1)
conv_gemm_kernel(const GemmParams p)
{
    if (gated_off(p.gate)) return;
    constexpr int A_TILE = BM * BK * 4;             // bytes of one hi (or lo) A tile
    constexpr int B_TILE = BN * BK * 4;
    constexpr int STAGE = 2 * (A_TILE + B_TILE);
    constexpr int STAGES = (STAGE * 4 <= 200 * 1024) ? 4 : (STAGE * 3 <= 200 * 1024 ? 3 : 2);
    constexpr int A_PER = BM * 8 / THREADS;         // 16-byte pieces per thread per k-block
    constexpr int B_PER = (BN * 8 + THREADS - 1) / THREADS;
    // The tensor core adds each MMA result into its fp32 accumulator with truncation, so a long chain of
    // accumulations drifts (error grows with the number of steps).  K-blocks are therefore dealt
    // round-robin to NACC independent TMEM accumulators, which the epilogue adds up in fp32: chains are
    // NACC times shorter and their partial sums smaller.
    constexpr int ACC_COLS = BN < 32 ? 32 : BN;
    constexpr int NACC = (512 / ACC_COLS) > 8 ? 8 : (512 / ACC_COLS);
    constexpr uint32_t TMEM_COLS = ACC_COLS * NACC;

    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t bars[STAGES + 1];           // stage-free barriers + accumulator-ready barrier
    __shared__ uint32_t tmem_base_s;
    __shared__ int pixtab[2][BK][2];                // WGRAD: (ih0, iw0) of the 32 pixels of a k-block, double buffered

    const int tid = threadIdx.x, warp = tid >> 5;
    const int m0 = blockIdx.x * BM;                 // first tile row
    const int n0 = blockIdx.y * BN;                 // first tile column
    const int split = blockIdx.z;                   // WGRAD: image range

    if (tid == 0) {
        for (int s = 0; s <= STAGES; ++s) mbar_init(smem_u32(bars + s), 1);
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(smem_u32(&tmem_base_s), TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;

    // ---- per-thread operand rows ------------------------------------------------------------------
    // A pieces: row = tid % 128, chunks kc = tid / 128 + 2 i.  B pieces: piece q = i * 256 + tid -> row q % BN, chunk q / BN.
    const int a_row = tid & (BM - 1);
    const int a_kc0 = tid >> 7;
    PixRow a_pix{nullptr, 0, 0};
    const float *a_rowptr = nullptr;                // WGRAD: gy row of this k_out (per image offset added later)
    if (OP != OP_WGRAD) {
        const int m = m0 + a_row;
        if (m < p.M_total) {
            const int img = m / p.pix_HW, pix = m - img * p.pix_HW;
            const int ph = pix / p.pix_W, pw = pix - ph * p.pix_W;
            a_pix.img = p.a_src + (size_t)img * p.g_C * p.g_H * p.g_W;
            a_pix.ih0 = ph * p.g_dH - p.g_padH;
            a_pix.iw0 = pw * p.g_dW - p.g_padW;
        }
    } else {
        const int m = m0 + a_row;
        if (m < p.M_total) a_rowptr = p.a_src + (size_t)m * p.pix_HW;   // + img * K * oHW
    }
    const bool b_vec = OP == OP_FWD && (p.Kd & 3) == 0 && ((uintptr_t)p.b_src & 15) == 0;
    const bool a_vec = OP == OP_WGRAD && (p.pix_HW & 3) == 0 && ((uintptr_t)p.a_src & 15) == 0;

    // Loads the pieces of k-block `kb` (CTA-local index) into registers.
    auto load_block = [&](int kb, float4 (&ra)[A_PER], float4 (&rb)[B_PER]) {
        if (OP != OP_WGRAD) {
            const int kbase = kb * BK;
#pragma unroll
            for (int i = 0; i < A_PER; ++i) ra[i] = gather_pix_chunk(p, a_pix, kbase + (a_kc0 + 2 * i) * 4);
#pragma unroll
            for (int i = 0; i < B_PER; ++i) {
                const int q = i * THREADS + tid;
                const int row = q % BN, kc = q / BN;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (kc < 8 && n0 + row < p.N_total) {
                    const int k0 = kbase + kc * 4;
                    if (OP == OP_FWD) {
                        v = rowmajor_chunk(p.b_src + (size_t)(n0 + row) * p.Kd, k0, p.Kd, b_vec);
                    } else {
                        // DGRAD: B[c][(ko,kh,kw)] = W[ko][c][kH-1-kh][kW-1-kw]
                        float t[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int k = k0 + j;
                            float x = 0.f;
                            if (k < p.Kd) {
                                int ko, kh, kw;
                                split_k(p, k, ko, kh, kw);
                                x = __ldg(p.b_src + (((size_t)ko * p.C + (n0 + row)) * p.kH + (p.kH - 1 - kh)) * p.kW + (p.kW - 1 - kw));
                            }
                            t[j] = x;
                        }
                        v = make_float4(t[0], t[1], t[2], t[3]);
                    }
                }
                rb[i] = v;
            }
        } else {
            // k runs over (image, pixel); a k-block never straddles images
            const int img = split * p.imgs_per_split + kb / p.pix_blocks;
            const int pb = kb - (kb / p.pix_blocks) * p.pix_blocks;
            const bool img_ok = img < p.n_img && kb / p.pix_blocks < p.imgs_per_split;
#pragma unroll
            for (int i = 0; i < A_PER; ++i) {
                const int k0 = pb * BK + (a_kc0 + 2 * i) * 4;
                ra[i] = rowmajor_chunk((img_ok && a_rowptr) ? a_rowptr + (size_t)img * p.K * p.pix_HW : nullptr, k0, p.pix_HW, a_vec);
            }
#pragma unroll
            for (int i = 0; i < B_PER; ++i) {
                const int q = i * THREADS + tid;
                const int row = q % BN, kc = q / BN;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                const int n = n0 + row;
                if (kc < 8 && n < p.N_total && img_ok) {
                    int c, kh, kw;
                    split_k(p, n, c, kh, kw);
                    const float *plane = p.b_src + ((size_t)img * p.C + c) * p.g_H * p.g_W;
                    const int k0 = pb * BK + kc * 4;
                    float t[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int pix = k0 + j;
                        float x = 0.f;
                        if (pix < p.pix_HW) {
                            const int ih = pixtab[kb & 1][kc * 4 + j][0] + kh, iw = pixtab[kb & 1][kc * 4 + j][1] + kw;
                            if ((unsigned)ih < (unsigned)p.g_H && (unsigned)iw < (unsigned)p.g_W) x = __ldg(plane + (size_t)ih * p.g_W + iw);
                        }
                        t[j] = x;
                    }
                    v = make_float4(t[0], t[1], t[2], t[3]);
                }
                rb[i] = v;
            }
        }
    };
    // WGRAD: window corners of the 32 pixels of k-block kb (same for every image)
    auto fill_pixtab = [&](int kb) {
        if (OP == OP_WGRAD && tid < BK) {
            const int pb = kb % p.pix_blocks;
            const int pix = pb * BK + tid;
            const int oh = pix / p.pix_W, ow = pix - oh * p.pix_W;
            pixtab[kb & 1][tid][0] = oh * p.g_dH - p.g_padH;
            pixtab[kb & 1][tid][1] = ow * p.g_dW - p.g_padW;
        }
    };
    auto store_block = [&](int stage, const float4 (&ra)[A_PER], const float4 (&rb)[B_PER]) {
        unsigned char *sa_hi = smem + (size_t)stage * STAGE;
        unsigned char *sa_lo = sa_hi + A_TILE;
        unsigned char *sb_hi = sa_lo + A_TILE;
        unsigned char *sb_lo = sb_hi + B_TILE;
#pragma unroll
        for (int i = 0; i < A_PER; ++i) store_split(sa_hi, sa_lo, a_row, a_kc0 + 2 * i, ra[i]);
#pragma unroll
        for (int i = 0; i < B_PER; ++i) {
            const int q = i * THREADS + tid;
            const int row = q % BN, kc = q / BN;
            if (kc < 8) store_split(sb_hi, sb_lo, row, kc, rb[i]);
        }
    };
    auto issue_mmas = [&](int stage, int kb) {
        const uint32_t d_tmem = tmem_base + (uint32_t)((kb % NACC) * ACC_COLS);
        const bool first = kb < NACC;   // first k-block of this accumulator overwrites it
        const uint32_t sa_hi = smem_u32(smem + (size_t)stage * STAGE);
        const uint32_t sa_lo = sa_hi + A_TILE, sb_hi = sa_lo + A_TILE, sb_lo = sb_hi + B_TILE;
        constexpr uint32_t idesc = instr_desc(BN < 16 ? 16 : BN);
#pragma unroll
        for (int j = 0; j < BK / 8; ++j) {
            const uint32_t koff = (uint32_t)j * 32;           // two 16-byte chunks per MMA; the swizzle is applied to the address
            const uint64_t ah = smem_desc(sa_hi + koff), al = smem_desc(sa_lo + koff);
            const uint64_t bh = smem_desc(sb_hi + koff), bl = smem_desc(sb_lo + koff);
            umma_tf32(d_tmem, al, bh, idesc, (first && j == 0) ? 0u : 1u);
            umma_tf32(d_tmem, ah, bl, idesc, 1u);
            umma_tf32(d_tmem, ah, bh, idesc, 1u);
        }
    };

    // ---- main loop: two k-blocks in flight in registers, STAGES in shared memory -------------------
    const int KB = p.kblocks;
    float4 ra0[A_PER], rb0[B_PER], ra1[A_PER], rb1[B_PER];
    bool ok = true;
    fill_pixtab(0);
    if (OP == OP_WGRAD) __syncthreads();
    if (KB > 0) load_block(0, ra0, rb0);
    fill_pixtab(1);
    if (OP == OP_WGRAD) __syncthreads();
    if (KB > 1) load_block(1, ra1, rb1);
    for (int kb = 0; kb < KB && ok; kb += 2) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int k = kb + half;
            if (k >= KB) break;
            const int stage = k % STAGES;
            if (k >= STAGES) {
                // the MMAs that read this stage (k-block k - STAGES) must have finished
                if (!mbar_wait(smem_u32(bars + stage), (uint32_t)(((k / STAGES) - 1) & 1), p.status)) { ok = false; break; }
            }
            if (half == 0) store_block(stage, ra0, rb0);
            else store_block(stage, ra1, rb1);
            fence_async_smem();          // generic-proxy stores -> visible to the tensor core's async proxy
            fill_pixtab(k + 2);          // (k + 2) & 1 == k & 1: this block's table is no longer needed after the sync below
            __syncthreads();
            if (tid == 0) {
                tc_fence_after();
                issue_mmas(stage, k);
                umma_commit(smem_u32(bars + stage));
            }
            if (k + 2 < KB) {
                if (half == 0) load_block(k + 2, ra0, rb0);
                else load_block(k + 2, ra1, rb1);
            }
        }
    }
    // ---- epilogue ----------------------------------------------------------------------------------
    if (tid == 0) umma_commit(smem_u32(bars + STAGES));      // arrives when every MMA above has completed
    if (ok && KB > 0) ok = mbar_wait(smem_u32(bars + STAGES), 0u, p.status);
    tc_fence_after();
    if (ok) {
        const int quarter = warp & 3;                // TMEM lanes this warp may read
        const int row = quarter * 32 + (tid & 31);   // tile row == TMEM lane
        const int m = m0 + row;
        constexpr int HALF = (BN >= 64) ? BN / 2 : BN;
        const int col_begin = (BN >= 64) ? (warp >> 2) * HALF : 0;
        const bool do_cols = (BN >= 64) || (warp < 4);
        size_t out_base = 0;
        if (OP != OP_WGRAD && m < p.M_total) {
            const int img = m / p.out_HW, pix = m - img * p.out_HW;
            out_base = (size_t)img * p.N_total * p.out_HW + pix;
        }
        if (do_cols) {
            for (int cc = col_begin; cc < col_begin + HALF; cc += 32) {
                float acc[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) acc[j] = 0.f;
                const int nacc = KB < NACC ? KB : NACC;   // accumulators that received at least one k-block
                for (int a = 0; a < nacc; ++a) {
                    uint32_t r[32];
                    tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(a * ACC_COLS + cc), r);
#pragma unroll
                    for (int j = 0; j < 32; ++j) acc[j] += __uint_as_float(r[j]);
                }
                if (m < p.M_total) {
                    if (OP != OP_WGRAD) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const int n = n0 + cc + j;
                            if (cc + j < BN && n < p.N_total) {
                                float v = acc[j];
                                if (OP == OP_FWD && p.bias) v += __ldg(p.bias + n);
                                p.out[out_base + (size_t)n * p.out_HW] = v;
                            }
                        }
                    } else {
                        float *dst = p.out + ((size_t)split * p.M_total + m) * p.N_total + n0 + cc;
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (cc + j < BN && n0 + cc + j < p.N_total) dst[j] = acc[j];
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, TMEM_COLS);
}

// The end of a parameter gradient that may have been done already (conv_split.h): adds those sums where the gate says so.
__device__ __forceinline__ bool add_sums(const int *gate, const float *sums, float *gw, long long n, float scale)
{
    if (!gated_off(gate)) return false;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) gw[i] = fmaf(scale, sums[i], gw[i]);
    return true;
}

// gW[i] += scale * sum_s partial[s][i], in split order.
__global__ void __launch_bounds__(256)
wgrad_reduce_kernel(const float *__restrict__ partial, float *__restrict__ gw, long long n, int splits, float scale, const int *gate,
                    const float *__restrict__ sums)
{
    if (add_sums(gate, sums, gw, n, scale)) return;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float s = 0.f;
        for (int k = 0; k < splits; ++k) s += __ldg(partial + (size_t)k * n + i);
        gw[i] += scale * s;
    }
}

// Bias gradient: gb[k] += scale * sum over images and pixels of gy[img][k][pix].  One CTA per (k, chunk).
__global__ void __launch_bounds__(256)
bias_partial_kernel(const float *__restrict__ gy, float *__restrict__ part, int n_img, int K, int HW, int chunks)
{
    __shared__ float sh[8];
    const int k = blockIdx.x / chunks, j = blockIdx.x % chunks;
    const int per = n_img / chunks, extra = n_img % chunks;
    const int i0 = j * per + min(j, extra), i1 = i0 + per + (j < extra ? 1 : 0);
    float s = 0.f;
    for (int img = i0; img < i1; ++img) {
        const float *g = gy + ((size_t)img * K + k) * HW;
        for (int i = threadIdx.x; i < HW; i += blockDim.x) s += __ldg(g + i);
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w];
        part[blockIdx.x] = t;
    }
}
__global__ void __launch_bounds__(128)
bias_finish_kernel(const float *__restrict__ part, float *__restrict__ gb, int K, int chunks, float scale)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    double s = 0.0;
    for (int j = 0; j < chunks; ++j) s += (double)part[k * chunks + j];
    gb[k] = (float)((double)gb[k] + (double)scale * s);
}

// Both reductions of a weight-gradient pass in one launch: gW[i] += scale * sum_s partial[s][i] for i < n, and
// gb[k] += scale * sum_j bias_part[k][j] for the K threads after them (bias_part may be null).
__global__ void __launch_bounds__(256)
wgrad_bias_reduce_kernel(const float *__restrict__ partial, float *__restrict__ gw, long long n, int splits, float scale,
                         const float *__restrict__ bias_part, float *__restrict__ gb, int K, const int *gate, const float *__restrict__ sums)
{
    if (add_sums(gate, sums, gw, n, scale)) return;
    const long long total = n + (bias_part ? K : 0);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        if (i < n) {
            float s = 0.f;
            for (int k = 0; k < splits; ++k) s += __ldg(partial + (size_t)k * n + i);
            gw[i] += scale * s;
        } else {
            const int k = (int)(i - n);
            double s = 0.0;
            for (int j = 0; j < splits; ++j) s += (double)bias_part[(size_t)k * splits + j];
            gb[k] = (float)((double)gb[k] + (double)scale * s);
        }
    }
}

// The same for many splits: eight threads share an output, each adds every eighth split, and their sums are added in order.
__global__ void __launch_bounds__(256)
wgrad_bias_reduce_wide_kernel(const float *__restrict__ partial, float *__restrict__ gw, long long n, int splits, float scale,
                              const float *__restrict__ bias_part, float *__restrict__ gb, int K, const int *gate, const float *__restrict__ sums)
{
    if (add_sums(gate, sums, gw, n, scale)) return;
    __shared__ float part_s[8][32];
    __shared__ double bias_s[8][32];
    const long long total = n + (bias_part ? K : 0);
    const int lane = threadIdx.x & 31, group = threadIdx.x >> 5;
    for (long long base = blockIdx.x * 32LL; base < total; base += gridDim.x * 32LL) {
        const long long i = base + lane;
        float s = 0.f;
        double b = 0.0;
        if (i < n) {
#pragma unroll 4
            for (int k = group; k < splits; k += 8) s += __ldg(partial + (size_t)k * n + i);
        } else if (i < total) {
            for (int k = group; k < splits; k += 8) b += (double)__ldg(bias_part + (size_t)(i - n) * splits + k);
        }
        part_s[group][lane] = s;
        bias_s[group][lane] = b;
        __syncthreads();
        if (group == 0 && i < total) {
            if (i < n) {
                float t = 0.f;
#pragma unroll
                for (int g = 0; g < 8; ++g) t += part_s[g][lane];
                gw[i] += scale * t;
            } else {
                double t = 0.0;
#pragma unroll
                for (int g = 0; g < 8; ++g) t += bias_s[g][lane];
                gb[i - n] = (float)((double)gb[i - n] + (double)scale * t);
            }
        }
        __syncthreads();
    }
}

// y[img][q][pix] += bias[q]: the bias of a transposed convolution, whose product comes out of the input-gradient kernels.
__global__ void __launch_bounds__(256)
add_plane_bias_kernel(float *__restrict__ y, const float *__restrict__ bias, int Q, int HW, long long total, const int *gate)
{
    if (gated_off(gate)) return;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x)
        y[i] += __ldg(bias + (int)((i / HW) % Q));
}

// ---------------------------------------------------------------------------
// Pointwise convolutions (1x1, stride 1, no padding): persistent kernel
// ---------------------------------------------------------------------------
//
// A 1x1 convolution is a plain matrix product per image and every operand is already laid out the way the
// tensor core can take it, so nothing is gathered element by element:
//
//   forward      D[pixel, ko] = sum_c  x[img][c][pix]   * W[ko][c]      A: 4 pixels of one channel = 16 contiguous bytes (M-major)
//                                                                        B: 4 channels of one filter = 16 contiguous bytes (K-major)
//   input grad   D[pixel, c]  = sum_ko gy[img][ko][pix] * W[ko][c]      A: M-major as above;  B: 4 channels c of one ko (N-major)
//   weight grad  D[ko, c]     = sum_{img,pix} gy[img][ko][pix] * x[img][c][pix]      A, B: 4 pixels of one row (K-major);
//                                                                        k runs over the (image, pixel)s of this tile's split
//
// tcgen05.mma takes M/N-major operands through the major bits of the instruction descriptor, so a 16-byte
// asynchronous copy lands an operand piece in shared memory in its final place, no transposition.  One CTA per SM
// walks a strided list of tiles; operand copies run three k-blocks ahead of the MMAs ACROSS tile boundaries, and
// four epilogue warps drain finished accumulators to global memory while the next tile is being produced (when the
// accumulators fit twice in TMEM the MMAs of the next tile run under it as well).
namespace pw {

constexpr int PRODUCERS = 512;           // threads that copy, split and run the epilogue (16 warps)
constexpr int EPILOGUE_WARPS = 4;         // warps that only drain accumulators: TMEM -> registers -> global memory
constexpr int THREADS = PRODUCERS + 32 + 32 * EPILOGUE_WARPS;   // + one warp that only issues the MMAs
constexpr int TILE = 128 * 128;          // 128 rows x 32 k values (16 KiB) in either layout
constexpr int MN_ATOM = 512;             // M/N-major tile: bytes of one swizzle atom (32 rows x 4 k values)
constexpr int MN_KATOM = 4 * MN_ATOM;    // ... bytes from one group of 4 k values to the next (4 atoms cover 128 rows)
constexpr int RAW_STAGES = 4;            // raw fp32 tiles (A, B) filled by asynchronous copies; split in place they become the hi tiles
constexpr int LO_BUFS = 2;               // lo tiles (A, B) of the k-blocks whose MMAs are in flight
constexpr int PREFETCH = 3;              // k-blocks the copies run ahead of the MMAs
constexpr int STAGE_COLS = 64;           // output columns staged at a time for the bulk-store epilogue (x 128 rows x 4 bytes)
constexpr size_t OUT_STAGE = (size_t)STAGE_COLS * BM * 4;
constexpr size_t SMEM = (size_t)(RAW_STAGES + LO_BUFS) * 2 * TILE + OUT_STAGE + 1024;
static_assert(8 * MN_KATOM == TILE, "both layouts fill the tile");

struct Params {
    const float *a, *b, *bias;
    float *out;        // FWD: y; DGRAD: gx; WGRAD: partial sums [splits][M_total][N_total]
    float *bias_part;  // WGRAD: [M_total][splits] row sums of gy, or null
    int *status;
    const int *gate;   // null, or see gated_off
    int HW;            // pixels per image plane
    int M_total, N_total, Kd;
    int n_tiles, tiles_per_split, total_tiles;   // tile = (split * m_tiles + m_tile) * n_tiles + n_tile
    int kblocks;       // k-blocks per tile
    int n_img, splits;         // WGRAD: split s sums the k-blocks [s, s + 1) * kblocks of all images
    int vec_a, vec_b;  // 16-byte global loads allowed for A / B
    // kernels larger than 1x1 (KS != 1): the unfolded operand is gathered from a [g_C, g_H, g_W] image tensor, the
    // pixel grid that drives the gather is pix_W wide (HW = its size)
    int g_C, g_H, g_W, kH, kW, dH, dW, padH, padW, pix_W;
    int dilH, dilW;    // distance between kernel taps (SpatialDilatedConvolution; 1 for SpatialConvolutionMM)
    int nacc, sets;    // accumulators per tile (nacc - 1 for the hi*hi products, k-blocks round-robin, + 1 for the cross terms), accumulator sets in TMEM (1 or 2)
    int bulk_out;      // FWD/DGRAD: planes of >= 1024 pixels (a multiple of 4), 16-byte aligned output: the columns of a tile leave as bulk stores
    int gpi;           // tensor-map kernels: groups of 32 pixels per image, ceil(HW / 32)
};

// 3xTF32 split of a raw fp32 tile in place.  The tensor core reads only the upper 19 bits of a tf32 operand,
// so the raw value itself serves as hi = v with the low 13 mantissa bits dropped; lo = v - hi is exact in fp32
// and is the only tile that has to be written.
__device__ __forceinline__ float lo_part(float v) { return v - __uint_as_float(__float_as_uint(v) & 0xffffe000u); }
__device__ __forceinline__ void store_lo_at(unsigned char *lo_tile, uint32_t off, const float4 &v)
{
    *reinterpret_cast<float4 *>(lo_tile + off) = make_float4(lo_part(v.x), lo_part(v.y), lo_part(v.z), lo_part(v.w));
}
// 3xTF32 split of a 16-byte piece in place, with rounding: hi = v to 11 bits, lo = v - hi to 11 bits.  Truncating instead (the raw
// value as hi, as store_lo_at does it) saves a store, but lo then has the sign of v, and lo * lo and the bits that lo loses add up
// to -4e-7 of the sum whatever its length; rounded parts lose 2^-24 with either sign.
// The rounding is an addition to the bits, so it stops short of the values whose bits it would carry over: finite ones within 2^-12 of the
// largest (they would become infinite), infinities and NaN (0x7fffffff, the NaN that the GPU's own arithmetic makes, would become zero).
// A piece that may hold one is truncated; lo of an infinity or a NaN is inf - inf or NaN then, and every sum that reads one is NaN.
// (cvt.rna.tf32 for both parts, or a branch instead of the select, made a 7x7 layer's forward pass 5 and 6 % slower.)
__device__ __forceinline__ void split_rounded(unsigned char *hi_tile, unsigned char *lo_tile, uint32_t off, float4 v)
{
    const uint32_t half = (fabsf(v.x) + fabsf(v.y)) + (fabsf(v.z) + fabsf(v.w)) < 0x1.ffep127f ? 0x1000u : 0u;
    float4 l;
    auto part = [&](float &x, float &lo) {
        const float h = __uint_as_float((__float_as_uint(x) + half) & 0xffffe000u);
        lo = __uint_as_float(__float_as_uint(x - h) + half);             // the tensor core drops the low 13 bits
        x = h;
    };
    part(v.x, l.x); part(v.y, l.y); part(v.z, l.z); part(v.w, l.w);
    *reinterpret_cast<float4 *>(hi_tile + off) = v;
    *reinterpret_cast<float4 *>(lo_tile + off) = l;
}
__device__ __forceinline__ uint64_t desc_of(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
// M/N-major operand in the 128B-base-32B swizzle: leading offset = atom to atom along M/N, stride offset = along K.
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr)
{
    return desc_of(addr, MN_ATOM, MN_KATOM) | (1ull << 61);
}
__host__ __device__ constexpr uint32_t idesc_of(int n, bool a_mn, bool b_mn)
{
    return (1u << 4) | (2u << 7) | (2u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}
__device__ __forceinline__ float4 ldg4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }

// Asynchronous 16- and 4-byte copies global -> shared; `on` false writes zeros without reading `src`.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool on)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src, bool on)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(on ? 4u : 0u) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// 1-D bulk copy shared -> global through the TMA unit (16-byte aligned addresses, size a multiple of 16 bytes).
__device__ __forceinline__ void bulk_s2g_nocommit(void *dst, uint32_t src_smem, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src_smem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// Barrier among the producer warps only (hardware barrier 2).
__device__ __forceinline__ void producers_sync() { asm volatile("bar.sync 2, %0;" ::"n"(PRODUCERS) : "memory"); }
// Barrier among the epilogue warps only (hardware barrier 1; barrier 0 is __syncthreads).
__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * EPILOGUE_WARPS) : "memory"); }

// Where the operand loads of one thread stand: tile, k-block and the thread's element offsets inside that tile.
// M/N-major pieces: lane = group of 4 rows, k = warp + 16 i.  K-major pieces: chunk kc = tid & 7, rows (tid >> 3) + 64 i.
// KS = 1: pointwise.  KS = 3 / 0: 3x3 / any kernel of up to 32 taps (weight gradient: 256), any stride and padding: the same tiles, but
// the unfolded operand is gathered with 4-byte copies (zero-filled outside the image).
template <int OP, int BN, int KS>
struct Loader {
    int tile, kb;
    int a_off[4];       // FWD/DGRAD: element offsets of the thread's 4 pixels (channel 0); WGRAD: [0..1] row offsets
    int b_off[2];       // FWD: offsets of the thread's two filter rows (+ chunk); DGRAD: [0] first column; WGRAD: row offsets
    unsigned a_mask, b_mask;
    int img, pix;            // WGRAD: image and pixel of the thread's chunk in the current k-block; images >= n_img read as zeros
    unsigned tapmask[4];     // KS != 1, FWD/DGRAD: bit t set when tap t of pixel j lies inside the image
    int img2, pix2;          // KS != 1, WGRAD: image and pixel of this lane's column (k = lane) of the unfolded operand

    __device__ __forceinline__ int taps(const Params &p) const { return KS == 3 ? 9 : p.kH * p.kW; }
    __device__ __forceinline__ int kcols(const Params &p) const { return KS == 3 ? 3 : p.kW; }

    // rowtab (KS != 1, WGRAD): shared table of the tile's 128 unfolded rows: x = offset of the row's tap inside an image
    // (-1: row outside the problem), y = tap row offset | tap column offset << 16 (dilation applied)
    __device__ __forceinline__ void setup(const Params &p, int t, int2 *rowtab)
    {
        const int tid = threadIdx.x, lane = tid & 31;
        tile = t;
        kb = 0;
        a_mask = b_mask = 0;
        if (OP != OP_WGRAD) {
            const int m_tile = t / p.n_tiles, n_tile = t - m_tile * p.n_tiles;
            const int m = m_tile * BM + lane * 4, n0 = n_tile * BN;
            if (KS != 1) {
                // gathered operand: this lane's four rows are lane, lane + 32, lane + 64, lane + 96, so that one copy
                // instruction of the warp covers 32 consecutive pixels (and 128 consecutive bytes of shared memory)
                const int kk = taps(p), kw_n = kcols(p);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    a_off[j] = 0;
                    tapmask[j] = 0;
                    const int mj = m_tile * BM + lane + 32 * j;
                    if (mj < p.M_total) {
                        const int im = mj / p.HW, r = mj - im * p.HW;
                        const int ph = r / p.pix_W, pw_ = r - ph * p.pix_W;
                        const int ih0 = ph * p.dH - p.padH, iw0 = pw_ * p.dW - p.padW;
                        a_off[j] = im * p.g_C * p.g_H * p.g_W + ih0 * p.g_W + iw0;
                        a_mask |= 1u << j;
                        for (int t2 = 0; t2 < kk; ++t2) {
                            const int kh = t2 / kw_n, kw = t2 - kh * kw_n;
                            if ((unsigned)(ih0 + kh * p.dilH) < (unsigned)p.g_H && (unsigned)(iw0 + kw * p.dilW) < (unsigned)p.g_W) tapmask[j] |= 1u << t2;
                        }
                    }
                }
            } else if (p.vec_a) {
                if (m < p.M_total) {
                    const int im = m / p.HW;
                    a_off[0] = im * p.Kd * p.HW + (m - im * p.HW);
                    a_mask = 15u;
                }
            } else {
                // pixels lane + 32 j, as for gathered operands: one copy instruction covers 32 consecutive pixels (four consecutive ones
                // per lane spread it over 512 bytes, with four-way bank conflicts)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    a_off[j] = 0;
                    const int mj = m_tile * BM + lane + 32 * j;
                    if (mj < p.M_total) {
                        const int im = mj / p.HW;
                        a_off[j] = im * p.Kd * p.HW + (mj - im * p.HW);
                        a_mask |= 1u << j;
                    }
                }
            }
            if (OP == OP_FWD) {
                const int kc = tid & 7;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int row = (tid >> 3) + 64 * i, n = n0 + row;
                    b_off[i] = n * p.Kd + kc * 4;
                    if (row < BN && n < p.N_total) b_mask |= 1u << i;
                }
            } else {
                if (KS != 1) {
                    b_off[0] = n0 + lane;                  // gathered: columns lane + 32 j
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (lane + 32 * j < BN && n0 + lane + 32 * j < p.N_total) b_mask |= 1u << j;
                } else {
                    const int col = n0 + lane * 4;
                    b_off[0] = col;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (lane * 4 < BN && col + j < p.N_total) b_mask |= 1u << j;
                }
            }
        } else {
            const int split = t / p.tiles_per_split, r = t - split * p.tiles_per_split;
            const int m_tile = r / p.n_tiles, n_tile = r - m_tile * p.n_tiles;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int row = (tid >> 3) + 64 * i;
                const int m = m_tile * BM + row, n = n_tile * BN + row;
                a_off[i] = m * p.HW;
                b_off[i] = n * p.HW;
                if (m < p.M_total) a_mask |= 1u << i;
                if (row < BN && n < p.N_total) b_mask |= 1u << i;
            }
            const int p0 = split * p.kblocks * BK;               // the split's first pixel in the flat (image, pixel) sequence
            img = p0 / p.HW;
            pix = p0 - img * p.HW;
            if (KS != 1) {
                // every producer has issued the copies of the previous tile before the table changes
                producers_sync();
                if (tid < BM) {
                    const int n = n_tile * BN + tid;
                    int2 e = make_int2(-1, 0);
                    if (tid < BN && n < p.N_total) {
                        // unfolded row n = (channel, kh, kw)
                        const int kk = taps(p), kw_n = kcols(p);
                        const int c = n / kk, t2 = n - c * kk, kh = t2 / kw_n, kw = t2 - kh * kw_n;
                        e.x = (c * p.g_H + kh * p.dilH) * p.g_W + kw * p.dilW;
                        e.y = (kh * p.dilH) | ((kw * p.dilW) << 16);
                    }
                    rowtab[tid] = e;
                }
                producers_sync();
                img2 = img;
                pix2 = pix + lane;
                while (pix2 >= p.HW) { pix2 -= p.HW; ++img2; }
            }
            pix += (tid & 7) * 4;
            while (pix >= p.HW) { pix -= p.HW; ++img; }
        }
    }

    // Moves to the next k-block of this CTA's tile list.
    __device__ __forceinline__ void advance(const Params &p, int2 *rowtab)
    {
        if (++kb == p.kblocks) {
            const int t = tile + (int)gridDim.x;
            if (t < p.total_tiles) setup(p, t, rowtab);
            else tile = t;
        } else if (OP == OP_WGRAD) {
            pix += BK;
            while (pix >= p.HW) { pix -= p.HW; ++img; }
            if (KS != 1) {
                pix2 += BK;
                while (pix2 >= p.HW) { pix2 -= p.HW; ++img2; }
            }
        }
    }

    // Copies four consecutive pixels of one row, starting at this thread's (image, pixel), to shared memory.
    __device__ __forceinline__ void row_chunk(const Params &p, uint32_t dst, const float *base, int stride, bool vec, bool on) const
    {
        if (vec) {
            const bool ok = on && img < p.n_img;
            cp_async16(dst, ok ? base + (size_t)img * stride + pix : base, ok);
            return;
        }
        int ij = img, pj = pix;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            while (pj >= p.HW) { pj -= p.HW; ++ij; }
            const bool ok = on && ij < p.n_img;
            cp_async4(dst + 4 * j, ok ? base + (size_t)ij * stride + pj : base, ok);
            ++pj;
        }
    }

    // Issues the asynchronous copies of this thread's pieces of the current k-block into the raw tiles at
    // shared-memory addresses sa / sb (+ the piece offsets); masked pieces are zero-filled.
    __device__ __forceinline__ void issue(const Params &p, uint32_t sa, uint32_t sb, const uint32_t (&a_so)[2],
                                          const uint32_t (&b_so)[2], const bool (&b_store)[2], const uint32_t (&g_so)[2],
                                          const int2 *rowtab) const
    {
        const int tid = threadIdx.x, warp = tid >> 5;
        if (tile >= p.total_tiles) return;
        if (OP != OP_WGRAD) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int k = kb * BK + warp + 16 * i;
                const bool kok = k < p.Kd;
                if (KS != 1) {
                    const int kk = taps(p), kw_n = kcols(p);
                    const int c = k / kk, t2 = k - c * kk, kh = t2 / kw_n, kw = t2 - kh * kw_n;
                    const int koff = (c * p.g_H + kh * p.dilH) * p.g_W + kw * p.dilW;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const bool ok = kok && (tapmask[j] >> t2 & 1u);
                        cp_async4(sa + g_so[i] + MN_ATOM * j, ok ? p.a + (a_off[j] + koff) : p.a, ok);
                    }
                } else if (p.vec_a) {
                    const bool ok = kok && a_mask;
                    cp_async16(sa + a_so[i], ok ? p.a + a_off[0] + k * p.HW : p.a, ok);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const bool ok = kok && (a_mask >> j & 1u);
                        cp_async4(sa + g_so[i] + MN_ATOM * j, ok ? p.a + a_off[j] + k * p.HW : p.a, ok);
                    }
                }
            }
            if (OP == OP_FWD) {
                const int k0 = kb * BK + (tid & 7) * 4;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (!b_store[i]) continue;
                    const float *src = p.b + b_off[i] + kb * BK;
                    const bool rok = (b_mask >> i & 1u) != 0;
                    if (p.vec_b) {
                        const bool ok = rok && k0 < p.Kd;
                        cp_async16(sb + b_so[i], ok ? src : p.b, ok);
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const bool ok = rok && k0 + j < p.Kd;
                            cp_async4(sb + b_so[i] + 4 * j, ok ? src + j : p.b, ok);
                        }
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int k = kb * BK + warp + 16 * i;
                    const bool kok = k < p.Kd;
                    if (KS != 1) {
                        // B[c][(ko, kh, kw)] = W[ko][c][kH-1-kh][kW-1-kw]: the tap index runs backwards
                        const int kk = taps(p);
                        const int ko = k / kk, t2 = k - ko * kk;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const bool ok = kok && (b_mask >> j & 1u);
                            cp_async4(sb + g_so[i] + MN_ATOM * j, ok ? p.b + ((size_t)(ko * p.N_total + b_off[0] + 32 * j) * kk + (kk - 1 - t2)) : p.b, ok);
                        }
                        continue;
                    }
                    if (!b_store[i]) continue;
                    const float *src = p.b + (size_t)(kok ? k : 0) * p.N_total + b_off[0];
                    if (p.vec_b) {
                        const bool ok = kok && b_mask;
                        cp_async16(sb + b_so[i], ok ? src : p.b, ok);
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const bool ok = kok && (b_mask >> j & 1u);
                            cp_async4(sb + b_so[i] + 4 * j, ok ? src + j : p.b, ok);
                        }
                    }
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                row_chunk(p, sa + a_so[i], p.a + a_off[i], p.M_total * p.HW, p.vec_a != 0, (a_mask >> i & 1u) != 0);
                if (KS == 1 && b_store[i]) row_chunk(p, sb + b_so[i], p.b + b_off[i], p.N_total * p.HW, p.vec_b != 0, (b_mask >> i & 1u) != 0);
            }
            if (KS != 1) {
                // unfolded operand: this lane owns column k = lane (one output pixel) of rows warp, warp + 16, ...:
                // x[img][c][oh * dH - padH + kh * dilH][ow * dW - padW + kw * dilW]; one copy instruction of the warp
                // fills the 128 bytes of one tile row
                const int lane = tid & 31;
                const int oh = pix2 / p.pix_W, ow = pix2 - oh * p.pix_W;
                const int ih = oh * p.dH - p.padH, iw = ow * p.dW - p.padW;
                const bool pix_ok = img2 < p.n_img;
                const float *img_base = p.b + (size_t)(pix_ok ? img2 : 0) * p.g_C * p.g_H * p.g_W + (ih * p.g_W + iw);
                const uint32_t dst0 = sb + (uint32_t)(warp * 128 + (((lane >> 2) ^ (warp & 7)) << 4) + (lane & 3) * 4);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int row = warp + 16 * q;
                    if (row >= BN) break;
                    const int2 e = rowtab[row];
                    const bool ok = pix_ok && e.x >= 0 && (unsigned)(ih + (e.y & 0xffff)) < (unsigned)p.g_H &&
                                    (unsigned)(iw + (e.y >> 16)) < (unsigned)p.g_W;
                    cp_async4(dst0 + (uint32_t)q * 2048u, ok ? img_base + e.x : p.b, ok);
                }
            }
        }
    }
};

// ROUND (weight gradients): split_rounded instead of the truncating split, bias sums in fp64; see rounds_wgrad.
template <int OP, int BN, int KS, bool ROUND = false>
__global__ void __launch_bounds__(THREADS, 1)
pw_gemm_kernel(const Params p)
{
    if (gated_off(p.gate)) return;
    using BiasSum = typename std::conditional<ROUND, double, float>::type;
    constexpr bool A_MN = OP != OP_WGRAD;     // A is M-major (forward, input gradient)
    constexpr bool B_MN = OP == OP_DGRAD;     // B is N-major (input gradient)
    constexpr int ACC_COLS = BN < 32 ? 32 : BN;
    constexpr uint32_t TMEM_COLS = 512;
    constexpr uint32_t idesc = idesc_of(BN, A_MN, B_MN);

    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t bars[RAW_STAGES + 2]; // MMAs-of-this-stage-done barriers, then one accumulators-ready barrier per set
    __shared__ uint64_t full[RAW_STAGES];     // stage split and visible to the tensor core: one arrival per producer warp
    __shared__ uint64_t accfree[2];           // accumulator set drained: one arrival per epilogue warp
    __shared__ uint32_t tmem_base_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < RAW_STAGES + 2; ++s) mbar_init(smem_u32(bars + s), 1);
        for (int s = 0; s < RAW_STAGES; ++s) mbar_init(smem_u32(full + s), PRODUCERS / 32);
        for (int s = 0; s < 2; ++s) mbar_init(smem_u32(accfree + s), EPILOGUE_WARPS);
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(smem_u32(&tmem_base_s), TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;

    const int KB = p.kblocks;
    const int my_tiles = ((int)blockIdx.x < p.total_tiles) ? (p.total_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int total_it = my_tiles * KB;
    const int nhi_used = KB < p.nacc - 1 ? KB : p.nacc - 1;   // hi accumulators that received a k-block; the lo one always did
    const uint32_t set_cols = (uint32_t)(p.nacc * ACC_COLS);

    // shared-memory offsets of this thread's pieces (same for every stage)
    uint32_t a_so[2], b_so[2], g_so[2];
    bool b_store[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int k = warp + 16 * i;                    // M/N-major: k inside the block
        const int row = (tid >> 3) + 64 * i;            // K-major: tile row
        // 128-byte rows of 32 consecutive M/N values, four k rows per 512-byte atom, the 32-byte chunk index
        // XORed with the row index (the tensor core's 128B-base-32B swizzle, the only M/N-major form for tf32)
        const uint32_t mn = (uint32_t)((lane >> 3) * MN_ATOM + (k >> 2) * MN_KATOM + (k & 3) * 128 +
                                       ((((lane & 7) >> 1) ^ (k & 3)) << 5) + ((lane & 1) << 4));
        const uint32_t km = piece_offset(row, tid & 7);   // K-major: 128-byte swizzle
        a_so[i] = A_MN ? mn : km;
        b_so[i] = B_MN ? mn : km;
        b_store[i] = B_MN ? (lane * 4 < BN) : (row < BN);
        if (OP == OP_WGRAD && KS != 1) {
            // gathered K-major operand: warp w copies rows w, w + 16, ... element by element, so it also splits them:
            // this lane takes chunks (lane & 3) * 2 + i of row w + 16 * (lane >> 2)
            const int grow = warp + 16 * (lane >> 2);
            b_so[i] = piece_offset(grow, (lane & 3) * 2 + i);
            b_store[i] = grow < BN;
        }
        // gathered M/N-major operand (KS != 1): this lane copies element (row = lane + 32 j, k), 4 bytes each; j adds
        // one 512-byte atom.  The 32 lanes of one copy instruction fill one 128-byte row of an atom.
        g_so[i] = (uint32_t)((k >> 2) * MN_KATOM + (k & 3) * 128 + (((lane >> 3) ^ (k & 3)) << 5) + (((lane >> 2) & 1) << 4) + (lane & 3) * 4);
    }

    BiasSum bsum[2] = {0, 0};                           // WGRAD: running row sums of gy (bias gradient)
    unsigned char *const lo_base = smem + (size_t)RAW_STAGES * 2 * TILE;
    // Splits this thread's own pieces of raw stage `rs` (its copies have landed): the raw tile is the hi tile,
    // lo goes to the same offset of lo buffer `lb`.
    auto split_block = [&](int rs, int lb) {
        unsigned char *a_hi = smem + (size_t)rs * 2 * TILE, *b_hi = a_hi + TILE;
        unsigned char *a_lo = lo_base + (size_t)lb * 2 * TILE, *b_lo = a_lo + TILE;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float4 va = *reinterpret_cast<const float4 *>(a_hi + a_so[i]);
            if (ROUND) split_rounded(a_hi, a_lo, a_so[i], va);
            else store_lo_at(a_lo, a_so[i], va);
            if (OP == OP_WGRAD) bsum[i] += ((BiasSum)va.x + (BiasSum)va.y) + ((BiasSum)va.z + (BiasSum)va.w);
            if (b_store[i]) {
                const float4 vb = *reinterpret_cast<const float4 *>(b_hi + b_so[i]);
                if (ROUND) split_rounded(b_hi, b_lo, b_so[i], vb);
                else store_lo_at(b_lo, b_so[i], vb);
            }
        }
    };
    // hi*hi products go to accumulator d_hi, the two small cross terms to d_lo: the tensor core truncates when it
    // accumulates, and the error of a chain scales with the magnitude it carries, so the large terms get the short
    // chains (k-blocks round-robin over nacc - 1 accumulators) and all cross terms share one.
    // Epilogue warps: reads the accumulators of tile `t` (the `count`-th tile of this CTA), writes the warp's 32
    // rows of the output and hands the accumulator set back to the MMA warp.
    auto epilogue = [&](int t, int count) -> bool {
        const int set = (p.sets == 2) ? (count & 1) : 0;
        const uint32_t parity = (uint32_t)(((p.sets == 2) ? (count >> 1) : count) & 1);
        if (!mbar_wait(smem_u32(bars + RAW_STAGES + set), parity, p.status)) return false;
        tc_fence_after();
        const int quarter = warp & 3;                            // the TMEM lanes this warp may read
        const int row = quarter * 32 + lane;
        int m, n_tile0;
        size_t dst_off = 0;
        if (OP != OP_WGRAD) {
            const int m_tile = t / p.n_tiles, n_tile = t - m_tile * p.n_tiles;
            m = m_tile * BM + row;
            n_tile0 = n_tile * BN;
            if (m < p.M_total) {
                const int im = m / p.HW;
                dst_off = (size_t)im * p.N_total * p.HW + (m - im * p.HW) + (size_t)n_tile0 * p.HW;
            }
        } else {
            const int split = t / p.tiles_per_split, r2 = t - split * p.tiles_per_split;
            const int m_tile = r2 / p.n_tiles, n_tile = r2 - m_tile * p.n_tiles;
            m = m_tile * BM + row;
            n_tile0 = n_tile * BN;
            dst_off = ((size_t)split * p.M_total + m) * p.N_total + n_tile0;
        }
        if (OP != OP_WGRAD) {
            // Whole tile inside the problem and planes long enough: stage 64 columns x 128 pixels in shared memory
            // ([column][pixel], so a column is 512 contiguous bytes of one output plane) and let the TMA unit write
            // each column as one bulk store (two when the tile crosses into the next image).
            const int m_tile0 = (t / p.n_tiles) * BM;
            if (p.bulk_out && m_tile0 + BM <= p.M_total) {
                float *stage = reinterpret_cast<float *>(smem + (size_t)(RAW_STAGES + LO_BUFS) * 2 * TILE);
                const int e = tid - (PRODUCERS + 32);            // 0 .. 127
                const int im0 = m_tile0 / p.HW, pix0 = m_tile0 - im0 * p.HW;
                const int len0 = min(BM, p.HW - pix0);
#pragma unroll 1
                for (int cbase = 0; cbase < BN; cbase += STAGE_COLS) {
                    bulk_wait_read_all();                        // this thread's earlier bulk stores have left the buffer
                    epilogue_sync();
#pragma unroll 1
                    for (int c0 = cbase; c0 < cbase + STAGE_COLS && c0 < BN; c0 += 16) {
                        float acc[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[j] = (OP == OP_FWD && p.bias && n_tile0 + c0 + j < p.N_total) ? __ldg(p.bias + n_tile0 + c0 + j) : 0.f;
                        for (int a2 = 0; a2 <= nhi_used; ++a2) {
                            const int a = a2 < nhi_used ? a2 : p.nacc - 1;
                            uint32_t r[16];
                            tmem_ld16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)set * set_cols + (uint32_t)(a * ACC_COLS + c0), r);
#pragma unroll
                            for (int j = 0; j < 16; ++j) acc[j] += __uint_as_float(r[j]);
                        }
#pragma unroll
                        for (int j = 0; j < 16; ++j) stage[(c0 - cbase + j) * BM + row] = acc[j];
                    }
                    fence_async_smem();                          // staged values -> visible to the bulk copy engine
                    epilogue_sync();
                    const int col = cbase + e, n = n_tile0 + col;
                    if (e < STAGE_COLS && col < BN && n < p.N_total) {
                        const uint32_t src = smem_u32(stage + e * BM);
                        float *dst = p.out + ((size_t)im0 * p.N_total + n) * p.HW + pix0;
                        bulk_s2g_nocommit(dst, src, (uint32_t)len0 * 4u);
                        if (len0 < BM) bulk_s2g_nocommit(p.out + ((size_t)(im0 + 1) * p.N_total + n) * p.HW, src + (uint32_t)len0 * 4u, (uint32_t)(BM - len0) * 4u);
                        bulk_commit();
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(accfree + set));
                return true;
            }
        }
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 16) {                    // 16 columns at a time keeps the register count down
            float acc[16];
#pragma unroll
            for (int j = 0; j < 16; ++j)                         // the bias loads are in flight while TMEM is read
                acc[j] = (OP == OP_FWD && p.bias && n_tile0 + c0 + j < p.N_total) ? __ldg(p.bias + n_tile0 + c0 + j) : 0.f;
            for (int a2 = 0; a2 <= nhi_used; ++a2) {
                const int a = a2 < nhi_used ? a2 : p.nacc - 1;
                uint32_t r[16];
                tmem_ld16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)set * set_cols + (uint32_t)(a * ACC_COLS + c0), r);
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[j] += __uint_as_float(r[j]);
            }
            if (m < p.M_total) {
                const int n0 = n_tile0 + c0;
                if (OP != OP_WGRAD) {
                    float *dst = p.out + dst_off + (size_t)c0 * p.HW;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (n0 + j < p.N_total) dst[(size_t)j * p.HW] = acc[j];
                    }
                } else {
                    float *dst = p.out + dst_off + c0;
                    if ((p.N_total & 3) == 0) {
#pragma unroll
                        for (int j = 0; j < 16; j += 4)
                            if (n0 + j < p.N_total) *reinterpret_cast<float4 *>(dst + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (n0 + j < p.N_total) dst[j] = acc[j];
                    }
                }
            }
        }
        tc_fence_before();                                       // the TMEM reads above are ordered before the arrival
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(accfree + set));
        return true;
    };

    bool ok = true;
    if (warp == PRODUCERS / 32) {
        // ---- MMA warp: waits for a split stage, issues its twelve MMAs, commits them to the stage's barrier.  The tensor
        // pipe takes one of these MMAs every 64 clocks only if the issuing thread keeps up: every instruction between two
        // tcgen05.mma of this one thread is time the pipe idles.  So one lane runs the whole loop, descriptors are a
        // constant upper word + a lower word that advances by additions, ring positions and barrier parities are carried
        // incrementally, and the steady state uses the form without a predicate. ----
        if (lane == 0) {
            constexpr uint32_t A_LOW = A_MN ? ((uint32_t)(MN_ATOM >> 4) << 16) : (1u << 16);
            constexpr uint32_t B_LOW = B_MN ? ((uint32_t)(MN_ATOM >> 4) << 16) : (1u << 16);
            constexpr uint32_t A_HIGH = (A_MN ? (uint32_t)(MN_KATOM >> 4) : (uint32_t)(SBO >> 4)) | (1u << 14) | ((A_MN ? 1u : 2u) << 29);
            constexpr uint32_t B_HIGH = (B_MN ? (uint32_t)(MN_KATOM >> 4) : (uint32_t)(SBO >> 4)) | (1u << 14) | ((B_MN ? 1u : 2u) << 29);
            constexpr uint32_t A_STEP = A_MN ? (uint32_t)(2 * MN_KATOM >> 4) : 2u;     // 8 k values further, in 16-byte units
            constexpr uint32_t B_STEP = B_MN ? (uint32_t)(2 * MN_KATOM >> 4) : 2u;
            constexpr uint32_t STAGE_STEP = (uint32_t)(2 * TILE >> 4);
            const uint32_t raw0 = (smem_u32(smem) >> 4) & 0x3fffu, lo0 = (smem_u32(lo_base) >> 4) & 0x3fffu;
            auto desc = [](uint32_t low, uint32_t high) { return ((uint64_t)high << 32) | low; };
            const int nhi = p.nacc - 1;
            int rs = 0, lb = 0, kb = 0, set = 0, hi_slot = 0;
            uint32_t full_parity = 0, free_parity = 0;             // accfree is first awaited on the second use of a set (its phase 0)
            bool first_round = true;
            uint32_t acc0 = tmem_base;
            for (int i = 0; i < total_it; ++i) {
                if (!mbar_wait(smem_u32(full + rs), full_parity, p.status)) break;
                if (kb == 0 && !first_round) {
                    // the epilogue warps must have drained the tile that used this accumulator set before
                    if (!mbar_wait(smem_u32(accfree + set), free_parity, p.status)) break;
                }
                tc_fence_after();
                const uint32_t d_hi = acc0 + (uint32_t)(hi_slot * ACC_COLS), d_lo = acc0 + (uint32_t)(nhi * ACC_COLS);
                const uint32_t ah = (raw0 + (uint32_t)rs * STAGE_STEP) | A_LOW, bh = (raw0 + (uint32_t)rs * STAGE_STEP + (uint32_t)(TILE >> 4)) | B_LOW;
                const uint32_t al = (lo0 + (uint32_t)lb * STAGE_STEP) | A_LOW, bl = (lo0 + (uint32_t)lb * STAGE_STEP + (uint32_t)(TILE >> 4)) | B_LOW;
                if (kb < nhi || kb == 0) {
                    // first k-blocks of a tile: the first MMA into an accumulator overwrites it
                    const uint32_t keep_lo = kb == 0 ? 0u : 1u, keep_hi = kb < nhi ? 0u : 1u;
#pragma unroll
                    for (int j = 0; j < BK / 8; ++j) {
                        umma_tf32(d_lo, desc(al + j * A_STEP, A_HIGH), desc(bh + j * B_STEP, B_HIGH), idesc, j == 0 ? keep_lo : 1u);
                        umma_tf32(d_lo, desc(ah + j * A_STEP, A_HIGH), desc(bl + j * B_STEP, B_HIGH), idesc, 1u);
                        umma_tf32(d_hi, desc(ah + j * A_STEP, A_HIGH), desc(bh + j * B_STEP, B_HIGH), idesc, j == 0 ? keep_hi : 1u);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < BK / 8; ++j) {
                        umma_tf32_acc(d_lo, desc(al + j * A_STEP, A_HIGH), desc(bh + j * B_STEP, B_HIGH), idesc);
                        umma_tf32_acc(d_lo, desc(ah + j * A_STEP, A_HIGH), desc(bl + j * B_STEP, B_HIGH), idesc);
                        umma_tf32_acc(d_hi, desc(ah + j * A_STEP, A_HIGH), desc(bh + j * B_STEP, B_HIGH), idesc);
                    }
                }
                umma_commit(smem_u32(bars + rs));
                if (++rs == RAW_STAGES) { rs = 0; full_parity ^= 1u; }
                if (++lb == LO_BUFS) lb = 0;
                if (++hi_slot == nhi) hi_slot = 0;
                if (++kb == KB) {
                    umma_commit(smem_u32(bars + RAW_STAGES + set));
                    kb = 0;
                    hi_slot = 0;
                    acc0 += set_cols;
                    if (++set == p.sets) { set = 0; acc0 = tmem_base; if (!first_round) free_parity ^= 1u; first_round = false; }
                }
            }
        }
    } else if (warp > PRODUCERS / 32) {
        // ---- epilogue warps: one pass over this CTA's tiles ----
        for (int count = 0; count < my_tiles; ++count) {
            if (!epilogue((int)blockIdx.x + count * (int)gridDim.x, count)) { ok = false; break; }
        }
        bulk_wait_read_all();                                    // shared memory must outlive the last bulk stores' reads
    } else {
        Loader<OP, BN, KS> L;
        L.tile = (int)blockIdx.x;
        L.kb = 0;
        int2 *rowtab = reinterpret_cast<int2 *>(smem + (size_t)(RAW_STAGES + LO_BUFS) * 2 * TILE);   // in the output staging area, which the weight gradient does not use
        if (my_tiles > 0) L.setup(p, L.tile, rowtab);
        const uint32_t smem_a0 = smem_u32(smem);
        // copies of the first PREFETCH k-blocks; one commit group per k-block, empty ones included, so that
        // "all but the newest PREFETCH - 1 groups" always means "k-block i has landed"
    #pragma unroll
        for (int i = 0; i < PREFETCH; ++i) {
            if (i < total_it) {
                L.issue(p, smem_a0 + (uint32_t)(i * 2 * TILE), smem_a0 + (uint32_t)(i * 2 * TILE + TILE), a_so, b_so, b_store, g_so, rowtab);
                L.advance(p, rowtab);
            }
            cp_async_commit();
        }

        int c_tile = (int)blockIdx.x, c_kb = 0;                // tile and k-block of the block being split
        for (int i = 0; i < total_it; ++i) {
            const int rs = i % RAW_STAGES, lb = i % LO_BUFS;
            cp_async_wait<PREFETCH - 1>();                     // this thread's pieces of k-block i are in shared memory
            if (i >= LO_BUFS) {
                // the MMAs of k-block i - 2 read this lo buffer
                const int j = i - LO_BUFS;
                if (!mbar_wait(smem_u32(bars + j % RAW_STAGES), (uint32_t)((j / RAW_STAGES) & 1), p.status)) { ok = false; break; }
            }
            if (KS != 1 || (A_MN && !p.vec_a)) __syncwarp();   // pieces copied element by element were filled by several lanes of this warp
            split_block(rs, lb);
            fence_async_smem();                                // generic-proxy stores -> visible to the tensor core's async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(full + rs));
            // refill the raw stage that k-block i - 1 used with k-block i + PREFETCH, once its MMAs have read it
            if (i + PREFETCH < total_it) {
                if (i >= 1) {
                    const int j = i - 1;
                    if (!mbar_wait(smem_u32(bars + j % RAW_STAGES), (uint32_t)((j / RAW_STAGES) & 1), p.status)) { ok = false; break; }
                }
                const int ns = (i + PREFETCH) % RAW_STAGES;
                L.issue(p, smem_a0 + (uint32_t)(ns * 2 * TILE), smem_a0 + (uint32_t)(ns * 2 * TILE + TILE), a_so, b_so, b_store, g_so, rowtab);
                L.advance(p, rowtab);
            }
            cp_async_commit();
            if (c_kb == KB - 1) {
                if (OP == OP_WGRAD) {
                    // bias gradient: the eight chunk lanes of a row hold its partial sums
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        BiasSum sum = bsum[r];
                        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
                        const int split = c_tile / p.tiles_per_split, r2 = c_tile - split * p.tiles_per_split;
                        const int m_tile = r2 / p.n_tiles, n_tile = r2 - m_tile * p.n_tiles;
                        const int m = m_tile * BM + (tid >> 3) + 64 * r;
                        if (p.bias_part && n_tile == 0 && (tid & 7) == 0 && m < p.M_total) p.bias_part[(size_t)m * p.splits + split] = (float)sum;
                        bsum[r] = 0;
                    }
                }
                c_kb = 0;
                c_tile += (int)gridDim.x;
            } else {
                ++c_kb;
            }
        }
        cp_async_wait<0>();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, TMEM_COLS);
}

}  // namespace pw

#include "pw_tma.cuh"
#include "conv_gather.cuh"

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

typedef void (*GemmKernel)(const GemmParams);

template <int OP>
static GemmKernel pick_kernel(int bn)
{
    switch (bn) {
        case 32: return conv_gemm_kernel<OP, 32>;
        case 64: return conv_gemm_kernel<OP, 64>;
        default: return conv_gemm_kernel<OP, 128>;
    }
}

static size_t smem_bytes(int bn)
{
    const size_t stage = 2 * ((size_t)BM * BK * 4 + (size_t)bn * BK * 4);
    const int stages = (stage * 4 <= 200 * 1024) ? 4 : (stage * 3 <= 200 * 1024 ? 3 : 2);
    return stage * stages + 1024;   // + alignment slack
}

static int pick_bn_for(int n_total) { return n_total <= 32 ? 32 : (n_total <= 64 ? 64 : 128); }

// With a gate (see gated_off) the launch does not wait for the kernel before.
static cudaError_t launch_gated(const void *kern, dim3 grid, dim3 threads, void **args, size_t smem, cudaStream_t stream, const int *gate)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gate ? 1 : 0;
    return cudaLaunchKernelExC(&cfg, kern, args);
}
static int launch(GemmKernel kern, const GemmParams &p, dim3 grid, int bn, cudaStream_t stream)
{
    const size_t smem = smem_bytes(bn);
    CUNN_CUDA(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    void *args[] = {(void *)&p};
    CUNN_CUDA(launch_gated((const void *)kern, grid, dim3(THREADS), args, smem, stream, p.gate));
    return 0;
}

static int check(int N, int C, int H, int W, int K, int kH, int kW, int dH, int dW, int padH, int padW, int *oH, int *oW,
                 int dilH = 1, int dilW = 1)
{
    CUNN_CHECK_ARG(kW > 0 && kH > 0, "kernel size should be greater than zero, but got kH: %d kW: %d", kH, kW);
    CUNN_CHECK_ARG(dW > 0 && dH > 0, "stride should be greater than zero, but got dH: %d dW: %d", dH, dW);
    CUNN_CHECK_ARG(dilW > 0 && dilH > 0, "dilation should be greater than zero, but got dilationH: %d, dilationW: %d", dilH, dilW);
    CUNN_CHECK_ARG(N >= 0 && C > 0 && K > 0 && H > 0 && W > 0 && padH >= 0 && padW >= 0, "bad convolution sizes");
    const int spanH = dilH * (kH - 1) + 1, spanW = dilW * (kW - 1) + 1;   // extent of the dilated kernel
    CUNN_CHECK_ARG(spanH < (1 << 15) && spanW < (1 << 15), "dilated kernel extent too large");
    *oH = (H + 2 * padH - spanH) / dH + 1;
    *oW = (W + 2 * padW - spanW) / dW + 1;
    CUNN_CHECK_ARG(H + 2 * padH >= spanH && W + 2 * padW >= spanW && *oH >= 1 && *oW >= 1,
                   "Given input size: (%d x %d x %d). Calculated output size: (%d x %d x %d). Output size is too small", C, H,
                   W, K, *oH, *oW);
    CUNN_CHECK_ARG((long long)N * C * (long long)H * W < (1LL << 31) && (long long)N * K * (long long)(*oH) * (*oW) < (1LL << 31) &&
                       (long long)C * kH * kW < (1 << 24),
                   "tensors of 2^31 or more elements are not supported");
    return 0;
}

static void wgrad_plan(int N, int C, int K, int kk, int oHW, int *bn, int *splits, int *imgs_per_split, int *pix_blocks)
{
    *bn = pick_bn_for(C * kk);
    const int tiles = ceil_div(K, BM) * ceil_div(C * kk, *bn);
    int s = std::max(1, std::min(N, (2 * sm_count()) / std::max(1, tiles)));
    *imgs_per_split = ceil_div(N, s);
    *splits = ceil_div(N, *imgs_per_split);
    *pix_blocks = ceil_div(oHW, BK);
}


// ---- pointwise path ----------------------------------------------------------------------------------
static bool pw_applies(int kH, int kW, int dH, int dW, int padH, int padW)
{
    return kH == 1 && kW == 1 && dH == 1 && dW == 1 && padH == 0 && padW == 0;
}
static bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

typedef void (*PwKernel)(const pw::Params);
template <int OP, int KS, bool ROUND = false>
static PwKernel pw_pick_bn(int bn)
{
    switch (bn) {
        case 32: return pw::pw_gemm_kernel<OP, 32, KS, ROUND>;
        case 64: return pw::pw_gemm_kernel<OP, 64, KS, ROUND>;
        default: return pw::pw_gemm_kernel<OP, 128, KS, ROUND>;
    }
}
template <int OP>
static PwKernel pw_pick(int bn, int ks = 1)
{
    if (ks == 1) return pw_pick_bn<OP, 1>(bn);
    if (ks == 3) return pw_pick_bn<OP, 3>(bn);
    return pw_pick_bn<OP, 0>(bn);
}
// With rounding, 3x3 kernels take the loader for any size: they are short reductions.
static PwKernel pw_pick_rounded(int bn, int ks) { return ks == 1 ? pw_pick_bn<OP_WGRAD, 1, true>(bn) : pw_pick_bn<OP_WGRAD, 0, true>(bn); }
// Kernels of up to 32 taps run on the same persistent kernel with a gathering loader.
static bool gather_applies(int kH, int kW) { return kH * kW <= 32; }
// Kernels of up to 16 x 16 taps: any number of taps on the weight gradient's loader and on conv_gather.cuh.
static bool small_kernel(int kH, int kW) { return kH <= pwg::MAX_KERNEL && kW <= pwg::MAX_KERNEL; }
// The weight gradient's gathering loader takes both kinds.
static bool gathered_wgrad(int kH, int kW) { return gather_applies(kH, kW) || small_kernel(kH, kW); }
// loader variant of the gathering path: 3x3 has its own instantiation, everything else (a strided or padded 1x1
// included) the one with run-time kernel sizes
static int gather_ks(int kH, int kW) { return (kH == 3 && kW == 3) ? 3 : 0; }
static void set_geometry(pw::Params &q, int gC, int gH, int gW, int kH, int kW, int dH, int dW, int padH, int padW, int pixW,
                         int dilH, int dilW)
{
    q.g_C = gC; q.g_H = gH; q.g_W = gW; q.kH = kH; q.kW = kW; q.dH = dH; q.dW = dW; q.padH = padH; q.padW = padW; q.pix_W = pixW;
    q.dilH = dilH; q.dilW = dilW;
}
static int pw_bn_for(int n_total) { return n_total <= 32 ? 32 : (n_total <= 64 ? 64 : 128); }
// Column-tile width of a GEMM with `rows` rows: narrower tiles while the wide ones leave half of the SMs without one.  Such a launch
// lasts as long as one tile, and a tile's k-block costs less the narrower it is (one image through 512 -> 512 at 14 x 14: 8 tiles of
// 128 columns 18.9 us, 32 of 32 columns 15.5 us).
static int pw_bn_for(int n_total, long long rows)
{
    int bn = pw_bn_for(n_total);
    while (bn > 32 && ceil_div_ll(rows, BM) * ceil_div(n_total, bn) * 2 <= sm_count()) bn /= 2;
    return bn;
}

// Accumulators per tile and accumulator sets: the hi*hi products of the k-blocks are dealt round-robin to `nacc - 1`
// accumulators to keep the tensor core's truncating accumulation chains short, the cross terms share the last one; two sets (epilogue overlapped with the next tile) when
// they fit in the 512 TMEM columns.
static void pw_accumulators(int bn, int kblocks, int *nacc, int *sets, bool wgrad = false, int tiles = 0)
{
    if (wgrad && tiles <= sm_count()) {
        // a CTA's only tile has nothing to overlap with: all columns for short chains
        *nacc = std::min(8, 512 / std::max(bn, 32));
        *sets = 1;
    } else if (bn == 128 && wgrad) {
        // sums over pixels of random-sign products cancel: the weight gradient is the pass most sensitive to the
        // accumulation chains, and its long k loops make the epilogue a small share anyway
        if (kblocks <= 8) { *nacc = 2; *sets = 2; }
        else { *nacc = 4; *sets = 1; }
    } else if (bn == 128) {
        // two sets let the MMAs of the next tile run while the epilogue warps drain this one; beyond 16 k-blocks the
        // chains (12 MMAs per k-block and accumulator) get long enough to need four accumulators for the 1e-4 bar
        if (kblocks <= 16) { *nacc = 2; *sets = 2; }
        else { *nacc = 4; *sets = 1; }
    } else if (bn == 64) {
        if (kblocks <= 48) { *nacc = 4; *sets = 2; }
        else { *nacc = 8; *sets = 1; }
    } else {
        *nacc = 8; *sets = 2;
    }
}

static int pw_launch(PwKernel kern, pw::Params &p, cudaStream_t stream)
{
    const int grid = std::min(p.total_tiles, sm_count());
    CUNN_CUDA(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pw::SMEM));
    void *args[] = {(void *)&p};
    CUNN_CUDA(launch_gated((const void *)kern, dim3(grid), dim3(pw::THREADS), args, pw::SMEM, stream, p.gate));
    return 0;
}

// ---- tensor-map kernels (pw_tma.cuh) -----------------------------------------------------------------------------
static int g_use_tma = 1;

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// The driver's encoder, looked up through the runtime so that the library does not link libcuda.
static EncodeTiledFn encode_tiled()
{
    static EncodeTiledFn fn = [] {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            ptr = nullptr;
        return (EncodeTiledFn)ptr;
    }();
    return fn;
}
// fp32 tensor [d2][d1][d0] (d0 contiguous; d2 = 0: two dimensions), boxes of box0 x box1 (x 1), zero fill outside.
static int make_map(CUtensorMap *m, const float *base, long long d0, long long d1, long long d2, int box0, int box1, CUtensorMapSwizzle swz)
{
    const cuuint32_t rank = d2 ? 3 : 2;
    cuuint64_t dims[3] = {(cuuint64_t)d0, (cuuint64_t)d1, (cuuint64_t)(d2 ? d2 : 1)};
    cuuint64_t strides[2] = {(cuuint64_t)d0 * 4, (cuuint64_t)d0 * (cuuint64_t)d1 * 4};
    cuuint32_t box[3] = {(cuuint32_t)box0, (cuuint32_t)box1, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = encode_tiled()(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, rank, (void *)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                      swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail("cuTensorMapEncodeTiled failed with code %d", (int)r);
    return 0;
}
static bool tma_applies(const void *a, const void *b, const void *c, int HW, int C)
{
    return g_use_tma && HW % 4 == 0 && C % 4 == 0 && aligned16(a) && aligned16(b) && aligned16(c) && encode_tiled() != nullptr;
}
// Accumulator plan of the tensor-map kernels: tiles of one or two k-blocks put all products into one accumulator and
// use up to four accumulator sets, so that the MMA warp runs several tiles ahead of the epilogue warps; longer tiles, and
// launches with a tile per CTA, follow pw_accumulators, which keeps the small products apart from the large ones.
static void tma_accumulators(int bn, int kblocks, int *nacc, int *sets, bool wgrad, int tiles)
{
    const int cols = std::max(bn, 32);
    if (kblocks <= 2 && tiles > sm_count()) {
        *nacc = 1;
        *sets = std::min((int)pwt::MAX_SETS, 512 / cols);
        return;
    }
    pw_accumulators(bn, kblocks, nacc, sets, wgrad, tiles);
}
typedef void (*PwTmaKernel)(const pw::Params, const CUtensorMap, const CUtensorMap, const CUtensorMap);
// 4 splitter + 8 epilogue warps for every tile length: measured against 8 + 4 and 16 + 4 on tiles of 8, 16 and 32 k-blocks,
// 4 + 8 was never slower (16 + 4 runs at 80 registers and was 4-14 % slower).
template <int OP>
static PwTmaKernel pw_tma_pick(int bn)
{
    switch (bn) {
        case 32: return pwt::pw_tma_kernel<OP, 32, 4, 8, 4, 2>;
        case 64: return pwt::pw_tma_kernel<OP, 64, 4, 8, 4, 2>;
        default: return pwt::pw_tma_kernel<OP, 128, 4, 8, 4, 2>;
    }
}
// CTAs that share a tile of a launch whose tiles (of 32 columns) leave most SMs idle: four, where the reduction is ten k-blocks or longer, two
// where four do not fit, eight for the longest.  A share's start, and adding up through the others' shared memory, cost what four k-blocks do.
// Forward, one CTA / two / four / eight a tile, in us: 512 -> 512 on one 14 x 14 image (32 tiles, 16 k-blocks) 15.9 / 14.5 / 10.4 / -,
// 1024 -> 1024 at 8 x 8 24.7 / 18.6 / 12.9 / 13.1, 512 -> 512 at 8 x 8 15.2 / 14.0 / 10.4 / 14.5, 768 -> 768 at 14 x 14 20.6 / 16.5 / - / -,
// 4096 -> 64 at 4 x 4 (128 k-blocks) 80 / - / - / 17.6; but 256 -> 256 (8 k-blocks) on three 14 x 14 images 10.4 / 12.4 / - / -, 128 -> 128 at
// 28 x 28 8.3 / 10.4 / - / -.  The sums are in the order of the ranks, whatever finishes first; shorter chains: errors 5.2e-7 -> 4.3e-7.
static int pw_cluster(int bn, int tiles, int kblocks)
{
    const int sms = sm_count();
    if (bn != 32 || kblocks < 10) return 1;
    if (kblocks >= 64 && tiles * 8 <= sms) return 8;
    if (tiles * 4 <= sms) return 4;
    return kblocks >= 16 && tiles * 2 <= sms ? 2 : 1;
}
template <int OP>
static int pw_cluster_launch(pw::Params &p, int ranks, CUtensorMap &ma, CUtensorMap &mb, cudaStream_t stream)
{
    const void *kern = (const void *)pwt::pw_tma_kernel<OP, 32, 4, 8, 4, 2, true>;
    CUNN_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pw::SMEM));
    p.kblocks = ceil_div(p.kblocks, ranks);
    void *args[] = {(void *)&p, (void *)&ma, (void *)&mb, (void *)&ma};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.total_tiles * ranks));
    cfg.blockDim = dim3((unsigned)pwt::tma_threads(4, 8));
    cfg.dynamicSmemBytes = pw::SMEM;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CUNN_CUDA(cudaLaunchKernelExC(&cfg, kern, args));
    return 0;
}
// `mo` is the map of the output tensor for the bulk-store epilogue (forward / input gradient); kernels that do not use
// it get a copy of `ma`.
static int pw_tma_launch(PwTmaKernel kern, pw::Params &p, CUtensorMap &ma, CUtensorMap &mb, CUtensorMap &mo, cudaStream_t stream)
{
    const int grid = std::min(p.total_tiles, sm_count());
    const size_t smem_bytes = pw::SMEM;
    const int threads = pwt::tma_threads(4, 8);          // every configuration has 14 warps
    CUNN_CUDA(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes));
    void *args[] = {(void *)&p, (void *)&ma, (void *)&mb, (void *)&mo};
    CUNN_CUDA(launch_gated((const void *)kern, dim3(grid), dim3(threads), args, smem_bytes, stream, p.gate));
    return 0;
}

// k-blocks of a reduction over N images of HW pixels: flat (element copies), or whole groups of 32 per image (tensor maps).
static long long wgrad_kblocks(int N, int HW, bool groups)
{
    return groups ? (long long)N * ceil_div(HW, BK) : ceil_div_ll((long long)N * HW, BK);
}
// Weight gradients whose operands are split with rounding, for 8 to 11 % of their time.  Kernels of more than 32 taps came from a kernel that
// rounds and sums each image apart, with an error that grows with the image: 1.4e-7 to 4.6e-7 for up to 16 x 16 outputs, where truncated
// operands alone are 4.2e-7 off (rounded ones and their chains 1.3e-7 to 2.6e-7), but 1.35e-6 at 28 x 28 against 0.6e-6 to 1.1e-6 with
// truncated ones, and 2.2e-5 against 2.4e-6 at 112 x 112.  Reductions of up to 64 k-blocks are split below the image, where the truncating
// split's error and a chain's add up (fully connected layers 3.8e-7 -> 4.3e-7, 1.2e-7 with rounding); their launches wait for memory, and the
// extra stores cost nothing.
static bool rounds_wgrad(int kk, int N, int HW) { return kk > 32 ? HW < 784 : wgrad_kblocks(N, HW, false) <= 64; }
// k-blocks whose large products meet in one accumulator of a tile: the error of a weight gradient grows with them.
static int wgrad_chain(int bn, long long kb, long long tiles)
{
    int nacc, sets;
    pw_accumulators(bn, (int)kb, &nacc, &sets, true, (int)std::min<long long>(tiles, 1 << 30));
    return (int)ceil_div_ll(kb, nacc - 1);
}
// Splits of the weight gradient's reduction on the persistent kernels: a tile sums `kb_per_split` of the k-blocks of all images.
// Candidates fill one to sixteen waves of the persistent grid (and one to four splits, when one already fills it); they are
// scored by waves x k-blocks per tile — the time of the slowest CTA, plus about six k-blocks for a tile's prologue and its 64 KB of
// partial sums — and by what the reduction reads.  Splits end anywhere in an image: with whole images per split, 48 of 148 SMs had work at
// 12 x 144 x 37 x 29 -> 200 and 64 at 32 x 3 x 224 x 224, 7x7.
// The best split into whole images (tiles longer than 128 k-blocks avoided) bounds the accumulation chains: none is longer than its.  Of 4,000
// layers drawn over 16 to 1024 channels a tenth had longer ones without that bound (37 x 64 x 17 x 17, 4x4: 1.2e-6 off, 7.6e-7 with
// it), which is worth 0.4 % of the scored time.
static void pw_wgrad_plan(int C, int K, int kk, int N, int HW, bool groups, int *bn, int *splits, int *kb_per_split)
{
    C *= kk;
    *bn = pw_bn_for(C);
    const long long tiles_mn = (long long)ceil_div(K, BM) * ceil_div(C, *bn), kb_total = wgrad_kblocks(N, HW, groups);
    const int grid = sm_count();
    auto score = [&](long long kb, long long used) {
        const double cost = (double)ceil_div_ll(tiles_mn * used, grid) * ((double)kb + 6.0);
        return kb > 128 ? cost * (1.0 + 0.25 * (double)(kb - 128) / 128.0) : cost;
    };
    long long whole = kb_total;                                             // k-blocks of a tile of whole images
    const bool bounded = kk <= 32 && !rounds_wgrad(kk, N, HW);
    if (bounded) {
        double best = -1.0;
        for (int images = 1; images <= N; ++images) {
            const long long used = ceil_div(N, images);
            const double cost = score((long long)images * ceil_div(HW, BK), used);
            if (best < 0.0 || cost < best * 0.999) { best = cost; whole = wgrad_kblocks(images, HW, groups); }
            if (tiles_mn * used <= grid) break;                             // one wave: more images a tile only make it longer
        }
    }
    const int chain = wgrad_chain(*bn, whole, 1LL << 30);
    double best = -1.0;
    for (int i = bounded ? 0 : 1; i <= 20; ++i) {
        const long long want = i <= 16 ? (long long)i * grid / tiles_mn : i - 16;
        const long long kb = i ? ceil_div_ll(kb_total, std::max(1LL, std::min(want, kb_total))) : whole, used = ceil_div_ll(kb_total, kb);
        if (i && bounded && wgrad_chain(*bn, kb, tiles_mn * used) > chain) continue;
        const double cost = score(kb, used) + (double)used * K * C * 4.0 / 8e6;                   // a k-block lasts as long as 8 MB of L2 reads
        if (best < 0.0 || cost < best * 0.999) { best = cost; *splits = (int)used; *kb_per_split = (int)kb; }
    }
}
// Workspace for the partial sums of the splits and their bias sums.
static size_t wgrad_partial_bytes(int C, int K, int kk, int N, int HW, bool groups)
{
    int bn, splits, kb;
    pw_wgrad_plan(C, K, kk, N, HW, groups, &bn, &splits, &kb);
    return (size_t)splits * K * C * kk * sizeof(float) + (size_t)K * splits * sizeof(float) + 256;
}

// ---- gathered operand, register accumulation (conv_gather.cuh) -------------------------------------------------------
typedef void (*GatherKernel)(const pwg::GatherParams);
template <int OP>
static GatherKernel gather_pick(int bn)
{
    switch (bn) {
        case 32: return pwg::gather_gemm_kernel<OP, 32>;
        case 64: return pwg::gather_gemm_kernel<OP, 64>;
        default: return pwg::gather_gemm_kernel<OP, 128>;
    }
}
static uint32_t magic_of(int d) { return d == 1 ? 0u : (uint32_t)((1ull << 32) / (unsigned)d + 1u); }
template <int OP>
static int launch_gather(pwg::GatherParams &p, int bn, cudaStream_t stream)
{
    p.n_tiles = ceil_div(p.N_total, bn);
    p.total_tiles = 0;
    for (int i = 0; i < p.n_phases; ++i) {
        pwg::Phase &f = p.ph[i];
        f.tile0 = p.total_tiles;
        f.kblocks = ceil_div(f.Kd, BK);
        f.taps_magic = magic_of(f.taps);
        f.kW_magic = magic_of(f.kW);
        p.total_tiles += ceil_div(f.M_total, BM) * p.n_tiles;
    }
    const GatherKernel kern = gather_pick<OP>(bn);
    CUNN_CUDA(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pwg::GSMEM));
    void *args[] = {(void *)&p};
    CUNN_CUDA(launch_gated((const void *)kern, dim3(std::min(p.total_tiles, sm_count())), dim3(pwg::GTHREADS), args, pwg::GSMEM, stream, p.gate));
    return 0;
}

static int most_taps(const std::vector<AxisPhase> &v)
{
    int most = 0;
    for (const AxisPhase &a : v) most = std::max(most, a.taps);
    return most;
}
// The tensor-core kernel's limits: sixteen rows and columns of taps, and a reduction whose index magic_div divides by the taps.
static bool residue_gemm_takes(int K, int tapsH, int tapsW)
{
    const long long taps = (long long)tapsH * tapsW, Kd = ceil_div_ll(K * taps, BK) * BK;
    return tapsH <= pwg::MAX_KERNEL && tapsW <= pwg::MAX_KERNEL && Kd < (1LL << 31) && Kd * taps < (1LL << 32);
}
static int launch_phase_fma(pwg::FmaParams &q, const std::vector<AxisPhase> &ah, const std::vector<AxisPhase> &aw, cudaStream_t stream)
{
    q.groups = ceil_div(q.C, pwg::CH);
    for (size_t at = 0; at < ah.size(); at += pwg::MAX_AXIS)
        for (size_t bt = 0; bt < aw.size(); bt += pwg::MAX_AXIS) {
            const int nh = (int)std::min<size_t>(pwg::MAX_AXIS, ah.size() - at), nw = (int)std::min<size_t>(pwg::MAX_AXIS, aw.size() - bt);
            long long rows = 0, cols = 0;
            for (int i = 0; i < nh; ++i) { q.rows[i] = ah[at + i]; rows = std::max<long long>(rows, q.rows[i].n); }
            for (int i = 0; i < nw; ++i) { q.cols[i] = aw[bt + i]; cols = std::max<long long>(cols, q.cols[i].n); }
            const long long pixels = q.N * rows * cols;
            const int threads = (int)std::min(256LL, ceil_div_ll(pixels, 32) * 32);
            pwg::phase_fma_kernel<<<dim3((unsigned)(ceil_div_ll(pixels, threads) * q.groups), nh, nw), threads, 0, stream>>>(q);
            CUNN_LAUNCH_CHECK("convmm grad input (fp32 residues)");
        }
    return 0;
}

// Kernels as long as their stride (patch embeddings) have a residue per tap, with few pixels each: sixteen of them are one launch of the
// residue GEMM, which lasts as long as its longest tile however few of its 128 rows are pixels, and ones of three channels fill a
// tenth of the columns.  Estimates in us, from 500 layers of 1 to 64 images: 2.1 per k-block of the longest tile or 2.2 per k-block and SM,
// and 8 for the rest of a launch; the fp32 kernel takes 2.6 products per ps once it is full.  Input gradient of 3 filters of 64 x 64 on
// one 64 x 64 image, fp32 residues / residue GEMM / every tap scanned: 5 / 2640 / 125 us; 45 x 3 x 224 x 224, 358 filters of 16 x 16:
// 0.92 / 2.4 / 40.5 ms; 3 x 61 x 196 x 196, 378 filters of 14 x 14: 0.87 / 0.61 / 43.8 ms.
static bool fp32_residues_are_faster(int N, int C, int K, const std::vector<AxisPhase> &ah, const std::vector<AxisPhase> &aw)
{
    if (ah.size() * aw.size() <= (size_t)pwg::MAX_PHASES) return false;
    double products = 0, tile_kblocks = 0, longest = 0, rows = 0;
    for (const AxisPhase &a : ah)
        for (const AxisPhase &b : aw) {
            const double m = (double)N * a.n * b.n, kd = (double)K * a.taps * b.taps, kb = std::ceil(kd / BK);
            products += m * kd * C;
            tile_kblocks += std::ceil(m / BM) * kb;
            longest = std::max(longest, kb);
            rows += m;
        }
    const double launches = std::ceil((double)(ah.size() * aw.size()) / pwg::MAX_PHASES);
    const int bn = pw_bn_for(C, (long long)(rows / launches));
    const double gemm = launches * (8.0 + std::max(2.1 * longest, tile_kblocks / launches * ceil_div(C, bn) * 2.2 / sm_count()));
    return 4.0 + products / 2.6e6 < gemm;
}

// Input gradient of a convolution with any stride, padding and dilation, plus `bias` per input channel (null: none): the
// forward pass of a transposed convolution has one.
static int phased_grad_input(const float *gy, const float *weight, const float *bias, float *gx, int N, int C, int H, int W, int K,
                             int kH, int kW, int dH, int dW, int padH, int padW, int dilH, int dilW, int oH, int oW, const int *gate,
                             cudaStream_t stream)
{
    bool gaps = false;
    std::vector<AxisPhase> ah = axis_phases(H, kH, dH, padH, dilH, false, &gaps), aw = axis_phases(W, kW, dW, padW, dilW, false, &gaps);
    const int mostH = most_taps(ah), mostW = most_taps(aw);
    // residues whose sums are short are taken in fp32, and all of them where the tensor-core kernel cannot take the longest or is slower
    const bool all_fma = !residue_gemm_takes(K, mostH, mostW) || (long long)K * mostH * mostW < pwg::SHORT_SUM ||
                         fp32_residues_are_faster(N, C, K, ah, aw);
    bool any_fma = all_fma;
    for (const AxisPhase &a : ah)
        for (const AxisPhase &b : aw) any_fma |= (long long)K * a.taps * b.taps < pwg::SHORT_SUM;
    if (gaps && all_fma && std::min(dH, H) <= pwg::MAX_AXIS && std::min(dW, W) <= pwg::MAX_AXIS) {
        // one launch writes every residue
        ah = axis_phases(H, kH, dH, padH, dilH, true, &gaps);
        aw = axis_phases(W, kW, dW, padW, dilW, true, &gaps);
    } else if (gaps) {
        // pixels that no tap reaches: one pass over the tensor however many residues they are
        const long long total = (long long)N * C * H * W;
        const int blocks = (int)std::max(1LL, std::min(ceil_div_ll(total, 256), (long long)sm_count() * 16));
        pwg::plane_fill_kernel<<<blocks, 256, 0, stream>>>(gx, bias, C, H * W, total);
        CUNN_LAUNCH_CHECK("convmm grad input (pixels without taps)");
    }
    if (any_fma) {
        pwg::FmaParams q{};
        q.gy = gy; q.w = weight; q.bias = bias; q.gx = gx; q.gate = gate;
        q.N = N; q.C = C; q.H = H; q.W = W; q.K = K; q.kW = kW; q.kk = kH * kW; q.dH = dH; q.dW = dW; q.oH = oH; q.oW = oW;
        q.only_short = !all_fma;
        const int rc = launch_phase_fma(q, ah, aw, stream);
        if (rc || all_fma) return rc;
    }
    std::vector<pwg::Phase> ph;
    for (const AxisPhase &a : ah)
        for (const AxisPhase &b : aw) {
            if ((long long)K * a.taps * b.taps < pwg::SHORT_SUM) continue;
            pwg::Phase f{};
            f.HW = a.n * b.n; f.pix_W = b.n; f.M_total = N * f.HW;
            f.taps = a.taps * b.taps; f.kW = b.taps; f.Kd = K * f.taps;
            f.dH = f.dW = 1;
            f.padH = -a.o0; f.padW = -b.o0; f.dilH = -a.ostep; f.dilW = -b.ostep;
            f.w_base = a.k0 * kW + b.k0; f.w_sH = a.kstep * kW; f.w_sW = b.kstep;
            f.o_off = a.h0 * W + b.h0; f.o_sH = a.n > 1 ? dH * W : 0; f.o_sW = b.n > 1 ? dW : 0;
            ph.push_back(f);
        }
    // longest reductions first: the persistent grid deals tiles round-robin, so the last wave is made of the short ones
    std::stable_sort(ph.begin(), ph.end(), [](const pwg::Phase &a, const pwg::Phase &b) { return a.taps > b.taps; });
    for (size_t at = 0; at < ph.size(); at += pwg::MAX_PHASES) {
        pwg::GatherParams q{};
        q.a = gy; q.b = weight; q.bias = bias; q.out = gx; q.status = device_status_ptr(); q.gate = gate;
        q.g_C = K; q.g_H = oH; q.g_W = oW; q.N_total = C; q.w_kk = kH * kW; q.o_HW = H * W;
        q.n_phases = (int)std::min<size_t>(pwg::MAX_PHASES, ph.size() - at);
        for (int i = 0; i < q.n_phases; ++i) q.ph[i] = ph[at + i];
        long long rows = 0;
        for (int i = 0; i < q.n_phases; ++i) rows += q.ph[i].M_total;
        if (launch_gather<OP_DGRAD>(q, pw_bn_for(C, rows), stream)) return 1;
    }
    return 0;
}

}  // namespace mm
}  // namespace cunn

using namespace cunn;
using namespace cunn::mm;

// Scratch memory of the kernels in conv_split.cu, or 0 where they do not take the pass.
enum Pass : int { PASS_FORWARD = 0, PASS_GRAD_INPUT = 1, PASS_GRAD_WEIGHT = 2 };
static size_t conv_acc_grad_workspace(int N, int C, int H, int W, int K, int kH, int kW, int dH, int dW, int padH, int padW,
                                      int dilH, int dilW);
static size_t gathered_workspace(const split::Geometry &g)
{
    return conv_acc_grad_workspace(g.N, g.C, g.H, g.W, g.K, g.kH, g.kW, g.dH, g.dW, g.padH, g.padW, g.dilH, g.dilW);
}
static size_t split_scratch(int pass, const split::Geometry &g)
{
    if (!g_use_tma || g.N == 0 || (g.H == 1 && g.W == 1)) return 0;
    // 1x1 layers that read few values stay on the kernels without scratch: the estimates were fitted to larger ones.  Of 60 each that they
    // would take, without scratch / with it: forward 2.14 / 1.60 ms, up to 1.4 times slower; input gradients 1.94 / 1.46 ms, up to 2.4 times; parameter
    // gradients 1.88 / 2.61 ms, all but four slower.
    const long long read = pass == PASS_GRAD_INPUT ? (long long)g.N * g.K * g.oH * g.oW : (long long)g.N * g.C * g.H * g.W;
    if (g.kH * g.kW == 1 && read < CUNN_B200_CONV_POINT_VALUES) return 0;
    return pass == PASS_FORWARD ? split::forward_scratch(g) : pass == PASS_GRAD_INPUT ? split::grad_input_scratch(g)
                                                                                      : split::grad_weight_scratch(g, gathered_workspace);
}
static bool split_applies(int pass, const split::Geometry &g, const void *scratch, size_t scratch_bytes)
{
    const size_t need = scratch && aligned16(scratch) ? split_scratch(pass, g) : 0;
    return need && scratch_bytes >= need;
}

// `gate`: null, or the kernels do nothing where it is 0 (no scratch memory then).
static int conv_forward(const float *x, const float *weight, const float *bias, float *y, int N, int C, int H, int W, int K,
                        int kH, int kW, int dH, int dW, int padH, int padW, int dilH, int dilW, cunn_stream_t stream_,
                        void *scratch = nullptr, size_t scratch_bytes = 0, const int *gate = nullptr)
{
    clear_error();
    cudaStream_t stream = (cudaStream_t)stream_;
    int oH, oW;
    if (check(N, C, H, W, K, kH, kW, dH, dW, padH, padW, &oH, &oW, dilH, dilW)) return 1;
    if (N == 0) return 0;
    CUNN_CHECK_ARG(x && weight && y, "null tensor pointer");
    const bool dilated = dilH != 1 || dilW != 1;
    CUNN_CHECK_ARG(!dilated || gather_applies(kH, kW), "dilated kernels of more than 32 taps are not supported");
    if (!dilated && stem::applies(C, K, kH, kW)) return stem::forward(x, weight, bias, y, N, H, W, oH, oW, dH, dW, padH, padW, stream);
    const split::Geometry geo{N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW, oH, oW};
    if (split_applies(PASS_FORWARD, geo, scratch, scratch_bytes)) {
        auto again = [&](int first, int n, const int *wide) {
            return conv_forward(x + (size_t)first * C * H * W, weight, bias, y + (size_t)first * K * oH * oW, n, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH,
                                dilW, stream_, nullptr, 0, wide);
        };
        return split::forward(geo, x, weight, bias, y, split::fallback_of(again), scratch, stream);
    }
    if (pw_applies(kH, kW, dH, dW, padH, padW) && H * W == 1 && K % 4 == 0 && tma_applies(x, weight, y, C, 4)) {
        // a fully connected layer: y[n][k] = sum_c x[n][c] W[k][c], two K-major matrices, i.e. the weight gradient's GEMM over one
        // "image" of C pixels (with element copies of single-pixel planes, 128 x 1024 -> 1000 took 129 us)
        pw::Params q{};
        q.a = x; q.b = weight; q.bias = bias; q.out = y; q.status = device_status_ptr(); q.gate = gate;
        q.HW = C; q.gpi = ceil_div(C, 32); q.M_total = N; q.N_total = K; q.kblocks = q.gpi;
        const int bn = pw_bn_for(K, N);
        q.n_tiles = ceil_div(K, bn); q.tiles_per_split = q.total_tiles = ceil_div(N, BM) * q.n_tiles;
        q.n_img = 1; q.splits = 1;
        tma_accumulators(bn, q.kblocks, &q.nacc, &q.sets, true, q.total_tiles);
        alignas(64) CUtensorMap ma, mb;
        if (make_map(&ma, x, C, N, 1, 32, BM, CU_TENSOR_MAP_SWIZZLE_128B)) return 1;
        if (make_map(&mb, weight, C, K, 1, 32, bn, CU_TENSOR_MAP_SWIZZLE_128B)) return 1;
        return pw_tma_launch(pw_tma_pick<OP_WGRAD>(bn), q, ma, mb, ma, stream);
    }
    if (pw_applies(kH, kW, dH, dW, padH, padW)) {
        pw::Params q{};
        q.a = x; q.b = weight; q.bias = bias; q.out = y; q.status = device_status_ptr(); q.gate = gate;
        q.HW = H * W; q.M_total = N * H * W; q.N_total = K; q.Kd = C; q.kblocks = ceil_div(C, BK);
        const int bn = pw_bn_for(K, q.M_total);
        q.n_tiles = ceil_div(K, bn); q.tiles_per_split = 0; q.total_tiles = ceil_div(q.M_total, BM) * q.n_tiles;
        q.n_img = N; q.splits = 1;
        if (tma_applies(x, weight, y, q.HW, C)) {
            alignas(64) CUtensorMap ma, mb, mo;
            q.gpi = ceil_div(q.HW, 32); q.M_total = N * q.gpi * 32; q.total_tiles = ceil_div(q.M_total, BM) * q.n_tiles;
            q.bulk_out = (q.HW % 32 == 0) && q.HW >= 8 * BM;
            tma_accumulators(bn, q.kblocks, &q.nacc, &q.sets, false, q.total_tiles);
            if (make_map(&ma, x, q.HW, C, N, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B)) return 1;
            if (make_map(&mb, weight, C, K, 0, 32, bn, CU_TENSOR_MAP_SWIZZLE_128B)) return 1;
            if (const int ranks = pw_cluster(bn, q.total_tiles, q.kblocks); ranks > 1) return pw_cluster_launch<OP_FWD>(q, ranks, ma, mb, stream);
            if (q.bulk_out) { if (make_map(&mo, y, q.HW, K, N, BM, pwt::HALF_STAGE_COLS, CU_TENSOR_MAP_SWIZZLE_NONE)) return 1; }
            else mo = ma;
            return pw_tma_launch(pw_tma_pick<OP_FWD>(bn), q, ma, mb, mo, stream);
        }
        q.vec_a = (q.HW % 4 == 0) && aligned16(x); q.vec_b = (C % 4 == 0) && aligned16(weight);
        q.bulk_out = (q.HW % 4 == 0) && q.HW >= 8 * BM && aligned16(y);
        pw_accumulators(bn, q.kblocks, &q.nacc, &q.sets);
        return pw_launch(pw_pick<OP_FWD>(bn), q, stream);
    }
    if (gather_applies(kH, kW)) {
        pw::Params q{};
        q.a = x; q.b = weight; q.bias = bias; q.out = y; q.status = device_status_ptr(); q.gate = gate;
        q.HW = oH * oW; q.M_total = N * oH * oW; q.N_total = K; q.Kd = C * kH * kW; q.kblocks = ceil_div(q.Kd, BK);
        set_geometry(q, C, H, W, kH, kW, dH, dW, padH, padW, oW, dilH, dilW);
        const int bn = pw_bn_for(K, q.M_total);
        q.n_tiles = ceil_div(K, bn); q.tiles_per_split = 0; q.total_tiles = ceil_div(q.M_total, BM) * q.n_tiles;
        q.n_img = N; q.splits = 1;
        q.vec_a = 0; q.vec_b = (q.Kd % 4 == 0) && aligned16(weight);
        q.bulk_out = (q.HW % 4 == 0) && q.HW >= 8 * BM && aligned16(y);
        pw_accumulators(bn, q.kblocks, &q.nacc, &q.sets);
        return pw_launch(pw_pick<OP_FWD>(bn, gather_ks(kH, kW)), q, stream);
    }
    if (small_kernel(kH, kW)) {
        pwg::GatherParams q{};
        q.a = x; q.b = weight; q.bias = bias; q.out = y; q.status = device_status_ptr(); q.gate = gate;
        q.g_C = C; q.g_H = H; q.g_W = W; q.N_total = K; q.w_kk = kH * kW; q.o_HW = oH * oW;
        q.vec_b = (C * kH * kW) % 4 == 0 && aligned16(weight);
        q.n_phases = 1;
        pwg::Phase &f = q.ph[0];
        f.HW = oH * oW; f.pix_W = oW; f.M_total = N * f.HW;
        f.taps = kH * kW; f.kW = kW; f.Kd = C * f.taps;
        f.dH = dH; f.dW = dW; f.padH = padH; f.padW = padW; f.dilH = f.dilW = 1;
        f.o_sH = oW; f.o_sW = 1;
        return launch_gather<OP_FWD>(q, pw_bn_for(K, f.M_total), stream);
    }
    GemmParams p{};
    p.a_src = x; p.b_src = weight; p.bias = bias; p.out = y; p.status = device_status_ptr(); p.gate = gate;
    p.g_C = C; p.g_H = H; p.g_W = W; p.g_padH = padH; p.g_padW = padW; p.g_dH = dH; p.g_dW = dW; p.kH = kH; p.kW = kW;
    p.pix_W = oW; p.pix_HW = oH * oW; p.C = C; p.K = K; p.n_img = N;
    p.M_total = N * oH * oW; p.N_total = K; p.Kd = C * kH * kW; p.kblocks = ceil_div(p.Kd, BK); p.out_HW = oH * oW;
    const int bn = pick_bn_for(K);
    dim3 grid(ceil_div(p.M_total, BM), ceil_div(K, bn), 1);
    return launch(pick_kernel<OP_FWD>(bn), p, grid, bn, stream);
}

// `bias` (null: none) is added to every plane of gx: a transposed convolution's forward pass is this one plus its bias.
static int conv_grad_input(const float *gy, const float *weight, const float *bias, float *gx, int N, int C, int H, int W, int K,
                           int kH, int kW, int dH, int dW, int padH, int padW, int dilH, int dilW, cunn_stream_t stream_,
                           void *scratch = nullptr, size_t scratch_bytes = 0, const int *gate = nullptr)
{
    clear_error();
    // the stride-1 kernels leave the bias to a pass of its own
    auto add_bias = [&](int rc) {
        if (rc || !bias) return rc;
        const long long total = (long long)N * C * H * W;
        const int blocks = (int)std::max(1LL, std::min(ceil_div_ll(total, 256), (long long)sm_count() * 16));
        add_plane_bias_kernel<<<blocks, 256, 0, (cudaStream_t)stream_>>>(gx, bias, C, H * W, total, gate);
        CUNN_LAUNCH_CHECK("full convolution bias");
        return 0;
    };
    cudaStream_t stream = (cudaStream_t)stream_;
    int oH, oW;
    if (check(N, C, H, W, K, kH, kW, dH, dW, padH, padW, &oH, &oW, dilH, dilW)) return 1;
    if (N == 0) return 0;
    CUNN_CHECK_ARG(gy && weight && gx, "null tensor pointer");
    const bool dilated = dilH != 1 || dilW != 1;
    CUNN_CHECK_ARG(!dilated || gather_applies(kH, kW), "dilated kernels of more than 32 taps are not supported");
    const split::Geometry geo{N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW, oH, oW};
    try {
        if (split_applies(PASS_GRAD_INPUT, geo, scratch, scratch_bytes)) {
            auto again = [&](int first, int n, const int *wide) {
                return conv_grad_input(gy + (size_t)first * K * oH * oW, weight, bias, gx + (size_t)first * C * H * W, n, C, H, W, K, kH, kW, dH, dW, padH,
                                       padW, dilH, dilW, stream_, nullptr, 0, wide);
            };
            return split::grad_input(geo, gy, weight, bias, gx, split::fallback_of(again), scratch, stream);
        }
    } catch (const std::bad_alloc &) {
        return fail("convmm grad input: out of host memory");
    }
    if (pw_applies(kH, kW, dH, dW, padH, padW) && H * W == 1 && K % 4 == 0 && K < (1 << 24) && (long long)K * C < (1LL << 31) &&
        tma_applies(gy, weight, gx, C, K))
        // a fully connected layer: gx[n][c] = sum_k gy[n][k] W[k][c] is the 1x1 convolution of the one "image" W (K channels of C
        // pixels) with the N filters gy, within the limits of an image and of a filter
        return add_bias(conv_forward(weight, gy, nullptr, gx, 1, K, 1, C, N, 1, 1, 1, 1, 0, 0, 1, 1, stream_));
    if (pw_applies(kH, kW, dH, dW, padH, padW)) {
        pw::Params q{};
        q.a = gy; q.b = weight; q.bias = nullptr; q.out = gx; q.status = device_status_ptr(); q.gate = gate;
        q.HW = H * W; q.M_total = N * H * W; q.N_total = C; q.Kd = K; q.kblocks = ceil_div(K, BK);
        const int bn = pw_bn_for(C, q.M_total);
        q.n_tiles = ceil_div(C, bn); q.tiles_per_split = 0; q.total_tiles = ceil_div(q.M_total, BM) * q.n_tiles;
        q.n_img = N; q.splits = 1;
        if (tma_applies(gy, weight, gx, q.HW, C)) {
            alignas(64) CUtensorMap ma, mb, mo;
            q.gpi = ceil_div(q.HW, 32); q.M_total = N * q.gpi * 32; q.total_tiles = ceil_div(q.M_total, BM) * q.n_tiles;
            q.bulk_out = (q.HW % 32 == 0) && q.HW >= 8 * BM;
            tma_accumulators(bn, q.kblocks, &q.nacc, &q.sets, false, q.total_tiles);
            if (make_map(&ma, gy, q.HW, K, N, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B)) return 1;
            if (make_map(&mb, weight, C, K, 0, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B)) return 1;
            if (const int ranks = pw_cluster(bn, q.total_tiles, q.kblocks); ranks > 1)
                return add_bias(pw_cluster_launch<OP_DGRAD>(q, ranks, ma, mb, stream));
            if (q.bulk_out) { if (make_map(&mo, gx, q.HW, C, N, BM, pwt::HALF_STAGE_COLS, CU_TENSOR_MAP_SWIZZLE_NONE)) return 1; }
            else mo = ma;
            return add_bias(pw_tma_launch(pw_tma_pick<OP_DGRAD>(bn), q, ma, mb, mo, stream));
        }
        q.vec_a = (q.HW % 4 == 0) && aligned16(gy); q.vec_b = (C % 4 == 0) && aligned16(weight);
        q.bulk_out = (q.HW % 4 == 0) && q.HW >= 8 * BM && aligned16(gx);
        pw_accumulators(bn, q.kblocks, &q.nacc, &q.sets);
        return add_bias(pw_launch(pw_pick<OP_DGRAD>(bn), q, stream));
    }
    if (dH == 1 && dW == 1 && padH <= dilH * (kH - 1) && padW <= dilW * (kW - 1) && (gather_applies(kH, kW) || !small_kernel(kH, kW))) {
        // stride 1: a convolution of gy with the kernel rotated by 180 degrees and padding dil (k - 1) - pad
        if (gather_applies(kH, kW)) {
            pw::Params q{};
            q.a = gy; q.b = weight; q.bias = nullptr; q.out = gx; q.status = device_status_ptr(); q.gate = gate;
            q.HW = H * W; q.M_total = N * H * W; q.N_total = C; q.Kd = K * kH * kW; q.kblocks = ceil_div(q.Kd, BK);
            set_geometry(q, K, oH, oW, kH, kW, 1, 1, dilH * (kH - 1) - padH, dilW * (kW - 1) - padW, W, dilH, dilW);
            const int bn = pw_bn_for(C, q.M_total);
            q.n_tiles = ceil_div(C, bn); q.tiles_per_split = 0; q.total_tiles = ceil_div(q.M_total, BM) * q.n_tiles;
            q.n_img = N; q.splits = 1;
            q.vec_a = 0; q.vec_b = 0;
            q.bulk_out = (q.HW % 4 == 0) && q.HW >= 8 * BM && aligned16(gx);
            pw_accumulators(bn, q.kblocks, &q.nacc, &q.sets);
            return add_bias(pw_launch(pw_pick<OP_DGRAD>(bn, gather_ks(kH, kW)), q, stream));
        }
        GemmParams p{};
        p.a_src = gy; p.b_src = weight; p.bias = nullptr; p.out = gx; p.status = device_status_ptr(); p.gate = gate;
        p.g_C = K; p.g_H = oH; p.g_W = oW; p.g_padH = kH - 1 - padH; p.g_padW = kW - 1 - padW; p.g_dH = 1; p.g_dW = 1;
        p.kH = kH; p.kW = kW; p.pix_W = W; p.pix_HW = H * W; p.C = C; p.K = K; p.n_img = N;
        p.M_total = N * H * W; p.N_total = C; p.Kd = K * kH * kW; p.kblocks = ceil_div(p.Kd, BK); p.out_HW = H * W;
        const int bn = pick_bn_for(C);
        dim3 grid(ceil_div(p.M_total, BM), ceil_div(C, bn), 1);
        return add_bias(launch(pick_kernel<OP_DGRAD>(bn), p, grid, bn, stream));
    }
    try {
        return phased_grad_input(gy, weight, bias, gx, N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW, oH, oW, gate, stream);
    } catch (const std::bad_alloc &) {
        return fail("convmm grad input: out of host memory");
    }
}

static int reduce_partials(const float *partial, float *gw, long long n, int splits, float scale, const float *bias_part, float *gb, int K,
                           const int *gate, const float *sums, cudaStream_t stream)
{
    const long long total = n + (bias_part ? K : 0);
    // eight threads per output where one per output would leave SMs short of warps: 9,408 outputs of 148 splits 6.8 us; 295,000 outputs
    // of 37 splits take 18 us that way and 7 us with a thread each
    const bool wide = splits >= 16 && total < 128LL * 1024;
    const int blocks = (int)std::max(1LL, std::min(ceil_div_ll(total, wide ? 32 : 256), (long long)sm_count() * 8));
    void *args[] = {&partial, &gw, &n, &splits, &scale, &bias_part, &gb, &K, &gate, &sums};
    CUNN_CUDA(launch_gated(wide ? (const void *)wgrad_bias_reduce_wide_kernel : (const void *)wgrad_bias_reduce_kernel, dim3(blocks), dim3(256), args, 0, stream,
                           gate));
    return 0;
}

static size_t conv_acc_grad_workspace(int N, int C, int H, int W, int K, int kH, int kW, int dH, int dW, int padH, int padW,
                                      int dilH, int dilW)
{
    int oH, oW;
    if (check(N, C, H, W, K, kH, kW, dH, dW, padH, padW, &oH, &oW, dilH, dilW) || N == 0) return 0;
    const bool dilated = dilH != 1 || dilW != 1;
    if (!dilated && stem::applies(C, K, kH, kW)) return stem::wgrad_workspace_bytes();
    if (pw_applies(kH, kW, dH, dW, padH, padW))
        return std::max(wgrad_partial_bytes(C, K, 1, N, H * W, false), wgrad_partial_bytes(C, K, 1, N, H * W, true));
    if (gathered_wgrad(kH, kW)) return wgrad_partial_bytes(C, K, kH * kW, N, oH * oW, false);
    int bn, splits, ips, pb;
    wgrad_plan(N, C, K, kH * kW, oH * oW, &bn, &splits, &ips, &pb);
    const int chunks = std::max(1, std::min(N, ceil_div(sm_count() * 4, K)));
    return (size_t)splits * K * C * kH * kW * sizeof(float) + (size_t)K * chunks * sizeof(float) + 256;
}

static int conv_acc_grad(const float *x, const float *gy, float *grad_weight, float *grad_bias, int N, int C, int H, int W, int K,
                         int kH, int kW, int dH, int dW, int padH, int padW, int dilH, int dilW, float scale, void *workspace,
                         size_t workspace_bytes, cunn_stream_t stream_, const int *gate = nullptr, const float *sums = nullptr)
{
    clear_error();
    cudaStream_t stream = (cudaStream_t)stream_;
    int oH, oW;
    if (check(N, C, H, W, K, kH, kW, dH, dW, padH, padW, &oH, &oW, dilH, dilW)) return 1;
    if (N == 0) return 0;
    CUNN_CHECK_ARG(x && gy && grad_weight, "null tensor pointer");
    const bool dilated = dilH != 1 || dilW != 1;
    CUNN_CHECK_ARG(!dilated || gather_applies(kH, kW), "dilated kernels of more than 32 taps are not supported");
    const size_t need = conv_acc_grad_workspace(N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW);
    CUNN_CHECK_ARG(workspace && workspace_bytes >= need && ((uintptr_t)workspace & 15) == 0,
                   "convmm acc_grad needs %zu bytes of 16-byte aligned workspace, got %zu", need,
                   workspace ? workspace_bytes : (size_t)0);
    int bn, splits, ips, pb, kb;
    const int kk = kH * kW;
    if (!dilated && stem::applies(C, K, kH, kW)) {
        const int ctas = stem::wgrad_ctas();
        const long long n = (long long)K * C * kk;
        float *partial = (float *)workspace, *bias_part = partial + (size_t)ctas * n;
        if (stem::weight_grad_partials(x, gy, partial, grad_bias ? bias_part : nullptr, N, H, W, oH, oW, dH, dW, padH, padW, stream)) return 1;
        return reduce_partials(partial, grad_weight, n, ctas, scale, grad_bias ? bias_part : nullptr, grad_bias, K, gate, sums, stream);
    }
    const split::Geometry geo{N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW, oH, oW};
    if (!gate && split_applies(PASS_GRAD_WEIGHT, geo, workspace, workspace_bytes)) {
        auto again = [&](int first, int n, const int *wide) {
            const size_t head = split::grad_weight_head(geo);
            return conv_acc_grad(x + (size_t)first * C * H * W, gy + (size_t)first * K * oH * oW, grad_weight, nullptr, n, C, H, W, K, kH, kW, dH, dW, padH, padW,
                                 dilH, dilW, scale, (char *)workspace + head, workspace_bytes - head, stream_, wide, split::grad_weight_sums(geo, workspace));
        };
        return split::grad_weight(geo, x, gy, grad_bias, scale, split::fallback_of(again), workspace, stream);
    }
    if (pw_applies(kH, kW, dH, dW, padH, padW)) {
        const bool tma = tma_applies(gy, x, workspace, H * W, 4);
        pw_wgrad_plan(C, K, 1, N, H * W, tma, &bn, &splits, &kb);
        const long long n = (long long)K * C;
        pw::Params q{};
        q.a = gy; q.b = x; q.bias = nullptr; q.out = (float *)workspace; q.status = device_status_ptr(); q.gate = gate;
        q.bias_part = grad_bias ? (float *)workspace + (size_t)splits * n : nullptr;
        q.HW = H * W; q.M_total = K; q.N_total = C; q.Kd = 0; q.kblocks = kb;
        q.n_tiles = ceil_div(C, bn); q.tiles_per_split = ceil_div(K, BM) * q.n_tiles; q.total_tiles = q.tiles_per_split * splits;
        q.n_img = N; q.splits = splits;
        q.vec_a = (q.HW % 4 == 0) && aligned16(gy); q.vec_b = (q.HW % 4 == 0) && aligned16(x);
        if (tma) {
            alignas(64) CUtensorMap ma, mb;
            q.gpi = ceil_div(q.HW, 32);
            tma_accumulators(bn, q.kblocks, &q.nacc, &q.sets, true, q.total_tiles);
            if (make_map(&ma, gy, q.HW, K, N, 32, BM, CU_TENSOR_MAP_SWIZZLE_128B)) return 1;
            if (make_map(&mb, x, q.HW, C, N, 32, bn, CU_TENSOR_MAP_SWIZZLE_128B)) return 1;
            if (pw_tma_launch(pw_tma_pick<OP_WGRAD>(bn), q, ma, mb, ma, stream)) return 1;
        } else {
            pw_accumulators(bn, q.kblocks, &q.nacc, &q.sets, true, q.total_tiles);
            if (pw_launch(rounds_wgrad(1, N, H * W) ? pw_pick_rounded(bn, 1) : pw_pick<OP_WGRAD>(bn), q, stream)) return 1;
        }
        return reduce_partials((const float *)workspace, grad_weight, n, splits, scale, q.bias_part, grad_bias, K, gate, sums, stream);
    }
    if (gathered_wgrad(kH, kW)) {
        const int oHW = oH * oW;
        pw_wgrad_plan(C, K, kk, N, oHW, false, &bn, &splits, &kb);
        const long long n = (long long)K * C * kk;
        pw::Params q{};
        q.a = gy; q.b = x; q.bias = nullptr; q.out = (float *)workspace; q.status = device_status_ptr(); q.gate = gate;
        q.bias_part = grad_bias ? (float *)workspace + (size_t)splits * n : nullptr;
        q.HW = oHW; q.M_total = K; q.N_total = C * kk; q.Kd = 0; q.kblocks = kb;
        set_geometry(q, C, H, W, kH, kW, dH, dW, padH, padW, oW, dilH, dilW);
        q.n_tiles = ceil_div(C * kk, bn); q.tiles_per_split = ceil_div(K, BM) * q.n_tiles; q.total_tiles = q.tiles_per_split * splits;
        q.n_img = N; q.splits = splits;
        q.vec_a = (oHW % 4 == 0) && aligned16(gy); q.vec_b = 0;
        pw_accumulators(bn, q.kblocks, &q.nacc, &q.sets, true, q.total_tiles);
        const int ks = gather_ks(kH, kW);
        if (pw_launch(rounds_wgrad(kk, N, oHW) ? pw_pick_rounded(bn, ks) : pw_pick<OP_WGRAD>(bn, ks), q, stream)) return 1;
        return reduce_partials((const float *)workspace, grad_weight, n, splits, scale, q.bias_part, grad_bias, K, gate, sums, stream);
    }
    wgrad_plan(N, C, K, kk, oH * oW, &bn, &splits, &ips, &pb);
    GemmParams p{};
    p.a_src = gy; p.b_src = x; p.bias = nullptr; p.out = (float *)workspace; p.status = device_status_ptr(); p.gate = gate;
    p.g_C = C; p.g_H = H; p.g_W = W; p.g_padH = padH; p.g_padW = padW; p.g_dH = dH; p.g_dW = dW; p.kH = kH; p.kW = kW;
    p.pix_W = oW; p.pix_HW = oH * oW; p.C = C; p.K = K; p.n_img = N;
    p.M_total = K; p.N_total = C * kk; p.Kd = 0; p.kblocks = ips * pb; p.out_HW = 0;
    p.imgs_per_split = ips; p.pix_blocks = pb;
    dim3 grid(ceil_div(K, BM), ceil_div(C * kk, bn), splits);
    if (launch(pick_kernel<OP_WGRAD>(bn), p, grid, bn, stream)) return 1;
    const long long n = (long long)K * C * kk;
    const int rblocks = (int)std::max(1LL, std::min(ceil_div_ll(n, 256), (long long)sm_count() * 8));
    wgrad_reduce_kernel<<<rblocks, 256, 0, stream>>>((const float *)workspace, grad_weight, n, splits, scale, gate, sums);
    CUNN_LAUNCH_CHECK("convmm acc grad reduce");
    if (grad_bias) {
        const int chunks = std::max(1, std::min(N, ceil_div(sm_count() * 4, K)));
        float *part = (float *)workspace + (size_t)splits * n;
        bias_partial_kernel<<<K * chunks, 256, 0, stream>>>(gy, part, N, K, oH * oW, chunks);
        CUNN_LAUNCH_CHECK("convmm bias gradient");
        bias_finish_kernel<<<ceil_div(K, 128), 128, 0, stream>>>(part, grad_bias, K, chunks, scale);
        CUNN_LAUNCH_CHECK("convmm bias gradient finish");
    }
    return 0;
}

extern "C" CUNN_API void cunn_b200_convmm_set_tma(int on) { cunn::mm::g_use_tma = on ? 1 : 0; }
extern "C" CUNN_API int cunn_b200_convmm_get_tma(void) { return cunn::mm::g_use_tma; }

extern "C" CUNN_API int cunn_b200_convmm_forward(const float *x, const float *weight, const float *bias, float *y, int N,
                                                 int C, int H, int W, int K, int kH, int kW, int dH, int dW, int padH,
                                                 int padW, cunn_stream_t stream)
{
    return conv_forward(x, weight, bias, y, N, C, H, W, K, kH, kW, dH, dW, padH, padW, 1, 1, stream);
}

extern "C" CUNN_API int cunn_b200_convmm_grad_input(const float *gy, const float *weight, float *gx, int N, int C, int H,
                                                    int W, int K, int kH, int kW, int dH, int dW, int padH, int padW,
                                                    cunn_stream_t stream)
{
    return conv_grad_input(gy, weight, nullptr, gx, N, C, H, W, K, kH, kW, dH, dW, padH, padW, 1, 1, stream);
}

extern "C" CUNN_API size_t cunn_b200_convmm_acc_grad_workspace(int N, int C, int H, int W, int K, int kH, int kW, int dH,
                                                               int dW, int padH, int padW)
{
    return conv_acc_grad_workspace(N, C, H, W, K, kH, kW, dH, dW, padH, padW, 1, 1);
}

extern "C" CUNN_API int cunn_b200_convmm_acc_grad(const float *x, const float *gy, float *grad_weight, float *grad_bias,
                                                  int N, int C, int H, int W, int K, int kH, int kW, int dH, int dW,
                                                  int padH, int padW, float scale, void *workspace, size_t workspace_bytes,
                                                  cunn_stream_t stream)
{
    return conv_acc_grad(x, gy, grad_weight, grad_bias, N, C, H, W, K, kH, kW, dH, dW, padH, padW, 1, 1, scale, workspace,
                         workspace_bytes, stream);
}

extern "C" CUNN_API size_t cunn_b200_conv_scratch(int pass, int N, int C, int H, int W, int K, int kH, int kW, int dH, int dW, int padH,
                                                  int padW, int dilH, int dilW)
{
    int oH, oW;
    if (pass < PASS_FORWARD || pass > PASS_GRAD_WEIGHT || check(N, C, H, W, K, kH, kW, dH, dW, padH, padW, &oH, &oW, dilH, dilW)) {
        clear_error();
        return 0;
    }
    if (dilH == 1 && dilW == 1 && pass != PASS_GRAD_INPUT && stem::applies(C, K, kH, kW)) return 0;
    try {
        return split_scratch(pass, split::Geometry{N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW, oH, oW});
    } catch (const std::bad_alloc &) {
        return 0;
    }
}

extern "C" CUNN_API int cunn_b200_conv_forward_scratch(const float *x, const float *weight, const float *bias, float *y, int N, int C, int H,
                                                       int W, int K, int kH, int kW, int dH, int dW, int padH, int padW, int dilH,
                                                       int dilW, void *scratch, size_t scratch_bytes, cunn_stream_t stream)
{
    return conv_forward(x, weight, bias, y, N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW, stream, scratch, scratch_bytes);
}

extern "C" CUNN_API int cunn_b200_conv_grad_input_scratch(const float *gy, const float *weight, float *gx, int N, int C, int H, int W, int K,
                                                          int kH, int kW, int dH, int dW, int padH, int padW, int dilH, int dilW,
                                                          void *scratch, size_t scratch_bytes, cunn_stream_t stream)
{
    return conv_grad_input(gy, weight, nullptr, gx, N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW, stream, scratch, scratch_bytes);
}

extern "C" CUNN_API int cunn_b200_dilated_conv_forward(const float *x, const float *weight, const float *bias, float *y, int N,
                                                       int C, int H, int W, int K, int kH, int kW, int dH, int dW, int padH,
                                                       int padW, int dilH, int dilW, cunn_stream_t stream)
{
    return conv_forward(x, weight, bias, y, N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW, stream);
}

extern "C" CUNN_API int cunn_b200_dilated_conv_grad_input(const float *gy, const float *weight, float *gx, int N, int C,
                                                          int H, int W, int K, int kH, int kW, int dH, int dW, int padH,
                                                          int padW, int dilH, int dilW, cunn_stream_t stream)
{
    return conv_grad_input(gy, weight, nullptr, gx, N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW, stream);
}

extern "C" CUNN_API size_t cunn_b200_dilated_conv_acc_grad_workspace(int N, int C, int H, int W, int K, int kH, int kW,
                                                                     int dH, int dW, int padH, int padW, int dilH, int dilW)
{
    return conv_acc_grad_workspace(N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW);
}

extern "C" CUNN_API int cunn_b200_dilated_conv_acc_grad(const float *x, const float *gy, float *grad_weight, float *grad_bias,
                                                        int N, int C, int H, int W, int K, int kH, int kW, int dH, int dW,
                                                        int padH, int padW, int dilH, int dilW, float scale, void *workspace,
                                                        size_t workspace_bytes, cunn_stream_t stream)
{
    return conv_acc_grad(x, gy, grad_weight, grad_bias, N, C, H, W, K, kH, kW, dH, dW, padH, padW, dilH, dilW, scale, workspace,
                         workspace_bytes, stream);
}

// ---------------------------------------------------------------------------
// SpatialFullDilatedConvolution (transposed convolution): x [N,P,H,W], weight [P,Q,kH,kW], y [N,Q,OH,OW].
// It is the adjoint of the convolution that maps [N,Q,OH,OW] to [N,P,H,W] with the same weight array read as
// [K = P][C = Q][kH][kW], so its forward is that convolution's input gradient (plus bias), its input gradient is that
// convolution's forward, and its weight gradient is that convolution's weight gradient with the roles of the
// activations and the output gradient exchanged.
// ---------------------------------------------------------------------------

static int full_check(int N, int P, int H, int W, int Q, int kH, int kW, int dH, int dW, int padH, int padW, int dilH, int dilW,
                      int adjH, int adjW, int *OH, int *OW)
{
    CUNN_CHECK_ARG(kW > 0 && kH > 0, "kernel size should be greater than zero, but got kH: %d kW: %d", kH, kW);
    CUNN_CHECK_ARG(dW > 0 && dH > 0, "stride should be greater than zero, but got dH: %d dW: %d", dH, dW);
    CUNN_CHECK_ARG(dilW > 0 && dilH > 0, "dilation should be greater than zero, but got dilationH: %d, dilationW: %d", dilH, dilW);
    CUNN_CHECK_ARG(adjH >= 0 && adjW >= 0 && (adjW < dW || adjW < dilW) && (adjH < dH || adjH < dilH),
                   "output padding must be smaller than either stride or dilation, but got adjH: %d adjW: %d dH: %d dW: %d "
                   "dilationH: %d dilationW: %d", adjH, adjW, dH, dW, dilH, dilW);
    CUNN_CHECK_ARG(adjH < dH && adjW < dW, "output padding of at least the stride is not supported (adjH: %d adjW: %d dH: %d dW: %d)",
                   adjH, adjW, dH, dW);
    CUNN_CHECK_ARG(N >= 0 && P > 0 && Q > 0 && H > 0 && W > 0 && padH >= 0 && padW >= 0, "bad convolution sizes");
    const long long oh = (long long)(H - 1) * dH - 2 * padH + (dilH * (kH - 1) + 1) + adjH;
    const long long ow = (long long)(W - 1) * dW - 2 * padW + (dilW * (kW - 1) + 1) + adjW;
    CUNN_CHECK_ARG(oh >= 1 && ow >= 1 && oh < (1 << 24) && ow < (1 << 24),
                   "Given input size: (%d x %d x %d). Calculated output size: (%d x %lld x %lld). Output size is too small", P, H, W,
                   Q, oh, ow);
    *OH = (int)oh; *OW = (int)ow;
    return 0;
}

static int bias_chunks(int N, int Q) { return std::max(1, std::min(N, ceil_div(sm_count() * 4, Q))); }
static size_t round256(size_t v) { return (v + 255) & ~(size_t)255; }
// The transposed convolution's bias sums, at the head of its parameter gradient's workspace.
static size_t full_bias_bytes(int N, int Q) { return round256((size_t)Q * bias_chunks(N, Q) * sizeof(float)); }

extern "C" CUNN_API int cunn_b200_full_conv_forward(const float *x, const float *weight, const float *bias, float *y, int N,
                                                    int P, int H, int W, int Q, int kH, int kW, int dH, int dW, int padH,
                                                    int padW, int dilH, int dilW, int adjH, int adjW, cunn_stream_t stream_)
{
    clear_error();
    int OH, OW;
    if (full_check(N, P, H, W, Q, kH, kW, dH, dW, padH, padW, dilH, dilW, adjH, adjW, &OH, &OW)) return 1;
    return conv_grad_input(x, weight, bias, y, N, Q, OH, OW, P, kH, kW, dH, dW, padH, padW, dilH, dilW, stream_);
}

extern "C" CUNN_API int cunn_b200_full_conv_grad_input(const float *gy, const float *weight, float *gx, int N, int P, int H,
                                                       int W, int Q, int kH, int kW, int dH, int dW, int padH, int padW,
                                                       int dilH, int dilW, int adjH, int adjW, cunn_stream_t stream_)
{
    clear_error();
    int OH, OW;
    if (full_check(N, P, H, W, Q, kH, kW, dH, dW, padH, padW, dilH, dilW, adjH, adjW, &OH, &OW)) return 1;
    return conv_forward(gy, weight, nullptr, gx, N, Q, OH, OW, P, kH, kW, dH, dW, padH, padW, dilH, dilW, stream_);
}

extern "C" CUNN_API size_t cunn_b200_full_conv_scratch(int pass, int N, int P, int H, int W, int Q, int kH, int kW, int dH, int dW, int padH,
                                                       int padW, int dilH, int dilW, int adjH, int adjW)
{
    int OH, OW;
    if (pass < PASS_FORWARD || pass > PASS_GRAD_WEIGHT ||
        full_check(N, P, H, W, Q, kH, kW, dH, dW, padH, padW, dilH, dilW, adjH, adjW, &OH, &OW)) {
        clear_error();
        return 0;
    }
    // the adjoint convolution: its input gradient is this forward pass
    const int of = pass == PASS_FORWARD ? PASS_GRAD_INPUT : pass == PASS_GRAD_INPUT ? PASS_FORWARD : PASS_GRAD_WEIGHT;
    const size_t bytes = cunn_b200_conv_scratch(of, N, Q, OH, OW, P, kH, kW, dH, dW, padH, padW, dilH, dilW);
    return bytes && of == PASS_GRAD_WEIGHT ? full_bias_bytes(N, Q) + bytes : bytes;
}

extern "C" CUNN_API int cunn_b200_full_conv_forward_scratch(const float *x, const float *weight, const float *bias, float *y, int N, int P, int H,
                                                            int W, int Q, int kH, int kW, int dH, int dW, int padH, int padW, int dilH,
                                                            int dilW, int adjH, int adjW, void *scratch, size_t scratch_bytes,
                                                            cunn_stream_t stream)
{
    clear_error();
    int OH, OW;
    if (full_check(N, P, H, W, Q, kH, kW, dH, dW, padH, padW, dilH, dilW, adjH, adjW, &OH, &OW)) return 1;
    return conv_grad_input(x, weight, bias, y, N, Q, OH, OW, P, kH, kW, dH, dW, padH, padW, dilH, dilW, stream, scratch, scratch_bytes);
}

extern "C" CUNN_API int cunn_b200_full_conv_grad_input_scratch(const float *gy, const float *weight, float *gx, int N, int P, int H, int W,
                                                               int Q, int kH, int kW, int dH, int dW, int padH, int padW, int dilH,
                                                               int dilW, int adjH, int adjW, void *scratch, size_t scratch_bytes,
                                                               cunn_stream_t stream)
{
    clear_error();
    int OH, OW;
    if (full_check(N, P, H, W, Q, kH, kW, dH, dW, padH, padW, dilH, dilW, adjH, adjW, &OH, &OW)) return 1;
    return conv_forward(gy, weight, nullptr, gx, N, Q, OH, OW, P, kH, kW, dH, dW, padH, padW, dilH, dilW, stream, scratch, scratch_bytes);
}

extern "C" CUNN_API size_t cunn_b200_full_conv_acc_grad_workspace(int N, int P, int H, int W, int Q, int kH, int kW, int dH,
                                                                  int dW, int padH, int padW, int dilH, int dilW, int adjH,
                                                                  int adjW)
{
    int OH, OW;
    if (full_check(N, P, H, W, Q, kH, kW, dH, dW, padH, padW, dilH, dilW, adjH, adjW, &OH, &OW) || N == 0) return 0;
    return full_bias_bytes(N, Q) + round256(conv_acc_grad_workspace(N, Q, OH, OW, P, kH, kW, dH, dW, padH, padW, dilH, dilW)) + 256;
}

extern "C" CUNN_API int cunn_b200_full_conv_acc_grad(const float *x, const float *gy, float *grad_weight, float *grad_bias,
                                                     int N, int P, int H, int W, int Q, int kH, int kW, int dH, int dW,
                                                     int padH, int padW, int dilH, int dilW, int adjH, int adjW, float scale,
                                                     void *workspace, size_t workspace_bytes, cunn_stream_t stream_)
{
    clear_error();
    int OH, OW;
    if (full_check(N, P, H, W, Q, kH, kW, dH, dW, padH, padW, dilH, dilW, adjH, adjW, &OH, &OW)) return 1;
    if (N == 0) return 0;
    const int chunks = bias_chunks(N, Q);
    const size_t head = full_bias_bytes(N, Q), need = cunn_b200_full_conv_acc_grad_workspace(N, P, H, W, Q, kH, kW, dH, dW, padH, padW, dilH, dilW, adjH, adjW);
    CUNN_CHECK_ARG(workspace && workspace_bytes >= need && ((uintptr_t)workspace & 15) == 0,
                   "full convolution acc_grad needs %zu bytes of 16-byte aligned workspace, got %zu", need,
                   workspace ? workspace_bytes : (size_t)0);
    // the adjoint convolution's "input" is gy and its "output gradient" is x
    if (conv_acc_grad(gy, x, grad_weight, nullptr, N, Q, OH, OW, P, kH, kW, dH, dW, padH, padW, dilH, dilW, scale,
                      (char *)workspace + head, workspace_bytes - head, stream_))
        return 1;
    if (grad_bias) {
        cudaStream_t stream = (cudaStream_t)stream_;
        float *part = (float *)workspace;
        bias_partial_kernel<<<Q * chunks, 256, 0, stream>>>(gy, part, N, Q, OH * OW, chunks);
        CUNN_LAUNCH_CHECK("full convolution bias gradient");
        bias_finish_kernel<<<ceil_div(Q, 128), 128, 0, stream>>>(part, grad_bias, Q, chunks, scale);
        CUNN_LAUNCH_CHECK("full convolution bias gradient finish");
    }
    return 0;
}
