// Implicit GEMM with a gathered image operand, partial sums kept in registers: strided input gradients (and with them the
// forward pass of transposed convolutions) and kernels of more than 32 taps.
//
//   input grad  D[pixel, c]  = sum_{ko, tap}  gy(pixel; ko, tap) * W[ko][c][tap]
//   forward     D[pixel, ko] = sum_{c, tap}   x(pixel; c, tap)   * W[ko][c][tap]
//
// A strided input gradient is taken apart into dH x dW phases: the input pixels with (h + padH) mod dH = a and
// (w + padW) mod dW = b are reached by the taps of that residue only, and for them the sum is a stride-1 convolution of gy
// with those taps.  A phase is therefore an ordinary GEMM whose rows are the phase's pixels and whose reduction runs over
// (ko, the phase's taps); no product with a zero is formed.  All phases are tiles of one launch, longest reduction first, but for those
// whose sums are short, or which fill too little of a tile: phase_fma_kernel takes them in fp32.
//
// Tiles, split (3xTF32), descriptors and the copies' ring are those of pw::pw_gemm_kernel.  What differs is the
// accumulation: the tensor core truncates when it adds to an accumulator, and an error of about 1e-7 of the result grows
// with every k-block that a chain holds (1.1e-6 at 1024 and 2.1e-6 at 2304 products in chains of 11 and 24 k-blocks; a chain of
// fp32 FMAs, which these passes used before, is 5e-7 off).  Here a chain is ONE k-block: its eight cross-term MMAs come first, while the
// accumulator is 2^-11 of its final size, then the four hi*hi ones; the 16 producer warps read the finished block back
// (32 columns each, two TMEM buffers in turn) and add it to fp32 registers with rounding.  The producers' waits already order
// everything: k-block i is drained before its producer hands over k-block i + 2, which is the next one to use its TMEM buffer, so
// no further barrier exists.
//
// Bound by the producers: 4-byte copies of the gathered operands (128 + up to 128 warp instructions per k-block, those of the weights
// 9 to 10 cache lines each) and the split; the tensor pipe needs 768 of the 4,400 clocks that a k-block takes.  Input gradient of
// 64 x 128 x 56 x 56, 256 filters 3x3 stride 2: 44.9 ms with a thread per pixel, 0.43 ms here (69 TFLOP/s); forward of the transposed
// 64 x 256 x 14 x 14 -> 128 x 28 x 28, 4x4: 26.9 ms and 0.245 ms (54 TFLOP/s).
// Relative error (2-norm) of those two: 4.7e-7 and 5.6e-7 before, 1.6e-7 and 1.7e-7 now; over sums of 48 to 9216 products 1.3e-7 to
// 1.6e-6 before and 1.2e-7 to 3.3e-7 now; shorter ones are the same sums as before.
#pragma once

namespace pwg {

using namespace pw;

constexpr int MAX_PHASES = 16;
constexpr int GTHREADS = PRODUCERS + 32;                              // 16 producer warps + one that issues the MMAs
constexpr size_t GSMEM = (size_t)(RAW_STAGES + LO_BUFS) * 2 * TILE + 1024;
constexpr int MAX_KERNEL = 16;                                        // rows and columns of taps: 16 + 16 validity bits per pixel

// One sub-problem: pixels (r / pix_W, r % pix_W) of its grid read the gathered tensor at
// (row * dH - padH + th * dilH, col * dW - padW + tw * dilW) for taps (th, tw), with the weight of tap
// w_base + th * w_sH + tw * w_sW, and are written at o_off + row * o_sH + col * o_sW of an output plane.
struct Phase {
    int tile0;                    // first tile of the phase in the launch
    int HW, pix_W, M_total;       // pixels per image, row length, pixels in all
    int Kd, kblocks;              // reduction length, k-blocks
    int taps, kW;                 // taps, columns of taps
    uint32_t taps_magic, kW_magic;
    int dH, dW, padH, padW, dilH, dilW;
    int w_base, w_sH, w_sW;
    int o_off, o_sH, o_sW;
};
struct GatherParams {
    const float *a, *b, *bias;    // gathered tensor, weights, bias or null
    float *out;
    int *status;
    const int *gate;              // null, or see gated_off
    int g_C, g_H, g_W;            // channels, rows and columns of the gathered tensor
    int N_total, n_tiles, total_tiles, n_phases;
    int w_kk;                     // taps of the whole kernel
    int o_HW;                     // pixels of an output plane
    int vec_b;                    // forward: 16-byte copies of the weights allowed
    Phase ph[MAX_PHASES];
};

// k / d for k * d < 2^32 by multiplication: magic = floor(2^32 / d) + 1, 0 for d = 1.  The error k / 2^32 of the product's
// fraction stays below 1 / d then.  The forward pass has k < 2^24 and d <= 256; input gradients beyond the bound go to phase_fma_kernel.
__device__ __forceinline__ int magic_div(int k, uint32_t magic) { return magic ? (int)__umulhi((uint32_t)k, magic) : k; }

template <int OP, int BN>
struct GatherLoader {
    int tile, kb, phase, KB;
    int a_off[4];            // element offsets of the thread's pixels lane + 32 j (tap 0, channel 0)
    uint32_t valid[4];       // bit th: tap row th inside the image; bit 16 + tw: tap column tw
    int b_off[2];            // forward: weight rows of the thread's two pieces; input gradient: [0] first column
    unsigned b_mask;

    __device__ __forceinline__ void setup(const GatherParams &p, int t)
    {
        const int tid = threadIdx.x, lane = tid & 31;
        tile = t;
        kb = 0;
        while (phase + 1 < p.n_phases && t >= p.ph[phase + 1].tile0) ++phase;
        const Phase &f = p.ph[phase];
        KB = f.kblocks;
        const int r0 = t - f.tile0, m_tile = r0 / p.n_tiles, n0 = (r0 - m_tile * p.n_tiles) * BN;
        const int kH_n = f.taps / f.kW;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            a_off[j] = 0;
            valid[j] = 0;
            const int m = m_tile * BM + lane + 32 * j;
            if (m < f.M_total) {
                const int im = m / f.HW, r = m - im * f.HW;
                const int ph = r / f.pix_W, pw_ = r - ph * f.pix_W;
                const int ih0 = ph * f.dH - f.padH, iw0 = pw_ * f.dW - f.padW;
                a_off[j] = im * p.g_C * p.g_H * p.g_W + ih0 * p.g_W + iw0;
                for (int th = 0; th < kH_n; ++th)
                    if ((unsigned)(ih0 + th * f.dilH) < (unsigned)p.g_H) valid[j] |= 1u << th;
                for (int tw = 0; tw < f.kW; ++tw)
                    if ((unsigned)(iw0 + tw * f.dilW) < (unsigned)p.g_W) valid[j] |= 0x10000u << tw;
            }
        }
        b_mask = 0;
        if (OP == OP_FWD) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int row = (tid >> 3) + 64 * i, n = n0 + row;
                b_off[i] = n * f.Kd + (tid & 7) * 4;
                if (row < BN && n < p.N_total) b_mask |= 1u << i;
            }
        } else {
            b_off[0] = n0 + lane;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (lane + 32 * j < BN && n0 + lane + 32 * j < p.N_total) b_mask |= 1u << j;
        }
    }
    __device__ __forceinline__ void advance(const GatherParams &p)
    {
        if (++kb < KB) return;
        const int t = tile + (int)gridDim.x;
        if (t < p.total_tiles) setup(p, t);
        else tile = t;
    }
    // Issues the copies of this thread's elements of the current k-block into the raw tiles at sa / sb.
    __device__ __forceinline__ void issue(const GatherParams &p, uint32_t sa, uint32_t sb, const uint32_t (&g_so)[2],
                                          const uint32_t (&b_so)[2]) const
    {
        const int tid = threadIdx.x, warp = tid >> 5;
        const Phase &f = p.ph[phase];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int k = kb * BK + warp + 16 * i;
            const bool kok = k < f.Kd;
            const int c = magic_div(k, f.taps_magic), t2 = k - c * f.taps;
            const int th = magic_div(t2, f.kW_magic), tw = t2 - th * f.kW;
            const int koff = (c * p.g_H + th * f.dilH) * p.g_W + tw * f.dilW;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool ok = kok && ((valid[j] >> th) & (valid[j] >> (16 + tw)) & 1u);
                cp_async4(sa + g_so[i] + MN_ATOM * j, ok ? p.a + (a_off[j] + koff) : p.a, ok);
            }
            if (OP == OP_DGRAD) {
                const float *wk = p.b + ((size_t)(kok ? c : 0) * p.N_total + b_off[0]) * p.w_kk + (f.w_base + th * f.w_sH + tw * f.w_sW);
#pragma unroll
                for (int j = 0; j < BN / 32; ++j) {
                    const bool ok = kok && (b_mask >> j & 1u);
                    cp_async4(sb + g_so[i] + MN_ATOM * j, ok ? wk + (size_t)(32 * j) * p.w_kk : p.b, ok);
                }
            }
        }
        if (OP == OP_FWD) {
            const int k0 = kb * BK + (tid & 7) * 4;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if ((tid >> 3) + 64 * i >= BN) continue;
                const float *src = p.b + b_off[i] + kb * BK;
                const bool rok = (b_mask >> i & 1u) != 0;
                if (p.vec_b) {
                    const bool ok = rok && k0 < f.Kd;
                    cp_async16(sb + b_so[i], ok ? src : p.b, ok);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const bool ok = rok && k0 + j < f.Kd;
                        cp_async4(sb + b_so[i] + 4 * j, ok ? src + j : p.b, ok);
                    }
                }
            }
        }
    }
};

// One warp: COLS accumulator columns of its 32 TMEM lanes, on top of acc (first: in place of it).
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
template <int COLS>
__device__ __forceinline__ void drain_block(float (&acc)[COLS], uint32_t taddr, bool first)
{
    if (first) {
#pragma unroll
        for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
    }
    if constexpr (COLS == 8) {
        uint32_t r[8];
        tmem_ld8(taddr, r);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += __uint_as_float(r[j]);
    } else {
#pragma unroll
        for (int c = 0; c < COLS; c += 16) {
            uint32_t r[16];
            tmem_ld16(taddr + (uint32_t)c, r);
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(r[j]);
        }
    }
}

// One input-gradient pixel in plain fp32.  The parts of infinities, and the zeros in place of taps outside gy, form products that are
// NaN where the definition has none, so sums that came out as NaN are taken again this way.
// That takes as long as the fp32 form takes (a warp's 32 pixels in step, gy in consecutive words), so it is done after the CTA's last
// k-block: no warp then waits on a barrier with a limit for this one's arrivals.
__device__ __forceinline__ float gather_scalar(const GatherParams &p, const Phase &f, int im, int row, int col, int n)
{
    const int channels = f.Kd / f.taps, kH_n = f.taps / f.kW;
    const float *src = p.a + (size_t)im * p.g_C * p.g_H * p.g_W;
    float s = 0.f;
#pragma unroll 1
    for (int th = 0; th < kH_n; ++th) {
        const int ih = row * f.dH - f.padH + th * f.dilH;
        if ((unsigned)ih >= (unsigned)p.g_H) continue;
#pragma unroll 1
        for (int tw = 0; tw < f.kW; ++tw) {
            const int iw = col * f.dW - f.padW + tw * f.dilW;
            if ((unsigned)iw >= (unsigned)p.g_W) continue;
#pragma unroll 8
            for (int c = 0; c < channels; ++c)
                s = fmaf(__ldg(p.b + ((size_t)c * p.N_total + n) * p.w_kk + f.w_base + th * f.w_sH + tw * f.w_sW),
                         __ldg(src + ((size_t)c * p.g_H + ih) * p.g_W + iw), s);
        }
    }
    return s;
}

template <int OP, int BN>
__global__ void __launch_bounds__(GTHREADS, 1)
gather_gemm_kernel(const __grid_constant__ GatherParams p)
{
    constexpr bool B_MN = OP == OP_DGRAD;
    constexpr uint32_t TMEM_COLS = 2 * BN;                                 // two buffers of one k-block's sums
    constexpr int COLS = BN / 4;                                           // columns per producer warp
    constexpr uint32_t idesc = idesc_of(BN, true, B_MN);

    if (gated_off(p.gate)) return;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t done[RAW_STAGES];     // the MMAs of this stage's k-block have finished
    __shared__ uint64_t full[RAW_STAGES];     // stage split and visible to the tensor core: one arrival per producer warp
    __shared__ uint32_t tmem_base_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < RAW_STAGES; ++s) {
            mbar_init(smem_u32(done + s), 1);
            mbar_init(smem_u32(full + s), PRODUCERS / 32);
        }
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(smem_u32(&tmem_base_s), TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;
    unsigned char *const lo_base = smem + (size_t)RAW_STAGES * 2 * TILE;

    // k-blocks of this CTA's tiles blockIdx.x, blockIdx.x + gridDim.x, ...
    int total_it = 0;
    for (int t = (int)blockIdx.x, f = 0; t < p.total_tiles; t += (int)gridDim.x) {
        while (f + 1 < p.n_phases && t >= p.ph[f + 1].tile0) ++f;
        total_it += p.ph[f].kblocks;
    }

    if (warp == PRODUCERS / 32) {
        if (lane == 0) {
            constexpr uint32_t A_LOW = (uint32_t)(MN_ATOM >> 4) << 16, B_LOW = B_MN ? ((uint32_t)(MN_ATOM >> 4) << 16) : (1u << 16);
            constexpr uint32_t A_HIGH = (uint32_t)(MN_KATOM >> 4) | (1u << 14) | (1u << 29);
            constexpr uint32_t B_HIGH = (B_MN ? (uint32_t)(MN_KATOM >> 4) : (uint32_t)(SBO >> 4)) | (1u << 14) | ((B_MN ? 1u : 2u) << 29);
            constexpr uint32_t A_STEP = (uint32_t)(2 * MN_KATOM >> 4), B_STEP = B_MN ? (uint32_t)(2 * MN_KATOM >> 4) : 2u;
            constexpr uint32_t STAGE_STEP = (uint32_t)(2 * TILE >> 4);
            const uint32_t raw0 = (smem_u32(smem) >> 4) & 0x3fffu, lo0 = (smem_u32(lo_base) >> 4) & 0x3fffu;
            auto desc = [](uint32_t low, uint32_t high) { return ((uint64_t)high << 32) | low; };
            int rs = 0, lb = 0;
            uint32_t parity = 0;
            for (int i = 0; i < total_it; ++i) {
                if (!mbar_wait(smem_u32(full + rs), parity, p.status)) break;
                tc_fence_after();
                const uint32_t d = tmem_base + (uint32_t)((i & 1) * BN);
                const uint32_t ah = (raw0 + (uint32_t)rs * STAGE_STEP) | A_LOW, bh = (raw0 + (uint32_t)rs * STAGE_STEP + (uint32_t)(TILE >> 4)) | B_LOW;
                const uint32_t al = (lo0 + (uint32_t)lb * STAGE_STEP) | A_LOW, bl = (lo0 + (uint32_t)lb * STAGE_STEP + (uint32_t)(TILE >> 4)) | B_LOW;
                umma_tf32(d, desc(al, A_HIGH), desc(bh, B_HIGH), idesc, 0u);       // overwrites the buffer
#pragma unroll
                for (int j = 1; j < BK / 8; ++j) umma_tf32_acc(d, desc(al + j * A_STEP, A_HIGH), desc(bh + j * B_STEP, B_HIGH), idesc);
#pragma unroll
                for (int j = 0; j < BK / 8; ++j) umma_tf32_acc(d, desc(ah + j * A_STEP, A_HIGH), desc(bl + j * B_STEP, B_HIGH), idesc);
#pragma unroll
                for (int j = 0; j < BK / 8; ++j) umma_tf32_acc(d, desc(ah + j * A_STEP, A_HIGH), desc(bh + j * B_STEP, B_HIGH), idesc);
                umma_commit(smem_u32(done + rs));
                if (++rs == RAW_STAGES) { rs = 0; parity ^= 1u; }
                if (++lb == LO_BUFS) lb = 0;
            }
        }
    } else {
        // shared-memory offsets of this thread's pieces (same for every stage): mn_so 16-byte pieces of an M/N-major tile, g_so the
        // elements lane + 32 j that it copies (512 bytes apart), b_so pieces of a K-major tile.  Either way a warp owns rows
        // k = warp and warp + 16 of the M/N-major tiles, so that it splits what it copied.
        uint32_t mn_so[2], g_so[2], b_so[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int k = warp + 16 * i;
            const uint32_t krow = (uint32_t)((k >> 2) * MN_KATOM + (k & 3) * 128);
            mn_so[i] = krow + (uint32_t)((lane >> 3) * MN_ATOM + ((((lane & 7) >> 1) ^ (k & 3)) << 5) + ((lane & 1) << 4));
            g_so[i] = krow + (uint32_t)((((lane >> 3) ^ (k & 3)) << 5) + (((lane >> 2) & 1) << 4) + (lane & 3) * 4);
            b_so[i] = B_MN ? mn_so[i] : piece_offset((tid >> 3) + 64 * i, tid & 7);
        }
        const uint32_t smem_a0 = smem_u32(smem);
        GatherLoader<OP, BN> L;
        L.phase = 0;
        L.KB = 0;
        L.tile = (int)blockIdx.x;
        if (total_it > 0) L.setup(p, L.tile);
#pragma unroll
        for (int i = 0; i < PREFETCH; ++i) {
            if (i < total_it) {
                L.issue(p, smem_a0 + (uint32_t)(i * 2 * TILE), smem_a0 + (uint32_t)(i * 2 * TILE + TILE), g_so, b_so);
                L.advance(p);
            }
            cp_async_commit();
        }
        const int quarter = warp & 3, cg = warp >> 2;                        // TMEM lanes this warp may read; its columns
        const uint32_t tsrc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(cg * COLS);
        float acc[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
        int d_tile = (int)blockIdx.x, d_kb = 0, d_phase = 0;                 // the k-block to drain next
        while (d_phase + 1 < p.n_phases && d_tile >= p.ph[d_phase + 1].tile0) ++d_phase;
        // This lane's pixel of a tile, and the tile's first column for this warp; null: no pixel.
        auto locate = [&](int tile, const Phase &f, int &n0, int &im, int &row, int &col) -> float * {
            const int r0 = tile - f.tile0, m_tile = r0 / p.n_tiles, m = m_tile * BM + quarter * 32 + lane;
            n0 = (r0 - m_tile * p.n_tiles) * BN + cg * COLS;
            im = m / f.HW;
            const int r = m - im * f.HW;
            row = r / f.pix_W;
            col = r - row * f.pix_W;
            return m < f.M_total ? p.out + ((size_t)im * p.N_total + n0) * p.o_HW + (f.o_off + row * f.o_sH + col * f.o_sW) : nullptr;
        };
        bool nan_seen = false;
        // Adds k-block i's sums (its MMAs are done) to the registers; after a tile's last one, writes the tile.
        auto drain = [&](int i) {
            tc_fence_after();
            drain_block<COLS>(acc, tsrc + (uint32_t)((i & 1) * BN), d_kb == 0);
            tc_fence_before();
            const Phase &f = p.ph[d_phase];
            if (++d_kb < f.kblocks) return;
            int n0, im, row, col;
            if (float *dst = locate(d_tile, f, n0, im, row, col)) {
#pragma unroll
                for (int j = 0; j < COLS; ++j)
                    if (n0 + j < p.N_total) {
                        nan_seen |= acc[j] != acc[j];
                        dst[(size_t)j * p.o_HW] = acc[j] + (p.bias ? __ldg(p.bias + n0 + j) : 0.f);
                    }
            }
            d_kb = 0;
            d_tile += (int)gridDim.x;
            while (d_phase + 1 < p.n_phases && d_tile >= p.ph[d_phase + 1].tile0) ++d_phase;
        };
        bool ok = true;
        for (int i = 0; i < total_it; ++i) {
            const int rs = i % RAW_STAGES, lb = i % LO_BUFS;
            cp_async_wait<PREFETCH - 1>();                     // this thread's elements of k-block i are in shared memory
            if (i >= LO_BUFS) {
                // the MMAs of k-block i - 2 read this lo buffer; their sums are taken before k-block i is handed over
                const int j = i - LO_BUFS;
                if (!mbar_wait(smem_u32(done + j % RAW_STAGES), (uint32_t)((j / RAW_STAGES) & 1), p.status)) { ok = false; break; }
                drain(j);
            }
            __syncwarp();                                      // pieces were filled by several lanes of this warp
            unsigned char *a_hi = smem + (size_t)rs * 2 * TILE, *b_hi = a_hi + TILE;
            unsigned char *a_lo = lo_base + (size_t)lb * 2 * TILE, *b_lo = a_lo + TILE;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                split_rounded(a_hi, a_lo, mn_so[h], *reinterpret_cast<const float4 *>(a_hi + mn_so[h]));
                const bool b_on = B_MN ? lane * 4 < BN : (tid >> 3) + 64 * h < BN;
                if (b_on) split_rounded(b_hi, b_lo, b_so[h], *reinterpret_cast<const float4 *>(b_hi + b_so[h]));
            }
            fence_async_smem();                                // generic-proxy stores -> visible to the tensor core's async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(full + rs));
            // refill the raw stage that k-block i - 1 used with k-block i + PREFETCH, once its MMAs have read it
            if (i + PREFETCH < total_it) {
                if (i >= 1) {
                    const int j = i - 1;
                    if (!mbar_wait(smem_u32(done + j % RAW_STAGES), (uint32_t)((j / RAW_STAGES) & 1), p.status)) { ok = false; break; }
                }
                const uint32_t dst = smem_a0 + (uint32_t)((i + PREFETCH) % RAW_STAGES) * (2 * TILE);
                L.issue(p, dst, dst + TILE, g_so, b_so);
                L.advance(p);
            }
            cp_async_commit();
        }
        for (int j = max(0, total_it - LO_BUFS); ok && j < total_it; ++j) {
            if (!mbar_wait(smem_u32(done + j % RAW_STAGES), (uint32_t)((j / RAW_STAGES) & 1), p.status)) { ok = false; break; }
            drain(j);
        }
        cp_async_wait<0>();
        if (OP == OP_DGRAD && __any_sync(0xffffffffu, ok && nan_seen)) {
#pragma unroll 1
            for (int t = (int)blockIdx.x, f_i = 0; t < p.total_tiles; t += (int)gridDim.x) {
                while (f_i + 1 < p.n_phases && t >= p.ph[f_i + 1].tile0) ++f_i;
                const Phase &f = p.ph[f_i];
                int n0, im, row, col;
                float *dst = locate(t, f, n0, im, row, col);
                if (!dst) continue;
#pragma unroll 1
                for (int j = 0; j < COLS && n0 + j < p.N_total; ++j) {
                    const float b = p.bias ? __ldg(p.bias + n0 + j) : 0.f;
                    if (isnan(dst[(size_t)j * p.o_HW]) && !isnan(b)) dst[(size_t)j * p.o_HW] = gather_scalar(p, f, im, row, col, n0 + j) + b;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, TMEM_COLS);
}

// Sums of fewer products are taken in fp32.  The split and the truncation of a k-block's chain cost 8e-8 to 1.2e-7 of a sum however
// short it is, a chain of n fp32 FMAs about 1.8e-8 sqrt(n + 1): 7.4e-8 (fp32) and 9.3e-8 (tensor cores) at 16 products, 1.15e-7 and
// 1.19e-7 at 40, 1.27e-7 and 1.17e-7 at 48, 2.0e-7 and 1.3e-7 at 128 (2-norm, normal gy, weights of either sign).
constexpr int SHORT_SUM = 48;

// The same sums in plain fp32, products in the order tap row, tap column, filter: short ones, and what the tensor-core kernel does not take.
// blockIdx.y and z are the residues of the rows and columns, blockIdx.x a group of CH channels of blockDim.x of the residue's pixels.
// A thread reads one value of gy (neighbours in consecutive words) and CH weights (the same ones in a whole warp) for CH products.
constexpr int CH = 4, MAX_AXIS = 64;
struct FmaParams {
    const float *gy, *w, *bias;
    float *gx;
    const int *gate;
    int N, C, H, W, K, kW, kk, dH, dW, oH, oW, groups;
    int only_short;                                             // leave residues of SHORT_SUM products or more alone
    AxisPhase rows[MAX_AXIS], cols[MAX_AXIS];
};
__global__ void __launch_bounds__(256)
phase_fma_kernel(const __grid_constant__ FmaParams p)
{
    if (gated_off(p.gate)) return;
    const AxisPhase &a = p.rows[blockIdx.y], &b = p.cols[blockIdx.z];
    if (p.only_short && (long long)p.K * a.taps * b.taps >= SHORT_SUM) return;
    const int part = (int)blockIdx.x / p.groups, n0 = ((int)blockIdx.x - part * p.groups) * CH;
    const long long m = (long long)part * blockDim.x + threadIdx.x;
    const int pixels = a.n * b.n;
    if (m >= (long long)p.N * pixels) return;
    const int im = (int)(m / pixels), r = (int)(m - (long long)im * pixels), i = r / b.n, j = r - i * b.n;
    const float *src = p.gy + (size_t)im * p.K * p.oH * p.oW;
    int plane[CH];                                              // channels past the last repeat it
#pragma unroll
    for (int q = 0; q < CH; ++q) plane[q] = min(n0 + q, p.C - 1) * p.kk;
    float s[CH];
#pragma unroll
    for (int q = 0; q < CH; ++q) s[q] = 0.f;
#pragma unroll 1
    for (int th = 0; th < a.taps; ++th) {
        const int oh = a.o0 + i - th * a.ostep;
        if ((unsigned)oh >= (unsigned)p.oH) continue;
#pragma unroll 1
        for (int tw = 0; tw < b.taps; ++tw) {
            const int ow = b.o0 + j - tw * b.ostep;
            if ((unsigned)ow >= (unsigned)p.oW) continue;
            const float *g = src + oh * p.oW + ow, *w = p.w + (a.k0 + th * a.kstep) * p.kW + b.k0 + tw * b.kstep;
#pragma unroll 4
            for (int k = 0; k < p.K; ++k, g += p.oH * p.oW, w += (size_t)p.C * p.kk) {
                const float v = __ldg(g);
#pragma unroll
                for (int q = 0; q < CH; ++q) s[q] = fmaf(__ldg(w + plane[q]), v, s[q]);
            }
        }
    }
    float *dst = p.gx + ((size_t)im * p.C + n0) * p.H * p.W + (size_t)(a.h0 + i * p.dH) * p.W + (b.h0 + j * p.dW);
#pragma unroll
    for (int q = 0; q < CH; ++q)
        if (n0 + q < p.C) dst[(size_t)q * p.H * p.W] = s[q] + (p.bias ? __ldg(p.bias + n0 + q) : 0.f);
}

// Every pixel of every plane: the bias, or zero.
__global__ void __launch_bounds__(256)
plane_fill_kernel(float *__restrict__ out, const float *__restrict__ bias, int C, int HW, long long total)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x)
        out[i] = bias ? __ldg(bias + (int)((i / HW) % C)) : 0.f;
}

}  // namespace pwg
