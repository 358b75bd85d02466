// Depthwise convolution by staged planes: square 3x3, 5x5 and 7x7 kernels with stride 1 or 2, any padding, depth multiplier,
// map size and alignment — what the bulk-copy path (3x3, pad 1, multiplier 1, rows of 16-byte multiples) does not take.
//
// The passes move 4 bytes per element of x and y and do k * k multiply-adds per output.  The kernels for any shape read every tap
// through the cache with a bounds check (25 loads and 50 comparisons per output of a 5x5), and their parameter gradient reads
// both tensors once per tap.  Here a CTA copies the rows it needs once, asynchronously and with the padding as zeros, into
// shared memory, and a thread takes strips of TH = 4 outputs of one column: every staged value of the strip's columns is
// read once (40 reads for 100 multiply-adds of a 5x5 at stride 1, 55 at stride 2), taps and weights are unrolled registers and no
// bounds are checked.  At stride 2 even and odd columns are staged apart, so that a warp reads consecutive words.
//   forward      a tile is P consecutive planes of one image, or a band of rows of one plane
//   input grad   in padded coordinates h + pad = S q + a: gx[S q + a][S r + b] = sum_{t,u} w[a + S t][b + S u] gy[q - t][r - u];
//                a thread takes TH consecutive q of one r and writes their S * S residues, so no product with a zero is formed
//   param grad   a cluster of up to eight CTAs per filter shares the images; every thread keeps the k * k sums of its strips in
//                registers for at most kChain terms, then they go through fp64: the thread (3x3) or the warp (WarpSums), the CTA, the
//                cluster and onto the gradient; the bias sum is fp64 throughout.  The order is fixed, so results do not depend on timing.  Over 40 layers of
//                16 to 600 channels the error is that of the kernel for any shape, which has fp64 across threads and images: 3.5e-8 to
//                6e-8 against 3.5e-8 to 1.2e-7 (2-norm; chains of 32 terms: 4.3e-8 to 1.1e-7).
//
// Forward / input gradient / parameter gradient on a cold cache, in us: 32 x 96 x 57 x 43, 5x5 stride 2: 21 / 16 / 34 (38 MB a pass: 6 us;
// 35 / 30 / 52 with bounds and addresses worked out row by row, 671 in all for any shape); 12 x 144 x 37 x 29, 3x3 stride 1 (rows of an odd
// length): 10 / 10 / 14 (13 / 16 / 31).  What bounds them is issue and shared memory: 54 to 64 % of the issue slots, and forward 58 % of the
// cycles of shared memory, for 3,500 / 3,000 / 6,400 warp instructions a plane of 57 x 43 (7,900 / 4,800 / 10,600 before).  Two tiles in flight per CTA
// were 15 % slower; planes as they lie in memory, by bulk copies into a ring, took half the instructions and were faster for small planes
// (17 / 19 / 27) but up to twice slower for wide ones, which leave such a CTA few warps.
#pragma once

namespace plane {

constexpr int TH = 4;                        // outputs (forward, parameter gradient) or q rows (input gradient) per strip
constexpr int THREADS = 256;
constexpr int kTileFloats = 6144;            // staged floats per tile to aim at: 24 KB, so that several CTAs share an SM
constexpr int kMaxFloats = 11264;            // ... and the most a tile may take (44 KB)
constexpr int kChain = 8;                    // fp32 terms per sum before it goes through fp64

// Division of 0 <= k < 2^31 by a multiplication (Granlund and Montgomery, Division by Invariant Integers using Multiplication, 1994).
struct Divisor {
    uint32_t mul, shift;                     // mul 0: by one
    __device__ __forceinline__ int operator()(int k) const { return mul ? (int)(__umulhi((uint32_t)k, mul) >> shift) : k; }
};
static Divisor divisor_of(int d)
{
    if (d == 1) return {0u, 0u};
    uint32_t bits = 1;
    while ((1LL << bits) < d) ++bits;
    return {(uint32_t)(((1ull << (31 + bits)) + (unsigned)d - 1) / (unsigned)d), bits - 1};
}

struct Params {
    const float *in, *gy, *w, *bias;         // forward, parameter gradient: in = x; input gradient: in = gy
    float *out, *gw, *gb;
    int N, C, M, H, W, oH, oW, padH, padW;
    int P, groups;                           // planes of a tile (parameter gradient: images), tiles that cover C (N)
    int R, bands;                            // strip rows of a band (a multiple of TH), bands
    int rows, cols, half, ld;                // staged rows and columns per plane; stride 2: columns of one parity; floats per row
    int lanes;                               // log2 of the lanes that stage a row
    int base_q, base_r, cols_out;            // input gradient: first q and r; columns of strips
    int strips;                              // strips per band
    int ranks;                               // parameter gradient: CTAs of a filter
    Divisor by_bands, by_groups, by_filters;  // by bands, groups and M
    uint32_t cols_magic, strips_magic;
    float scale;
};

__device__ __forceinline__ int mdiv(int k, uint32_t magic) { return magic ? (int)__umulhi((uint32_t)k, magic) : k; }
__device__ __forceinline__ void copy4(uint32_t dst, const float *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_land()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

// A double in another CTA's shared memory.
__device__ __forceinline__ double cluster_ld(const double *local, int rank)
{
    uint32_t a;
    double v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}

// Stages `count` planes (plane i at src + i * step, h x w) from row row0 and column col0 on, zeros outside.
// A group of `1 << p.lanes` lanes takes a row, a lane two columns of it; what is inside is known beforehand, so that a copy costs an
// address and little else.  (Rows one by one, each with bounds and addresses of its own, took 90 instructions a row of 47 columns, three
// quarters of what the forward pass executed.)
template <int S>
__device__ __forceinline__ void stage_planes(const Params &p, float *tile, const float *src, long long step, int count, int h, int w, int row0,
                                             int col0)
{
    // rows and columns that are inside
    const int lo = min(max(-row0, 0), p.rows), nv = max(min(p.rows, h - row0) - lo, 0);
    const int left = min(max(-col0, 0), p.cols), nc = max(min(p.cols, w - col0) - left, 0);
    const int lanes = 1 << p.lanes, lane = (int)threadIdx.x & (lanes - 1), group = (int)threadIdx.x >> p.lanes, groups = THREADS >> p.lanes;
    const uint32_t base = smem_u32(tile) + (uint32_t)(lo * p.ld) * 4u, pitch = (uint32_t)p.ld * 4u, next = (uint32_t)lanes * (S == 1 ? 4u : 2u);
    const float *first = src + (long long)(row0 + lo) * w + (col0 + left);
    for (int k = lane; k < nc; k += 2 * lanes) {
        const int j = left + k;
        const bool two = k + lanes < nc;
        const float *s = first + k;
        const uint32_t d = base + (uint32_t)(S == 1 ? j : (j & 1) * p.half + (j >> 1)) * 4u;
        if (count == 1 || nv >= 2 * groups) {
            for (int pl = 0; pl < count; ++pl) {
                const float *si = s + pl * step + group * w;
                uint32_t di = d + (uint32_t)(pl * p.rows + group) * pitch;
#pragma unroll 2
                for (int i = group; i < nv; i += groups, si += groups * w, di += (uint32_t)groups * pitch) {
                    copy4(di, si);
                    if (two) copy4(di + next, si + lanes);
                }
            }
        } else if (nv > 0) {
            const uint32_t magic = nv == 1 ? 0u : 0xffffffffu / (uint32_t)nv + 1u;                      // exact for the few rows of a tile
            for (int q = group; q < count * nv; q += groups) {
                const int pl = mdiv(q, magic), i = q - pl * nv;
                const float *si = s + pl * step + i * w;
                const uint32_t di = d + (uint32_t)(pl * p.rows + i) * pitch;
                copy4(di, si);
                if (two) copy4(di + next, si + lanes);
            }
        }
    }
    if (nc < p.cols)
        for (int q = threadIdx.x; q < count * p.rows; q += THREADS)
            for (int k = 0; k < p.cols - nc; ++k) {
                const int j = k < left ? k : k + nc;
                tile[q * p.ld + (S == 1 ? j : (j & 1) * p.half + (j >> 1))] = 0.f;
            }
    if (nv < p.rows) {
        const int above = lo * p.ld, zeros = (p.rows - nv) * p.ld, skip = nv * p.ld, stride = count == 1 ? THREADS : 32;
        for (int pl = count == 1 ? 0 : (int)threadIdx.x >> 5; pl < count; pl += THREADS / 32)
            for (int e = (int)threadIdx.x & (stride - 1); e < zeros; e += stride) tile[pl * p.rows * p.ld + e + (e < above ? 0 : skip)] = 0.f;
    }
}

// Weights of `count` channels from c0 on, all M filters of each: slot (p * M + j) * WS; bad[slot]: a weight that is not finite,
// whose product with a padding zero must not be formed.
template <int K>
struct Weights {
    static constexpr int KK = K * K, WS = (KK + 3) & ~3;
    __device__ __forceinline__ static void stage(const Params &p, float *wsm, int *bad, int c0, int count)
    {
        for (int s = threadIdx.x; s < count * p.M; s += THREADS) bad[s] = 0;
        __syncthreads();
        for (int e = threadIdx.x; e < count * p.M * KK; e += THREADS) {
            const int s = e / KK, i = e - s * KK, pl = p.by_filters(s), j = s - pl * p.M;
            const float v = __ldg(p.w + ((size_t)j * p.C + c0 + pl) * KK + i);
            wsm[s * WS + i] = v;
            if (!(fabsf(v) <= 3.402823466e38f)) bad[s] = 1;
        }
    }
    __device__ __forceinline__ static void load(const float *wsm, int slot, float (&w)[WS])
    {
        const float4 *q = reinterpret_cast<const float4 *>(wsm + slot * WS);
#pragma unroll
        for (int i = 0; i < WS / 4; ++i) {
            const float4 v = q[i];
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
    }
};

template <int K, int S>
__global__ void __launch_bounds__(THREADS, 3)
fwd_kernel(const __grid_constant__ Params p)
{
    using WT = Weights<K>;
    extern __shared__ __align__(16) float sm[];
    float *wsm = sm;                                           // [P * M][WS], then flags, then the tile
    int *bad = reinterpret_cast<int *>(wsm + p.P * p.M * WT::WS);
    float *tile = reinterpret_cast<float *>(bad + ((p.P * p.M + 3) & ~3));
    const int unit = (int)blockIdx.x, ng = p.by_bands(unit), band = unit - ng * p.bands, n = p.by_groups(ng), g = ng - n * p.groups;
    const int c0 = g * p.P, planes = min(p.P, p.C - c0), r0 = band * p.R;
    stage_planes<S>(p, tile, p.in + ((long long)n * p.C + c0) * p.H * p.W, (long long)p.H * p.W, planes, p.H, p.W, r0 * S - p.padH, -p.padW);
    WT::stage(p, wsm, bad, c0, planes);
    copies_land();
    const int items = planes * p.M * p.strips * p.oW;
    for (int it = threadIdx.x; it < items; it += THREADS) {
        const int t2 = mdiv(it, p.cols_magic), ow = it - t2 * p.oW;
        const int slot = mdiv(t2, p.strips_magic), t0 = (t2 - slot * p.strips) * TH;
        const int pl = p.by_filters(slot), j = slot - pl * p.M, c = c0 + pl;
        const int oh0 = r0 + t0, cnt = min(TH, p.oH - oh0);
        if (cnt <= 0) continue;
        const float b = p.bias ? __ldg(p.bias + (size_t)j * p.C + c) : 0.f;
        float *dst = p.out + (((long long)n * p.C + c) * p.M + j) * p.oH * p.oW + (long long)oh0 * p.oW + ow;
        if (bad[slot]) {
            for (int t = 0; t < cnt; ++t)
                dst[(long long)t * p.oW] = fwd_point(p.in + ((long long)n * p.C + c) * p.H * p.W, p.w + ((size_t)j * p.C + c) * WT::KK, b, p.H, p.W, K, K,
                                                     (oh0 + t) * S - p.padH, ow * S - p.padW);
            continue;
        }
        float w[WT::WS];
        WT::load(wsm, slot, w);
        float acc[TH];
#pragma unroll
        for (int t = 0; t < TH; ++t) acc[t] = b;
        // row by row, so that an output adds its taps in the order of fwd_point: the same bits
        const float *row = tile + (pl * p.rows + t0 * S) * p.ld + ow;
#pragma unroll
        for (int r = 0; r < (TH - 1) * S + K; ++r, row += p.ld) {
            float v[K];
#pragma unroll
            for (int kw = 0; kw < K; ++kw) v[kw] = row[S == 1 ? kw : (kw & 1) * p.half + (kw >> 1)];
#pragma unroll
            for (int t = 0; t < TH; ++t) {
                if (r - t * S < 0 || r - t * S >= K) continue;
#pragma unroll
                for (int kw = 0; kw < K; ++kw) acc[t] = fmaf(w[(r - t * S) * K + kw], v[kw], acc[t]);
            }
        }
#pragma unroll
        for (int t = 0; t < TH; ++t, dst += p.oW)
            if (t < cnt) *dst = acc[t];
    }
}

template <int K, int S>
__global__ void __launch_bounds__(THREADS, 3)
dgrad_kernel(const __grid_constant__ Params p)
{
    using WT = Weights<K>;
    constexpr int T = (K + S - 1) / S;                          // taps of a residue, at most
    extern __shared__ __align__(16) float sm[];
    float *wsm = sm;
    int *bad = reinterpret_cast<int *>(wsm + p.P * p.M * WT::WS);
    float *tile = reinterpret_cast<float *>(bad + ((p.P * p.M + 3) & ~3));
    const int unit = (int)blockIdx.x, ng = p.by_bands(unit), band = unit - ng * p.bands, n = p.by_groups(ng), g = ng - n * p.groups;
    const int c0 = g * p.P, planes = min(p.P, p.C - c0), q0 = p.base_q + band * p.R;
    stage_planes<1>(p, tile, p.in + ((long long)n * p.C + c0) * p.M * p.oH * p.oW, (long long)p.oH * p.oW, planes * p.M, p.oH, p.oW, q0 - (T - 1),
                    p.base_r - (T - 1));
    WT::stage(p, wsm, bad, c0, planes);
    copies_land();
    const int items = planes * p.strips * p.cols_out;
    for (int it = threadIdx.x; it < items; it += THREADS) {
        const int t2 = mdiv(it, p.cols_magic), ri = it - t2 * p.cols_out;
        const int pl = mdiv(t2, p.strips_magic), t0 = (t2 - pl * p.strips) * TH;
        float acc[TH][S][S];
#pragma unroll
        for (int t = 0; t < TH; ++t)
#pragma unroll
            for (int a = 0; a < S; ++a)
#pragma unroll
                for (int b = 0; b < S; ++b) acc[t][a][b] = 0.f;
        bool any_bad = false;
        for (int j = 0; j < p.M; ++j) {
            const int slot = pl * p.M + j;
            any_bad |= bad[slot] != 0;
            float w[WT::WS];
            WT::load(wsm, slot, w);
            const float *row0 = tile + (slot * p.rows + t0) * p.ld + ri;
#pragma unroll
            for (int u = 0; u < T; ++u) {
#pragma unroll
                for (int rr = 0; rr < TH + T - 1; ++rr) {
                    const float v = row0[rr * p.ld + (T - 1 - u)];
#pragma unroll
                    for (int t = 0; t < TH; ++t) {
                        const int tt = t + T - 1 - rr;
                        if (tt < 0 || tt >= T) continue;
#pragma unroll
                        for (int a = 0; a < S; ++a)
#pragma unroll
                            for (int b = 0; b < S; ++b)
                                if (a + S * tt < K && b + S * u < K) acc[t][a][b] = fmaf(w[(a + S * tt) * K + b + S * u], v, acc[t][a][b]);
                    }
                }
            }
        }
        const int h0 = (q0 + t0) * S - p.padH, w0 = (p.base_r + ri) * S - p.padW;
        float *plane = p.out + ((long long)n * p.C + c0 + pl) * p.H * p.W;
        if (any_bad) {
#pragma unroll 1
            for (int e = 0; e < TH * S * S; ++e) {
                const int h = h0 + e / S, wi = w0 + e % S;
                if ((unsigned)h < (unsigned)p.H && (unsigned)wi < (unsigned)p.W)
                    plane[(long long)h * p.W + wi] = dgrad_point(p.in, p.w, n, c0 + pl, h, wi, p.C, p.M, K, K, S, S, p.padH, p.padW, p.oH, p.oW);
            }
            continue;
        }
        float *dst = plane + (long long)h0 * p.W + w0;
#pragma unroll
        for (int r = 0; r < TH * S; ++r, dst += p.W) {
            if ((unsigned)(h0 + r) >= (unsigned)p.H) continue;
#pragma unroll
            for (int b = 0; b < S; ++b)
                if ((unsigned)(w0 + b) < (unsigned)p.W) dst[b] = acc[r / S][r % S][b];
        }
    }
}

// Sums over a warp of SUMS values per lane, added up in fp64: those of a 3x3 filter in registers of each lane, more of them (which would
// leave an SM two CTAs for three) across the warp each time.  Across the warp, each of the five steps halves the values as well as the
// lanes that they still have to meet: a lane passes on half of its values and keeps the other half, so that SUMS = 25 takes 46 shuffles
// (250 for a butterfly per value) and every lane ends up with a sum or two of its own.  Of 5x5, 32 x 96 x 57 x 43: 35 us across the warp,
// 45 in registers; of 3x3, 12 x 144 x 37 x 29: 27 and 26.
template <int SUMS>
struct WarpSums {
    static constexpr bool OWN = SUMS <= 9;
    static constexpr int P = SUMS <= 16 ? 16 : (SUMS <= 32 ? 32 : 64), KEEP = P > 32 ? 2 : 1, N = OWN ? SUMS : KEEP;
    double mine[N];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int q = 0; q < N; ++q) mine[q] = 0.0;
    }
    template <class T>
    __device__ __forceinline__ static void across(const T (&acc)[SUMS], double (&v)[P / 2])
    {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int i = 0; i < P / 2; ++i) {
            const T a = i < SUMS ? acc[i < SUMS ? i : 0] : T(0), b = i + P / 2 < SUMS ? acc[i + P / 2 < SUMS ? i + P / 2 : 0] : T(0);
            v[i] = (double)(lane & 16 ? b : a) + (double)__shfl_xor_sync(0xffffffffu, lane & 16 ? a : b, 16);
        }
        int count = P / 2;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            if (count > KEEP) {
                count /= 2;
#pragma unroll
                for (int i = 0; i < P / 4; ++i)
                    if (i < count) {
                        const double a = v[i], b = v[i + count];
                        v[i] = (lane & o ? b : a) + __shfl_xor_sync(0xffffffffu, lane & o ? a : b, o);
                    }
            } else {
#pragma unroll
                for (int q = 0; q < KEEP; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
            }
        }
    }
    __device__ __forceinline__ void add(float (&acc)[SUMS])
    {
        if constexpr (OWN) {
#pragma unroll
            for (int i = 0; i < SUMS; ++i) mine[i] += (double)acc[i];
        } else {
            double v[P / 2];
            across(acc, v);
#pragma unroll
            for (int q = 0; q < KEEP; ++q) mine[q] += v[q];
        }
#pragma unroll
        for (int i = 0; i < SUMS; ++i) acc[i] = 0.f;
    }
    __device__ __forceinline__ void store(double *dst) const
    {
        const int lane = threadIdx.x & 31;
        double v[P / 2];
        if constexpr (OWN) across(mine, v);
#pragma unroll
        for (int q = 0; q < KEEP; ++q) {
            const int i = P == 16 ? lane >> 1 : KEEP * lane + q;
            if (i < SUMS) dst[i] = OWN ? v[q] : mine[q];
        }
    }
};

template <int K, int S>
__global__ void __launch_bounds__(THREADS, K == 7 ? 2 : 3)
wgrad_kernel(const __grid_constant__ Params p)
{
    constexpr int KK = K * K, SUMS = KK + 1;                                // the taps and the bias
    extern __shared__ __align__(16) float tile[];
    __shared__ double warp_sums[THREADS / 32][SUMS];
    __shared__ double cta_sums[SUMS];
    const int rank = cluster_rank(), ranks = cluster_size();
    const int jc = (int)blockIdx.x / ranks, j = jc / p.C, c = jc - j * p.C;
    const int warp = threadIdx.x >> 5;
    WarpSums<KK> sums;
    sums.clear();
    float acc[KK];
#pragma unroll
    for (int i = 0; i < KK; ++i) acc[i] = 0.f;
    double bias = 0.0;
    int chain = 0;
    const long long units = (long long)p.groups * p.bands;                  // (image group, band)
    const int u_end = (int)(units * (rank + 1) / ranks);
    for (int u = (int)(units * rank / ranks); u < u_end; ++u) {
        const int group = p.by_bands(u), band = u - group * p.bands, n0 = group * p.P, imgs = min(p.P, p.N - n0), r0 = band * p.R;
        const int items = imgs * p.strips * p.oW;
        // an item's gy, and where its strip starts in the tile: read while the tile, or the strip before, is on its way
        float next[TH];
        int at_next = 0;
        auto fetch = [&](int it) {
            if (it >= items) return;
            const int t2 = mdiv(it, p.cols_magic), ow = it - t2 * p.oW;
            const int pl = mdiv(t2, p.strips_magic), t0 = (t2 - pl * p.strips) * TH, oh0 = r0 + t0;
            const float *gp = p.gy + (((long long)(n0 + pl) * p.C + c) * p.M + j) * p.oH * p.oW + (long long)oh0 * p.oW + ow;
#pragma unroll
            for (int t = 0; t < TH; ++t, gp += p.oW) next[t] = oh0 + t < p.oH ? __ldg(gp) : 0.f;
            at_next = (pl * p.rows + t0 * S) * p.ld + ow;
        };
        stage_planes<S>(p, tile, p.in + ((long long)n0 * p.C + c) * p.H * p.W, (long long)p.C * p.H * p.W, imgs, p.H, p.W, r0 * S - p.padH, -p.padW);
        fetch(threadIdx.x);
        copies_land();
        for (int it0 = 0; it0 < items; it0 += THREADS) {
            if (chain + TH > kChain) { sums.add(acc); chain = 0; }
            chain += TH;
            const int it = it0 + (int)threadIdx.x;
            if (it >= items) continue;
            float gv[TH];
#pragma unroll
            for (int t = 0; t < TH; ++t) gv[t] = next[t];
            const float *row0 = tile + at_next;
            fetch(it + THREADS);
#pragma unroll
            for (int t = 0; t < TH; ++t) bias += (double)gv[t];
#pragma unroll
            for (int kw = 0; kw < K; ++kw) {
                const float *col = row0 + (S == 1 ? kw : (kw & 1) * p.half + (kw >> 1));
#pragma unroll
                for (int r = 0; r < (TH - 1) * S + K; ++r, col += p.ld) {
                    const float v = *col;
#pragma unroll
                    for (int t = 0; t < TH; ++t)
                        if (r - t * S >= 0 && r - t * S < K) acc[(r - t * S) * K + kw] = fmaf(gv[t], v, acc[(r - t * S) * K + kw]);
                }
            }
        }
        __syncthreads();                                                    // the tile is read before the next one lands in its place
    }
    // The CTA's sums; true if one of the filter's is not finite.
    auto gather = [&]() {
        sums.add(acc);
        sums.store(warp_sums[warp]);
        bias = warp_sum(bias);
        if ((threadIdx.x & 31) == 0) warp_sums[warp][KK] = bias;
        __syncthreads();
        bool bad = false;
        for (int i = threadIdx.x; i < SUMS; i += THREADS) {
            double s = 0.0;
            for (int w = 0; w < THREADS / 32; ++w) s += warp_sums[w][i];
            cta_sums[i] = s;
            bad |= i < KK && !isfinite(s);
        }
        return __syncthreads_or(bad) != 0;
    };
    if (gather()) {
        // The staged form also multiplies the padding's zeros by gy and the zeros past the last output by x: an infinity or a NaN there
        // reaches taps that never read it.  This CTA's share again, product by product.
        sums.clear();
        bias = 0.0;
        chain = 0;
#pragma unroll 1
        for (int u = (int)(units * rank / ranks); u < u_end; ++u) {
            const int band = u % p.bands, n0 = (u / p.bands) * p.P, imgs = min(p.P, p.N - n0), r0 = band * p.R;
            const int rows = min(p.R, p.oH - r0), items = imgs * rows * p.oW;
#pragma unroll 1
            for (int it0 = 0; it0 < items; it0 += THREADS) {
                if (++chain > kChain) { sums.add(acc); chain = 1; }
                const int it = it0 + (int)threadIdx.x;
                if (it >= items) continue;
                const int t2 = it / p.oW, ow = it - t2 * p.oW, pl = t2 / rows, oh = r0 + t2 - pl * rows;
                const long long n = n0 + pl;
                const float g = __ldg(p.gy + ((n * p.C + c) * p.M + j) * p.oH * p.oW + (long long)oh * p.oW + ow);
                const float *xp = p.in + (n * p.C + c) * p.H * p.W;
                const int ih0 = oh * S - p.padH, iw0 = ow * S - p.padW;
                bias += (double)g;
#pragma unroll
                for (int kh = 0; kh < K; ++kh)
#pragma unroll
                    for (int kw = 0; kw < K; ++kw)
                        if ((unsigned)(ih0 + kh) < (unsigned)p.H && (unsigned)(iw0 + kw) < (unsigned)p.W)
                            acc[kh * K + kw] = fmaf(g, __ldg(xp + (long long)(ih0 + kh) * p.W + iw0 + kw), acc[kh * K + kw]);
            }
        }
        gather();
    }
    cluster_sync();
    if (rank == 0) {
        for (int i = threadIdx.x; i < SUMS; i += THREADS) {
            double s = 0.0;
            for (int r = 0; r < ranks; ++r) s += cluster_ld(&cta_sums[i], r);
            float *dst = i < KK ? p.gw + (size_t)jc * KK + i : (p.gb ? p.gb + jc : nullptr);
            if (dst) *dst = (float)((double)*dst + (double)p.scale * s);
        }
    }
    cluster_sync();                                                         // shared memory outlives rank 0's reads
}

static uint32_t magic_of(int d) { return d == 1 ? 0u : (uint32_t)((1ull << 32) / (unsigned)d + 1u); }

enum Pass { FWD, DGRAD, WGRAD };

// Whether a planned pass is faster than the kernel for any shape, by straight lines fitted to 1,500 layers (maps of 3 to 900 columns, 1 to
// 1024 channels, 1 to 128 images; us on a busy stream).  A few channels, or maps of a few pixels, are over sooner there: staging takes an
// instruction per row and warp however short the row is, and nothing can be computed before it has landed.
// Forward of 128 x 600 x 5 x 4, 5x5: 17 us for any shape, 23 staged; of 3 x 2 x 113 x 143, three 3x3 filters: 8.4 and 9.4; of
// 70 x 560 x 9 x 9, 5x5 stride 2: 29 and 23; of 32 x 96 x 57 x 43, 5x5 stride 2: 54 and 21; parameter gradient of 1 x 3 x 46 x 40, 7x7
// stride 2: 4.4 and 7.9.  Over 1,500 other layers the passes that the rule picks take 1.01 / 1.002 / 1.006 times what the faster ones would.
static bool faster_than_any_shape(const Params &p, Pass pass, int K)
{
    const double sms = sm_count(), kk = K * K;
    const double rows_per_warp = (double)p.P * (pass == DGRAD ? p.M : 1) * p.rows * ((p.cols + 31) / 32) / (THREADS / 32);
    const double strips = std::ceil((double)p.P * (pass == FWD ? p.M : 1) * p.strips * p.cols_out / THREADS);
    if (pass == WGRAD) {
        const double ctas = (double)p.C * p.M * (kk + 1) / (sms * 8), loops = std::ceil((double)p.oH * p.oW / 256) * p.N;
        const double units = std::ceil((double)p.groups * p.bands / p.ranks), waves = std::max(1.0, (double)p.C * p.M * p.ranks / (sms * 3));
        return 3.4 + waves * (units * (0.147 * rows_per_warp + 0.015 * strips * kk) + 0.047 * kk) <
               2.5 + loops * (0.43 + (ctas > 1.0 ? 0.63 * ctas : 0.0));
    }
    const double full = (double)p.N * p.groups * p.bands / (sms * 3), weights = (double)p.P * p.M * kk / THREADS;
    if (pass == FWD) {
        const double threads = (double)p.N * p.C * p.M * p.oH * p.oW / (sms * 2048);
        return 3.7 + rows_per_warp * (0.004 + 0.037 * full) + strips * kk * (0.017 + 0.028 * full) + 1.9 * full + 0.22 * weights <
               1.1 * (2.2 + 0.076 * K + kk * (0.078 + 0.10 * threads + 0.10 * std::max(0.0, threads - 1.0)) + 2.1 * threads);
    }
    const double threads = (double)p.N * p.C * p.H * p.W / (sms * 2048);
    const double any = 1.3 + 0.43 * K * p.M + kk * p.M * (0.16 + 0.46 * threads + 0.02 * std::max(0.0, threads - 1.0));
    return 3.7 + 0.04 * K + rows_per_warp * (0.026 + 0.035 * full) + strips * p.M * kk * (0.012 + 0.023 * full) + 2.2 * full + 0.04 * weights < 1.1 * any;
}

// Fills the tile plan of a pass; false when the shape is left to the kernels for any shape: other kernel sizes and strides, rows so
// long that a strip's do not fit a tile, or where they are faster.
static bool plan(Params &p, Pass pass, int N, int C, int H, int W, int M, int kH, int kW, int dH, int dW, int padH, int padW, int oH, int oW)
{
    if (kH != kW || dH != dW || (kH != 3 && kH != 5 && kH != 7) || (dH != 1 && dH != 2)) return false;
    const int K = kH, S = dH, T = (K + S - 1) / S;
    p = Params{};
    p.N = N; p.C = C; p.M = M; p.H = H; p.W = W; p.oH = oH; p.oW = oW; p.padH = padH; p.padW = padW;
    int rows_out, halo, step;                                   // strip rows of a plane; staged rows = (R - 1) * step + halo
    if (pass == DGRAD) {
        p.base_q = padH / S; p.base_r = padW / S;
        rows_out = (padH + H - 1) / S - p.base_q + 1;
        p.cols_out = (padW + W - 1) / S - p.base_r + 1;
        p.cols = p.cols_out + T - 1;
        p.ld = p.cols;
        halo = T; step = 1;
    } else {
        rows_out = oH;
        p.cols_out = oW;
        p.cols = (oW - 1) * S + K;
        p.half = (p.cols + 1) / 2;
        p.ld = S == 1 ? p.cols : 2 * p.half;
        halo = K; step = S;
    }
    const int per_plane = pass == DGRAD ? M : 1;                // staged planes per plane of the tile
    const int wfloats = pass == WGRAD ? 0 : M * (((K * K + 3) & ~3) + 1) + 4;
    auto floats = [&](long long planes, long long R) { return planes * (per_plane * ((R - 1) * step + halo) * p.ld + wfloats); };
    const int whole = (rows_out + TH - 1) / TH * TH;
    if (floats(1, whole) <= kTileFloats) {
        p.R = whole; p.bands = 1;
        // enough strips for every thread, as long as the planes fit
        const int strips = whole / TH, want = (THREADS + strips * p.cols_out * (pass == FWD ? M : 1) - 1) / (strips * p.cols_out * (pass == FWD ? M : 1));
        const int most = pass == WGRAD ? N : C;
        p.P = 1;
        while (p.P < want && p.P < most && floats(p.P + 1, whole) <= kTileFloats) ++p.P;
        const long long one = (long long)strips * p.cols_out * (pass == FWD ? M : 1);
        // up to four rounds of strips, while CTAs for 2.75 on each SM remain: what a CTA does once counts for less.  12 x 144 x 37 x 29, 3x3:
        // 13 / 14 us with one plane, 10 / 11 with two, 8.4 / 10 with four, 10 / 12 with eight (forward / input gradient)
        if (pass != WGRAD)
            while (p.P < most && floats(p.P + 1, whole) <= kMaxFloats && (p.P + 1) * one <= 4 * THREADS &&
                   (long long)N * ceil_div(C, p.P + 1) * 4 >= 11LL * sm_count())
                ++p.P;
        else p.P = (int)std::min<long long>(N, kTileFloats / floats(1, whole));
    } else {
        int R = whole;
        while (R > TH && floats(1, R) > kTileFloats) R -= TH;
        if (floats(1, R) > kMaxFloats) return false;
        p.bands = (rows_out + R - 1) / R;
        p.R = ((rows_out + p.bands - 1) / p.bands + TH - 1) / TH * TH;      // even bands
        p.bands = (rows_out + p.R - 1) / p.R;
        p.P = 1;
    }
    p.rows = (p.R - 1) * step + halo;
    p.strips = p.R / TH;
    p.lanes = 3;                                                 // two columns a lane, if there are enough
    while (p.lanes < 8 && (2 << p.lanes) < p.cols) ++p.lanes;
    if (pass == WGRAD) {
        // CTAs of a filter and images of a unit: the fewest microseconds with the units shared out evenly, a start of 1.5 and 0.6 a unit;
        // w warps on an SM issue w / (w + 10) of what it can (0.48 with 9, 0.65 with 21, 0.77 with 29).  16 x 512 x 14 x 14, 5x5: 41 us with
        // images for one round of strips and as many CTAs as there are units, 23 so; 32 x 96 x 57 x 43, 5x5 stride 2: 39 and 31
        const long long sms = sm_count();
        const int per_sm = K == 7 ? 2 : 3, fit = p.P;
        double best = 0.0;
        for (int ranks = 1; ranks <= 8; ranks *= 2) {
            int groups = ceil_div(N, fit);
            if (p.bands == 1) groups = std::min(N, ceil_div(groups, ranks) * ranks);
            const int P = ceil_div(N, groups);
            groups = ceil_div(N, P);
            if ((long long)groups * p.bands < ranks) break;
            const double unit = 0.6 + 0.015 * K * K * std::ceil((double)P * p.strips * oW / THREADS) + 0.06 * P * p.rows * ((p.cols + 31) / 32) / (THREADS / 32);
            const long long ctas = (long long)C * M * ranks, together = std::min<long long>(per_sm, ceil_div_ll(ctas, sms));
            const double cost = (double)ceil_div_ll(ctas, sms * per_sm) * (1.5 + unit * ceil_div_ll((long long)groups * p.bands, ranks)) * (double)(8 * together + 10);
            if (best == 0.0 || cost < best) { best = cost; p.P = P; p.ranks = ranks; }
        }
    }
    p.groups = ((pass == WGRAD ? N : C) + p.P - 1) / p.P;
    p.cols_magic = magic_of(p.cols_out);
    p.strips_magic = magic_of(p.strips);
    p.by_bands = divisor_of(p.bands);
    p.by_groups = divisor_of(p.groups);
    p.by_filters = divisor_of(M);
    const long long items = (long long)p.P * (pass == FWD ? M : 1) * p.strips * p.cols_out;
    // exact divisions: items * divisor < 2^32 (see magic_of); grids within the launch limits
    if (items * std::max(p.cols_out, p.strips) >= (1LL << 32) || p.cols_out >= (1 << 16)) return false;
    if (pass != WGRAD && (long long)N * p.groups * p.bands >= (1LL << 31)) return false;
    if (pass == WGRAD && (long long)C * M * 8 >= (1LL << 31)) return false;
    return faster_than_any_shape(p, pass, K);
}
static size_t smem_bytes(const Params &p, Pass pass, int K)
{
    const size_t t = (size_t)p.P * (pass == DGRAD ? p.M : 1) * p.rows * p.ld;
    if (pass == WGRAD) return t * 4;
    const size_t slots = (size_t)p.P * p.M;
    return (slots * ((K * K + 3) & ~3) + ((slots + 3) & ~(size_t)3) + t) * 4;
}

typedef void (*Kernel)(const Params);
template <int K, int S>
static Kernel pick_pass(Pass pass)
{
    return pass == FWD ? fwd_kernel<K, S> : pass == DGRAD ? dgrad_kernel<K, S> : wgrad_kernel<K, S>;
}
static Kernel pick(Pass pass, int K, int S)
{
    if (K == 3) return S == 1 ? pick_pass<3, 1>(pass) : pick_pass<3, 2>(pass);
    if (K == 5) return S == 1 ? pick_pass<5, 1>(pass) : pick_pass<5, 2>(pass);
    return S == 1 ? pick_pass<7, 1>(pass) : pick_pass<7, 2>(pass);
}
static int launch(const Params &p, Pass pass, int K, int S, cudaStream_t stream)
{
    void *args[] = {(void *)&p};
    const Kernel kern = pick(pass, K, S);
    if (pass != WGRAD) {
        CUNN_CUDA(cudaLaunchKernel((const void *)kern, dim3((unsigned)((long long)p.N * p.groups * p.bands)), dim3(THREADS), args, smem_bytes(p, pass, K), stream));
        return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.C * p.M * p.ranks));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem_bytes(p, pass, K);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CUNN_CUDA(cudaLaunchKernelExC(&cfg, (const void *)kern, args));
    return 0;
}

}  // namespace plane
