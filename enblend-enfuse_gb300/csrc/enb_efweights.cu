// enb_efweights.cu -- the weight pass of the fused enfuse (enb_efuse.cu) for
// 8/16-bit images: the weights of all K exposures, their normalisation into
// level 0 of the mask pyramids and the union alpha.
//
// Three kernels give the same values:
//   * k_ef_weights_point, RGB images without windows (exposure and saturation
//     weights): four pixels a thread, no tile;
//   * k_ef_weights_quad, RGB images with contrast and entropy windows of 3 or
//     5 (or off): 2x2 pixels a thread on 32x32 tiles, whose windows share
//     columns and sorted rows;
//   * k_ef_weights, everything else: gray images, cutoffs, other window sizes,
//     loaded masks.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "enb_device.cuh"
#include "enb_internal.h"
#include "enb_iweights.cuh"
#include "enb_pixels.cuh"

namespace enb {

// ---------------------------------------------------------------------------
// weights of all exposures, normalisation, level-0 masks, union alpha
// ---------------------------------------------------------------------------

template <typename TM>
struct EfWeightsArgs {
    int K, w, h, hard, mfrac;
    PixelView img[kEfuseMaxK];
    AlphaSrc alpha[kEfuseMaxK];
    const float* min[kEfuseMaxK];
    int64_t mipitch[kEfuseMaxK];
    WeightParams wp;
    WeightTables tab;
    TM* m0[kEfuseMaxK];
    int64_t mpitch;
    uint8_t* u0;
    int64_t upitch;
    int vec;  // the images' bases and pitches allow the pixel runs of the kernel
};

// Output tile of the weight pass: 32 x 16 pixels, a pair of horizontally
// adjacent pixels per thread.
constexpr int EWX = 32, EWY = 16;

// Left and top margins of the weight tile: the windows' halo, the left one
// rounded up to even so that pair keys are word loads.
__host__ __device__ inline int ef_halo_x(const WeightParams& wp) { return (iweight_halo(wp) + 1) & ~1; }

template <typename TM>
__global__ void __launch_bounds__(256, 3) k_ef_weights(const __grid_constant__ EfWeightsArgs<TM> a)
{
    extern __shared__ __align__(16) unsigned char esmem[];
    // the call's first kernel: its buffers may be ones that the launch before still reads
    griddep_wait();
    griddep_launch();
    const int halo = iweight_halo(a.wp), hx = ef_halo_x(a.wp);
    const int TW = EWX + 2 * hx, TH = EWY + 2 * halo;
    const ITile t = itile_carve_rect(esmem, TW, TH);
    long long* fx = reinterpret_cast<long long*>(esmem + ((itile_bytes_rect(TW, TH) + 15) & ~(size_t)15));  // [32]
    float2* wk = reinterpret_cast<float2*>(fx + 32) + threadIdx.x;  // [K][256]
    const int px = threadIdx.x % (EWX / 2), py = threadIdx.x / (EWX / 2);
    const int x = blockIdx.x * EWX + 2 * px, y = blockIdx.y * EWY + py;
    const bool in0 = x < a.w && y < a.h, in1 = x + 1 < a.w && y < a.h;
    const int cx = hx + 2 * px, cy = halo + py;
    const int ci = cy * TW + cx;
    const int K = a.K;
    const bool pair_path = iweight_pair_path(a.wp);
    if (a.wp.use_entropy && pair_path && (int)threadIdx.x <= a.wp.entropy_window * a.wp.entropy_window) {
        // the p log p terms of full windows (n = W * W)
        const int M = a.wp.entropy_window * a.wp.entropy_window;
        fx[threadIdx.x] = a.tab.plogp_fx[(int64_t)M * (M + 1) + threadIdx.x];
    }
    uint32_t ua0 = 0, ua1 = 0;
    for (int k = 0; k < K; ++k) {
        if (a.min[k]) {
            // --load-masks: the loaded weight replaces enfuseMask (src/enfuse.h:1288-1331)
            const float* mrow = a.min[k] + (int64_t)y * a.mipitch[k];
            wk[k * 256] = make_float2(in0 ? ld_dep(&mrow[x]) : 0.0f, in1 ? ld_dep(&mrow[x + 1]) : 0.0f);
            ua0 |= in0 ? (uint32_t)alpha_at(a.alpha[k], x, y) : 0u;
            ua1 |= in1 ? (uint32_t)alpha_at(a.alpha[k], x + 1, y) : 0u;
            continue;
        }
        // ends with a barrier (which also publishes fx)
        const int opaque = itile_load_rect(t, a.wp, a.img[k], a.alpha[k], blockIdx.x * EWX - hx, blockIdx.y * EWY - halo);
        float w0 = 0.0f, w1 = 0.0f;
        if (opaque && pair_path) {
            // every window of the tile is whole and opaque: both pixels at once
            pair_weights(t, a.wp, a.tab, fx, a.img[k].C, cx, cy, w0, w1);
        } else {
            w0 = in0 ? i_pixel_weight(t, a.wp, a.tab, a.img[k], ci, x, y) : 0.0f;
            w1 = in1 ? i_pixel_weight(t, a.wp, a.tab, a.img[k], ci + 1, x + 1, y) : 0.0f;
        }
        wk[k * 256] = make_float2(w0, w1);
        ua0 |= t.a[ci];
        ua1 |= t.a[ci + 1];
        __syncthreads();  // the next exposure's load overwrites the tile
    }
    // normalisation (src/enfuse.h:1382-1385 sum in exposure order, 1399-1442
    // hard mask, 1526-1535 soft mask: float 255 * w / sum, integer 255 / K
    // where every weight is 0), then fromRealPromote(m * 2^F) into the mask
    // pyramid's level 0
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        if (!(q == 0 ? in0 : in1)) {
            continue;
        }
        const float* wq = reinterpret_cast<const float*>(wk) + q;
        const int64_t o = (int64_t)y * a.mpitch + x + q;
        if (a.hard) {
            float mx = 0.0f;
            int mi = 0;
            for (int k = 0; k < K; ++k) {
                if (wq[k * 512] > mx) {
                    mx = wq[k * 512];
                    mi = k;
                }
            }
            const float fallback = __fdiv_rn(255.0f, (float)K);
            for (int k = 0; k < K; ++k) {
                const float m = mx == 0.0f ? fallback : (k == mi ? 255.0f : 0.0f);
                a.m0[k][o] = mask_to_fixed<TM>(m, a.mfrac);
            }
        } else {
            float norm = 0.0f;
            for (int k = 0; k < K; ++k) {
                norm = __fadd_rn(wq[k * 512], norm);
            }
            const float fallback = (float)(255 / K);
            for (int k = 0; k < K; ++k) {
                const float m = norm > 0.0f ? __fdiv_rn(__fmul_rn(255.0f, wq[k * 512]), norm) : fallback;
                a.m0[k][o] = mask_to_fixed<TM>(m, a.mfrac);
            }
        }
        a.u0[(int64_t)y * a.upitch + x + q] = (q == 0 ? ua0 : ua1) ? 255 : 0;
    }
}


// ---------------------------------------------------------------------------
// RGB images: the common parts
// ---------------------------------------------------------------------------

// Masks of N horizontally adjacent pixels (x a multiple of N) from their K
// weights wk[k * ws + i]: as the end of k_ef_weights, with the words of a
// pixel run stored at once (rows of the mask planes are padded beyond it).
template <int N, typename TM>
__device__ __forceinline__ void ef_masks(const EfWeightsArgs<TM>& a, const float* wk, int ws, int x, int y)
{
    const int K = a.K;
    const int64_t o = (int64_t)y * a.mpitch + x;
    const auto put = [&](int k, const float (&m)[N]) {
        union {
            TM m[N];
            typename PairWord<N * (int)sizeof(TM)>::type w;
        } u;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            u.m[i] = mask_to_fixed<TM>(m[i], a.mfrac);
        }
        *reinterpret_cast<typename PairWord<N * (int)sizeof(TM)>::type*>(a.m0[k] + o) = u.w;
    };
    if (a.hard) {
        float mx[N];
        int mi[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            mx[i] = 0.0f;
            mi[i] = 0;
        }
        for (int k = 0; k < K; ++k) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const float w = wk[k * ws + i];
                if (w > mx[i]) {
                    mx[i] = w;
                    mi[i] = k;
                }
            }
        }
        const float fallback = __fdiv_rn(255.0f, (float)K);
        for (int k = 0; k < K; ++k) {
            float m[N];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                m[i] = mx[i] == 0.0f ? fallback : (k == mi[i] ? 255.0f : 0.0f);
            }
            put(k, m);
        }
        return;
    }
    float norm[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        norm[i] = 0.0f;
    }
    for (int k = 0; k < K; ++k) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            norm[i] = __fadd_rn(wk[k * ws + i], norm[i]);
        }
    }
    const float fallback = (float)(255 / K);
    for (int k = 0; k < K; ++k) {
        float m[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            m[i] = norm[i] > 0.0f ? __fdiv_rn(__fmul_rn(255.0f, wk[k * ws + i]), norm[i]) : fallback;
        }
        put(k, m);
    }
}

// Loads N pixels from (x, y), zero outside the image.
template <typename TIn, int S, int N>
__device__ __forceinline__ void ef_load_run(const PixelView& img, int vec, int x, int y, TIn (&px)[N][S])
{
    const TIn* p = reinterpret_cast<const TIn*>(img.p) + (int64_t)y * img.pitch + (int64_t)x * S;
    const bool row = y >= 0 && y < img.h;
    if (vec && row && x >= 0 && x + N <= img.w) {
        PixelRun<TIn, S, N>::load(p, px);
        return;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const bool in = row && x + i >= 0 && x + i < img.w;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            px[i][s] = in ? ld_dep(p + i * S + s) : (TIn)0;
        }
    }
}

// Whether pixel (x, y) inside the image, of samples px, is opaque.
template <typename TIn, int S>
__device__ __forceinline__ int ef_alpha(const AlphaSrc& al, const TIn (&px)[S], int x, int y)
{
    if (al.mode == kAlphaOpaque) {
        return 1;
    }
    if (S == 4 && al.mode == kAlphaChannel3) {
        const uint32_t v = px[S - 1];
        return v >= al.lo && v <= al.hi;
    }
    return alpha_at(al, x, y);
}

// ---------------------------------------------------------------------------
// exposure and saturation weights: no windows
// ---------------------------------------------------------------------------

// Four adjacent pixels a thread, 128 x 8 a CTA; the K weights wait in shared
// memory for their sum.  A stream of the images with the arithmetic of the
// saturation (about 25 instructions) behind it.  3 x 1024x768 u8: 19 us; the
// tile kernel, which loaded sample by sample, took 46 us.
template <typename TIn, typename TM, int S>
__global__ void __launch_bounds__(256) k_ef_weights_point(const __grid_constant__ EfWeightsArgs<TM> a)
{
    extern __shared__ __align__(16) unsigned char esmem[];
    griddep_wait();
    griddep_launch();
    float* wk = reinterpret_cast<float*>(esmem) + 4 * threadIdx.x;  // [K][256][4]
    const int x = blockIdx.x * 128 + 4 * (threadIdx.x % 32), y = blockIdx.y * 8 + threadIdx.x / 32;
    if (x >= a.w || y >= a.h) {
        return;
    }
    uint32_t ua = 0;  // bit i: pixel i opaque in some exposure
    TIn next[4][S];
    ef_load_run<TIn, S, 4>(a.img[0], a.vec, x, y, next);
    for (int k = 0; k < a.K; ++k) {
        TIn px[4][S];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int s = 0; s < S; ++s) {
                px[i][s] = next[i][s];
            }
        }
        if (k + 1 < a.K) {
            ef_load_run<TIn, S, 4>(a.img[k + 1], a.vec, x, y, next);
        }
        float w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            w[i] = 0.0f;
            if (x + i < a.w && ef_alpha<TIn, S>(a.alpha[k], px[i], x + i, y)) {
                ua |= 1u << i;
                const uint32_t r = px[i][0], g = px[i][1], b = px[i][2];
                if (a.wp.use_exposure) {
                    w[i] = __ldg(&a.tab.exposure[gray_of(a.wp, r, g, b)]);
                }
                if (a.wp.use_saturation) {
                    w[i] = __fadd_rn(saturation_of(a.wp, r, g, b), w[i]);
                }
            }
        }
        *reinterpret_cast<float4*>(wk + k * 1024) = make_float4(w[0], w[1], w[2], w[3]);
    }
    ef_masks<4, TM>(a, wk, 1024, x, y);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (x + i < a.w) {
            a.u0[(int64_t)y * a.upitch + x + i] = (ua >> i) & 1u ? 255 : 0;
        }
    }
}

// ---------------------------------------------------------------------------
// contrast and entropy windows of 3 or 5
// ---------------------------------------------------------------------------

// The exact value of one window's channel, out of line: it is rarely needed.
template <int EW>
static __device__ __noinline__ uint32_t entropy_exact(const uint16_t* raw, const uint8_t* a, int TW, int ci,
                                                      const WeightTables& tab, uint32_t maxv)
{
    return entropy_window_int<EW>(raw, a, TW, ci, tab, maxv);
}

constexpr int EQX = 32, EQY = 32;  // output tile

constexpr int kQuadBlocks = 4;  // CTAs an SM

template <int CW, int EW>
struct EfQuadTile {
    static constexpr int HALO = (CW > EW ? CW : EW) / 2;
    static constexpr int HX = (HALO + 1) & ~1;  // even, so that pairs of columns are aligned words
    static constexpr int TW = EQX + 2 * HX, TH = EQY + 2 * HALO, TT = TW * TH;
    static constexpr int RUNS = TW / 2 * TH, NP = (RUNS + 255) / 256;
    static constexpr size_t TILE = ((size_t)TT * (sizeof(int32_t) + 3 * sizeof(uint16_t) + 1) + 15) & ~(size_t)15;
};

// Loads exposure k's tile at (x0, y0): gray (0 where transparent), the samples
// (0xffff where transparent, when there are entropy windows) and the opaque
// flags; the image's outside is transparent.  Ends with a barrier; nonzero when every pixel of
// the tile inside the image is opaque (then every window that counts, which
// lies inside the image, is).
template <typename TIn, int S, int CW, int EW, bool ALPHA, typename TM>
__device__ __forceinline__ int ef_quad_load(const ITile& t, const EfWeightsArgs<TM>& a, int k, int x0, int y0)
{
    typedef EfQuadTile<CW, EW> Q;
    TIn px[Q::NP][2][S];
#pragma unroll
    for (int j = 0; j < Q::NP; ++j) {
        const int i = (int)threadIdx.x + 256 * j, r = i / (Q::TW / 2), c = 2 * (i - r * (Q::TW / 2));
        if (j * 256 + 256 <= Q::RUNS || i < Q::RUNS) {
            ef_load_run<TIn, S, 2>(a.img[k], a.vec, x0 + c, y0 + r, px[j]);
        }
    }
    int mine = 1;
#pragma unroll
    for (int j = 0; j < Q::NP; ++j) {
        const int i = (int)threadIdx.x + 256 * j, r = i / (Q::TW / 2), c = 2 * (i - r * (Q::TW / 2));
        if (!(j * 256 + 256 <= Q::RUNS || i < Q::RUNS)) {
            continue;
        }
        int al[2];
        int32_t g[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int x = x0 + c + q, y = y0 + r;
            const bool in = x >= 0 && x < a.w && y >= 0 && y < a.h;
            al[q] = in ? (ALPHA ? ef_alpha<TIn, S>(a.alpha[k], px[j][q], x, y) : 1) : 0;
            mine &= al[q] || !in;
            g[q] = al[q] ? gray_of(a.wp, px[j][q][0], px[j][q][1], px[j][q][2]) : 0;
        }
        const int p = r * Q::TW + c;
        *reinterpret_cast<int2*>(t.gray + p) = make_int2(g[0], g[1]);
        *reinterpret_cast<uchar2*>(t.a + p) = make_uchar2((unsigned char)al[0], (unsigned char)al[1]);
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            uint32_t v = (uint32_t)px[j][0][s] | ((uint32_t)px[j][1][s] << 16);
            if (ALPHA && EW > 0) {
                v |= (al[0] ? 0u : 0xffffu) | (al[1] ? 0u : 0xffff0000u);
            }
            *reinterpret_cast<uint32_t*>(t.raw + s * Q::TT + p) = v;
        }
    }
    if (!ALPHA) {
        __syncthreads();
        return 1;
    }
    return __syncthreads_and(mine);
}

// Bound by instructions, the min/max pairs of the sorting networks first.
// 9 x 6000x4000 u16, all weights, 5x5 windows: 8.0 ms, 911 instructions a pixel
// and exposure (12.7 ms and 1,546 with pairs of pixels, each window sorted by
// itself and every channel's entropy rounded); 5 x 2047x1535 u16 with alpha,
// contrast alone: 0.21 ms (0.45 ms).  Before the two instances below, at 8.4
// ms: four CTAs an SM (64 registers) beat three (8.7 ms) and two (9.4 ms); not
// kept: the next exposure's pixels in flight while one is weighted, as
// unaligned words (8.8 ms; 0.25 ms).
// ALPHA: some exposure has alpha.  Tiles with transparent pixels weight their
// quads too, with the taps of each window counted; evaluating their entropy
// windows one by one had taken 2.5 times as long as a pixel a thread does on
// images of a few tiles (9 x 400x300 u8 with holes everywhere, entropy 5x5: 0.92
// ms a call, now 0.33).  Stacks without alpha have an instance without that
// code: in one kernel for both they took 8.7 ms.
template <typename TIn, typename TM, int CW, int EW, bool ALPHA>
__global__ void __launch_bounds__(256, kQuadBlocks) k_ef_weights_quad(const __grid_constant__ EfWeightsArgs<TM> a)
{
    typedef EfQuadTile<CW, EW> Q;
    extern __shared__ __align__(16) unsigned char esmem[];
    __shared__ EntropyTables et;
    griddep_wait();
    griddep_launch();
    ITile t;
    t.TW = Q::TW;
    t.TT = Q::TT;
    t.gray = reinterpret_cast<int32_t*>(esmem);
    t.raw = reinterpret_cast<uint16_t*>(t.gray + Q::TT);
    t.a = reinterpret_cast<uint8_t*>(t.raw + 3 * Q::TT);
    float* wk = reinterpret_cast<float*>(esmem + Q::TILE) + 2 * threadIdx.x;  // [K][2 rows][256][2]
    const int px = threadIdx.x % (EQX / 2), py = threadIdx.x / (EQX / 2);
    const int x = blockIdx.x * EQX + 2 * px, y = blockIdx.y * EQY + 2 * py;
    const int cx = Q::HX + 2 * px, cy = Q::HALO + 2 * py, ci = cy * Q::TW + cx;
    if (EW > 0) {
        entropy_tables_load<(EW > 0 ? EW : 3)>(et, a.tab);  // published by the first load's barrier
    }
    uint32_t ua = 0;
    for (int k = 0; k < a.K; ++k) {
        const int x0 = blockIdx.x * EQX - Q::HX, y0 = blockIdx.y * EQY - Q::HALO;
        const int loaded = a.img[k].stride == 3 ? ef_quad_load<TIn, 3, CW, EW, ALPHA, TM>(t, a, k, x0, y0)
                                                : ef_quad_load<TIn, 4, CW, EW, ALPHA, TM>(t, a, k, x0, y0);
        const bool opaque = !ALPHA || loaded;
        float w[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (x < a.w && y < a.h) {
            const auto inside = [&](int q, int b) {  // q's window of half-width b lies in the image
                const int xx = x + (q & 1), yy = y + (q >> 1);
                return xx >= b && xx < a.w - b && yy >= b && yy < a.h - b;
            };
            if (a.wp.use_exposure) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    w[q] = __ldg(&a.tab.exposure[t.gray[ci + (q >> 1) * Q::TW + (q & 1)]]);
                }
            }
            if constexpr (CW > 0) {
                uint32_t g[4];
                if (opaque) {
                    contrast_quad<CW, true>(t.gray, t.a, Q::TW, cx, cy, g);
                } else {
                    contrast_quad<CW, false>(t.gray, t.a, Q::TW, cx, cy, g);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    w[q] = __fadd_rn(__ldg(&a.tab.contrast[inside(q, CW / 2) ? g[q] & a.wp.maxv : 0u]), w[q]);
                }
            }
            if (a.wp.use_saturation) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint16_t* p = t.raw + ci + (q >> 1) * Q::TW + (q & 1);
                    w[q] = __fadd_rn(saturation_of(a.wp, p[0], p[Q::TT], p[2 * Q::TT]), w[q]);
                }
            }
            if constexpr (EW > 0) {
                uint64_t v[4] = {~0ull, ~0ull, ~0ull, ~0ull};
                uint32_t counts = 0u;  // opaque taps of the four windows, 0: all
                if (!opaque) {
                    int n[4];
                    opaque_quad<EW>(t.a, Q::TW, cx, cy, n);
                    counts = (uint32_t)(n[0] | n[1] << 8 | n[2] << 16 | n[3] << 24);
                }
#pragma unroll 1
                for (int c = 0; c < 3; ++c) {
                    entropy_quad<EW>(t.raw + c * Q::TT, Q::TW, cx, cy, et, counts, a.tab, v);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    // the rounding is monotone, so that of the least value is the least of the roundings
                    // (entropy_fx_round); near a half-integer every channel's exact value decides
                    const uint32_t frac = (uint32_t)v[q];
                    const uint32_t dist = frac >= 0x80000000u ? frac - 0x80000000u : 0x80000000u - frac;
                    uint32_t m = min((uint32_t)(v[q] >> 32) + (frac >> 31), a.wp.maxv);
                    const int cq = ci + (q >> 1) * Q::TW + (q & 1);
                    if (!inside(q, EW / 2)) {
                        m = 0u;
                    } else if (dist <= (uint32_t)((counts ? (int)((counts >> (8 * q)) & 255u) : EW * EW) + 8)) {
                        m = a.wp.maxv;
                        for (int c = 0; c < 3 && t.a[cq]; ++c) {
                            m = min(m, entropy_exact<EW>(t.raw + c * Q::TT, t.a, Q::TW, cq, a.tab, a.wp.maxv));
                        }
                    }
                    w[q] = __fadd_rn(__ldg(&a.tab.entropy[m]), w[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                w[q] = t.a[ci + (q >> 1) * Q::TW + (q & 1)] ? w[q] : 0.0f;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                ua |= (uint32_t)t.a[ci + (q >> 1) * Q::TW + (q & 1)] << q;
            }
        }
        *reinterpret_cast<float2*>(wk + k * 1024) = make_float2(w[0], w[1]);
        *reinterpret_cast<float2*>(wk + k * 1024 + 512) = make_float2(w[2], w[3]);
        __syncthreads();  // the next exposure's load overwrites the tile
    }
    if (x >= a.w) {
        return;
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (y + r < a.h) {
            ef_masks<2, TM>(a, wk + 512 * r, 1024, x, y + r);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (x + i < a.w) {
                    a.u0[(int64_t)(y + r) * a.upitch + x + i] = (ua >> (2 * r + i)) & 1u ? 255 : 0;
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

static inline double esz_b(int dt) { return dt == ENB_U8 ? 1.0 : 2.0; }

template <typename K_>
static void allow_smem(K_ kernel, size_t smem)
{
    if (smem > 48 * 1024) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }
}

// The sample type of the images whose masks are TM.
template <typename TM> struct EfSample { typedef uint16_t type; };
template <> struct EfSample<int16_t> { typedef uint8_t type; };

// Whether every image allows runs of N pixels.
template <typename TIn, int S, int N>
static int ef_runs_aligned(const EfuseHost& h)
{
    bool ok = true;
    for (int k = 0; k < h.K; ++k) {
        ok = ok && run_aligned<PixelRun<TIn, S, N>>(h.img[k].p, (size_t)h.img[k].pitch * sizeof(TIn));
    }
    return ok;
}

// The kernels of RGB images (no cutoff, no loaded masks, windows of 3 or 5).
template <typename TIn, typename TM>
static cudaError_t ef_weights_rgb(EfWeightsArgs<TM>& a, const EfuseHost& h, cudaStream_t st)
{
    const int cw = h.wp.use_contrast ? h.wp.contrast_window : 0, ew = h.wp.use_entropy ? h.wp.entropy_window : 0;
    if (cw == 0 && ew == 0) {
        a.vec = h.S == 4 ? ef_runs_aligned<TIn, 4, 4>(h) : ef_runs_aligned<TIn, 3, 4>(h);
        auto k = h.S == 4 ? k_ef_weights_point<TIn, TM, 4> : k_ef_weights_point<TIn, TM, 3>;
        const size_t smem = (size_t)h.K * 1024 * sizeof(float);
        allow_smem(k, smem);
        return launch_pdl_smem(k, dim3((unsigned)((h.w + 127) / 128), (unsigned)((h.h + 7) / 8)), dim3(256), smem, st, a);
    }
    a.vec = h.S == 4 ? ef_runs_aligned<TIn, 4, 2>(h) : ef_runs_aligned<TIn, 3, 2>(h);
    const dim3 g((unsigned)((h.w + EQX - 1) / EQX), (unsigned)((h.h + EQY - 1) / EQY));
#define ENB_EQ(CWV, EWV)                                                                                    \
    if (cw == CWV && ew == EWV) {                                                                           \
        auto k = alpha ? k_ef_weights_quad<TIn, TM, CWV, EWV, true> : k_ef_weights_quad<TIn, TM, CWV, EWV, false>; \
        const size_t smem = EfQuadTile<CWV, EWV>::TILE + (size_t)h.K * 1024 * sizeof(float);                \
        allow_smem(k, smem);                                                                                \
        return launch_pdl_smem(k, g, dim3(256), smem, st, a);                                               \
    }
    bool alpha = false;
    for (int k = 0; k < h.K; ++k) {
        alpha = alpha || h.alpha[k].mode != kAlphaOpaque;
    }
    ENB_EQ(5, 5) ENB_EQ(5, 3) ENB_EQ(3, 5) ENB_EQ(3, 3) ENB_EQ(0, 5) ENB_EQ(0, 3) ENB_EQ(5, 0) ENB_EQ(3, 0)
#undef ENB_EQ
    return cudaErrorInvalidValue;
}

template <typename TM>
static cudaError_t ef_weights_t(const EfuseHost& h, cudaStream_t st)
{
    EfWeightsArgs<TM> a{};
    a.K = h.K;
    a.w = h.w;
    a.h = h.h;
    a.hard = h.hard;
    a.mfrac = h.dtype == ENB_U8 ? 7 : 15;
    for (int k = 0; k < h.K; ++k) {
        a.img[k] = h.img[k];
        a.alpha[k] = h.alpha[k];
        a.min[k] = h.masks_in[k];
        a.mipitch[k] = h.mipitch[k];
        a.m0[k] = (TM*)h.m[k][0];
    }
    a.wp = h.wp;
    a.tab = h.tab;
    a.mpitch = h.pitch[0];
    a.u0 = h.u[0];
    a.upitch = h.upitch0;
    if (h.C == 3 && !h.masks_in[0] && iweight_pair_path(h.wp) && !(h.wp.use_contrast && h.wp.contrast_window == 7)) {
        return ef_weights_rgb<typename EfSample<TM>::type, TM>(a, h, st);
    }
    const int TW = EWX + 2 * ef_halo_x(h.wp), TH = EWY + 2 * iweight_halo(h.wp);
    const size_t smem = ((itile_bytes_rect(TW, TH) + 15) & ~(size_t)15) + 32 * sizeof(long long) +
                        (size_t)h.K * 256 * sizeof(float2);
    allow_smem(k_ef_weights<TM>, smem);
    const dim3 g((unsigned)((h.w + EWX - 1) / EWX), (unsigned)((h.h + EWY - 1) / EWY));
    return launch_pdl_smem(k_ef_weights<TM>, g, dim3(256), smem, st, a);
}

cudaError_t launch_ef_weights(const EfuseHost& h, cudaStream_t st)
{
    const double px = (double)h.w * h.h;
    double in = 0.0;
    for (int k = 0; k < h.K; ++k) {
        in += h.masks_in[k] ? 4.0 : h.S * esz_b(h.dtype) + (h.alpha[k].mode == kAlphaPlane ? 1.0 : 0.0);
    }
    note_launch("ef_weights", px * (in + h.K * (h.dtype == ENB_U8 ? 2.0 : 4.0) + 1.0));
    return h.dtype == ENB_U8 ? ef_weights_t<int16_t>(h, st) : ef_weights_t<int32_t>(h, st);
}

}  // namespace enb
