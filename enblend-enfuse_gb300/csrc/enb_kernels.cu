// enb_kernels.cu -- sm_103a kernels of the enblend/enfuse multiresolution path.
//
// Integer stages reproduce the reference's fixed-point arithmetic exactly
// (src/pyramid.h, src/fixmath.h, src/blend.h, src/enfuse.h:601-620).  Where the
// reference rounds an IEEE double expression, the kernels either evaluate it
// with the same round-to-nearest double operations (__dmul_rn/__dadd_rn/
// __ddiv_rn, never contracted into FMAs) or with an exact integer/float
// formulation that provably yields the same result, falling back to the double
// expression in the rare cases the fast path cannot decide.
#include <cuda_runtime.h>
#include <stdint.h>

#include "enb_device.cuh"
#include "enb_internal.h"
#include "enb_entropy.cuh"
#include "enb_iweights.cuh"
#include "enb_reduce.cuh"
#include "enb_pixels.cuh"
#include "enb_tiles.cuh"

namespace enb {

// ---------------------------------------------------------------------------
// Conversions to fixed point (src/fixmath.h:116-206)
// ---------------------------------------------------------------------------

template <typename TS, typename TD>
__global__ void __launch_bounds__(256) k_to_fixed(const TS* src, int64_t spitch, int stride, int C, TD* dst,
                                                  int64_t dpitch, int64_t dplane, int w, int h, int frac)
{
    griddep_wait();
    griddep_launch();
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w) {
        return;
    }
    const TS* s = src + (int64_t)y * spitch + (int64_t)x * stride;
    for (int c = 0; c < C; ++c) {
        dst[(int64_t)c * dplane + (int64_t)y * dpitch + x] = (TD)((int32_t)s[c] << frac);
    }
}

template <typename TD>
__global__ void __launch_bounds__(256) k_float_to_fixed(const float* __restrict__ src, int64_t spitch,
                                                        TD* __restrict__ dst, int64_t dpitch, int w, int h,
                                                        int frac)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w) {
        return;
    }
    const double v = __dmul_rn((double)src[(int64_t)y * spitch + x], (double)(1u << frac));
    dst[(int64_t)y * dpitch + x] = frp_store<TD>(v);
}

// Soft-mask normalisation fused with the conversion of the mask to fixed
// point (src/enfuse.h:1526-1535 then fixmath.h:189-195).
template <typename TD>
__global__ void __launch_bounds__(256) k_soft_mask_to_fixed(const float* __restrict__ mask, int64_t mpitch,
                                                            const float* __restrict__ norm, int64_t npitch,
                                                            float fallback, TD* __restrict__ dst,
                                                            int64_t dpitch, int w, int h, int frac)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w) {
        return;
    }
    const float n = norm[(int64_t)y * npitch + x];
    const float m = n > 0.0f ? __fdiv_rn(__fmul_rn(255.0f, mask[(int64_t)y * mpitch + x]), n) : fallback;
    dst[(int64_t)y * dpitch + x] = mask_to_fixed<TD>(m, frac);
}

template <typename TD>
__global__ void __launch_bounds__(256) k_bytes_to_fixed(const uint8_t* __restrict__ src, int64_t spitch,
                                                        TD* __restrict__ dst, int64_t dpitch, int w, int h,
                                                        int frac)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w) {
        return;
    }
    dst[(int64_t)y * dpitch + x] = (TD)((int32_t)src[(int64_t)y * spitch + x] << frac);
}

__global__ void __launch_bounds__(256) k_alpha_extract(AlphaSrc a, uint8_t* __restrict__ dst, int64_t dpitch,
                                                       int w, int h)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w) {
        return;
    }
    dst[(int64_t)y * dpitch + x] = alpha_at(a, x, y) ? 255 : 0;
}

// Reduce (src/pyramid.h:166-848): k_reduce in enb_reduce.cuh.

// ---------------------------------------------------------------------------
// Expand (src/pyramid.h:875-1457)
// ---------------------------------------------------------------------------
//
// Destination pixel (X, Y) is a separable interpolation of the source:
// horizontally (1,6,1) at even X and (4,4) at odd X, vertically (1,6,1) at
// even Y and (1,1) at odd Y, divided by the product of the in-image weight
// sums (64 or 16 inside the image; 56, 49, 14, 8, ... at the borders).  One
// thread handles the 2x2 destination quad of one source pixel.
//
// The levels of a pyramid are a chain of these launches, most of them far
// below a wave, so the launch latency and the two load latencies counted:
// a launch of the chain loads what the one before it does not write (the
// destination samples; the source too when it subtracts, as level l + 1 is
// only replaced by the next launch) and waits after that.  Border tiles share
// the interior's arithmetic (TileWindow, QuadDivisors), where a quad at a
// border had computed its weights and divided per sample.  The eight adding
// launches of a 1921x1081 Int32 pyramid went from 92 to 60 us with event
// overhead, the sixteen subtracting ones of two pyramids from 167 to 121 us.

// The destination's samples before the operation: the level itself, or (for
// level 0 of a Laplacian pyramid) the pixels it is the conversion of, which
// saves writing and reading the converted level.  PAIR: a pixel pair is read
// as words (PixelPair), the image's base and pitch being multiples of theirs.
struct FineLevel {
    template <typename T, int C>
    __device__ __forceinline__ void load(const T* d, int64_t o, int64_t o1, int64_t plane, int, int, int, bool pair,
                                         bool x1, int32_t (&f)[C][4]) const
    {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const T *p = d + c * plane + o, *q = d + c * plane + o1;
            if (pair) {
                ld2<T, true>(p, f[c][0], f[c][1]);
                ld2<T, true>(q, f[c][2], f[c][3]);
            } else {
                f[c][0] = (int32_t)p[0];
                f[c][2] = (int32_t)q[0];
                f[c][1] = x1 ? (int32_t)p[1] : 0;
                f[c][3] = x1 ? (int32_t)q[1] : 0;
            }
        }
    }
};

template <typename TIn, int S, bool PAIR>
struct FinePixels {
    const TIn* p;
    int64_t pitch;
    int frac;
    template <typename T, int C>
    __device__ __forceinline__ void load(const T*, int64_t, int64_t, int64_t, int X, int Y, int Y1, bool, bool x1,
                                         int32_t (&f)[C][4]) const
    {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const TIn* row = p + (int64_t)(r ? Y1 : Y) * pitch + (int64_t)X * S;
            TIn px[2][S];
            if (PAIR && x1) {
                PixelPair<TIn, S>::load(row, px);
            } else {
                ld_px<TIn, S, false>(row, px[0]);
                ld_px<TIn, S, false>(x1 ? row + S : row, px[1]);
            }
#pragma unroll
            for (int c = 0; c < C; ++c) {
                f[c][2 * r] = (int32_t)px[0][c] << frac;
                f[c][2 * r + 1] = (int32_t)px[1][c] << frac;
            }
        }
    }
};

template <typename T>
struct ExpandArgs {
    const T* src;
    T* dst;
    int64_t spitch, splane, dpitch, dplane;
    int sw, sh, dw, dh, wrap;
    int pairs;    // destination rows hold aligned pairs
    int chained;  // the launch before on the stream is another of the chain
};

template <typename T, int C, bool ADD, class FINE>
__global__ void __launch_bounds__(256) k_expand(const __grid_constant__ ExpandArgs<T> a, const FINE fine)
{
    __shared__ int32_t ss[C][ESH][ESW];
    if (!a.chained) {
        griddep_wait();
    }
    griddep_launch();
    const int X0 = blockIdx.x * ETW, Y0 = blockIdx.y * ETH, I0 = X0 >> 1, J0 = Y0 >> 1;
    const int qx = threadIdx.x % 32, qy = threadIdx.x / 32;
    const int X = 2 * (I0 + qx), Y = 2 * (J0 + qy);
    const bool on = X < a.dw && Y < a.dh, y1 = Y + 1 < a.dh;
    const int Xc = min(X, a.dw - 1), Yc = min(Y, a.dh - 1), Y1 = min(Y + 1, a.dh - 1);
    const bool x1 = Xc == X && X + 1 < a.dw, pair = a.pairs && x1;
    const int64_t o = (int64_t)Yc * a.dpitch + Xc, o1 = (int64_t)Y1 * a.dpitch + Xc;
    const TileWindow win(I0, J0, a.sw, a.sh, a.spitch, a.dw, a.wrap);
    int32_t v[C][2], f[C][4];
    if (!ADD) {
        win.load<T, C>(a.src, a.splane, v);
    }
    fine.template load<T, C>(a.dst, o, o1, a.dplane, Xc, Yc, Y1, pair, x1, f);
    griddep_wait();
    if (ADD) {
        win.load<T, C>(a.src, a.splane, v);
    }
    win.store<C>(ss, v);
    __syncthreads();
    const auto body = [&](const auto& div) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            int32_t e[4];
            expand_window<false>(ss[c], qx, qy, div, e);
            T r[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                r[q] = ADD ? (T)sat_store<T>(f[c][q] + e[q]) : cast_store<T>((int64_t)f[c][q] - e[q]);
            }
            T *p = a.dst + c * a.dplane + o, *q = a.dst + c * a.dplane + o1;
            if (pair) {
                st2<T>(p, r[0], r[1]);
                if (y1) {
                    st2<T>(q, r[2], r[3]);
                }
            } else {
                p[0] = r[0];
                if (x1) {
                    p[1] = r[1];
                }
                if (y1) {
                    q[0] = r[2];
                    if (x1) {
                        q[1] = r[3];
                    }
                }
            }
        }
    };
    if (!on) {
        return;
    }
    if (interior_tile(X0, Y0, a.dw, a.dh, I0, J0, a.sw, a.sh)) {
        body(QuadInside{});
    } else {
        body(QuadDivisors(X, Y, a.sw, a.sh, a.dw, a.wrap));
    }
}

// ---------------------------------------------------------------------------
// Merge operators
// ---------------------------------------------------------------------------

// CartesianBlendFunctor (src/blend.h:41-76) in place on the black levels,
// evaluated by blend_sample (exact integer rounding, double only at ties).
// All levels in one launch, a run of four pixels a thread: the pass is bound by
// memory (nothing is read where the mask is 0, white is copied where it is
// full), and one launch a level and one pixel a thread took 77 us where this
// takes 24 (nine levels of 1921x1081 Int32, with event overhead).
struct BlendLevel {
    const void *m, *w;
    void* b;
    int64_t mpitch, wpitch, wplane, bpitch, bplane;
    int width, h;
    int runs;        // a row's runs of four pixels
    unsigned first;  // block
};

struct BlendLevels {
    BlendLevel l[kMaxLevels];
    int n;
    int32_t white_value;
};

template <typename T>
__device__ __forceinline__ void load4(const T* p, int32_t (&v)[4], int n)
{
    if (n == 4 && ((uintptr_t)p & (4 * sizeof(T) - 1)) == 0) {
        if (sizeof(T) == 4) {
            const int4 t = *reinterpret_cast<const int4*>(p);
            v[0] = t.x;
            v[1] = t.y;
            v[2] = t.z;
            v[3] = t.w;
        } else {
            const int2 t = *reinterpret_cast<const int2*>(p);
            v[0] = (int32_t)(int16_t)(t.x & 0xffff);
            v[1] = t.x >> 16;
            v[2] = (int32_t)(int16_t)(t.y & 0xffff);
            v[3] = t.y >> 16;
        }
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v[q] = q < n ? (int32_t)p[q] : 0;
        }
    }
}

template <typename T, typename TM, int C>
__global__ void __launch_bounds__(256) k_blend(const __grid_constant__ BlendLevels a)
{
    griddep_wait();
    griddep_launch();
    int l = 0;
    while (l + 1 < a.n && blockIdx.x >= a.l[l + 1].first) {
        ++l;
    }
    const BlendLevel& b = a.l[l];
    const unsigned i = (blockIdx.x - b.first) * 256 + threadIdx.x;
    const int y = (int)(i / (unsigned)b.runs), x = 4 * (int)(i - (unsigned)y * (unsigned)b.runs);
    if (y >= b.h) {
        return;
    }
    const int n = min(4, b.width - x);
    int32_t m[4];
    load4((const TM*)b.m + (int64_t)y * b.mpitch + x, m, n);
    if (max(max(m[0], m[1]), max(m[2], m[3])) <= 0) {
        return;
    }
    const bool white = min(min(m[0], m[1]), min(m[2], m[3])) >= a.white_value;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        T* p = (T*)b.b + c * b.bplane + (int64_t)y * b.bpitch + x;
        int32_t w[4], k[4];
        load4((const T*)b.w + c * b.wplane + (int64_t)y * b.wpitch + x, w, n);
        if (!white) {
            load4(p, k, n);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                w[q] = blend_sample<T>(m[q], a.white_value, w[q], k[q]);
            }
        }
        store4(p, w, n);
    }
}

template <typename T, typename TM, int C, int F>
__global__ void __launch_bounds__(256) k_mask_mul_acc(const T* __restrict__ lp, int64_t lpitch, int64_t lplane,
                                                      const TM* __restrict__ mask, int64_t mpitch,
                                                      T* __restrict__ res, int64_t rpitch, int64_t rplane, int w,
                                                      int h, int accumulate)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w) {
        return;
    }
    const int32_t m = (int32_t)mask[(int64_t)y * mpitch + x];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const T v = mask_multiply<T, F>((int32_t)lp[(int64_t)c * lplane + (int64_t)y * lpitch + x], m);
        T* r = &res[(int64_t)c * rplane + (int64_t)y * rpitch + x];
        *r = accumulate ? cast_store<T>((int64_t)*r + v) : v;
    }
}

// Generic (non-constant divisor) variant for the primitive entry point.
template <typename T, typename TM, int C>
__global__ void __launch_bounds__(256) k_mask_mul_acc_generic(const T* __restrict__ lp, int64_t lpitch,
                                                              int64_t lplane, const TM* __restrict__ mask,
                                                              int64_t mpitch, int32_t divisor,
                                                              T* __restrict__ res, int64_t rpitch, int64_t rplane,
                                                              int w, int h, int accumulate)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w) {
        return;
    }
    const double coeff = __ddiv_rn((double)mask[(int64_t)y * mpitch + x], (double)divisor);
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const T v = frp_store<T>(__dmul_rn((double)lp[(int64_t)c * lplane + (int64_t)y * lpitch + x], coeff));
        T* r = &res[(int64_t)c * rplane + (int64_t)y * rpitch + x];
        *r = accumulate ? cast_store<T>((int64_t)*r + v) : v;
    }
}

// ---------------------------------------------------------------------------
// Conversion from fixed point (src/fixmath.h:241-277)
// ---------------------------------------------------------------------------

template <typename TS, typename TD>
__global__ void __launch_bounds__(256) k_from_fixed(const TS* src, int64_t spitch, int64_t splane, int C,
                                                    const uint8_t* alpha, int64_t apitch, TD* dst, int64_t dpitch,
                                                    int dstride, int w, int h, int frac, int dither, uint64_t seed,
                                                    int32_t maxv)
{
    griddep_wait();
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w || !alpha[(int64_t)y * apitch + x]) {
        return;
    }
    const uint32_t key = dither_key(seed);
    const uint64_t pix = (uint64_t)y * (uint64_t)w + (uint64_t)x;
    const uint32_t pixbits = mix32((uint32_t)pix ^ key);
    for (int c = 0; c < C; ++c) {
        const int32_t v = (int32_t)src[(int64_t)c * splane + (int64_t)y * spitch + x];
        const uint32_t bits = dither_sample_bits(key, pixbits, pix, C, c, frac);
        dst[(int64_t)y * dpitch + (int64_t)x * dstride + c] =
            (TD)dither_rule(v, frac, dither == ENB_DITHER_NEAREST, bits, maxv);
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_copy_pixels(const T* __restrict__ src, int64_t spitch,
                                                     T* __restrict__ dst, int64_t dpitch, int rowlen, int h)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x < rowlen) {
        dst[(int64_t)y * dpitch + x] = src[(int64_t)y * spitch + x];
    }
}

// 4th component of an RGBA result: the union alpha scaled to the sample type,
// as the output writer stores the alpha image (src/assemble.h:133-225).
template <typename T>
__global__ void __launch_bounds__(256) k_alpha_component(const uint8_t* __restrict__ a, int64_t apitch,
                                                         T* __restrict__ dst, int64_t dpitch, int w, int h, T maxv)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x < w) {
        dst[(int64_t)y * dpitch + (int64_t)x * 4 + 3] = a[(int64_t)y * apitch + x] ? maxv : (T)0;
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_copy_level0(const T* __restrict__ src, int64_t spitch, int64_t splane,
                                                     int C, int32_t* __restrict__ dst, int w, int h)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w) {
        return;
    }
    for (int c = 0; c < C; ++c) {
        dst[((int64_t)y * w + x) * C + c] = (int32_t)src[(int64_t)c * splane + (int64_t)y * spitch + x];
    }
}

// ---------------------------------------------------------------------------
// enfuse weights (src/enfuse.h:962-1212)
// ---------------------------------------------------------------------------

// 32 x 16 output pixels per CTA, a pair of horizontally adjacent pixels per
// thread: fully opaque tiles take the pair path (enb_iweights.cuh), the
// others the per-pixel weight.
constexpr int EMX = 32, EMY = 16;

__host__ __device__ inline int emask_halo_x(const WeightParams& wp) { return (iweight_halo(wp) + 1) & ~1; }

__global__ void __launch_bounds__(256, 3) k_enfuse_mask(PixelView img, AlphaSrc alpha, WeightParams wp,
                                                        WeightTables tab, float* __restrict__ out, int64_t opitch)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int halo = iweight_halo(wp), hx = emask_halo_x(wp);
    const int TW = EMX + 2 * hx, TH = EMY + 2 * halo;
    const ITile t = itile_carve_rect(smem, TW, TH);
    long long* fx = reinterpret_cast<long long*>(smem + ((itile_bytes_rect(TW, TH) + 15) & ~(size_t)15));  // [32]
    const bool pair_path = iweight_pair_path(wp);
    if (wp.use_entropy && pair_path && (int)threadIdx.x <= wp.entropy_window * wp.entropy_window) {
        const int M = wp.entropy_window * wp.entropy_window;
        fx[threadIdx.x] = tab.plogp_fx[(int64_t)M * (M + 1) + threadIdx.x];
    }
    // ends with a barrier (which also publishes fx)
    const int opaque = itile_load_rect(t, wp, img, alpha, blockIdx.x * EMX - hx, blockIdx.y * EMY - halo);
    const int px = threadIdx.x % (EMX / 2), py = threadIdx.x / (EMX / 2);
    const int x = blockIdx.x * EMX + 2 * px, y = blockIdx.y * EMY + py;
    const int cx = hx + 2 * px, cy = halo + py;
    if (opaque && pair_path) {
        float w0, w1;
        pair_weights(t, wp, tab, fx, img.C, cx, cy, w0, w1);
        out[(int64_t)y * opitch + x] = w0;
        out[(int64_t)y * opitch + x + 1] = w1;
        return;
    }
    const int ci = cy * TW + cx;
    if (y < img.h && x < img.w) {
        out[(int64_t)y * opitch + x] = i_pixel_weight(t, wp, tab, img, ci, x, y);
    }
    if (y < img.h && x + 1 < img.w) {
        out[(int64_t)y * opitch + x + 1] = i_pixel_weight(t, wp, tab, img, ci + 1, x + 1, y);
    }
}

__global__ void __launch_bounds__(256) k_norm_accumulate(const float* __restrict__ m, int64_t mpitch,
                                                         float* __restrict__ norm, int64_t npitch, int w, int h,
                                                         int first)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w) {
        return;
    }
    const float v = m[(int64_t)y * mpitch + x];
    float* n = &norm[(int64_t)y * npitch + x];
    *n = first ? __fadd_rn(v, 0.0f) : __fadd_rn(v, *n);
}

__global__ void __launch_bounds__(256) k_union_alpha(const uint8_t* __restrict__ a, int64_t apitch,
                                                     uint8_t* __restrict__ u, int64_t upitch, int w, int h,
                                                     int first)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w) {
        return;
    }
    const uint8_t v = a[(int64_t)y * apitch + x];
    uint8_t* d = &u[(int64_t)y * upitch + x];
    if (first) {
        *d = v;
    } else if (v) {
        *d = v;
    }
}

constexpr int kMaxHardMasks = 64;
struct HardMaskArgs {
    float* p[kMaxHardMasks];
    int64_t pitch[kMaxHardMasks];
};

// Hard mask: argmax (first maximum) -> 255, others 0; all-zero -> 255/K
// (src/enfuse.h:1402-1442).
__global__ void __launch_bounds__(256) k_hard_mask(HardMaskArgs m, int K, int w, int h)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w) {
        return;
    }
    float mx = 0.0f;
    int mi = 0;
    for (int k = 0; k < K; ++k) {
        const float v = m.p[k][(int64_t)y * m.pitch[k] + x];
        if (v > mx) {
            mx = v;
            mi = k;
        }
    }
    const float fallback = __fdiv_rn(255.0f, (float)K);
    for (int k = 0; k < K; ++k) {
        m.p[k][(int64_t)y * m.pitch[k] + x] = mx == 0.0f ? fallback : (k == mi ? 255.0f : 0.0f);
    }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------

static inline dim3 row_grid(int w, int h) { return dim3((unsigned)((w + 255) / 256), (unsigned)h); }

LaunchInfo& last_launch()
{
    static thread_local LaunchInfo li{"", 0.0, 1};
    return li;
}

static inline double esz(int dt) { return dt == ENB_U8 ? 1.0 : ((dt == ENB_U16 || dt == ENB_I16) ? 2.0 : 4.0); }
static inline double npix(int w, int h) { return (double)w * (double)h; }
static inline double planar_bytes(const PlanarView& v) { return npix(v.w, v.h) * v.C * esz(v.dtype); }
static inline void note(const char* name, double bytes) { last_launch() = LaunchInfo{name, bytes, 1}; }

cudaError_t launch_to_fixed(const PixelView& s, const PlanarView& d, int frac, cudaStream_t st)
{
    if (s.dtype == ENB_F32 || d.dtype == ENB_F32) {
        if (s.dtype != d.dtype) {
            return cudaErrorInvalidValue;
        }
        return launch_f_to_pyramid(FloatPixelView{(const float*)s.p, s.pitch, s.w, s.h, s.C, s.stride}, d, st);
    }
    note("to_fixed", npix(s.w, s.h) * s.C * esz(s.dtype) + planar_bytes(d));
    const dim3 g = row_grid(s.w, s.h);
    if (s.dtype == ENB_U8 && d.dtype == ENB_I16) {
        (void)launch_pdl(k_to_fixed<uint8_t, int16_t>, g, dim3(256), st,
                         (const uint8_t*)s.p, s.pitch, s.stride, s.C, (int16_t*)d.p, d.pitch, d.plane, s.w, s.h, frac);
    } else if (s.dtype == ENB_U8 && d.dtype == ENB_I32) {
        (void)launch_pdl(k_to_fixed<uint8_t, int32_t>, g, dim3(256), st,
                         (const uint8_t*)s.p, s.pitch, s.stride, s.C, (int32_t*)d.p, d.pitch, d.plane, s.w, s.h, frac);
    } else if (s.dtype == ENB_U16 && d.dtype == ENB_I32) {
        (void)launch_pdl(k_to_fixed<uint16_t, int32_t>, g, dim3(256), st,
                         (const uint16_t*)s.p, s.pitch, s.stride, s.C, (int32_t*)d.p, d.pitch, d.plane, s.w, s.h, frac);
    } else if (s.dtype == ENB_U16 && d.dtype == ENB_I16) {
        (void)launch_pdl(k_to_fixed<uint16_t, int16_t>, g, dim3(256), st,
                         (const uint16_t*)s.p, s.pitch, s.stride, s.C, (int16_t*)d.p, d.pitch, d.plane, s.w, s.h, frac);
    } else {
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_bytes_to_fixed(const BytePlane& s, const PlanarView& d, int frac, cudaStream_t st)
{
    note("bytes_to_fixed", npix(s.w, s.h) + planar_bytes(d));
    const dim3 g = row_grid(s.w, s.h);
    if (d.dtype == ENB_I16) {
        k_bytes_to_fixed<int16_t><<<g, 256, 0, st>>>(s.p, s.pitch, (int16_t*)d.p, d.pitch, s.w, s.h, frac);
    } else {
        k_bytes_to_fixed<int32_t><<<g, 256, 0, st>>>(s.p, s.pitch, (int32_t*)d.p, d.pitch, s.w, s.h, frac);
    }
    return cudaGetLastError();
}

cudaError_t launch_float_to_fixed(const FloatPlane& s, const PlanarView& d, int frac, cudaStream_t st)
{
    note("float_to_fixed", 4.0 * npix(s.w, s.h) + planar_bytes(d));
    const dim3 g = row_grid(s.w, s.h);
    if (d.dtype == ENB_I16) {
        k_float_to_fixed<int16_t><<<g, 256, 0, st>>>(s.p, s.pitch, (int16_t*)d.p, d.pitch, s.w, s.h, frac);
    } else {
        k_float_to_fixed<int32_t><<<g, 256, 0, st>>>(s.p, s.pitch, (int32_t*)d.p, d.pitch, s.w, s.h, frac);
    }
    return cudaGetLastError();
}

cudaError_t launch_soft_mask_to_fixed(const FloatPlane& m, const FloatPlane& n, int K, const PlanarView& d,
                                      int frac, cudaStream_t st)
{
    note("soft_mask_to_fixed", 8.0 * npix(m.w, m.h) + planar_bytes(d));
    const dim3 g = row_grid(m.w, m.h);
    const float fallback = (float)(255 / K);  // integer division, src/enfuse.h:1534
    if (d.dtype == ENB_I16) {
        k_soft_mask_to_fixed<int16_t><<<g, 256, 0, st>>>(m.p, m.pitch, n.p, n.pitch, fallback, (int16_t*)d.p, d.pitch,
                                                         m.w, m.h, frac);
    } else {
        k_soft_mask_to_fixed<int32_t><<<g, 256, 0, st>>>(m.p, m.pitch, n.p, n.pitch, fallback, (int32_t*)d.p, d.pitch,
                                                         m.w, m.h, frac);
    }
    return cudaGetLastError();
}

cudaError_t launch_alpha_extract(const AlphaSrc& a, const BytePlane& d, cudaStream_t st)
{
    note("alpha_extract", npix(d.w, d.h) * (a.mode == kAlphaChannel3 ? 1.0 + esz(a.pix.dtype) : 1.0));
    k_alpha_extract<<<row_grid(d.w, d.h), 256, 0, st>>>(a, d.p, d.pitch, d.w, d.h);
    return cudaGetLastError();
}

template <typename T, int C>
static void reduce_dispatch(int wrap, const PlanarView& s, const BytePlane* sa, const PlanarView& d, const BytePlane* da,
                            cudaStream_t st)
{
    if (sa) {
        using Src = PlanarSource<T, C, true>;
        ReduceJobs<Src, T> jobs{};
        jobs.j[0] = ReduceJob<Src, T>{Src{(const T*)s.p, s.pitch, s.plane, sa->p, sa->pitch}, (T*)d.p, d.pitch, d.plane,
                                      da->p, da->pitch};
        launch_reduce_jobs<Src, T, C, true>(jobs, 1, s.w, s.h, d.w, d.h, wrap, st);
    } else {
        using Src = PlanarSource<T, C, false>;
        ReduceJobs<Src, T> jobs{};
        jobs.j[0] = ReduceJob<Src, T>{Src{(const T*)s.p, s.pitch, s.plane, nullptr, 0}, (T*)d.p, d.pitch, d.plane,
                                      nullptr, 0};
        launch_reduce_jobs<Src, T, C, false>(jobs, 1, s.w, s.h, d.w, d.h, wrap, st);
    }
}

cudaError_t launch_reduce(int wrap, const PlanarView& s, const BytePlane* sa, const PlanarView& d,
                          const BytePlane* da, cudaStream_t st)
{
    if (s.dtype != d.dtype || s.C != d.C || (sa == nullptr) != (da == nullptr)) {
        return cudaErrorInvalidValue;
    }
    note(sa ? "reduce_alpha" : "reduce",
         planar_bytes(s) + planar_bytes(d) + (sa ? npix(s.w, s.h) + npix(d.w, d.h) : 0.0));
    if (s.dtype == ENB_F32) {
        s.C == 1 ? reduce_dispatch<float, 1>(wrap, s, sa, d, da, st) : reduce_dispatch<float, 3>(wrap, s, sa, d, da, st);
    } else if (s.dtype == ENB_I16) {
        s.C == 1 ? reduce_dispatch<int16_t, 1>(wrap, s, sa, d, da, st) : reduce_dispatch<int16_t, 3>(wrap, s, sa, d, da, st);
    } else {
        s.C == 1 ? reduce_dispatch<int32_t, 1>(wrap, s, sa, d, da, st) : reduce_dispatch<int32_t, 3>(wrap, s, sa, d, da, st);
    }
    return cudaGetLastError();
}

template <typename T, typename TM, int C>
static void reduce_img2_mask_t(int wrap, const PlanarView& s0, const BytePlane& sa0, const PlanarView& d0,
                               const BytePlane& da0, const PlanarView& s1, const BytePlane& sa1, const PlanarView& d1,
                               const BytePlane& da1, const PlanarView& ms, const PlanarView& md, cudaStream_t st)
{
    using SrcI = PlanarSource<T, C, true>;
    using SrcM = PlanarSource<TM, 1, false>;
    ReduceJobs<SrcI, T> img{};
    img.j[0] = ReduceJob<SrcI, T>{SrcI{(const T*)s0.p, s0.pitch, s0.plane, sa0.p, sa0.pitch}, (T*)d0.p, d0.pitch,
                                  d0.plane, da0.p, da0.pitch};
    img.j[1] = ReduceJob<SrcI, T>{SrcI{(const T*)s1.p, s1.pitch, s1.plane, sa1.p, sa1.pitch}, (T*)d1.p, d1.pitch,
                                  d1.plane, da1.p, da1.pitch};
    const ReduceJob<SrcM, TM> msk{SrcM{(const TM*)ms.p, ms.pitch, ms.plane, nullptr, 0}, (TM*)md.p, md.pitch, md.plane,
                                  nullptr, 0};
    const dim3 g((unsigned)((d0.w + RDW - 1) / RDW), (unsigned)reduce_tile_rows(d0.h), 3u);
    (void)launch_pdl(k_reduce_img2_mask<SrcI, T, C, SrcM, TM>, g, dim3(RTHREADS), st, img, msk, s0.w, s0.h, d0.w,
                     d0.h, wrap);
}

cudaError_t launch_reduce_img2_mask(int wrap, const PlanarView& s0, const BytePlane& sa0, const PlanarView& d0,
                                    const BytePlane& da0, const PlanarView& s1, const BytePlane& sa1,
                                    const PlanarView& d1, const BytePlane& da1, const PlanarView& ms,
                                    const PlanarView& md, cudaStream_t st)
{
    const bool same = s0.w == s1.w && s0.h == s1.h && s0.w == ms.w && s0.h == ms.h && d0.w == d1.w && d0.h == d1.h &&
                      d0.w == md.w && d0.h == md.h && s0.dtype == s1.dtype && s0.dtype == d0.dtype &&
                      d1.dtype == d0.dtype && s0.C == s1.C && s0.C == d0.C && d1.C == d0.C && ms.C == 1 && md.C == 1 &&
                      ms.dtype == md.dtype && (s0.dtype == ENB_I16 || s0.dtype == ENB_I32) &&
                      (ms.dtype == ENB_I16 || ms.dtype == ENB_I32) && (s0.C == 1 || s0.C == 3);
    if (!same) {
        return cudaErrorInvalidValue;
    }
    note("reduce_level", planar_bytes(s0) + planar_bytes(d0) + planar_bytes(s1) + planar_bytes(d1) +
                             2.0 * (npix(s0.w, s0.h) + npix(d0.w, d0.h)) + planar_bytes(ms) + planar_bytes(md));
#define ENB_RIM(T, TM, CC) reduce_img2_mask_t<T, TM, CC>(wrap, s0, sa0, d0, da0, s1, sa1, d1, da1, ms, md, st)
    const bool m16 = ms.dtype == ENB_I16;
    if (s0.dtype == ENB_I16) {
        if (s0.C == 1) {
            if (m16) ENB_RIM(int16_t, int16_t, 1); else ENB_RIM(int16_t, int32_t, 1);
        } else {
            if (m16) ENB_RIM(int16_t, int16_t, 3); else ENB_RIM(int16_t, int32_t, 3);
        }
    } else {
        if (s0.C == 1) {
            if (m16) ENB_RIM(int32_t, int16_t, 1); else ENB_RIM(int32_t, int32_t, 1);
        } else {
            if (m16) ENB_RIM(int32_t, int16_t, 3); else ENB_RIM(int32_t, int32_t, 3);
        }
    }
#undef ENB_RIM
    return cudaGetLastError();
}

template <typename T, int C>
static cudaError_t reduce_tail_t(int wrap, int n, const PlanarView* s, const BytePlane* al, cudaStream_t st)
{
    TailJobs<T, T> j{};
    j.g.n = n;
    j.images = 1;
    for (int i = 0; i < n; ++i) {
        j.g.w[i] = s[i].w;
        j.g.h[i] = s[i].h;
        j.g.pitch[i] = s[i].pitch;
        j.img[0][i] = (T*)s[i].p;
        if (al) {
            j.g.apitch[i] = al[i].pitch;
            j.a[0][i] = al[i].p;
        }
    }
    return al ? launch_reduce_tail<T, C, T, kReduceAlpha, kReduceClamp>(j, 0, wrap, st)
              : launch_reduce_tail<T, C, T, kReduceClamp, kReduceClamp>(j, 0, wrap, st);
}

// A pyramid of the caller's may be of any shape and depth: the level's row of
// column sums has to fit, and the last kTailLevels levels are enough.
int pyramid_tail_level(const int* lw, const int* lh, int L, int dtype)
{
    int l = L > kTailLevels ? L - kTailLevels : 1;
    while (l < L && ((int64_t)lw[l] * lh[l] > kTailPixels || lw[l] > 512)) {
        ++l;
    }
    return dtype != ENB_F32 && l + 2 < L ? l : L;
}

cudaError_t launch_reduce_tail_levels(int wrap, int n, const PlanarView* s, const BytePlane* al, cudaStream_t st)
{
    bool fits = n >= 2 && n <= kTailLevels && s[0].dtype != ENB_F32;
    for (int i = 0; i < n && fits; ++i) {
        fits = (int64_t)s[i].w * s[i].h <= kTailPixels && s[i].w <= 512 && s[i].plane == s[i].pitch * s[i].h;
    }
    if (!fits) {
        return cudaErrorInvalidValue;
    }
    note("reduce_tail", 0.0);
    if (s[0].dtype == ENB_I16) {
        return s[0].C == 1 ? reduce_tail_t<int16_t, 1>(wrap, n, s, al, st) : reduce_tail_t<int16_t, 3>(wrap, n, s, al, st);
    }
    return s[0].C == 1 ? reduce_tail_t<int32_t, 1>(wrap, n, s, al, st) : reduce_tail_t<int32_t, 3>(wrap, n, s, al, st);
}

int enb_tail_level(const int* lw, const int* lh, int L) { return tail_level(lw, lh, L); }

template <typename T, typename TM, int C>
static cudaError_t reduce_img2_mask_tail_t(int wrap, int n, const PlanarView* s0, const BytePlane* a0, const PlanarView* s1,
                                           const BytePlane* a1, const PlanarView* ms, cudaStream_t st)
{
    TailJobs<T, TM> j{};
    j.g.n = n;
    j.images = 2;
    for (int i = 0; i < n; ++i) {
        j.g.w[i] = s0[i].w;
        j.g.h[i] = s0[i].h;
        j.g.pitch[i] = s0[i].pitch;
        j.g.apitch[i] = a0[i].pitch;
        j.img[0][i] = (T*)s0[i].p;
        j.img[1][i] = (T*)s1[i].p;
        j.a[0][i] = a0[i].p;
        j.a[1][i] = a1[i].p;
        j.msk[0][i] = (TM*)ms[i].p;
    }
    return launch_reduce_tail<T, C, TM, kReduceAlpha, kReduceClamp>(j, 1, wrap, st);
}

cudaError_t launch_reduce_img2_mask_tail(int wrap, int n, const PlanarView* s0, const BytePlane* a0, const PlanarView* s1,
                                         const BytePlane* a1, const PlanarView* ms, cudaStream_t st)
{
    // one geometry and row pitch a level for all three pyramids and both alphas
    bool same = n >= 2 && n <= kTailLevels && (int64_t)s0[0].w * s0[0].h <= kTailPixels;
    for (int i = 0; i < n; ++i) {
        same = same && s0[i].pitch == s1[i].pitch && s0[i].pitch == ms[i].pitch && a0[i].pitch == a1[i].pitch &&
               s0[i].plane == s0[i].pitch * s0[i].h && s1[i].plane == s0[i].plane;
    }
    if (!same) {
        return cudaErrorInvalidValue;
    }
    note("reduce_tail", 0.0);
#define ENB_RIT(T, TM, CC) return reduce_img2_mask_tail_t<T, TM, CC>(wrap, n, s0, a0, s1, a1, ms, st)
    if (s0[0].dtype == ENB_I16) {
        if (s0[0].C == 1) {
            ENB_RIT(int16_t, int16_t, 1);
        }
        ENB_RIT(int16_t, int16_t, 3);
    }
    if (s0[0].C == 1) {
        ENB_RIT(int32_t, int32_t, 1);
    }
    ENB_RIT(int32_t, int32_t, 3);
#undef ENB_RIT
}

template <typename T>
static ExpandArgs<T> expand_args(const PlanarView& s, const PlanarView& d, int wrap, bool chained)
{
    const bool pairs = (uintptr_t)d.p % (2 * sizeof(T)) == 0 && d.pitch % 2 == 0 && d.plane % 2 == 0;
    return ExpandArgs<T>{(const T*)s.p, (T*)d.p, s.pitch, s.plane, d.pitch, d.plane, s.w, s.h,
                         d.w, d.h, wrap, pairs, chained};
}

template <typename T, int C>
static cudaError_t expand_dispatch(int add, int wrap, const PlanarView& s, const PlanarView& d, bool chained,
                                   cudaStream_t st)
{
    const ExpandArgs<T> a = expand_args<T>(s, d, wrap, chained);
    return launch_pdl(add ? k_expand<T, C, true, FineLevel> : k_expand<T, C, false, FineLevel>,
                      grid2d(d.w, d.h, ETW, ETH), dim3(256), st, a, FineLevel{});
}

cudaError_t launch_expand(int add, int wrap, const PlanarView& s, const PlanarView& d, cudaStream_t st, bool chained)
{
    if (s.dtype != d.dtype || s.C != d.C) {
        return cudaErrorInvalidValue;
    }
    if (s.dtype == ENB_F32) {
        return launch_f_expand(add, wrap, s, d, st);
    }
    note(add ? "expand_add" : "expand_sub", planar_bytes(s) + 2.0 * planar_bytes(d));
    if (s.dtype == ENB_I16) {
        return s.C == 1 ? expand_dispatch<int16_t, 1>(add, wrap, s, d, chained, st)
                        : expand_dispatch<int16_t, 3>(add, wrap, s, d, chained, st);
    }
    return s.C == 1 ? expand_dispatch<int32_t, 1>(add, wrap, s, d, chained, st)
                    : expand_dispatch<int32_t, 3>(add, wrap, s, d, chained, st);
}

template <typename TIn, typename T, int C, int S>
static cudaError_t laplacian0_dispatch(const PixelView& px, int frac, int wrap, const PlanarView& g1, const PlanarView& l0,
                                       cudaStream_t st)
{
    const ExpandArgs<T> a = expand_args<T>(g1, l0, wrap, false);
    const dim3 g = grid2d(l0.w, l0.h, ETW, ETH);
    const TIn* p = (const TIn*)px.p;
    if (run_aligned<PixelPair<TIn, S>>(p, (size_t)px.pitch * sizeof(TIn))) {
        return launch_pdl(k_expand<T, C, false, FinePixels<TIn, S, true>>, g, dim3(256), st, a,
                          FinePixels<TIn, S, true>{p, px.pitch, frac});
    }
    return launch_pdl(k_expand<T, C, false, FinePixels<TIn, S, false>>, g, dim3(256), st, a,
                      FinePixels<TIn, S, false>{p, px.pitch, frac});
}

bool laplacian_takes_pixels(int px_dtype, int C, int stride, int dtype, int frac)
{
    const bool value = (px_dtype == ENB_U8 && dtype == ENB_I16 && frac <= 7) ||
                       (px_dtype == ENB_U16 && dtype == ENB_I32 && frac <= 15);
    return value && ((C == 1 && stride == 1) || (C == 3 && (stride == 3 || stride == 4)));
}

cudaError_t launch_laplacian0(const PixelView& px, int frac, int wrap, const PlanarView& g1, const PlanarView& l0,
                              cudaStream_t st)
{
    if (g1.dtype != l0.dtype || g1.C != l0.C || px.C != l0.C ||
        !laplacian_takes_pixels(px.dtype, px.C, px.stride, l0.dtype, frac)) {
        return cudaErrorInvalidValue;
    }
    note("laplacian0", npix(px.w, px.h) * px.stride * esz(px.dtype) + planar_bytes(g1) + planar_bytes(l0));
    if (px.dtype == ENB_U8) {
        return px.C == 1 ? laplacian0_dispatch<uint8_t, int16_t, 1, 1>(px, frac, wrap, g1, l0, st)
               : px.stride == 3 ? laplacian0_dispatch<uint8_t, int16_t, 3, 3>(px, frac, wrap, g1, l0, st)
                                : laplacian0_dispatch<uint8_t, int16_t, 3, 4>(px, frac, wrap, g1, l0, st);
    }
    return px.C == 1 ? laplacian0_dispatch<uint16_t, int32_t, 1, 1>(px, frac, wrap, g1, l0, st)
           : px.stride == 3 ? laplacian0_dispatch<uint16_t, int32_t, 3, 3>(px, frac, wrap, g1, l0, st)
                            : laplacian0_dispatch<uint16_t, int32_t, 3, 4>(px, frac, wrap, g1, l0, st);
}

cudaError_t launch_blend(int n, const PlanarView* m, const PlanarView* wt, const PlanarView* b, int32_t wv,
                         cudaStream_t st)
{
    double bytes = 0.0;
    for (int i = 0; i < n; ++i) {
        if (wt[i].dtype != b[0].dtype || wt[i].C != b[0].C || b[i].dtype != b[0].dtype || b[i].C != b[0].C ||
            m[i].dtype != m[0].dtype) {
            return cudaErrorInvalidValue;
        }
        bytes += planar_bytes(m[i]) + planar_bytes(wt[i]) + 2.0 * planar_bytes(b[i]);
    }
    if (n < 1 || n > kMaxLevels) {
        return cudaErrorInvalidValue;
    }
    if (b[0].dtype == ENB_F32) {
        for (int i = 0; i < n; ++i) {
            const cudaError_t e = m[i].dtype == ENB_I32 ? launch_f_blend(m[i], wt[i], b[i], wv, st) : cudaErrorInvalidValue;
            if (e != cudaSuccess) {
                return e;
            }
        }
        last_launch() = LaunchInfo{"blend", bytes, n};
        return cudaSuccess;
    }
    BlendLevels a{};
    a.n = n;
    a.white_value = wv;
    unsigned blocks = 0;
    for (int i = 0; i < n; ++i) {
        const int runs = (b[i].w + 3) / 4;
        a.l[i] = BlendLevel{m[i].p, wt[i].p, b[i].p, m[i].pitch, wt[i].pitch, wt[i].plane,
                            b[i].pitch, b[i].plane, b[i].w, b[i].h, runs, blocks};
        blocks += (unsigned)(((int64_t)runs * b[i].h + 255) / 256);
    }
    note("blend", bytes);
    const dim3 g(blocks), t(256);
    const bool m16 = m[0].dtype == ENB_I16;
    if (b[0].dtype == ENB_I16) {
        if (b[0].C == 1) {
            return launch_pdl(m16 ? k_blend<int16_t, int16_t, 1> : k_blend<int16_t, int32_t, 1>, g, t, st, a);
        }
        return launch_pdl(m16 ? k_blend<int16_t, int16_t, 3> : k_blend<int16_t, int32_t, 3>, g, t, st, a);
    }
    if (b[0].C == 1) {
        return launch_pdl(m16 ? k_blend<int32_t, int16_t, 1> : k_blend<int32_t, int32_t, 1>, g, t, st, a);
    }
    return launch_pdl(m16 ? k_blend<int32_t, int16_t, 3> : k_blend<int32_t, int32_t, 3>, g, t, st, a);
}

template <typename T, typename TM, int C>
static void mma_dispatch(const PlanarView& lp, const PlanarView& m, int32_t divisor, const PlanarView& r, int acc,
                         cudaStream_t st)
{
    const dim3 g = row_grid(lp.w, lp.h);
    if (divisor == (255 << 15)) {
        k_mask_mul_acc<T, TM, C, 15><<<g, 256, 0, st>>>((const T*)lp.p, lp.pitch, lp.plane, (const TM*)m.p, m.pitch,
                                                        (T*)r.p, r.pitch, r.plane, lp.w, lp.h, acc);
    } else if (divisor == (255 << 7)) {
        k_mask_mul_acc<T, TM, C, 7><<<g, 256, 0, st>>>((const T*)lp.p, lp.pitch, lp.plane, (const TM*)m.p, m.pitch,
                                                       (T*)r.p, r.pitch, r.plane, lp.w, lp.h, acc);
    } else {
        k_mask_mul_acc_generic<T, TM, C><<<g, 256, 0, st>>>((const T*)lp.p, lp.pitch, lp.plane, (const TM*)m.p,
                                                            m.pitch, divisor, (T*)r.p, r.pitch, r.plane, lp.w, lp.h,
                                                            acc);
    }
}

cudaError_t launch_mask_mul_acc(const PlanarView& lp, const PlanarView& m, int32_t divisor, const PlanarView& r,
                                int acc, cudaStream_t st)
{
    if (lp.dtype != r.dtype || lp.C != r.C) {
        return cudaErrorInvalidValue;
    }
    if (lp.dtype == ENB_F32) {
        return m.dtype == ENB_I32 ? launch_f_mask_mul_acc(lp, m, divisor, r, acc, st) : cudaErrorInvalidValue;
    }
    note("mask_mul_acc", planar_bytes(lp) + planar_bytes(m) + (acc ? 2.0 : 1.0) * planar_bytes(r));
    const bool m16 = m.dtype == ENB_I16;
    if (lp.dtype == ENB_I16) {
        if (lp.C == 1) {
            m16 ? mma_dispatch<int16_t, int16_t, 1>(lp, m, divisor, r, acc, st) : mma_dispatch<int16_t, int32_t, 1>(lp, m, divisor, r, acc, st);
        } else {
            m16 ? mma_dispatch<int16_t, int16_t, 3>(lp, m, divisor, r, acc, st) : mma_dispatch<int16_t, int32_t, 3>(lp, m, divisor, r, acc, st);
        }
    } else {
        if (lp.C == 1) {
            m16 ? mma_dispatch<int32_t, int16_t, 1>(lp, m, divisor, r, acc, st) : mma_dispatch<int32_t, int32_t, 1>(lp, m, divisor, r, acc, st);
        } else {
            m16 ? mma_dispatch<int32_t, int16_t, 3>(lp, m, divisor, r, acc, st) : mma_dispatch<int32_t, int32_t, 3>(lp, m, divisor, r, acc, st);
        }
    }
    return cudaGetLastError();
}

cudaError_t launch_from_fixed(const PlanarView& s, const BytePlane& a, void* dst, int64_t dpitch, int ddtype,
                              int dstride, int frac, int dither, uint64_t seed, cudaStream_t st)
{
    if (s.dtype == ENB_F32 || ddtype == ENB_F32) {
        if (s.dtype != ddtype) {
            return cudaErrorInvalidValue;
        }
        return launch_f_from_pyramid(s, a, (float*)dst, dpitch, dstride, st);
    }
    note("from_fixed", planar_bytes(s) + npix(s.w, s.h) * (1.0 + s.C * esz(ddtype)));
    const dim3 g = row_grid(s.w, s.h);
    if (s.dtype == ENB_I16) {
        if (ddtype == ENB_U8) {
            (void)launch_pdl(k_from_fixed<int16_t, uint8_t>, g, dim3(256), st,
                             (const int16_t*)s.p, s.pitch, s.plane, s.C, a.p, a.pitch, (uint8_t*)dst, dpitch, dstride,
                             s.w, s.h, frac, dither, seed, 255);
        } else {
            (void)launch_pdl(k_from_fixed<int16_t, uint16_t>, g, dim3(256), st,
                             (const int16_t*)s.p, s.pitch, s.plane, s.C, a.p, a.pitch, (uint16_t*)dst, dpitch, dstride,
                             s.w, s.h, frac, dither, seed, 65535);
        }
    } else {
        if (ddtype == ENB_U8) {
            (void)launch_pdl(k_from_fixed<int32_t, uint8_t>, g, dim3(256), st,
                             (const int32_t*)s.p, s.pitch, s.plane, s.C, a.p, a.pitch, (uint8_t*)dst, dpitch, dstride,
                             s.w, s.h, frac, dither, seed, 255);
        } else {
            (void)launch_pdl(k_from_fixed<int32_t, uint16_t>, g, dim3(256), st,
                             (const int32_t*)s.p, s.pitch, s.plane, s.C, a.p, a.pitch, (uint16_t*)dst, dpitch, dstride,
                             s.w, s.h, frac, dither, seed, 65535);
        }
    }
    return cudaGetLastError();
}

cudaError_t launch_copy_pixels(const PixelView& s, void* dst, int64_t dpitch, cudaStream_t st)
{
    const int rowlen = s.w * s.stride;
    note("copy_pixels", 2.0 * npix(rowlen, s.h) * esz(s.dtype));
    const dim3 g = row_grid(rowlen, s.h);
    if (s.dtype == ENB_U8) {
        k_copy_pixels<uint8_t><<<g, 256, 0, st>>>((const uint8_t*)s.p, s.pitch, (uint8_t*)dst, dpitch, rowlen, s.h);
    } else if (s.dtype == ENB_F32) {
        k_copy_pixels<uint32_t><<<g, 256, 0, st>>>((const uint32_t*)s.p, s.pitch, (uint32_t*)dst, dpitch, rowlen, s.h);
    } else {
        k_copy_pixels<uint16_t><<<g, 256, 0, st>>>((const uint16_t*)s.p, s.pitch, (uint16_t*)dst, dpitch, rowlen, s.h);
    }
    return cudaGetLastError();
}

cudaError_t launch_alpha_component(const BytePlane& a, void* dst, int64_t dpitch, int ddtype, cudaStream_t st)
{
    note("alpha_component", npix(a.w, a.h) * (1.0 + esz(ddtype)));
    const dim3 g = row_grid(a.w, a.h);
    if (ddtype == ENB_U8) {
        k_alpha_component<uint8_t><<<g, 256, 0, st>>>(a.p, a.pitch, (uint8_t*)dst, dpitch, a.w, a.h, (uint8_t)255);
    } else if (ddtype == ENB_F32) {
        // AlphaTraits<float>::max() = 1.0 (src/numerictraits.h:247)
        k_alpha_component<float><<<g, 256, 0, st>>>(a.p, a.pitch, (float*)dst, dpitch, a.w, a.h, 1.0f);
    } else {
        k_alpha_component<uint16_t><<<g, 256, 0, st>>>(a.p, a.pitch, (uint16_t*)dst, dpitch, a.w, a.h, (uint16_t)65535);
    }
    return cudaGetLastError();
}

cudaError_t launch_copy_level0(const PlanarView& s, int32_t* dst, cudaStream_t st)
{
    if (s.dtype == ENB_F32) {
        return launch_f_copy_level0(s, reinterpret_cast<float*>(dst), st);
    }
    note("copy_level0", planar_bytes(s) + 4.0 * npix(s.w, s.h) * s.C);
    const dim3 g = row_grid(s.w, s.h);
    if (s.dtype == ENB_I16) {
        k_copy_level0<int16_t><<<g, 256, 0, st>>>((const int16_t*)s.p, s.pitch, s.plane, s.C, dst, s.w, s.h);
    } else {
        k_copy_level0<int32_t><<<g, 256, 0, st>>>((const int32_t*)s.p, s.pitch, s.plane, s.C, dst, s.w, s.h);
    }
    return cudaGetLastError();
}

cudaError_t launch_enfuse_mask(const PixelView& img, const AlphaSrc& alpha, const WeightParams& wp,
                               const WeightTables& tab, const FloatPlane& out, cudaStream_t st)
{
    const int TW = EMX + 2 * emask_halo_x(wp), TH = EMY + 2 * iweight_halo(wp);
    const size_t smem = ((itile_bytes_rect(TW, TH) + 15) & ~(size_t)15) + 32 * sizeof(long long);
    note("enfuse_mask", npix(img.w, img.h) * (img.stride * esz(img.dtype) + (alpha.mode == kAlphaPlane ? 1.0 : 0.0) + 4.0));
    if (smem > 48 * 1024) {
        cudaFuncSetAttribute(k_enfuse_mask, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }
    k_enfuse_mask<<<grid2d(img.w, img.h, EMX, EMY), 256, smem, st>>>(img, alpha, wp, tab, out.p, out.pitch);
    return cudaGetLastError();
}

cudaError_t launch_norm_accumulate(const FloatPlane& m, const FloatPlane& n, int first, cudaStream_t st)
{
    note("norm_accumulate", npix(m.w, m.h) * (first ? 8.0 : 12.0));
    k_norm_accumulate<<<row_grid(m.w, m.h), 256, 0, st>>>(m.p, m.pitch, n.p, n.pitch, m.w, m.h, first);
    return cudaGetLastError();
}

cudaError_t launch_union_alpha(const BytePlane& a, const BytePlane& u, int first, cudaStream_t st)
{
    note("union_alpha", npix(a.w, a.h) * (first ? 2.0 : 3.0));
    k_union_alpha<<<row_grid(a.w, a.h), 256, 0, st>>>(a.p, a.pitch, u.p, u.pitch, a.w, a.h, first);
    return cudaGetLastError();
}

cudaError_t launch_hard_mask(const FloatPlane* masks, int K, cudaStream_t st)
{
    if (K > kMaxHardMasks) {
        return cudaErrorInvalidValue;
    }
    note("hard_mask", 8.0 * K * npix(masks[0].w, masks[0].h));
    HardMaskArgs a;
    for (int k = 0; k < K; ++k) {
        a.p[k] = masks[k].p;
        a.pitch[k] = masks[k].pitch;
    }
    k_hard_mask<<<row_grid(masks[0].w, masks[0].h), 256, 0, st>>>(a, K, masks[0].w, masks[0].h);
    return cudaGetLastError();
}

}  // namespace enb
