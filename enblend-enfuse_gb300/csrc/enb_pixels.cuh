// enb_pixels.cuh -- interleaved pixel I/O shared by the fused enblend and
// enfuse kernels: vector pixel loads and stores, the pixel's alpha (8-bit
// plane, opaque, or the thresholded 4th component, src/assemble.h:240-253)
// and the reduce source that converts pixels to fixed point on the fly.
#pragma once

#include <stdint.h>

#include "enb_device.cuh"

namespace enb {

// ---------------------------------------------------------------------------
// Pixel I/O
// ---------------------------------------------------------------------------

// Interleaved pixel load/store; VEC packs the 4 samples of an RGBA pixel in
// one 4- or 8-byte access (the caller checks the alignment).
template <typename TIn, int S, bool VEC>
__device__ __forceinline__ void ld_px(const TIn* p, TIn (&o)[S])
{
    if (VEC && S == 4 && sizeof(TIn) == 2) {
        const uint2 v = ld_dep(reinterpret_cast<const uint2*>(p));
        o[0] = (TIn)(v.x & 0xffffu);
        o[1] = (TIn)(v.x >> 16);
        o[2] = (TIn)(v.y & 0xffffu);
        o[S - 1] = (TIn)(v.y >> 16);
    } else if (VEC && S == 4 && sizeof(TIn) == 1) {
        const uint32_t v = ld_dep(reinterpret_cast<const uint32_t*>(p));
        o[0] = (TIn)(v & 0xffu);
        o[1] = (TIn)((v >> 8) & 0xffu);
        o[2] = (TIn)((v >> 16) & 0xffu);
        o[S - 1] = (TIn)(v >> 24);
    } else {
#pragma unroll
        for (int c = 0; c < S; ++c) {
            o[c] = ld_dep(&p[c]);
        }
    }
}

template <typename TIn, int S, bool VEC>
__device__ __forceinline__ void st_px(TIn* p, const TIn (&o)[S])
{
    if (VEC && S == 4 && sizeof(TIn) == 2) {
        uint2 v;
        v.x = (uint32_t)o[0] | ((uint32_t)o[1] << 16);
        v.y = (uint32_t)o[2] | ((uint32_t)o[S - 1] << 16);
        *reinterpret_cast<uint2*>(p) = v;
    } else if (VEC && S == 4 && sizeof(TIn) == 1) {
        *reinterpret_cast<uint32_t*>(p) =
            (uint32_t)o[0] | ((uint32_t)o[1] << 8) | ((uint32_t)o[2] << 16) | ((uint32_t)o[S - 1] << 24);
    } else {
#pragma unroll
        for (int c = 0; c < S; ++c) {
            p[c] = o[c];
        }
    }
}

// N (2 or 4) horizontally adjacent pixels (the first at a multiple of N) of an
// interleaved image as N*S*sizeof(TIn) / UNIT words of UNIT bytes (UNIT: the
// largest power of two, at most 16, dividing the run's size; the caller
// checks that the image's base and row pitch are multiples of it).
template <int U> struct PairWord;
template <> struct PairWord<2> { typedef uint16_t type; };
template <> struct PairWord<4> { typedef uint32_t type; };
template <> struct PairWord<8> { typedef uint2 type; };
template <> struct PairWord<16> { typedef uint4 type; };

template <typename TIn, int S, int N>
struct PixelRun {
    static constexpr int BYTES = N * S * (int)sizeof(TIn);
    static constexpr int UNIT = (BYTES % 16 == 0) ? 16 : (BYTES % 8 == 0) ? 8 : (BYTES % 4 == 0) ? 4 : 2;
    static constexpr int NW = BYTES / UNIT;
    typedef typename PairWord<UNIT>::type W;
    __device__ __forceinline__ static void load(const TIn* p, TIn (&px)[N][S])
    {
        union {
            W w[NW];
            TIn s[N * S];
        } u;
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            u.w[i] = ld_dep(reinterpret_cast<const W*>(p) + i);
        }
#pragma unroll
        for (int i = 0; i < N * S; ++i) {
            px[i / S][i % S] = u.s[i];
        }
    }
    __device__ __forceinline__ static void store(TIn* p, const TIn (&px)[N][S])
    {
        union {
            W w[NW];
            TIn s[N * S];
        } u;
#pragma unroll
        for (int i = 0; i < N * S; ++i) {
            u.s[i] = px[i / S][i % S];
        }
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            reinterpret_cast<W*>(p)[i] = u.w[i];
        }
    }
};

template <typename TIn, int S>
using PixelPair = PixelRun<TIn, S, 2>;

// Whether an image's base and row pitch (bytes) allow RUN's words.
template <class RUN>
inline bool run_aligned(const void* p, size_t pitch)
{
    return (uintptr_t)p % (size_t)RUN::UNIT == 0 && pitch % (size_t)RUN::UNIT == 0;
}

// Alpha of an interleaved pixel: 8-bit plane (AM 0), opaque (AM 1) or the
// thresholded 4th component (AM 2, src/assemble.h:240-253).
template <int AM, typename TIn, int S>
__device__ __forceinline__ int pixel_alpha(const TIn (&px)[S], const uint8_t* ap, int64_t apitch, int x, int y,
                                           uint32_t alo, uint32_t ahi)
{
    if (AM == 0) {
        return ld_dep(&ap[(int64_t)y * apitch + x]) != 0;
    }
    if (AM == 1) {
        return 1;
    }
    const uint32_t v = px[S - 1];
    return v >= alo && v <= ahi;
}

// Source of the tiled reduce: interleaved pixels converted to fixed point
// on the fly (copyToPyramidImage, src/fixmath.h:197-202).
template <typename TIn, int C, int S, int AM, bool VEC>
struct PixelSourceV {
    const TIn* p;
    int64_t pitch;
    const uint8_t* a;
    int64_t apitch;
    uint32_t lo, hi;
    int frac;
    __device__ __forceinline__ void load(int gy, int gx, int32_t (&v)[C], int& al) const
    {
        TIn px[S];
        ld_px<TIn, S, VEC>(p + (int64_t)gy * pitch + (int64_t)gx * S, px);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            v[c] = (int32_t)px[c] << frac;
        }
        al = pixel_alpha<AM, TIn, S>(px, a, apitch, gx, gy, lo, hi);
    }
};

}  // namespace enb
