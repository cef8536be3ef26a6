// enb_efuse.cu -- fused level passes of enfuse for 8/16-bit images.
//
// The reference (src/enfuse.h:1281-1617) computes each exposure's weight
// map, sums them, then per exposure builds the full Laplacian pyramid of the
// image and the Gaussian pyramid of its normalised mask, multiplies them
// level by level and adds the product into the result pyramid, and finally
// collapses it: the result pyramid is read and written once per exposure and
// every level of every pyramid is materialised.  Here
//   * one pass (enb_efweights.cu) computes the weights of all K exposures,
//     their sum, the normalised (or hard) masks as level 0 of the mask pyramids
//     and the union alpha;
//   * level 0 of no image pyramid is stored: the level-1 reduce reads the
//     interleaved pixels and converts them to fixed point on the fly; each
//     reduce launch covers the K exposures (blockIdx.z);
//   * each level l >= 1 is one pass: R_l = fromPromote(sum_k
//     fromRealPromote((G_k,l - E(G_k,l+1)) * M_k,l / D) + E(R_l+1)), the sum
//     wrapping in the pyramid type as the reference's accumulation does (the
//     order of the exposures does not change a modular sum);
//   * level 0 is one pass from the K images and level-0 masks and the
//     level-1 pyramids straight to the dithered output pixels.
// Every value is the same integer the reference computes: only the order of
// the passes over memory changes.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "enb_device.cuh"
#include "enb_internal.h"
#include "enb_pixels.cuh"
#include "enb_reduce.cuh"
#include "enb_tiles.cuh"

namespace enb {

// ---------------------------------------------------------------------------
// the top level and pixel pairs
// ---------------------------------------------------------------------------

// R of the top level, sum_k fromRealPromote(G_k M_k / D), at the thread's
// taps, from the staged windows of the K image pyramids (one level of a
// few pixels, not worth a launch and a trip through memory)
template <typename T, typename TM, int C, int F>
__device__ __forceinline__ void ef_top(const TileWindow& win, int32_t (*ss)[ESH][ESW], const TM* const* m, int K,
                                       int32_t (&v)[C][2])
{
#pragma unroll
    for (int c = 0; c < C; ++c) {
        v[c][0] = v[c][1] = 0;
    }
    for (int k = 0; k < K; ++k) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (win.f[u] == 0 || (u == 1 && !win.two)) {
                continue;
            }
            const int32_t mv = (int32_t)ld_dep(&m[k][win.o[u]]);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int32_t g = (&ss[k * C + c][0][0])[threadIdx.x + 256 * u] / win.f[u];
                v[c][u] += (int32_t)mask_multiply<T, F>(g, mv);
            }
        }
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
        v[c][0] = (int32_t)cast_store<T>(v[c][0]);
        v[c][1] = (int32_t)cast_store<T>(v[c][1]);
    }
}

// Two adjacent samples of a planar level or mask (x even).
template <typename T>
__device__ __forceinline__ void ld_pair(const T* p, int32_t& a, int32_t& b)
{
    ld2<T, true>(p, a, b);
}

// ---------------------------------------------------------------------------
// levels L-2 .. 1: Laplacians, mask products, accumulation and collapse
// ---------------------------------------------------------------------------

template <typename T, typename TM>
struct EfLevelArgs {
    int K, dw, dh, cw, ch, wrap;
    const T* g[kEfuseMaxK];   // level l of the image pyramids
    const T* gc[kEfuseMaxK];  // level l + 1
    const TM* m[kEfuseMaxK];  // level l of the mask pyramids
    const T* rc;              // R[l + 1]
    const TM* mc[kEfuseMaxK]; // level l + 1 of the mask pyramids
    T* r;                     // R[l]
    int64_t pitch, plane, cpitch, cplane;
};

// One 64x16 tile of level l (256 threads, one 2x2 quad each): the K coarse
// windows of every channel are staged together (one barrier), the exposures'
// products summed, and only then the launch waits for its predecessor, which
// wrote R_l+1.  The first of these launches (FOLD) waits for the reduces
// before it lets the next start, the others let theirs start at once: every
// input but R_l+1 is complete by then, the small levels' sums run side by
// side, and from level to level only the expansion of R remains.  ss holds
// (K + 1) * C windows.
// Bound by instructions, about a hundred per exposure, channel and quad; one
// division table entry per quad serves every border expansion, so that the
// small levels, all border, cost no more than the large ones.  The eight
// levels of 9 x 6000x4000 u16 take 0.46 ms (3.2 TB/s; 1.28 ms with a staging
// loop per window, per-position border weights and the wait up front), the six
// of 3 x 1024x768 u8 75 us with event overhead (157 us).
// FOLD: level l + 1 is the top and its R is formed here.
template <typename T, typename TM, int C, int F, bool FOLD>
__global__ void __launch_bounds__(256, 3) k_ef_up(const __grid_constant__ EfLevelArgs<T, TM> a)
{
    extern __shared__ __align__(16) int32_t ewin[];
    int32_t (*ss)[ESH][ESW] = reinterpret_cast<int32_t (*)[ESH][ESW]>(ewin);
    if (FOLD) {
        griddep_wait();  // the launch before wrote the top level
    }
    griddep_launch();
    const int K = a.K;
    const int X0 = blockIdx.x * ETW, Y0 = blockIdx.y * ETH;
    const int I0 = X0 >> 1, J0 = Y0 >> 1;
    const int qx = threadIdx.x % 32, qy = threadIdx.x / 32;
    const int X = 2 * (I0 + qx), Y = 2 * (J0 + qy);
    const bool on = X < a.dw && Y < a.dh;
    // the quad's first pixel, its second row (the first again below the level);
    // both pixels of a quad row in one paired load where x + 1 is inside
    const int64_t off = (int64_t)min(Y, a.dh - 1) * a.pitch + min(X, a.dw - 1);
    const int64_t off2 = Y + 1 < a.dh ? off + a.pitch : off;
    const bool pair = X + 1 < a.dw;
    // the fine values of exposure k: mask m[4], image g[C][4]
    const auto fetch = [&](int k, int32_t (&m)[4], int32_t (&g)[C][4]) {
        if (pair) {
            ld_pair<TM>(a.m[k] + off, m[0], m[1]);
            ld_pair<TM>(a.m[k] + off2, m[2], m[3]);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                ld_pair<T>(a.g[k] + c * a.plane + off, g[c][0], g[c][1]);
                ld_pair<T>(a.g[k] + c * a.plane + off2, g[c][2], g[c][3]);
            }
        } else {  // the last column of an odd level: only pixels 0 and 2 exist
            m[0] = m[1] = (int32_t)ld_dep(&a.m[k][off]);
            m[2] = m[3] = (int32_t)ld_dep(&a.m[k][off2]);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                g[c][0] = g[c][1] = (int32_t)ld_dep(&a.g[k][c * a.plane + off]);
                g[c][2] = g[c][3] = (int32_t)ld_dep(&a.g[k][c * a.plane + off2]);
            }
        }
    };
    int32_t m[4], g[C][4];
    fetch(0, m, g);
    const TileWindow win(I0, J0, a.cw, a.ch, a.cpitch, a.dw, a.wrap);
    win.stage<T, C>(ss, a.gc, a.cplane, K);
    const bool interior = interior_tile(X0, Y0, a.dw, a.dh, I0, J0, a.cw, a.ch);
    __syncthreads();
    int32_t acc[C][4] = {};
    const auto sum = [&](const auto& div) {
        for (int k = 0; k < K; ++k) {
            int32_t mn[4], gn[C][4];
            fetch(min(k + 1, K - 1), mn, gn);  // in flight while exposure k is merged
#pragma unroll
            for (int c = 0; c < C; ++c) {
                int32_t e[4];
                expand_window<true>(ss[k * C + c], qx, qy, div, e);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int32_t lp = (int32_t)cast_store<T>((int64_t)g[c][q] - e[q]);
                    acc[c][q] += (int32_t)mask_multiply<T, F>(lp, m[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                m[q] = mn[q];
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    g[c][q] = gn[c][q];
                }
            }
        }
    };
    if (on) {
        if (interior) {
            sum(QuadInside());
        } else {
            sum(QuadDivisors(X, Y, a.cw, a.ch, a.dw, a.wrap));
        }
    }
    griddep_wait();
    {
        int32_t v[C][2];
        if constexpr (FOLD) {
            ef_top<T, TM, C, F>(win, ss, a.mc, K, v);
        } else {
            win.load<T, C>(a.rc, a.cplane, v);
        }
        win.store<C>(ss + K * C, v);
    }
    __syncthreads();
    if (!on) {
        return;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
        int32_t e[4];
        if (interior) {
            expand_window<false>(ss[K * C + c], qx, qy, QuadInside(), e);
        } else {
            expand_window<false>(ss[K * C + c], qx, qy, QuadDivisors(X, Y, a.cw, a.ch, a.dw, a.wrap), e);
        }
        T r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            r[q] = sat_store<T>((int32_t)cast_store<T>(acc[c][q]) + e[q]);
        }
        T* dst = a.r + c * a.plane + off;
        if (pair) {
            st2<T>(dst, r[0], r[1]);
        } else {
            *dst = r[0];
        }
        if (Y + 1 < a.dh) {
            if (pair) {
                st2<T>(dst + a.pitch, r[2], r[3]);
            } else {
                dst[a.pitch] = r[2];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// level 0: from the K images and level-0 masks to the output pixels
// ---------------------------------------------------------------------------

template <typename TIn, typename T, typename TM>
struct EfOut0Args {
    int K, w, h, cw, ch, wrap;
    const TIn* img[kEfuseMaxK];
    int64_t ipitch[kEfuseMaxK];  // elements
    const TM* m0[kEfuseMaxK];
    int64_t mpitch;
    const T* g1[kEfuseMaxK];
    const T* r1;
    const TM* mc[kEfuseMaxK];  // level 1 of the mask pyramids
    int64_t cpitch, cplane;
    const uint8_t* u0;
    int64_t upitch;
    TIn* out;
    int64_t opitch;
    int32_t* level0;
    int dither;
    uint32_t key;
    int32_t maxv;
    int vec;   // the images' bases and pitches allow the paired pixel loads
    int ovec;  // the output's the paired stores
};

// As k_ef_up, with the image samples in place of level 0 of the image
// pyramids and the output pixels in place of R_0 (stored in words of the
// pair's size where the rows allow it).  9 x 6000x4000 u16: 1.21 ms
// (2.5 TB/s), 2.73 ms before the changes named at k_ef_up.
template <typename TIn, typename T, typename TM, int C, int S, int F, bool FOLD>
__global__ void __launch_bounds__(256, 3) k_ef_out0(const __grid_constant__ EfOut0Args<TIn, T, TM> a)
{
    extern __shared__ __align__(16) int32_t ewin[];
    int32_t (*ss)[ESH][ESW] = reinterpret_cast<int32_t (*)[ESH][ESW]>(ewin);
    if (FOLD) {
        griddep_wait();  // the launch before wrote the top level
        griddep_launch();
    }
    const int K = a.K;
    const int X0 = blockIdx.x * ETW, Y0 = blockIdx.y * ETH;
    const int I0 = X0 >> 1, J0 = Y0 >> 1;
    const int qx = threadIdx.x % 32, qy = threadIdx.x / 32;
    const int X = 2 * (I0 + qx), Y = 2 * (J0 + qy);
    const bool on = X < a.w && Y < a.h;
    // the quad's rows and columns, clamped to the image
    const int Xc = min(X, a.w - 1), X1 = min(X + 1, a.w - 1), Yc = min(Y, a.h - 1), Y1 = min(Y + 1, a.h - 1);
    // both pixels of a quad row in one paired load where x + 1 is inside and
    // the images are aligned for it
    const bool pair = a.vec && X + 1 < a.w;
    const auto fetch = [&](int k, int32_t (&m)[4], TIn (&px)[4][S]) {
        if (pair) {
            ld_pair<TM>(a.m0[k] + (int64_t)Yc * a.mpitch + X, m[0], m[1]);
            ld_pair<TM>(a.m0[k] + (int64_t)Y1 * a.mpitch + X, m[2], m[3]);
            TIn pp[2][S];
            PixelPair<TIn, S>::load(a.img[k] + (int64_t)Yc * a.ipitch[k] + (int64_t)X * S, pp);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                px[0][s] = pp[0][s];
                px[1][s] = pp[1][s];
            }
            PixelPair<TIn, S>::load(a.img[k] + (int64_t)Y1 * a.ipitch[k] + (int64_t)X * S, pp);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                px[2][s] = pp[0][s];
                px[3][s] = pp[1][s];
            }
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int x = q & 1 ? X1 : Xc, y = q & 2 ? Y1 : Yc;
                m[q] = (int32_t)ld_dep(&a.m0[k][(int64_t)y * a.mpitch + x]);
                const TIn* p = a.img[k] + (int64_t)y * a.ipitch[k] + (int64_t)x * S;
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    px[q][s] = ld_dep(&p[s]);
                }
            }
        }
    };
    int32_t m[4];
    TIn px[4][S];
    fetch(0, m, px);
    const TileWindow win(I0, J0, a.cw, a.ch, a.cpitch, a.w, a.wrap);
    win.stage<T, C>(ss, a.g1, a.cplane, K);
    const bool interior = interior_tile(X0, Y0, a.w, a.h, I0, J0, a.cw, a.ch);
    __syncthreads();
    int32_t acc[C][4] = {};
    const auto sum = [&](const auto& div) {
        for (int k = 0; k < K; ++k) {
            int32_t mn[4];
            TIn pn[4][S];
            fetch(min(k + 1, K - 1), mn, pn);  // in flight while exposure k is merged
#pragma unroll
            for (int c = 0; c < C; ++c) {
                int32_t e[4];
                expand_window<true>(ss[k * C + c], qx, qy, div, e);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    // copyToPyramidImage: v << 7 (src/fixmath.h:197-202)
                    const int32_t lp = (int32_t)cast_store<T>((int64_t)((int32_t)px[q][c] << 7) - e[q]);
                    acc[c][q] += (int32_t)mask_multiply<T, F>(lp, m[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                m[q] = mn[q];
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    px[q][s] = pn[q][s];
                }
            }
        }
    };
    if (on) {
        if (interior) {
            sum(QuadInside());
        } else {
            sum(QuadDivisors(X, Y, a.cw, a.ch, a.w, a.wrap));
        }
    }
    griddep_wait();
    griddep_launch();
    {
        int32_t v[C][2];
        if constexpr (FOLD) {
            ef_top<T, TM, C, F>(win, ss, a.mc, K, v);
        } else {
            win.load<T, C>(a.r1, a.cplane, v);
        }
        win.store<C>(ss + K * C, v);
    }
    __syncthreads();
    if (!on) {
        return;
    }
    int32_t res[C][4];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        int32_t e[4];
        if (interior) {
            expand_window<false>(ss[K * C + c], qx, qy, QuadInside(), e);
        } else {
            expand_window<false>(ss[K * C + c], qx, qy, QuadDivisors(X, Y, a.cw, a.ch, a.w, a.wrap), e);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            res[c][q] = (int32_t)sat_store<T>((int32_t)cast_store<T>(acc[c][q]) + e[q]);
        }
    }
    TIn o[4][S];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int x = q & 1 ? X1 : X, y = q & 2 ? Y1 : Y;
        const int64_t pix = (int64_t)y * a.w + x;
        if (a.level0 && X + (q & 1) < a.w && Y + (q >> 1) < a.h) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                a.level0[pix * C + c] = res[c][q];
            }
        }
        // copyFromPyramidImageIf (src/fixmath.h:2158-2294): the dither rule
        // where the union alpha is set, 0 elsewhere; an RGBA result's 4th
        // component is the union alpha
        const bool set = ld_dep(&a.u0[(int64_t)y * a.upitch + x]) != 0;
        const uint32_t pixbits = mix32((uint32_t)pix ^ a.key);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const uint32_t bits = dither_sample_bits(a.key, pixbits, (uint64_t)pix, C, c, 7);
            o[q][c] = set ? (TIn)dither_rule(res[c][q], 7, a.dither == ENB_DITHER_NEAREST, bits, a.maxv) : (TIn)0;
        }
        if (S == 4) {
            o[q][S - 1] = set ? (TIn)a.maxv : (TIn)0;
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (Y + r >= a.h) {
            break;
        }
        TIn* dst = a.out + (int64_t)(Y + r) * a.opitch + (int64_t)X * S;
        if (a.ovec && X + 1 < a.w) {
            PixelPair<TIn, S>::store(dst, reinterpret_cast<const TIn(&)[2][S]>(o[2 * r]));
            continue;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (X + q < a.w) {
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    dst[q * S + s] = o[2 * r + q][s];
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

static inline double esz_b(int dt) { return dt == ENB_U8 ? 1.0 : 2.0; }

static size_t win_smem(int K, int C) { return (size_t)(K + 1) * C * ESH * ESW * sizeof(int32_t); }

template <typename K_>
static void allow_smem(K_ kernel, size_t smem)
{
    if (smem > 48 * 1024) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }
}

// No exposure has alpha: the pyramids need no alpha planes (kReduceOpaque).
static bool ef_opaque(const EfuseHost& h)
{
    bool opaque = true;
    for (int k = 0; k < h.K; ++k) {
        opaque = opaque && h.alpha[k].mode == kAlphaOpaque;
    }
    return opaque;
}

// The mask pyramids' jobs from level l to l + 1 (A: with the union alpha).
template <typename TM, bool A>
static ReduceJobsN<PlanarSource<TM, 1, A>, TM> ef_mask_jobs(const EfuseHost& h, int l)
{
    using Src = PlanarSource<TM, 1, A>;
    ReduceJobsN<Src, TM> jobs{};
    const int64_t ap = l == 0 ? h.upitch0 : h.apitch[l];
    for (int k = 0; k < h.K; ++k) {
        jobs.j[k] = ReduceJob<Src, TM>{Src{(const TM*)h.m[k][l], h.pitch[l], h.pitch[l] * h.lh[l], h.u[l], ap},
                                       (TM*)h.m[k][l + 1], h.pitch[l + 1], h.pitch[l + 1] * h.lh[l + 1], h.u[l + 1],
                                       h.apitch[l + 1]};
    }
    return jobs;
}

// Level 1 of the K image pyramids straight from the pixels (PixelSourceV) and
// of the mask pyramids.
struct EfReduce0 {
    const EfuseHost& h;
    cudaStream_t st;
    cudaError_t err;
    template <typename TIn, typename T, int C, int S, int AM, bool VEC>
    void operator()()
    {
        using Src = PixelSourceV<TIn, C, S, AM, VEC>;
        constexpr bool A = AM != 1;
        ReduceJobsN<Src, T> jobs{};
        for (int k = 0; k < h.K; ++k) {
            const AlphaSrc& al = h.alpha[k];
            jobs.j[k] = ReduceJob<Src, T>{
                Src{(const TIn*)h.img[k].p, h.img[k].pitch, al.mode == kAlphaPlane ? al.plane.p : nullptr,
                    al.mode == kAlphaPlane ? al.plane.pitch : 0, al.lo, al.hi, 7},
                (T*)h.g[k][1], h.pitch[1], h.pitch[1] * h.lh[1], h.a[k][1], h.apitch[1]};
        }
        err = launch_reduce_joint<Src, T, C, PlanarSource<T, 1, A>, T, A ? kReduceAlpha : kReduceOpaque>(
            jobs, ef_mask_jobs<T, A>(h, 0), h.K, h.w, h.h, h.lw[1], h.lh[1], h.wrap, st);
    }
};

template <typename T, int C, bool A>
static cudaError_t ef_reduce_level(const EfuseHost& h, int l, cudaStream_t st)
{
    using Src = PlanarSource<T, C, A>;
    ReduceJobsN<Src, T> jobs{};
    for (int k = 0; k < h.K; ++k) {
        jobs.j[k] = ReduceJob<Src, T>{Src{(const T*)h.g[k][l], h.pitch[l], h.pitch[l] * h.lh[l], h.a[k][l], h.apitch[l]},
                                      (T*)h.g[k][l + 1], h.pitch[l + 1], h.pitch[l + 1] * h.lh[l + 1], h.a[k][l + 1],
                                      h.apitch[l + 1]};
    }
    return launch_reduce_joint<Src, T, C, PlanarSource<T, 1, A>, T, A ? kReduceAlpha : kReduceOpaque>(
        jobs, ef_mask_jobs<T, A>(h, l), h.K, h.lw[l], h.lh[l], h.lw[l + 1], h.lh[l + 1], h.wrap, st);
}

// Level l + 1 of the K image pyramids and the K mask pyramids.
cudaError_t launch_ef_reduce(const EfuseHost& h, int l, cudaStream_t st)
{
    const double sp = (double)h.lw[l] * h.lh[l], dp = (double)h.lw[l + 1] * h.lh[l + 1];
    const double ps = h.dtype == ENB_U8 ? 2.0 : 4.0;
    const bool opaque = ef_opaque(h);
    const double as = opaque ? 0.0 : 1.0;
    const double masks = h.K * (sp + dp) * ps + as * (sp + h.K * dp);
    if (l == 0) {
        double in = 0.0;
        for (int k = 0; k < h.K; ++k) {
            in += sp * (h.S * esz_b(h.dtype) + (h.alpha[k].mode == kAlphaPlane ? 1.0 : 0.0));
        }
        note_launch("ef_reduce0", in + h.K * dp * (h.C * ps + as) + masks);
        const PixelView& v = h.img[0];
        bool vec = h.S == 4;
        for (int k = 0; k < h.K; ++k) {
            const size_t px = (size_t)h.S * (size_t)esz_b(h.dtype);
            vec = vec && ((uintptr_t)h.img[k].p % px) == 0 && ((size_t)h.img[k].pitch * (size_t)esz_b(h.dtype)) % px == 0;
        }
        const int am = h.alpha[0].mode == kAlphaPlane ? 0 : (h.alpha[0].mode == kAlphaOpaque ? 1 : 2);
        EfReduce0 f{h, st, cudaErrorInvalidValue};
#define ENB_EF_CASE(TIN, TP, CC, SS, AMM, VV)                  \
    if (v.C == CC && h.S == SS && am == AMM && vec == VV) {    \
        f.template operator()<TIN, TP, CC, SS, AMM, VV>();     \
        return f.err;                                          \
    }
#define ENB_EF_TYPE(TIN, TP)                                   \
    ENB_EF_CASE(TIN, TP, 1, 1, 0, false)                       \
    ENB_EF_CASE(TIN, TP, 1, 1, 1, false)                       \
    ENB_EF_CASE(TIN, TP, 3, 3, 0, false)                       \
    ENB_EF_CASE(TIN, TP, 3, 3, 1, false)                       \
    ENB_EF_CASE(TIN, TP, 3, 4, 0, false)                       \
    ENB_EF_CASE(TIN, TP, 3, 4, 1, false)                       \
    ENB_EF_CASE(TIN, TP, 3, 4, 2, false)                       \
    ENB_EF_CASE(TIN, TP, 3, 4, 0, true)                        \
    ENB_EF_CASE(TIN, TP, 3, 4, 1, true)                        \
    ENB_EF_CASE(TIN, TP, 3, 4, 2, true)
        if (h.dtype == ENB_U8) {
            ENB_EF_TYPE(uint8_t, int16_t)
        } else {
            ENB_EF_TYPE(uint16_t, int32_t)
        }
#undef ENB_EF_TYPE
#undef ENB_EF_CASE
        return cudaErrorInvalidValue;
    }
    note_launch("ef_reduce", h.K * (sp + dp) * (h.C * ps + as) + masks);
    if (h.dtype == ENB_U8) {
        if (opaque) {
            return h.C == 1 ? ef_reduce_level<int16_t, 1, false>(h, l, st) : ef_reduce_level<int16_t, 3, false>(h, l, st);
        }
        return h.C == 1 ? ef_reduce_level<int16_t, 1, true>(h, l, st) : ef_reduce_level<int16_t, 3, true>(h, l, st);
    }
    if (opaque) {
        return h.C == 1 ? ef_reduce_level<int32_t, 1, false>(h, l, st) : ef_reduce_level<int32_t, 3, false>(h, l, st);
    }
    return h.C == 1 ? ef_reduce_level<int32_t, 1, true>(h, l, st) : ef_reduce_level<int32_t, 3, true>(h, l, st);
}

// The levels after l of all pyramids in one launch.
template <typename T, int C, bool A>
static cudaError_t ef_tail(const EfuseHost& h, int l, cudaStream_t st)
{
    constexpr int M = A ? kReduceAlpha : kReduceOpaque;
    TailJobs<T, T> j{};
    j.g.n = h.L - l;
    j.images = h.K;
    for (int i = 0; i < j.g.n; ++i) {
        j.g.w[i] = h.lw[l + i];
        j.g.h[i] = h.lh[l + i];
        j.g.pitch[i] = h.pitch[l + i];
        j.g.apitch[i] = h.apitch[l + i];
        j.u[i] = h.u[l + i];
        for (int k = 0; k < h.K; ++k) {
            j.img[k][i] = (T*)h.g[k][l + i];
            j.a[k][i] = h.a[k][l + i];
            j.msk[k][i] = (T*)h.m[k][l + i];
        }
    }
    return launch_reduce_tail<T, C, T, M, M>(j, h.K, h.wrap, st);
}

int ef_tail_level(const EfuseHost& h) { return tail_level(h.lw, h.lh, h.L); }

cudaError_t launch_ef_reduce_tail(const EfuseHost& h, int l, cudaStream_t st)
{
    note_launch("ef_reduce_tail", 0.0);
    const bool opaque = ef_opaque(h);
    if (h.dtype == ENB_U8) {
        if (h.C == 1) {
            return opaque ? ef_tail<int16_t, 1, false>(h, l, st) : ef_tail<int16_t, 1, true>(h, l, st);
        }
        return opaque ? ef_tail<int16_t, 3, false>(h, l, st) : ef_tail<int16_t, 3, true>(h, l, st);
    }
    if (h.C == 1) {
        return opaque ? ef_tail<int32_t, 1, false>(h, l, st) : ef_tail<int32_t, 1, true>(h, l, st);
    }
    return opaque ? ef_tail<int32_t, 3, false>(h, l, st) : ef_tail<int32_t, 3, true>(h, l, st);
}

template <typename T, typename TM>
static EfLevelArgs<T, TM> level_args(const EfuseHost& h, int l)
{
    EfLevelArgs<T, TM> a{};
    a.K = h.K;
    a.dw = h.lw[l];
    a.dh = h.lh[l];
    a.cw = h.lw[l + 1];
    a.ch = h.lh[l + 1];
    a.wrap = h.wrap;
    for (int k = 0; k < h.K; ++k) {
        a.g[k] = (const T*)h.g[k][l];
        a.gc[k] = (const T*)h.g[k][l + 1];
        a.m[k] = (const TM*)h.m[k][l];
        a.mc[k] = (const TM*)h.m[k][l + 1];
    }
    a.rc = (const T*)h.r[l + 1];
    a.r = (T*)h.r[l];
    a.pitch = h.pitch[l];
    a.plane = h.pitch[l] * h.lh[l];
    a.cpitch = h.pitch[l + 1];
    a.cplane = h.pitch[l + 1] * h.lh[l + 1];
    return a;
}

template <typename T, typename TM, int C, int F>
static cudaError_t ef_up_t(const EfuseHost& h, int l, cudaStream_t st)
{
    const size_t smem = win_smem(h.K, C);
    auto k = l + 2 == h.L ? k_ef_up<T, TM, C, F, true> : k_ef_up<T, TM, C, F, false>;
    allow_smem(k, smem);
    const dim3 g((unsigned)((h.lw[l] + ETW - 1) / ETW), (unsigned)((h.lh[l] + ETH - 1) / ETH));
    return launch_pdl_smem(k, g, dim3(256), smem, st, level_args<T, TM>(h, l));
}

cudaError_t launch_ef_up(const EfuseHost& h, int l, cudaStream_t st)
{
    const double px = (double)h.lw[l] * h.lh[l], cp = (double)h.lw[l + 1] * h.lh[l + 1];
    const double ps = h.dtype == ENB_U8 ? 2.0 : 4.0;
    note_launch("ef_up", px * (h.K * (h.C * ps + ps) + h.C * ps) + cp * (h.K + 1) * h.C * ps);
    if (h.dtype == ENB_U8) {
        return h.C == 1 ? ef_up_t<int16_t, int16_t, 1, 7>(h, l, st) : ef_up_t<int16_t, int16_t, 3, 7>(h, l, st);
    }
    return h.C == 1 ? ef_up_t<int32_t, int32_t, 1, 15>(h, l, st) : ef_up_t<int32_t, int32_t, 3, 15>(h, l, st);
}

template <typename TIn, typename T, typename TM, int C, int S, int F>
static cudaError_t ef_out0_t(const EfuseHost& h, cudaStream_t st)
{
    EfOut0Args<TIn, T, TM> a{};
    a.K = h.K;
    a.w = h.w;
    a.h = h.h;
    a.cw = h.lw[1];
    a.ch = h.lh[1];
    a.wrap = h.wrap;
    for (int k = 0; k < h.K; ++k) {
        a.img[k] = (const TIn*)h.img[k].p;
        a.ipitch[k] = h.img[k].pitch;
        a.m0[k] = (const TM*)h.m[k][0];
        a.g1[k] = (const T*)h.g[k][1];
        a.mc[k] = (const TM*)h.m[k][1];
    }
    a.mpitch = h.pitch[0];
    a.r1 = (const T*)h.r[1];
    a.cpitch = h.pitch[1];
    a.cplane = h.pitch[1] * h.lh[1];
    a.u0 = h.u[0];
    a.upitch = h.upitch0;
    a.out = (TIn*)h.out;
    a.opitch = h.opitch;
    a.level0 = h.level0;
    a.dither = h.dither;
    a.key = dither_key(h.seed);
    a.maxv = sizeof(TIn) == 1 ? 255 : 65535;
    a.vec = 1;
    for (int k = 0; k < h.K; ++k) {
        const size_t unit = (size_t)PixelPair<TIn, S>::UNIT;
        a.vec &= ((uintptr_t)h.img[k].p % unit) == 0 && ((size_t)h.img[k].pitch * sizeof(TIn)) % unit == 0;
    }
    a.ovec = (uintptr_t)h.out % (size_t)PixelPair<TIn, S>::UNIT == 0 &&
             ((size_t)h.opitch * sizeof(TIn)) % (size_t)PixelPair<TIn, S>::UNIT == 0;
    const size_t smem = win_smem(h.K, C);
    auto k = h.L == 2 ? k_ef_out0<TIn, T, TM, C, S, F, true> : k_ef_out0<TIn, T, TM, C, S, F, false>;
    allow_smem(k, smem);
    const dim3 g((unsigned)((h.w + ETW - 1) / ETW), (unsigned)((h.h + ETH - 1) / ETH));
    return launch_pdl_smem(k, g, dim3(256), smem, st, a);
}

cudaError_t launch_ef_out0(const EfuseHost& h, cudaStream_t st)
{
    const double px = (double)h.w * h.h, cp = (double)h.lw[1] * h.lh[1];
    const double ps = h.dtype == ENB_U8 ? 2.0 : 4.0, ss = esz_b(h.dtype);
    note_launch("ef_out0", px * (h.K * (h.S * ss + ps) + 1.0 + h.S * ss) + cp * (h.K + 1) * h.C * ps +
                               (h.level0 ? px * h.C * 4.0 : 0.0));
#define ENB_EF_OUT(TIN, TP, CC, SS, FF)                                    \
    if (h.C == CC && h.S == SS) {                                          \
        return ef_out0_t<TIN, TP, TP, CC, SS, FF>(h, st);                  \
    }
    if (h.dtype == ENB_U8) {
        ENB_EF_OUT(uint8_t, int16_t, 1, 1, 7)
        ENB_EF_OUT(uint8_t, int16_t, 3, 3, 7)
        ENB_EF_OUT(uint8_t, int16_t, 3, 4, 7)
    } else {
        ENB_EF_OUT(uint16_t, int32_t, 1, 1, 15)
        ENB_EF_OUT(uint16_t, int32_t, 3, 3, 15)
        ENB_EF_OUT(uint16_t, int32_t, 3, 4, 15)
    }
#undef ENB_EF_OUT
    return cudaErrorInvalidValue;
}

}  // namespace enb
