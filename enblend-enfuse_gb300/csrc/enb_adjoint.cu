// enb_adjoint.cu -- adjoint of the float enfuse (no counterpart in the
// reference): gradients of a mean-squared loss against a target image with
// respect to the exposure-weight parameters (optimum, width), the weight
// coefficients (exposure, saturation, contrast) and a per-exposure additive
// logit map.
//
// The differentiated forward model is enfuseMain's float path
// (src/enfuse.h:1217-1617) with continuous masks: per exposure the weight
// w_k = W_exp f((y - opt) / width') + W_con sigma + W_sat s of
// src/enfuse.h:623-829, w~_k = w_k exp(a_k) with the logit map a_k,
// m_k = w~_k / sum_j w~_j (the soft mask, src/enfuse.h:1526-1535, without
// its 9.15 fixed-point quantisation), the mask Gaussian pyramids and image
// Laplacian pyramids of the opaque images (src/pyramid.h:1468-1747), the
// merge R[l] = sum_k LP_k[l] M_k[l] (src/enfuse.h:601-620, 1576-1588), the
// collapse (src/pyramid.h:1758-1784) and the mapping back
// (src/fixmath.h:320-329).  Entropy weights, hard masks and wrap-around are
// not differentiated.
//
// Backward, for each level from the output down the pyramids:
//   gC0 = dL/dout phi'(C0); gR[l] = gC[l], gC[l+1] = E^T gC[l]  (collapse)
//   gM_k[l] = sum_c gR[l]_c LP_k[l]_c                          (merge)
//   gm_k = gM_k[0] + Rd^T(gM_k[1] + Rd^T(...))                  (mask pyramid)
//   gw~_k = (gm_k - sum_j gm_j m_j) / S, ga_k = gw~_k w~_k     (normalisation)
//   gw_k = gw~_k exp(a_k) -> d/d(opt, width, W_exp, W_sat, W_con)
// where E^T and Rd^T are the transposes of the expand and of the
// normalised (opaque) reduce, written as gathers with the forward
// operators' per-position weights and divisors.
//
// The image pyramids hold G - 1 rather than the log-mapped G itself
// (log1p(v) for v >= 0, v / (1 - v) below): reduce and expand are
// normalised, so every level and every Laplacian but the top one is the
// same, the collapse yields C - 1 and the top level's Laplacian differs by
// the same amount for every exposure, which the normalisation's backward
// cancels.  In FP32 this keeps the fine Laplacians, small differences of
// values near 1 to 1.7, a few times more accurate.
//
// Every launch covers all K exposures of a level; the Gaussian levels of all
// exposures stay in memory (no Laplacian is ever stored, both sweeps form it
// from two Gaussian levels), and the mask pyramids' buffers hold their
// adjoints in the backward.  8 x 2048x2048: 38 launches and
// 1.95 ms; one exposure at a time, with stored Laplacians and one pixel a
// thread, took 515 launches and 7.44 ms.
#include <cuda_runtime.h>
#include <stdint.h>

#include "enb_device.cuh"
#include "enb_fpair.cuh"
#include "enb_fweights.cuh"
#include "enb_internal.h"
#include "enb_reduce.cuh"
#include "enb_tiles.cuh"

namespace enb {

namespace {

inline dim3 row_grid(int w, int h) { return dim3((unsigned)((w + 255) / 256), (unsigned)h); }
inline double npix(int w, int h) { return (double)w * (double)h; }

// log1p(v) for v >= 0, v / (1 - v) below: the log mapping less 1.
__device__ __forceinline__ float log_offset(float v) { return v >= 0.0f ? log1pf(v) : __fdiv_rn(v, 1.0f - v); }

// Planes of a level.
__device__ __forceinline__ int64_t level_plane(const AdjGeometry& g, int l) { return (int64_t)g.pitch[l] * g.lh[l]; }
__device__ __forceinline__ float* g_level(const AdjGeometry& g, int k, int l)
{
    return g.g + (int64_t)k * 3 * g.s + 3 * g.off[l];
}
__device__ __forceinline__ float* m_level(const AdjGeometry& g, int k, int l) { return g.m + (int64_t)k * g.s + g.off[l]; }

// The coarse windows of a 64x16 tile in floats: a thread's one or two taps of
// the (ESH x ESW) window at (I0 - 1, J0 - 1); taps outside the level are 0.
struct AdjWindow {
    int64_t o[2];
    float f[2];  // 1, or 0 outside the level
    bool two;
    __device__ __forceinline__ AdjWindow(int I0, int J0, int cw, int ch, int64_t cpitch)
    {
        two = threadIdx.x + 256 < ESH * ESW;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int k = min((int)threadIdx.x + 256 * u, ESH * ESW - 1);
            const int j = J0 - 1 + k / ESW, i = I0 - 1 + k % ESW;
            f[u] = j >= 0 && j < ch && i >= 0 && i < cw ? 1.0f : 0.0f;
            o[u] = (int64_t)min(max(j, 0), ch - 1) * cpitch + min(max(i, 0), cw - 1);
        }
    }
    // the mask adjoint's taps: divided by the reduce's divisors of the tap
    __device__ __forceinline__ void scale_by_reduce(int I0, int J0, int fw, int fh)
    {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int k = min((int)threadIdx.x + 256 * u, ESH * ESW - 1);
            const int j = J0 - 1 + k / ESW, i = I0 - 1 + k % ESW;
            f[u] = f[u] != 0.0f ? 1.0f / (float)(reduce_den1(i, fw) * reduce_den1(j, fh)) : 0.0f;
        }
    }
    template <int P>
    __device__ __forceinline__ void load(const float* p, int64_t plane, float (&v)[P][2]) const
    {
#pragma unroll
        for (int c = 0; c < P; ++c) {
            v[c][0] = ld_dep(&p[c * plane + o[0]]);
            v[c][1] = ld_dep(&p[c * plane + o[1]]);
        }
    }
    template <int P>
    __device__ __forceinline__ void store(float (*ss)[ESH][ESW], const float (&v)[P][2]) const
    {
#pragma unroll
        for (int c = 0; c < P; ++c) {
            // a select, so that nothing outside the level (NaN, infinities) enters
            (&ss[c][0][0])[threadIdx.x] = f[0] != 0.0f ? v[c][0] * f[0] : 0.0f;
            if (two) {
                (&ss[c][0][0])[threadIdx.x + 256] = f[1] != 0.0f ? v[c][1] * f[1] : 0.0f;
            }
        }
    }
};

// Numerators of a quad's expansion from the staged window, without the (4,4)
// taps' common factor 4.
__device__ __forceinline__ void adj_numerators(const float (*s)[ESW], int qx, int qy, float (&n)[4])
{
    float e[3], o[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float *v = &s[qy + r][qx];
        const float v0 = v[0], v1 = v[1], v2 = v[2];
        e[r] = fmaf(6.0f, v1, v0) + v2;
        o[r] = v1 + v2;
    }
    n[0] = fmaf(6.0f, e[1], e[0]) + e[2];
    n[1] = fmaf(6.0f, o[1], o[0]) + o[2];
    n[2] = e[1] + e[2];
    n[3] = o[1] + o[2];
}

// 1 / divisor of a quad's expansions (exact away from the borders).
__device__ __forceinline__ void adj_inverse(int X, int Y, int cw, int ch, int dw, float (&inv)[4])
{
    int w[3], he, ho, ve, vo;
    expand_hweights(X, cw, dw, 0, w, he);
    expand_hweights(X + 1, cw, dw, 0, w, ho);
    expand_vweights(Y, ch, w, ve);
    expand_vweights(Y + 1, ch, w, vo);
    ho >>= 2;
    inv[0] = 1.0f / (float)(he * ve);
    inv[1] = 1.0f / (float)(ho * ve);
    inv[2] = 1.0f / (float)(he * vo);
    inv[3] = 1.0f / (float)(ho * vo);
}

// A thread's quad of a level: pixel offsets, clamped at the level's ends.
struct AdjQuad {
    int X, Y;
    bool on, pair, row2;  // any pixel inside, both columns inside, second row inside
    int64_t off, off2;
    __device__ __forceinline__ AdjQuad(int X_, int Y_, int w, int h, int64_t pitch) : X(X_), Y(Y_)
    {
        on = X < w && Y < h;
        pair = X + 1 < w;
        row2 = Y + 1 < h;
        off = (int64_t)min(Y, h - 1) * pitch + min(X, w - 1);
        off2 = row2 ? off + pitch : off;
    }
    __device__ __forceinline__ void load(const float* p, float (&v)[4]) const
    {
        if (pair) {  // X is even and rows start on 128-byte boundaries
            const float2 a = ld_dep(reinterpret_cast<const float2*>(p + off)), b = ld_dep(reinterpret_cast<const float2*>(p + off2));
            v[0] = a.x;
            v[1] = a.y;
            v[2] = b.x;
            v[3] = b.y;
        } else {
            v[0] = v[1] = ld_dep(p + off);
            v[2] = v[3] = ld_dep(p + off2);
        }
    }
    __device__ __forceinline__ void store(float* p, const float (&v)[4]) const
    {
        if (pair) {
            *reinterpret_cast<float2*>(p + off) = make_float2(v[0], v[1]);
        } else {
            p[off] = v[0];
        }
        if (row2) {
            if (pair) {
                *reinterpret_cast<float2*>(p + off2) = make_float2(v[2], v[3]);
            } else {
                p[off2] = v[2];
            }
        }
    }
};

}  // namespace

// ---- forward pieces ---------------------------------------------------------

// Weights of one exposure (blockIdx.z) on a 32x16 tile, two pixels a thread
// (enb_fpair.cuh), and level 0 of its image pyramid, so that each image is
// read once.
template <int CW>
__global__ void __launch_bounds__(FPT, 5) k_adj_weights(const __grid_constant__ AdjGeometry g, FloatWeightParams wp,
                                                        WeightTables tab)
{
    constexpr int HALO = fpair_halo(CW, 0), HX = fpair_halo_x(HALO);
    constexpr int TW = fpair_tw(CW, 0), TT = TW * fpair_th(CW, 0), NP = (TT + FPT - 1) / FPT;
    extern __shared__ __align__(16) unsigned char asmem[];
    griddep_wait();
    griddep_launch();
    const FTileP t = fpair_carve(asmem, TW, TT, 0, 0);
    const int k = blockIdx.z, w = g.lw[0], h = g.lh[0];
    const AdjExposure& e = g.exposures[k];
    const int opaque = fpair_load<NP, 3, TW, TT>(t, wp, e.img, e.ipitch, e.stride, w, h, nullptr, 0,
                                                 blockIdx.x * FPX - HX, blockIdx.y * FPY - HALO);
    const int px = threadIdx.x % (FPX / 2), py = threadIdx.x / (FPX / 2);
    const int x = blockIdx.x * FPX + 2 * px, y = blockIdx.y * FPY + py;
    if (x >= w || y >= h) {
        return;
    }
    const int cx = HX + 2 * px, cy = HALO + py, ci = cy * TW + cx;
    float w0, w1;
    fpair_weights<CW, 0, 3>(t, wp, tab, cx, cy, x, y, w, h, opaque != 0, w0, w1);
    const int64_t plane = level_plane(g, 0), o = (int64_t)y * g.pitch[0] + x;
    float* wo = g.w + k * plane + o;
    float* g0 = g_level(g, k, 0) + o;
    if (x + 1 < w) {
        *reinterpret_cast<float2*>(wo) = make_float2(w0, w1);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            *reinterpret_cast<float2*>(g0 + c * plane) = make_float2(log_offset(t.raw[c * TT + ci]), log_offset(t.raw[c * TT + ci + 1]));
        }
    } else {
        *wo = w0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            g0[c * plane] = log_offset(t.raw[c * TT + ci]);
        }
    }
}

// Level 0 of the image pyramids alone (contrast windows outside the pair
// kernel, whose weights come from the per-image kernel).
__global__ void __launch_bounds__(256) k_adj_to_pyramid(const __grid_constant__ AdjGeometry g)
{
    griddep_wait();
    griddep_launch();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= g.lw[0]) {
        return;
    }
    const AdjExposure& e = g.exposures[blockIdx.z];
    const float* px = e.img + (int64_t)y * e.ipitch + (int64_t)x * e.stride;
    float* o = g_level(g, blockIdx.z, 0) + (int64_t)y * g.pitch[0] + x;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        o[c * level_plane(g, 0)] = log_offset(px[c]);
    }
}

// exp(a_k) of a pixel's logit, 1 without logits.
__device__ __forceinline__ float exp_logit(const AdjExposure& e, int x, int y)
{
    return e.logit ? expf(ld_dep(&e.logit[(int64_t)y * e.lpitch + x])) : 1.0f;
}

// w~_k = w_k exp(a_k), m_k = w~_k / S (S = sum_k w~_k; 1/K where S == 0) as
// level 0 of the mask pyramids.  KC > 0: at most KC exposures, their values in
// registers; 0: any number, read twice.
template <int KC>
__global__ void __launch_bounds__(256) k_adj_norm(const __grid_constant__ AdjGeometry g)
{
    griddep_wait();
    griddep_launch();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, K = g.K;
    if (x >= g.lw[0]) {
        return;
    }
    const int64_t o = (int64_t)y * g.pitch[0] + x, plane = level_plane(g, 0);
    const auto wt = [&](int k) { return g.w[k * plane + o] * exp_logit(g.exposures[k], x, y); };
    float v[KC > 0 ? KC : 1];
    float S = 0.0f;
    if (KC > 0) {
#pragma unroll
        for (int k = 0; k < KC; ++k) {
            v[k] = k < K ? wt(k) : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < KC; ++k) {
            S += v[k];
        }
    } else {
        for (int k = 0; k < K; ++k) {
            S += wt(k);
        }
    }
    const auto put = [&](int k, float t) { m_level(g, k, 0)[o] = S > 0.0f ? t / S : 1.0f / (float)K; };
    if (KC > 0) {
#pragma unroll
        for (int k = 0; k < KC; ++k) {
            if (k < K) {
                put(k, v[k]);
            }
        }
    } else {
        for (int k = 0; k < K; ++k) {
            put(k, wt(k));
        }
    }
}

// Level l + 1 of the K image pyramids (blockIdx.z < K) and mask pyramids.
__global__ void __launch_bounds__(RTHREADS, 3) k_adj_reduce(const __grid_constant__ AdjGeometry g, int l)
{
    __shared__ __align__(16) float V[ReduceSmem<3, false>::NV][RDH][RVP];
    griddep_wait();
    griddep_launch();
    const int sw = g.lw[l], sh = g.lh[l], dw = g.lw[l + 1], dh = g.lh[l + 1], z = blockIdx.z;
    const int64_t sp = level_plane(g, l), dp = level_plane(g, l + 1);
    if (z < g.K) {
        using Src = PlanarSource<float, 3, false>;
        const ReduceJob<Src, float> job{Src{g_level(g, z, l), g.pitch[l], sp, nullptr, 0}, g_level(g, z, l + 1),
                                        g.pitch[l + 1], dp, nullptr, 0};
        reduce_tile<Src, float, 3, kReduceOpaque, float>(job, blockIdx.x * RDW, blockIdx.y * RDH, sw, sh, dw, dh, 0, V);
    } else {
        using Src = PlanarSource<float, 1, false>;
        const ReduceJob<Src, float> job{Src{m_level(g, z - g.K, l), g.pitch[l], sp, nullptr, 0},
                                        m_level(g, z - g.K, l + 1), g.pitch[l + 1], dp, nullptr, 0};
        reduce_tile<Src, float, 1, kReduceOpaque, float>(job, blockIdx.x * RDW, blockIdx.y * RDH, sw, sh, dw, dh, 0, V);
    }
}

// Exposures whose windows a merge or mask-adjoint CTA stages at once.
constexpr int kAdjStage = 4;

// One 64x16 tile of level l: C[l] = sum_k (G_k[l] - E(G_k[l+1])) m_k[l] +
// E(C[l+1]) (no expand terms at the top).  L0: the loss, its gradient g0 =
// dL/dC0 and the output in place of C[0]: with u = C0 - 1, out = expm1(u)
// above 0 and u / (1 + u) below, loss += (out - T)^2, g0 = 2 (out - T) / N *
// phi'(C0).
template <bool L0>
__global__ void __launch_bounds__(256, 3) k_adj_up(const __grid_constant__ AdjGeometry g, int l, AdjLoss loss)
{
    __shared__ float ss[kAdjStage * 3][ESH][ESW];
    __shared__ double part[8];
    griddep_wait();
    griddep_launch();
    const bool top = l == g.L - 1;
    const int w = g.lw[l], h = g.lh[l], cw = top ? 1 : g.lw[l + 1], ch = top ? 1 : g.lh[l + 1];
    const int X0 = blockIdx.x * ETW, Y0 = blockIdx.y * ETH, I0 = X0 >> 1, J0 = Y0 >> 1;
    const int qx = threadIdx.x % 32, qy = threadIdx.x / 32;
    const AdjQuad q(2 * (I0 + qx), 2 * (J0 + qy), w, h, g.pitch[l]);
    const int64_t plane = level_plane(g, l), cplane = top ? 0 : level_plane(g, l + 1);
    const AdjWindow win(I0, J0, cw, ch, top ? 0 : g.pitch[l + 1]);
    float inv[4];
    adj_inverse(q.X, q.Y, cw, ch, w, inv);
    float acc[3][4] = {};
    for (int k0 = 0; k0 < g.K; k0 += kAdjStage) {
        if (!top) {
            float v[kAdjStage][3][2];
#pragma unroll
            for (int u = 0; u < kAdjStage; ++u) {
                win.load<3>(g_level(g, min(k0 + u, g.K - 1), l + 1), cplane, v[u]);
            }
            __syncthreads();  // the windows staged before are used up
#pragma unroll
            for (int u = 0; u < kAdjStage; ++u) {
                win.store<3>(ss + 3 * u, v[u]);
            }
            __syncthreads();
        }
        if (!q.on) {
            continue;
        }
        for (int u = 0; u < kAdjStage && k0 + u < g.K; ++u) {
            float m[4], f[3][4];
            q.load(m_level(g, k0 + u, l), m);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                q.load(g_level(g, k0 + u, l) + c * plane, f[c]);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                float n[4] = {};
                if (!top) {
                    adj_numerators(ss[3 * u + c], qx, qy, n);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    acc[c][i] += (f[c][i] - n[i] * inv[i]) * m[i];
                }
            }
        }
    }
    if (!top) {
        float v[3][2];
        win.load<3>(g.r + 3 * g.off[l + 1], cplane, v);
        __syncthreads();
        win.store<3>(ss, v);
        __syncthreads();
        if (q.on) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                float n[4];
                adj_numerators(ss[c], qx, qy, n);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    acc[c][i] += n[i] * inv[i];
                }
            }
        }
    }
    if (!L0) {
        if (q.on) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                q.store(g.r + 3 * g.off[l] + c * plane, acc[c]);
            }
        }
        return;
    }
    double sum = 0.0;
    if (q.on) {
        float g0[3][4] = {};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int x = q.X + (i & 1), y = q.Y + (i >> 1);
            if (x >= w || y >= h) {
                continue;
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float u = acc[c][i];
                const float ov = u >= 0.0f ? expm1f(u) : __fdiv_rn(u, 1.0f + u);
                const float d = ov - loss.target[(int64_t)y * loss.tpitch + (int64_t)x * loss.tstride + c];
                sum += (double)d * d;
                const float dphi = u >= 0.0f ? expf(u) : 1.0f / ((1.0f + u) * (1.0f + u));
                g0[c][i] = 2.0f * d * loss.inv_n * dphi;
                if (loss.out) {
                    loss.out[(int64_t)y * loss.opitch + (int64_t)x * loss.ostride + c] = ov;
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            q.store(g.gr + c * plane, g0[c]);
        }
    }
    for (int off = 16; off > 0; off >>= 1) {
        sum += __shfl_down_sync(0xffffffffu, sum, off);
    }
    if ((threadIdx.x & 31) == 0) {
        part[threadIdx.x >> 5] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < 8; ++i) {
            s += part[i];
        }
        atomicAdd(loss.sums, s);
    }
}

// ---- transposed operators -------------------------------------------------------

// Fine pixels of the transposed expand, scaled by 8 / divisor along each axis
// (1 but at the ends of the level), after which E^T is the zero-padded reduce
// with the taps [1 4 6 4 1] / 8.
struct ExpandTSource {
    const float* p;
    int64_t pitch, plane;
    int w, h, cw, ch;
    __device__ __forceinline__ static float scale(int X, int n)
    {
        const int i = X >> 1;
        if (X & 1) {
            return i + 1 < n ? 1.0f : 2.0f;
        }
        return (i == 0 || i + 1 >= n) ? (n == 1 ? 8.0f / 6.0f : 8.0f / 7.0f) : 1.0f;
    }
    template <typename AC>
    __device__ __forceinline__ void load(int gy, int gx, AC (&v)[3], int& al) const
    {
        const float f = scale(gx, cw) * scale(gy, ch);
        const int64_t o = (int64_t)gy * pitch + gx;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v[c] = ld_dep(&p[c * plane + o]) * f;
        }
        al = 1;
    }
};

// gR[l+1] = E^T gR[l].
__global__ void __launch_bounds__(RTHREADS, 3) k_adj_expand_T(const __grid_constant__ AdjGeometry g, int l)
{
    __shared__ __align__(16) float V[ReduceSmem<3, false>::NV][RDH][RVP];
    griddep_wait();
    griddep_launch();
    const int fw = g.lw[l], fh = g.lh[l], cw = g.lw[l + 1], ch = g.lh[l + 1];
    const ReduceJob<ExpandTSource, float> job{
        ExpandTSource{g.gr + 3 * g.off[l], g.pitch[l], level_plane(g, l), fw, fh, cw, ch}, g.gr + 3 * g.off[l + 1],
        g.pitch[l + 1], level_plane(g, l + 1), nullptr, 0};
    reduce_tile<ExpandTSource, float, 3, kReduceZeros, float>(job, blockIdx.x * RDW, blockIdx.y * RDH, fw, fh, cw, ch, 0, V);
}

// acc[l] = sum_c gR[l]_c LP_k[l]_c + Rd^T(acc[l+1]) of kAdjStage exposures
// (blockIdx.z): the mask pyramids' adjoint at one level, into the mask
// pyramids' buffers (the masks are not read again).  Rd^T spreads each coarse
// value, divided by the reduce's divisor there, with the taps (1,6,1)/(4,4)
// of the expand.
__global__ void __launch_bounds__(256, 3) k_adj_mask_level(const __grid_constant__ AdjGeometry g, int l)
{
    __shared__ float ss[kAdjStage * 4][ESH][ESW];
    griddep_wait();
    griddep_launch();
    const bool top = l == g.L - 1;
    const int w = g.lw[l], h = g.lh[l], cw = top ? 1 : g.lw[l + 1], ch = top ? 1 : g.lh[l + 1];
    const int X0 = blockIdx.x * ETW, Y0 = blockIdx.y * ETH, I0 = X0 >> 1, J0 = Y0 >> 1;
    const int qx = threadIdx.x % 32, qy = threadIdx.x / 32;
    const int k0 = blockIdx.z * kAdjStage;
    const AdjQuad q(2 * (I0 + qx), 2 * (J0 + qy), w, h, g.pitch[l]);
    const int64_t plane = level_plane(g, l);
    float gr[3][4];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        q.load(g.gr + 3 * g.off[l] + c * plane, gr[c]);
    }
    if (!top) {
        const int64_t cplane = level_plane(g, l + 1);
        AdjWindow win(I0, J0, cw, ch, g.pitch[l + 1]);
        {
            float v[kAdjStage][3][2];
#pragma unroll
            for (int u = 0; u < kAdjStage; ++u) {
                win.load<3>(g_level(g, min(k0 + u, g.K - 1), l + 1), cplane, v[u]);
            }
#pragma unroll
            for (int u = 0; u < kAdjStage; ++u) {
                win.store<3>(ss + 4 * u, v[u]);
            }
        }
        win.scale_by_reduce(I0, J0, w, h);
        float v[kAdjStage][1][2];
#pragma unroll
        for (int u = 0; u < kAdjStage; ++u) {
            win.load<1>(m_level(g, min(k0 + u, g.K - 1), l + 1), 0, v[u]);
        }
#pragma unroll
        for (int u = 0; u < kAdjStage; ++u) {
            win.store<1>(ss + 4 * u + 3, v[u]);
        }
        __syncthreads();
    }
    if (!q.on) {
        return;
    }
    float inv[4];
    adj_inverse(q.X, q.Y, cw, ch, w, inv);
    for (int u = 0; u < kAdjStage && k0 + u < g.K; ++u) {
        float f[3][4], acc[4] = {};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            q.load(g_level(g, k0 + u, l) + c * plane, f[c]);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float n[4] = {};
            if (!top) {
                adj_numerators(ss[4 * u + c], qx, qy, n);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc[i] += gr[c][i] * (f[c][i] - n[i] * inv[i]);
            }
        }
        if (!top) {
            float n[4];
            adj_numerators(ss[4 * u + 3], qx, qy, n);
            acc[0] += n[0];
            acc[1] += 4.0f * n[1];
            acc[2] += 4.0f * n[2];
            acc[3] += 16.0f * n[3];
        }
        q.store(m_level(g, k0 + u, l), acc);
    }
}

// ---- normalisation, logits and weight functions ---------------------------------

// gw~_k = (gm_k - sum_j gm_j m_j) / S; ga_k = gw~_k w~_k into the caller's
// planes; gw_k = gw~_k exp(a_k) in place of w_k.  KC as in k_adj_norm.
template <int KC>
__global__ void __launch_bounds__(256) k_adj_norm_bw(const __grid_constant__ AdjGeometry g)
{
    griddep_wait();
    griddep_launch();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, K = g.K;
    if (x >= g.lw[0]) {
        return;
    }
    const int64_t o = (int64_t)y * g.pitch[0] + x, plane = level_plane(g, 0);
    constexpr int N = KC > 0 ? KC : 1;
    float w[N], e[N], gm[N];
    float S = 0.0f, dot = 0.0f;
    if (KC > 0) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            w[k] = k < K ? g.w[k * plane + o] : 0.0f;
            e[k] = k < K ? exp_logit(g.exposures[k], x, y) : 1.0f;
            gm[k] = k < K ? m_level(g, k, 0)[o] : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < N; ++k) {
            S += w[k] * e[k];
        }
    } else {
        for (int k = 0; k < K; ++k) {
            S += g.w[k * plane + o] * exp_logit(g.exposures[k], x, y);
        }
    }
    const bool any = S > 0.0f;
    if (KC > 0) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            dot += any ? gm[k] * (w[k] * e[k] / S) : 0.0f;
        }
    } else {
        for (int k = 0; k < K && any; ++k) {
            dot += m_level(g, k, 0)[o] * (g.w[k * plane + o] * exp_logit(g.exposures[k], x, y) / S);
        }
    }
    const auto put = [&](int k, float wk, float ek, float gk) {
        const AdjExposure& ex = g.exposures[k];
        const float gwt = any ? (gk - dot) / S : 0.0f;
        g.w[k * plane + o] = gwt * ek;
        if (ex.glogit) {
            ex.glogit[(int64_t)y * ex.gpitch + x] = any ? gwt * wk * ek : 0.0f;
        }
    };
    if (KC > 0) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (k < K) {
                put(k, w[k], e[k], gm[k]);
            }
        }
    } else {
        for (int k = 0; k < K; ++k) {
            put(k, g.w[k * plane + o], exp_logit(g.exposures[k], x, y), m_level(g, k, 0)[o]);
        }
    }
}

// Derivative of the built-in exposure weight functions (src/exposure_weight.h:44-128).
__device__ __forceinline__ float exposure_dfdz(int fn, float z)
{
    switch (fn) {
    case ENB_EXP_LORENTZIAN: {
        const float q = 1.0f + 0.5f * z * z;
        return -z / (q * q);
    }
    case ENB_EXP_HALF_SINE: return fabsf(z) <= 1.57079632679489661923f ? -sinf(z) : 0.0f;
    case ENB_EXP_FULL_SINE: return fabsf(z) <= 3.14159265358979323846f ? -0.5f * sinf(z) : 0.0f;
    case ENB_EXP_BISQUARE: return fabsf(z) <= 1.0f ? -4.0f * z * z * z : 0.0f;
    default: return -z * expf(-0.5f * z * z);
    }
}

// A pixel's terms of d/d(optimum, width, W_exp, W_sat, W_con): gw = dL/dw_k
// times the partial derivatives of w_k.
__device__ __forceinline__ void adj_weight_terms(const FloatWeightParams& wp, float inv_width, float width, float w_exp, float gw,
                                                 float gray, float r, float g, float b, float sd, float (&s)[5])
{
    // exposure: z = (y - opt) / width'; dz/dopt = -1/width', dz/dwidth = -z/width
    const float yv = __fdiv_rn(gray, wp.range);
    const float z = (yv - (wp.opt_hi + wp.opt_lo)) * inv_width;
    const float df = exposure_dfdz(wp.exp_function, z);
    s[0] += gw * w_exp * df * (-inv_width);
    s[1] += gw * w_exp * df * (-z / width);
    s[2] += gw * exposure_f(wp, gray);
    // saturation (max_value 1.0)
    const float mx = fmaxf(r, fmaxf(g, b)), mn = fminf(r, fminf(g, b));
    float sat = 0.0f;
    if (mx != mn) {
        const float sum = mx + mn, diff = mx - mn;
        sat = __fdiv_rn(diff, sum <= 1.0f ? sum : (1.0f - mx) + (1.0f - mn));
    }
    s[3] += gw * sat;
    // contrast: the window's sample standard deviation (border strip 0)
    s[4] += gw * sd;
}

// The sums of those terms over all pixels and exposures, for the pair kernel's
// contrast windows: two pixels a thread on 32x16 tiles, the windows' deviation
// by the forward's arithmetic.  A CTA walks many tiles and adds its sums once
// (one addition per tile and sum to the same five doubles had cost as much as
// the arithmetic); a thread adds its pairs in a pair of floats each (TwoSum:
// more digits than the tiles' doubles of 32-term float sums had, and no FP64
// or shuffles in the loop).  8 x 2048x2048: 0.43 ms
// (1.02 ms one exposure a launch, one pixel a thread).
template <int CW>
__global__ void __launch_bounds__(FPT, 4) k_adj_weights_bw_pair(const __grid_constant__ AdjGeometry g, FloatWeightParams wp,
                                                                float inv_width, float width, float w_exp, int tx, int ty,
                                                                double* d)
{
    constexpr int HALO = fpair_halo(CW, 0), HX = fpair_halo_x(HALO), B = CW / 2;
    constexpr int TW = fpair_tw(CW, 0), TT = TW * fpair_th(CW, 0), NP = (TT + FPT - 1) / FPT;
    extern __shared__ __align__(16) unsigned char asmem[];
    __shared__ double part[5][FPT / 32];
    griddep_wait();
    griddep_launch();
    const FTileP t = fpair_carve(asmem, TW, TT, 0, 0);
    const int px = threadIdx.x % (FPX / 2), py = threadIdx.x / (FPX / 2);
    const int cx = HX + 2 * px, cy = HALO + py, ci = cy * TW + cx;
    const int w = g.lw[0], h = g.lh[0];
    float hi[5] = {}, lo[5] = {};
    for (int i = blockIdx.x; i < tx * ty * g.K; i += gridDim.x) {
        const int k = i / (tx * ty), tile = i - k * (tx * ty), bx = tile % tx, by = tile / tx;
        const AdjExposure& e = g.exposures[k];
        fpair_load<NP, 3, TW, TT>(t, wp, e.img, e.ipitch, e.stride, w, h, nullptr, 0, bx * FPX - HX, by * FPY - HALO);
        const int x = bx * FPX + 2 * px, y = by * FPY + py;
        float s[5] = {};
        if (x < w && y < h) {
            const bool rows = y >= B && y < h - B;
            const bool need0 = rows && x >= B && x < w - B, need1 = rows && x + 1 >= B && x + 1 < w - B;
            float sd[2] = {0.0f, 0.0f};
            if (need0 || need1) {
                fpair_contrast<CW, true>(t, cx, cy, t.gray[ci], sd);
            }
            const float* gw = g.w + k * level_plane(g, 0) + (int64_t)y * g.pitch[0] + x;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (x + q < w) {
                    adj_weight_terms(wp, inv_width, width, w_exp, gw[q], t.gray[ci + q], t.raw[ci + q], t.raw[TT + ci + q],
                                     t.raw[2 * TT + ci + q], (q == 0 ? need0 : need1) ? sd[q] : 0.0f, s);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            const float t1 = __fadd_rn(hi[j], s[j]), bb = __fsub_rn(t1, hi[j]);
            lo[j] += __fadd_rn(__fsub_rn(hi[j], __fsub_rn(t1, bb)), __fsub_rn(s[j], bb));
            hi[j] = t1;
        }
        __syncthreads();  // the next tile overwrites this one
    }
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        double v = (double)hi[j] + (double)lo[j];
        for (int off = 16; off > 0; off >>= 1) {
            v += __shfl_down_sync(0xffffffffu, v, off);
        }
        if ((threadIdx.x & 31) == 0) {
            part[j][threadIdx.x >> 5] = v;
        }
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        double v = 0.0;
        for (int j = 0; j < FPT / 32; ++j) {
            v += part[threadIdx.x][j];
        }
        atomicAdd(&d[threadIdx.x], v);
    }
}

// The same sums of one exposure for other contrast windows.  A 16x16
// tile of the image (with the contrast window's halo) is staged in shared
// memory as the per-image weight kernel stages it, and sigma is recomputed
// from it with that kernel's arithmetic.
__global__ void __launch_bounds__(256) k_adj_weights_bw(FloatPixelView img, const float* __restrict__ gw,
                                                        int64_t gpitch, FloatWeightParams wp, float inv_width,
                                                        float width, float w_exp, double* d)
{
    extern __shared__ __align__(16) unsigned char asmem[];
    __shared__ double part[5][8];
    const int halo = wp.contrast_window / 2;
    FloatWeightParams tp = wp;
    tp.repeat_slots = 0;
    const FTile t = ftile_carve(asmem, 16 + 2 * halo, 0);
    const int opaque = ftile_load(t, tp, img.p, img.pitch, img.stride, img.w, img.h, 3, nullptr, 0,
                                  blockIdx.x * 16 - halo, blockIdx.y * 16 - halo);
    const int lx = threadIdx.x % 16, ly = threadIdx.x / 16;
    const int x = blockIdx.x * 16 + lx, y = blockIdx.y * 16 + ly;
    // per pixel and per warp in float (a warp's sum of 32 terms: ~1e-6
    // relative), per block and across blocks in double
    float s[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (x < img.w && y < img.h) {
        const int ci = (ly + halo) * t.TW + (lx + halo);
        const float g = gw[(int64_t)y * gpitch + x];
        const int TT = t.TW * t.TW;
        float sd = 0.0f;
        if (x >= halo && x < img.w - halo && y >= halo && y < img.h - halo) {
            sd = window_stddev<0>(t, ci, halo, opaque != 0);
        }
        adj_weight_terms(wp, inv_width, width, w_exp, g, t.gray[ci], t.raw[ci], t.raw[TT + ci], t.raw[2 * TT + ci], sd, s);
    }
    for (int i = 0; i < 5; ++i) {
        for (int off = 16; off > 0; off >>= 1) {
            s[i] += __shfl_down_sync(0xffffffffu, s[i], off);
        }
    }
    if ((threadIdx.x & 31) == 0) {
        for (int i = 0; i < 5; ++i) {
            part[i][threadIdx.x >> 5] = (double)s[i];
        }
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        double tot = 0.0;
        for (int j = 0; j < (int)(blockDim.x >> 5); ++j) {
            tot += part[threadIdx.x][j];
        }
        atomicAdd(&d[threadIdx.x], tot);
    }
}

// ---- launchers ---------------------------------------------------------------------

static dim3 tiles_of(int w, int h, int tx, int ty, int z)
{
    return dim3((unsigned)((w + tx - 1) / tx), (unsigned)((h + ty - 1) / ty), (unsigned)z);
}

static bool adj_pair(const FloatWeightParams& wp) { return fpair_path(wp) && !wp.use_entropy; }

bool adj_weights_at_once(const FloatWeightParams& wp) { return adj_pair(wp); }

cudaError_t launch_adj_weights(const AdjGeometry& g, const FloatWeightParams& wp, const WeightTables& tab, cudaStream_t st)
{
    note_launch("adj_weights", npix(g.lw[0], g.lh[0]) * g.K * (12.0 + 4.0 + 12.0));
    const int cw = wp.use_contrast ? wp.contrast_window : 0;
    FloatWeightParams p = wp;
    p.repeat_slots = 0;
    const size_t smem = fpair_tile_bytes(fpair_tw(cw, 0) * fpair_th(cw, 0), 0, 0);
    auto k = cw == 5 ? k_adj_weights<5> : (cw == 3 ? k_adj_weights<3> : k_adj_weights<0>);
    return launch_pdl_smem(k, tiles_of(g.lw[0], g.lh[0], FPX, FPY, g.K), dim3(FPT), smem, st, g, p, tab);
}

cudaError_t launch_adj_to_pyramid(const AdjGeometry& g, cudaStream_t st)
{
    note_launch("adj_to_pyramid", npix(g.lw[0], g.lh[0]) * g.K * 24.0);
    return launch_pdl(k_adj_to_pyramid, tiles_of(g.lw[0], g.lh[0], 256, 1, g.K), dim3(256), st, g);
}

cudaError_t launch_adj_norm(const AdjGeometry& g, bool logits, cudaStream_t st)
{
    note_launch("adj_norm", npix(g.lw[0], g.lh[0]) * g.K * (logits ? 12.0 : 8.0));
    auto k = g.K <= 4 ? k_adj_norm<4> : (g.K <= 8 ? k_adj_norm<8> : k_adj_norm<0>);
    return launch_pdl(k, row_grid(g.lw[0], g.lh[0]), dim3(256), st, g);
}

cudaError_t launch_adj_reduce(const AdjGeometry& g, int l, cudaStream_t st)
{
    note_launch("adj_reduce", (npix(g.lw[l], g.lh[l]) + npix(g.lw[l + 1], g.lh[l + 1])) * g.K * 16.0);
    return launch_pdl(k_adj_reduce, tiles_of(g.lw[l + 1], g.lh[l + 1], RDW, RDH, 2 * g.K), dim3(RTHREADS), st, g, l);
}

cudaError_t launch_adj_up(const AdjGeometry& g, int l, const AdjLoss& loss, cudaStream_t st)
{
    const double up = l + 1 < g.L ? npix(g.lw[l + 1], g.lh[l + 1]) : 0.0;
    note_launch(l == 0 ? "adj_up0" : "adj_up", npix(g.lw[l], g.lh[l]) * (g.K * 16.0 + (l == 0 ? 24.0 + (loss.out ? 12.0 : 0.0) : 12.0)) +
                                                   up * (g.K + 1) * 12.0);
    return launch_pdl(l == 0 ? k_adj_up<true> : k_adj_up<false>, tiles_of(g.lw[l], g.lh[l], ETW, ETH, 1), dim3(256), st, g, l,
                      loss);
}

cudaError_t launch_adj_expand_T(const AdjGeometry& g, int l, cudaStream_t st)
{
    note_launch("adj_expand_T", 12.0 * (npix(g.lw[l], g.lh[l]) + npix(g.lw[l + 1], g.lh[l + 1])));
    return launch_pdl(k_adj_expand_T, tiles_of(g.lw[l + 1], g.lh[l + 1], RDW, RDH, 1), dim3(RTHREADS), st, g, l);
}

cudaError_t launch_adj_mask_level(const AdjGeometry& g, int l, cudaStream_t st)
{
    const double up = l + 1 < g.L ? npix(g.lw[l + 1], g.lh[l + 1]) : 0.0;
    note_launch("adj_mask_level", npix(g.lw[l], g.lh[l]) * (g.K * 16.0 + 12.0) + up * g.K * 16.0);
    return launch_pdl(k_adj_mask_level, tiles_of(g.lw[l], g.lh[l], ETW, ETH, (g.K + kAdjStage - 1) / kAdjStage), dim3(256), st,
                      g, l);
}

cudaError_t launch_adj_norm_bw(const AdjGeometry& g, bool logits, bool grad, cudaStream_t st)
{
    note_launch("adj_norm_bw", npix(g.lw[0], g.lh[0]) * g.K * (12.0 + (logits ? 4.0 : 0.0) + (grad ? 4.0 : 0.0)));
    auto k = g.K <= 4 ? k_adj_norm_bw<4> : (g.K <= 8 ? k_adj_norm_bw<8> : k_adj_norm_bw<0>);
    return launch_pdl(k, row_grid(g.lw[0], g.lh[0]), dim3(256), st, g);
}

cudaError_t launch_adj_weights_bw_pair(const AdjGeometry& g, const FloatWeightParams& wp, float inv_width, float width, float w_exp,
                                       int cwin, double* d, cudaStream_t st)
{
    note_launch("adj_weights_bw", npix(g.lw[0], g.lh[0]) * g.K * 16.0);
    FloatWeightParams p = wp;
    p.repeat_slots = 0;
    p.use_entropy = 0;
    const size_t smem = fpair_tile_bytes(fpair_tw(cwin, 0) * fpair_th(cwin, 0), 0, 0);
    const int tx = (g.lw[0] + FPX - 1) / FPX, ty = (g.lh[0] + FPY - 1) / FPY;
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t jobs = (int64_t)tx * ty * g.K;
    const dim3 grid((unsigned)(jobs < 4 * sms ? jobs : 4 * sms));
    return launch_pdl_smem(cwin == 5 ? k_adj_weights_bw_pair<5> : k_adj_weights_bw_pair<3>, grid, dim3(FPT), smem, st, g, p,
                           inv_width, width, w_exp, tx, ty, d);
}

cudaError_t launch_adj_weights_bw(const FloatPixelView& img, const float* gw, int64_t gpitch, const FloatWeightParams& wp,
                                  float inv_width, float width, float w_exp, int cwin, double* d, cudaStream_t st)
{
    note_launch("adj_weights_bw", npix(img.w, img.h) * (img.stride * 4.0 + 4.0));
    FloatWeightParams p = wp;
    p.contrast_window = cwin;
    const int TW = 16 + 2 * (cwin / 2);
    const size_t smem = ftile_bytes(TW, 0);
    const dim3 g((unsigned)((img.w + 15) / 16), (unsigned)((img.h + 15) / 16));
    if (smem > 48 * 1024) {
        cudaFuncSetAttribute(k_adj_weights_bw, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }
    k_adj_weights_bw<<<g, 256, smem, st>>>(img, gw, gpitch, p, inv_width, width, w_exp, d);
    return cudaGetLastError();
}

}  // namespace enb
