// enb_nft.cu -- enblend's nearest-feature seam mask (src/nearest.h:427-553)
// on the GPU: the mask of `enblend --fine-mask --no-optimize`
// (src/mask.h:1101-1180), 255 where the nearest pixel that only the white
// image covers is nearer than the nearest pixel that only the black image
// covers, else 0.
//
// The distances are the Euclidean distance transform of Felzenszwalb and
// Huttenlocher as the reference's OpenMP build computes it
// (src/openmp_vigra.h:257-433): a 1-D lower envelope of parabolas along
// every column of the feature image (0 on features, FLT_MAX elsewhere), then
// along every row of that result, then sqrt.  Every float operation is the
// reference's, in its order and rounding (no contraction into fused
// multiply-adds), so the masks are bit-identical.
//
// Columns of at most 4096 rows: q^2 and every other number of the column
// envelope is an integer below 2^24, exact in float, so the envelope of a
// 0 / FLT_MAX column is the distance to the nearest feature above or below
// (FLT_MAX without one) and k_nft_near scans for it with bit masks, half a warp
// per 16 columns x 1/32 of the rows.  Taller columns round and keep the
// sequential envelope (k_nft_columns, one thread a line).
//
// Rows: the sums round (q^2 beyond 2^24) and which vertex survives depends on
// it, so the envelope stays the reference's sequential walk, one lane a line
// (k_nft_envelope); the lookup of the surviving vertex of every pixel is
// parallel over the pixels (k_nft_select, a binary search of the line's
// boundaries) and ends in the mask.
//
// Wrap-around (--wrap horizontal): the reference transforms the image
// doubled horizontally and keeps, for x < w/2, column w + x and, for the
// other columns, column x (src/nearest.h:136-342).
#include <cuda_runtime.h>
#include <float.h>
#include <limits.h>
#include <math_constants.h>
#include <stdint.h>

#include "enb_internal.h"

namespace enb {

namespace {

// The 1-D transform of n samples f(q) (src/openmp_vigra.h:300-351); out(q,
// d) receives the squared distances.  v, z: this line's envelope in scratch
// with a stride of ss elements between consecutive entries.
template <class F, class Out>
__device__ __forceinline__ void fh_line(int n, const F& f, const Out& out, int* v, float* z, int64_t ss)
{
    int k = 0;
    v[0] = 0;
    z[0] = -CUDART_INF_F;
    z[ss] = CUDART_INF_F;
    for (int q = 1; q < n; ++q) {
        const float qf = (float)q;
        const float sum_q = __fadd_rn(f(q), __fmul_rn(qf, qf));
        int vk = v[k * ss];
        float s = __fdiv_rn(__fsub_rn(sum_q, __fadd_rn(f(vk), (float)(vk * vk))), (float)(2 * (q - vk)));
        while (s <= z[k * ss]) {
            --k;
            vk = v[k * ss];
            s = __fdiv_rn(__fsub_rn(sum_q, __fadd_rn(f(vk), (float)(vk * vk))), (float)(2 * (q - vk)));
        }
        ++k;
        v[k * ss] = q;
        z[k * ss] = s;
        z[(k + 1) * ss] = CUDART_INF_F;
    }
    k = 0;
    for (int q = 0; q < n; ++q) {
        while (z[(k + 1) * ss] < (float)q) {
            ++k;
        }
        const int vk = v[k * ss];
        out(q, __fadd_rn((float)((q - vk) * (q - vk)), f(vk)));
    }
}

struct NftArgs {
    const uint8_t* white;
    const uint8_t* black;
    int64_t wpitch, bpitch;
    int w, h;
    float* inter;        // [2][h][ipitch]: column pass of the two transforms
    int64_t ipitch;
    int* v;              // envelope scratch
    float* z;
    unsigned int* tally; // [2]: pixels only white covers, only black covers
};

// Whether (x, y) is a feature of transform t: covered by the white image
// only (t = 0, saturating white - black != 0) or by the black one only.
__device__ __forceinline__ bool nft_feature(const NftArgs& a, int t, int x, int y)
{
    const uint8_t wv = a.white[(int64_t)y * a.wpitch + x], bv = a.black[(int64_t)y * a.bpitch + x];
    return t == 0 ? wv > bv : bv > wv;
}

// Column pass of tall canvases: thread (x, t) for x < w, t = blockIdx.y.
// With wrap the doubled image's columns repeat, so each column is
// transformed once.
__global__ void __launch_bounds__(128) k_nft_columns(const NftArgs a)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = blockIdx.y;
    if (x >= a.w) {
        return;
    }
    const int64_t line = (int64_t)t * a.w + x, ss = 2 * (int64_t)a.w;
    int* v = a.v + line;
    float* z = a.z + line;
    unsigned int count = 0;
    const auto f = [&](int y) { return nft_feature(a, t, x, y) ? 0.0f : FLT_MAX; };
    float* col = a.inter + (int64_t)t * a.h * a.ipitch + x;
    fh_line(a.h, f, [&](int y, float d) { col[(int64_t)y * a.ipitch] = d; }, v, z, ss);
    for (int y = 0; y < a.h; ++y) {
        count += nft_feature(a, t, x, y) ? 1u : 0u;
    }
    atomicAdd(&a.tally[t], count);
}

// ---- columns of at most kNearRows rows --------------------------------------

constexpr int kNearRows = 4096;
constexpr uint16_t kNoFeature = 0xffff;
constexpr int kNearWords = kNearRows / 32 / 32;  // feature words of a half warp's rows

struct NearArgs {
    const uint8_t* white;
    const uint8_t* black;
    int64_t wpitch, bpitch;
    int w, h, rows;      // rows: rows of one half warp
    uint16_t* g;         // [2][h][pitch]: rows to the nearest feature, kNoFeature
    int64_t pitch;
    unsigned int* tally; // [2]
};

// Distance in rows to the nearest feature of the column, for both
// transforms.  A block covers 16 columns; half warp r takes the rows
// [r * rows, (r + 1) * rows), a lane keeps its rows' features as bits, the
// half warps exchange the last and first feature of their rows through shared
// memory, and every distance follows from the bits (clz / ffs) and the
// neighbours'.  16 columns and 512 threads fit three blocks on an SM, so that
// the 6963 columns of a panorama are one wave (32 columns and 1024 threads
// took 1.4 waves and 0.17 ms).  Bound by the instructions of the bit scans:
// 6963x3072 takes 0.11 ms (128 MB); the sequential envelope took 6.0 ms.
constexpr int kNearCols = 16;

__global__ void __launch_bounds__(32 * kNearCols, 3) k_nft_near(const NearArgs a)
{
    __shared__ int last[2][32][kNearCols], first[2][32][kNearCols];
    const int lane = threadIdx.x % kNearCols, r = threadIdx.x / kNearCols;
    const int x = blockIdx.x * kNearCols + lane, y0 = r * a.rows, y1 = min(a.h, y0 + a.rows);
    uint32_t bits[2][kNearWords];
    int lo[2] = {INT_MAX / 2, INT_MAX / 2}, hi[2] = {INT_MIN / 2, INT_MIN / 2};
    unsigned int count[2] = {0u, 0u};
#pragma unroll
    for (int i = 0; i < kNearWords; ++i) {
        bits[0][i] = bits[1][i] = 0u;
        if (y0 + 32 * i < y1 && x < a.w) {
#pragma unroll 16
            for (int b = 0; b < 32; ++b) {
                const int y = y0 + 32 * i + b;
                if (y < y1) {
                    const int wv = __ldg(&a.white[(int64_t)y * a.wpitch + x]), bv = __ldg(&a.black[(int64_t)y * a.bpitch + x]);
                    bits[0][i] |= (wv > bv ? 1u : 0u) << b;
                    bits[1][i] |= (bv > wv ? 1u : 0u) << b;
                }
            }
        }
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const uint32_t v = bits[t][i];
            if (v) {
                lo[t] = min(lo[t], y0 + 32 * i + __ffs(v) - 1);
                hi[t] = y0 + 32 * i + 31 - __clz(v);
                count[t] += __popc(v);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        first[t][r][lane] = lo[t];
        last[t][r][lane] = hi[t];
        const unsigned int n = __reduce_add_sync(0xffffffffu, count[t]);
        if (threadIdx.x % 32 == 0 && n) {
            atomicAdd(&a.tally[t], n);
        }
    }
    __syncthreads();
    if (x >= a.w) {
        return;
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        int above = INT_MIN / 2, below = INT_MAX / 2;  // nearest feature outside the half warp's rows
        for (int q = 0; q < r; ++q) {
            above = max(above, last[t][q][lane]);
        }
        for (int q = r + 1; q < 32; ++q) {
            below = min(below, first[t][q][lane]);
        }
        uint16_t* col = a.g + (int64_t)t * a.h * a.pitch + x;
#pragma unroll
        for (int i = 0; i < kNearWords; ++i) {
            int next = below;  // first feature after this word
#pragma unroll
            for (int j = kNearWords - 1; j > i; --j) {
                next = bits[t][j] ? y0 + 32 * j + __ffs(bits[t][j]) - 1 : next;
            }
            const int base = y0 + 32 * i;
            const uint32_t v = bits[t][i];
            for (int b = 0; b < 32 && base + b < y1; ++b) {
                const uint32_t up = v & (0xffffffffu >> (31 - b)), down = v >> b;
                const int u = up ? b - 31 + __clz(up) : base + b - above;
                const int d = down ? __ffs(down) - 1 : next - base - b;
                const int m = min(u, d);
                col[(int64_t)(base + b) * a.pitch] = m < kNearRows ? (uint16_t)m : kNoFeature;
            }
            above = v ? base + 31 - __clz(v) : above;
        }
    }
}

// ---- rows -------------------------------------------------------------------

// f(q) of a row, eight at a time: squared row distances as floats, or the
// distances of k_nft_near.  The planes' pitches are multiples of 32 samples,
// so a group of eight is aligned and lies inside the plane.
struct RowsF32 {
    typedef float T;
    __device__ __forceinline__ static float one(const float* p) { return *p; }
    struct Group {
        float4 a, b;
    };
    __device__ __forceinline__ static Group load(const float* p)
    {
        return Group{__ldg(reinterpret_cast<const float4*>(p)), __ldg(reinterpret_cast<const float4*>(p) + 1)};
    }
    __device__ __forceinline__ static float get(const Group& g, int i)
    {
        const float v[8] = {g.a.x, g.a.y, g.a.z, g.a.w, g.b.x, g.b.y, g.b.z, g.b.w};
        return v[i];
    }
};

struct RowsU16 {
    typedef uint16_t T;
    typedef uint4 Group;
    __device__ __forceinline__ static float of(uint32_t v)
    {
        return v == kNoFeature ? FLT_MAX : (float)(v * v);  // v < 4096: exact
    }
    __device__ __forceinline__ static float one(const uint16_t* p) { return of(*p); }
    __device__ __forceinline__ static Group load(const uint16_t* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
    __device__ __forceinline__ static float get(const Group& g, int i)
    {
        const uint32_t w = i < 2 ? g.x : (i < 4 ? g.y : (i < 6 ? g.z : g.w));
        return of((i & 1) ? w >> 16 : w & 0xffffu);
    }
};

// One vertex of a line's envelope: its column and the start of its range.
struct Vertex {
    int v;
    float z;
};

struct RowArgs {
    const void* f;       // [2][h][pitch]
    int64_t pitch;
    int w, h, wrap;
    Vertex* env;         // [2][h][n], n = w or 2 w
    int* count;          // [2][h] vertices
    uint8_t* mask;
    int64_t mpitch;
};

// The first loop of the 1-D transform (src/openmp_vigra.h:300-330) of row y,
// transform t: the envelope's vertices in order.  Lane l of a warp walks line
// blockIdx.x * kLines + l; the top of the stack is in registers, the entries
// just below it in a shared-memory ring (a pop there is one access), all of
// it in global memory, where pops beyond the ring read it back.
//   * Samples without a feature (FLT_MAX) after the first are skipped: such a
//     vertex is pushed with a boundary of 0 or FLT_MAX / (2 d), and the next
//     finite sample's intersection with it is -FLT_MAX / (2 d), which pops it
//     before anything else is compared; left at the end of the line, its range
//     starts beyond the line (or, over a first sample without a feature, gives
//     the same FLT_MAX).
//   * The division by 2 (q - v) of neighbours is an exact halving.
// Bound by the dependent chain of a line (about 470 cycles a sample), so a
// warp takes only kLines lines: fewer lanes diverge, and every SM holds
// several warps.  6963x3072, both transforms: 1.02 ms with 4 or 8 lines a
// warp, 1.18 / 1.11 / 1.24 ms with 2 / 16 / 32; the walk with the envelope in
// interleaved global scratch and the second loop in the same thread took
// 11.6 ms.  (Cutting the lines into 16 parts, each on an empty stack above a
// vertex later proven unpopped, took 1.40 ms: the lanes of a warp then walk
// unlike samples, and in the overlap of two footprints no vertex stands.)
constexpr int kLines = 8, kRing = 32;

template <class R>
__global__ void __launch_bounds__(32) k_nft_envelope(const RowArgs a)
{
    __shared__ int ring_v[kRing][kLines];
    __shared__ float ring_f[kRing][kLines], ring_z[kRing][kLines];
    const int lane = threadIdx.x;
    const int line = blockIdx.x * kLines + lane;
    if (lane >= kLines || line >= 2 * a.h) {
        return;
    }
    typedef typename R::T T;
    const T* row = static_cast<const T*>(a.f) + (int64_t)line * a.pitch;
    const int n = a.wrap ? 2 * a.w : a.w;
    Vertex* env = a.env + (int64_t)line * n;
    // f(v) + v^2 as the reference adds it for a vertex of the stack (an integer square)
    const auto lift = [](float f, int v) { return __fadd_rn(f, (float)(int)((unsigned)v * (unsigned)v)); };
    int k = 0, low = 0;  // top of the stack, lowest entry in the ring
    int vk = 0;
    float fk = lift(R::one(row), 0), zk = -CUDART_INF_F;
    const auto put = [&]() {
        ring_v[k % kRing][lane] = vk;
        ring_f[k % kRing][lane] = fk;
        ring_z[k % kRing][lane] = zk;
        env[k] = Vertex{vk, zk};
    };
    put();
    for (int pass = 0; pass * a.w < n; ++pass) {
        typename R::Group next = R::load(row);
        for (int x0 = 0; x0 < a.w; x0 += 8) {
            const typename R::Group g = next;
            if (x0 + 8 < a.w) {
                next = R::load(row + x0 + 8);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int q = pass * a.w + x0 + i;
                const float f = R::get(g, i);
                if (x0 + i >= a.w || q == 0 || f == FLT_MAX) {
                    continue;
                }
                const float qf = (float)q;
                const float sum = __fadd_rn(f, __fmul_rn(qf, qf));
                float num = __fsub_rn(sum, fk);
                float s = vk == q - 1 ? 0.5f * num : __fdiv_rn(num, (float)(2 * (q - vk)));
                while (s <= zk) {
                    --k;
                    if (k >= low) {
                        vk = ring_v[k % kRing][lane];
                        fk = ring_f[k % kRing][lane];
                        zk = ring_z[k % kRing][lane];
                    } else {
                        const Vertex e = env[k];
                        vk = e.v;
                        zk = e.z;
                        fk = lift(R::one(row + (vk < a.w ? vk : vk - a.w)), vk);
                        low = k;
                        ring_v[k % kRing][lane] = vk;
                        ring_f[k % kRing][lane] = fk;
                        ring_z[k % kRing][lane] = zk;
                    }
                    s = __fdiv_rn(__fsub_rn(sum, fk), (float)(2 * (q - vk)));
                }
                ++k;
                low = max(low, k - kRing + 1);
                vk = q;
                fk = lift(f, q);
                zk = s;
                put();
            }
        }
    }
    a.count[line] = k + 1;
}

// The second loop (src/openmp_vigra.h:333-351) and the comparison: pixel q of
// row y takes the last vertex whose range starts before q.  A thread finds it
// for the first of its eight columns by binary search and walks on from there.
template <class R>
__global__ void __launch_bounds__(128) k_nft_select(const RowArgs a)
{
    const int y = blockIdx.y;
    const int x0 = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (x0 >= a.w) {
        return;
    }
    typedef typename R::T T;
    const int n = a.wrap ? 2 * a.w : a.w, half = a.w / 2;
    float d[2][8];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int64_t line = (int64_t)t * a.h + y;
        const T* row = static_cast<const T*>(a.f) + line * a.pitch;
        const Vertex* env = a.env + line * n;
        const int m = a.count[line];
        int k = -1, v = 0;
        float next = 0.0f, f = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int x = min(x0 + i, a.w - 1);
            // the periodic transform keeps the doubled row's columns w/2 .. w + w/2 - 1
            const int q = a.wrap && x < half ? x + a.w : x;
            bool moved = false;
            if (k < 0 || (a.wrap && x == half)) {
                int lo = 0, hi = m;  // env[lo].z < q <= env[hi].z
                while (hi - lo > 1) {
                    const int mid = (lo + hi) / 2;
                    if (env[mid].z < (float)q) {
                        lo = mid;
                    } else {
                        hi = mid;
                    }
                }
                k = lo;
                moved = true;
                next = k + 1 < m ? env[k + 1].z : CUDART_INF_F;
            }
            while (next < (float)q) {
                ++k;
                moved = true;
                next = k + 1 < m ? env[k + 1].z : CUDART_INF_F;
            }
            if (moved) {
                v = env[k].v;
                f = R::one(row + (v < a.w ? v : v - a.w));
            }
            d[t][i] = __fsqrt_rn(__fadd_rn((float)((q - v) * (q - v)), f));
        }
    }
    uint8_t* out = a.mask + (int64_t)y * a.mpitch + x0;
    uint32_t o[2] = {0u, 0u};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        o[i / 4] |= (d[0][i] < d[1][i] ? 255u : 0u) << (8 * (i % 4));
    }
    if (x0 + 8 <= a.w && (reinterpret_cast<uintptr_t>(out) & 7) == 0) {
        *reinterpret_cast<uint2*>(out) = make_uint2(o[0], o[1]);
    } else {
        for (int i = 0; i < 8 && x0 + i < a.w; ++i) {
            out[i] = (uint8_t)(o[i / 4] >> (8 * (i % 4)));
        }
    }
}

}  // namespace

// Scratch of one call: the row pass's source planes (16-bit distances, or
// floats for tall columns), the envelopes and the vertex counts.
struct NftLayout {
    int64_t pitch, env, count, column_v, column_z, total;  // byte offsets
    NftLayout(int w, int h, int wrap)
    {
        const auto up = [](int64_t v) { return (v + 255) / 256 * 256; };
        const bool tall = h > kNearRows;
        pitch = (w + 31) / 32 * 32;
        env = up(2 * pitch * h * (tall ? (int64_t)sizeof(float) : (int64_t)sizeof(uint16_t)));
        count = up(env + 2 * (int64_t)h * (wrap ? 2 : 1) * w * (int64_t)sizeof(Vertex));
        column_v = up(count + 2 * (int64_t)h * (int64_t)sizeof(int));
        // the sequential column envelopes of tall canvases
        column_z = up(column_v + (tall ? 2 * (int64_t)w * (h + 1) * (int64_t)sizeof(int) : 0));
        total = up(column_z + (tall ? 2 * (int64_t)w * (h + 1) * (int64_t)sizeof(float) : 0));
    }
};

size_t nft_scratch_bytes(int w, int h, int wrap) { return (size_t)NftLayout(w, h, wrap).total; }

// Stage 0: the column pass and the tallies; 1: the row envelopes; 2: the
// nearest vertices and the mask.
cudaError_t launch_nft_stage(int stage, const BytePlane& white, const BytePlane& black, const BytePlane& mask,
                             int wrap, void* scratch, unsigned int* tally, cudaStream_t st)
{
    const int w = white.w, h = white.h;
    const NftLayout l(w, h, wrap);
    char* base = static_cast<char*>(scratch);
    const bool tall = h > kNearRows;
    const double sample = tall ? 4.0 : 2.0;
    if (stage == 0) {
        note_launch("nft_columns", 2.0 * w * h * (1.0 + sample));
        if (!tall) {
            const NearArgs a{white.p, black.p, white.pitch, black.pitch, w, h, (h + 31) / 32,
                             reinterpret_cast<uint16_t*>(base), l.pitch, tally};
            k_nft_near<<<(unsigned)((w + kNearCols - 1) / kNearCols), 32 * kNearCols, 0, st>>>(a);
            return cudaGetLastError();
        }
        NftArgs a{};
        a.white = white.p;
        a.black = black.p;
        a.wpitch = white.pitch;
        a.bpitch = black.pitch;
        a.w = w;
        a.h = h;
        a.ipitch = l.pitch;
        a.inter = reinterpret_cast<float*>(base);
        a.v = reinterpret_cast<int*>(base + l.column_v);
        a.z = reinterpret_cast<float*>(base + l.column_z);
        a.tally = tally;
        k_nft_columns<<<dim3((unsigned)((w + 127) / 128), 2), 128, 0, st>>>(a);
        return cudaGetLastError();
    }
    RowArgs a{base, l.pitch, w, h, wrap, reinterpret_cast<Vertex*>(base + l.env), reinterpret_cast<int*>(base + l.count),
              mask.p, mask.pitch};
    if (stage == 1) {
        note_launch("nft_rows", 2.0 * w * h * (sample + (wrap ? 16.0 : 8.0)));
        const unsigned blocks = (unsigned)((2 * h + kLines - 1) / kLines);
        if (tall) {
            k_nft_envelope<RowsF32><<<blocks, 32, 0, st>>>(a);
        } else {
            k_nft_envelope<RowsU16><<<blocks, 32, 0, st>>>(a);
        }
    } else {
        note_launch("nft_mask", 2.0 * w * h * (sample + 8.0) + (double)w * h);
        const dim3 grid((unsigned)((w + 1023) / 1024), (unsigned)h);
        if (tall) {
            k_nft_select<RowsF32><<<grid, 128, 0, st>>>(a);
        } else {
            k_nft_select<RowsU16><<<grid, 128, 0, st>>>(a);
        }
    }
    return cudaGetLastError();
}

}  // namespace enb
