// Gaussian blur of masks, sparse (boundary tiles only) and dense.
//
// Sparse (reference: gaussian_blur_cuda.cu:288-507).  The reference flags edge
// pixels, compacts them with cub, expands each to the 3x3 window of tiles
// (tile side kernel_size/2) around its tile, sorts and uniques those tile ids,
// and convolves only the pixels of the listed tiles; every other pixel keeps
// its input value.  Here pass 1 sets one byte per tile that holds an edge
// pixel; pass 2 writes every output pixel once: a pixel whose tile has an edge
// tile within one tile in x and y (the reference's clamped 3x3 window) gets the
// convolution, any other pixel the converted input.  No compaction, no sort,
// and the output is written in the same pass as the copy the reference makes
// with images.clone().
//
// The convolution keeps the reference's arithmetic: 2-D taps with the x
// offset outer and the y offset inner, weights expf(-(i^2+j^2)/(2 sigma^2))
// rounded to the output type, acc += w * v fused for float and double (nvcc
// contracts the reference's expression), c10::Half rounding after every
// operation for half, and division by the sum of the weights in the same
// order.  The weight table and its sum are computed once per call on the
// device with the same expression, so results are bit-identical per pixel.
//
// Dense (reference: :20-114, reflect pad + torch conv2d with the normalised
// kernel).  Same halo reads; the weights are normalised first as the
// reference does, and the sum is accumulated in float (double for double
// output).  The reference's conv2d order belongs to cuDNN, so dense output
// agrees within rounding, as the reference's own dense/sparse test allows.

#include <algorithm>
#include <cstring>

#include "th_common.cuh"
#include "th_internal.h"

namespace th
{

namespace
{

constexpr int kMaxTaps = 63 * 63;

template <int DT>
__device__ __forceinline__ double load_f64(const void* p, int64_t i)
{
    using T = typename Elem<DT>::T;
    if constexpr (DT == TH_FLOAT16)
        return static_cast<double>(__half2float(static_cast<const __half*>(p)[i]));
    else
        return static_cast<double>(static_cast<const T*>(p)[i]);
}

__device__ __forceinline__ float round_half(float v)
{
    return __half2float(__float2half_rn(v));
}

// Input element as the output type (static_cast<BlurredImageT>(ImageT)),
// returned widened to double; for half through float like c10::Half does.
template <int DT, int OT>
__device__ __forceinline__ double as_out(const void* p, int64_t i)
{
    if constexpr (OT == TH_FLOAT64)
        return load_f64<DT>(p, i);
    else if constexpr (OT == TH_FLOAT32)
        return static_cast<double>(load_f32<DT>(p, i));
    else
        return static_cast<double>(round_half(load_f32<DT>(p, i)));
}

template <int OT>
__device__ __forceinline__ void store_out(void* p, int64_t i, double v)
{
    if constexpr (OT == TH_FLOAT64)
        static_cast<double*>(p)[i] = v;
    else if constexpr (OT == TH_FLOAT32)
        static_cast<float*>(p)[i] = static_cast<float>(v);
    else
        static_cast<__half*>(p)[i] = __float2half_rn(static_cast<float>(v));
}

// image_utils.h:129-160
__device__ __forceinline__ int64_t reflect(int64_t y, int64_t n)
{
    if (n == 1)
        return 0;
    const int64_t m = n - 1;
    // one reflection, the usual case (halos narrower than the image)
    if (-m < y && y < 2 * m)
        return y < 0 ? -y : (y > m ? 2 * m - y : y);
    const int64_t flips = y / m + (y < 0 ? 1 : 0);
    int64_t rem = y % m;
    if (rem < 0)
        rem += m;
    return (flips % 2 == 0) ? rem : m - rem;
}

template <int DT>
__device__ __forceinline__ bool differ(typename Elem<DT>::T a, typename Elem<DT>::T b)
{
    if constexpr (DT == TH_FLOAT16)
        return __half2float(a) != __half2float(b);
    else
        return a != b;
}

template <class F>
__device__ __forceinline__ void dispatch_out_device(int odt, F&& f)
{
    if (odt == TH_FLOAT16)
        f.template operator()<TH_FLOAT16>();
    else if (odt == TH_FLOAT32)
        f.template operator()<TH_FLOAT32>();
    else
        f.template operator()<TH_FLOAT64>();
}

// edge_kernel (gaussian_blur_cuda.cu:116-142) folded into tile flags, and the
// copy of every pixel to the output (the pixels that are blurred are written
// again by the second pass).  A warp owns 32 * V columns of a band of
// kEdgeRows rows, V elements per lane (16 bytes where input and output have
// one type and 16-byte aligned rows, else one): it issues the band's loads at
// once and compares from registers, so every row is read once plus one per
// band, and index arithmetic is left to the few elements that are edges.
// Bound by the read and the write of the images: 32x1024^2 float32 61 us
// with the copy (one element per thread with 64-bit divisions took 146 us
// without it).
constexpr int kEdgeRows = 8;

template <int DT, int V>
__global__ void __launch_bounds__(256) edge_tiles_kernel(const void* __restrict__ img,
                                                         void* __restrict__ out,
                                                         int odt,
                                                         int64_t B,
                                                         int64_t H,
                                                         int64_t W,
                                                         int64_t ts,
                                                         int64_t TH,
                                                         int64_t TW,
                                                         uint8_t* __restrict__ tiles)
{
    using T = typename Elem<DT>::T;
    const T* src = static_cast<const T*>(img);
    const int64_t chunks = (W + 32 * V - 1) / (32 * V), bands = (H + kEdgeRows - 1) / kEdgeRows;
    const int64_t units = B * bands * chunks;
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t u = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; u < units; u += nwarps)
    {
        const int64_t chunk = u % chunks, bb = u / chunks;
        const int64_t band = bb % bands, b = bb / bands;
        const int64_t x = (chunk * 32 + lane) * V, y0 = band * kEdgeRows;
        if (x >= W)
            continue; // with V > 1, W is a multiple of V
        const int64_t at = (b * H + y0) * W + x;
        const T* p = src + at;
        const int rows = static_cast<int>(H - y0 < kEdgeRows + 1 ? H - y0 : kEdgeRows + 1); // with the row below
        const bool right = x + V < W;
        T v[kEdgeRows + 1][V], rn[kEdgeRows];
#pragma unroll
        for (int i = 0; i <= kEdgeRows; ++i)
        {
            // rows past the image repeat its last one: no difference there
            const T* q = p + static_cast<int64_t>(i < rows ? i : rows - 1) * W;
            if constexpr (V > 1)
            {
                const uint4 w = *reinterpret_cast<const uint4*>(q);
                memcpy(v[i], &w, sizeof(w));
            }
            else
                v[i][0] = *q;
            if (i < kEdgeRows)
                rn[i] = right ? q[V] : v[i][V - 1];
        }
        if constexpr (V > 1)
        {
#pragma unroll
            for (int i = 0; i < kEdgeRows; ++i)
            {
                uint4 w;
                memcpy(&w, v[i], sizeof(w));
                if (i < rows)
                    *reinterpret_cast<uint4*>(static_cast<T*>(out) + at + i * W) = w;
            }
        }
        else
            dispatch_out_device(odt, [&]<int OT>() {
#pragma unroll
                for (int i = 0; i < kEdgeRows; ++i)
                    if (i < rows)
                        store_out<OT>(out, at + i * W, as_out<DT, OT>(&v[i][0], 0));
            });
#pragma unroll
        for (int i = 0; i < kEdgeRows; ++i)
        {
            uint32_t m = 0;
#pragma unroll
            for (int e = 0; e < V; ++e)
            {
                // the comparison with itself at the right border is left out (a NaN differs from itself)
                const bool h = e + 1 < V ? differ<DT>(v[i][e], v[i][e + 1 < V ? e + 1 : e])
                                         : right && differ<DT>(v[i][e], rn[i]);
                const bool w = i + 1 < rows && differ<DT>(v[i][e], v[i + 1][e]);
                m |= (h || w ? 1u : 0u) << e;
            }
            if (m == 0 || i >= rows)
                continue;
            uint8_t* row = tiles + (b * TH + (y0 + i) / ts) * TW;
            for (; m; m &= m - 1)
            {
                uint8_t* t = row + (x + __ffs(m) - 1) / ts;
                if (*t == 0)
                    *t = 1;
            }
        }
    }
}

// Weight table (k*k, x offset major) and its sum, in the output type's
// arithmetic: block 0; the other blocks clear the tile flags (zero_bytes, a
// multiple of 16).  The weights come from all threads; the sum keeps the
// reference's order (tap by tap), so one thread adds them, from shared memory
// for up to kSumTaps taps.  i*i + j*j is symmetric, so the x-major and the
// y-major table are the same numbers.
constexpr int kSumTaps = 4096;

template <int OT>
__global__ void __launch_bounds__(256) weights_kernel(int k, float sigma, bool normalise, double* __restrict__ w, double* __restrict__ norm,
                                                      uint4* __restrict__ zero, int64_t zero_bytes, uint32_t* __restrict__ ticket)
{
    if (blockIdx.x > 0)
    {
        const int64_t n = zero_bytes / 16, stride = static_cast<int64_t>(gridDim.x - 1) * blockDim.x;
        for (int64_t i = static_cast<int64_t>(blockIdx.x - 1) * blockDim.x + threadIdx.x; i < n; i += stride)
            zero[i] = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    __shared__ float ev[kSumTaps];
    __shared__ float total;
    if (threadIdx.x == 0 && ticket)
        *ticket = 0;
    const int r = k / 2, taps = k * k;
    const float den = __fmul_rn(__fmul_rn(2.f, sigma), sigma);
    auto weight = [&](int t) {
        const int i = t / k - r, j = t % k - r;
        return expf(__fdiv_rn(-static_cast<float>(i * i + j * j), den));
    };
    // tile_convolution_kernel (:268-283) rounds each weight to the output type
    // and sums in it; create_gaussian_kernel (:20-71) sums the rounded weights
    // in float32 and divides by that sum.
    for (int t = threadIdx.x; t < taps; t += blockDim.x)
    {
        const float e = weight(t);
        const float er = OT == TH_FLOAT16 ? round_half(e) : e;
        if (t < kSumTaps)
            ev[t] = er;
        if (!normalise)
            w[t] = static_cast<double>(er);
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double s = 0.0;
        float sf = 0.f;
#pragma unroll 8
        for (int t = 0; t < taps; ++t)
        {
            float e;
            if (t < kSumTaps)
                e = ev[t];
            else
                e = OT == TH_FLOAT16 ? round_half(weight(t)) : weight(t);
            if (!normalise && OT == TH_FLOAT64)
                s = __dadd_rn(s, static_cast<double>(e));
            else if (!normalise && OT == TH_FLOAT16)
                sf = round_half(__fadd_rn(sf, e));
            else
                sf = __fadd_rn(sf, e);
        }
        *norm = normalise ? 1.0 : (OT == TH_FLOAT64 ? s : static_cast<double>(sf));
        total = sf;
    }
    if (!normalise)
        return;
    __syncthreads();
    const float sum = total;
    for (int t = threadIdx.x; t < taps; t += blockDim.x)
    {
        const float e = weight(t);
        if constexpr (OT == TH_FLOAT64)
            w[t] = __ddiv_rn(static_cast<double>(e), static_cast<double>(sum));
        else if constexpr (OT == TH_FLOAT32)
            w[t] = static_cast<double>(__fdiv_rn(e, sum));
        else
            w[t] = static_cast<double>(round_half(__fdiv_rn(round_half(e), sum)));
    }
}

struct BlurGeom
{
    int64_t B, H, W, ts, TH, TW;
    int k;
};

__device__ __forceinline__ bool tile_active(const uint8_t* tiles, const BlurGeom& g, int64_t b, int64_t y, int64_t x)
{
    const int64_t tx = x / g.ts, ty = y / g.ts;
    for (int64_t dy = -1; dy <= 1; ++dy)
    {
        const int64_t yy = ty + dy;
        if (yy < 0 || yy >= g.TH)
            continue;
        for (int64_t dx = -1; dx <= 1; ++dx)
        {
            const int64_t xx = tx + dx;
            if (xx < 0 || xx >= g.TW)
                continue;
            if (tiles[(b * g.TH + yy) * g.TW + xx])
                return true;
        }
    }
    return false;
}

// One output pixel per thread.  SPARSE: only pixels of active tiles are
// convolved (reference arithmetic); DENSE: all pixels, normalised weights.
template <int DT, int OT, bool SPARSE>
__global__ void __launch_bounds__(256) blur_kernel(const void* __restrict__ img,
                                                   void* __restrict__ out,
                                                   BlurGeom g,
                                                   const uint8_t* __restrict__ tiles,
                                                   const double* __restrict__ wtab,
                                                   const double* __restrict__ norm_ptr)
{
    __shared__ double w[kMaxTaps > 1024 ? 1024 : kMaxTaps];
    const int taps = g.k * g.k;
    const bool smem_w = taps <= 1024;
    if (smem_w)
    {
        for (int i = threadIdx.x; i < taps; i += blockDim.x)
            w[i] = wtab[i];
        __syncthreads();
    }
    const double norm = *norm_ptr;
    const int r = g.k / 2;
    const int64_t n = g.B * g.H * g.W;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
    {
        const int64_t x = i % g.W, y = i / g.W % g.H, b = i / (g.W * g.H);
        if (SPARSE && !tile_active(tiles, g, b, y, x))
        {
            store_out<OT>(out, i, as_out<DT, OT>(img, i));
            continue;
        }
        const int64_t img_base = b * g.H * g.W;
        if constexpr (OT == TH_FLOAT64)
        {
            double acc = 0.0;
            for (int dx = -r; dx <= r; ++dx)
            {
                const int64_t xx = reflect(x + dx, g.W);
                for (int dy = -r; dy <= r; ++dy)
                {
                    const int64_t yy = reflect(y + dy, g.H);
                    const int t = (dx + r) * g.k + (dy + r);
                    const double kv = smem_w ? w[t] : wtab[t];
                    acc = __fma_rn(kv, load_f64<DT>(img, img_base + yy * g.W + xx), acc);
                }
            }
            store_out<OT>(out, i, SPARSE ? __ddiv_rn(acc, norm) : acc);
        }
        else if constexpr (OT == TH_FLOAT32)
        {
            float acc = 0.f;
            for (int dx = -r; dx <= r; ++dx)
            {
                const int64_t xx = reflect(x + dx, g.W);
                for (int dy = -r; dy <= r; ++dy)
                {
                    const int64_t yy = reflect(y + dy, g.H);
                    const int t = (dx + r) * g.k + (dy + r);
                    const float kv = static_cast<float>(smem_w ? w[t] : wtab[t]);
                    acc = __fmaf_rn(kv, load_f32<DT>(img, img_base + yy * g.W + xx), acc);
                }
            }
            store_out<OT>(out, i, SPARSE ? static_cast<double>(__fdiv_rn(acc, static_cast<float>(norm))) : acc);
        }
        else
        {
            float acc = 0.f;
            for (int dx = -r; dx <= r; ++dx)
            {
                const int64_t xx = reflect(x + dx, g.W);
                for (int dy = -r; dy <= r; ++dy)
                {
                    const int64_t yy = reflect(y + dy, g.H);
                    const int t = (dx + r) * g.k + (dy + r);
                    const float kv = static_cast<float>(smem_w ? w[t] : wtab[t]);
                    const float iv = round_half(load_f32<DT>(img, img_base + yy * g.W + xx));
                    if (SPARSE)
                        acc = round_half(__fadd_rn(acc, round_half(__fmul_rn(kv, iv))));
                    else
                        acc = __fmaf_rn(kv, iv, acc);
                }
            }
            const float res = SPARSE ? round_half(__fdiv_rn(acc, static_cast<float>(norm))) : acc;
            store_out<OT>(out, i, static_cast<double>(res));
        }
    }
}

// The device side of dispatch_image_dtype (a block-uniform branch).
template <class F>
__device__ __forceinline__ void dispatch_device(int dt, F&& f)
{
    switch (dt)
    {
    case TH_UINT8:
        f.template operator()<TH_UINT8>();
        break;
    case TH_INT8:
        f.template operator()<TH_INT8>();
        break;
    case TH_INT16:
        f.template operator()<TH_INT16>();
        break;
    case TH_INT32:
        f.template operator()<TH_INT32>();
        break;
    case TH_INT64:
        f.template operator()<TH_INT64>();
        break;
    case TH_FLOAT16:
        f.template operator()<TH_FLOAT16>();
        break;
    case TH_FLOAT32:
        f.template operator()<TH_FLOAT32>();
        break;
    default:
        f.template operator()<TH_FLOAT64>();
        break;
    }
}

// ---- blocks of 32 x 32 output pixels ---------------------------------------
//
// The block stages its pixels and a halo of k/2 in shared memory, converted
// once to the type the taps are accumulated in (reflected at the image's
// borders); a thread owns eight pixels of a column and keeps a sliding window
// of that column in registers, so a shared load serves eight taps.  Per pixel
// the taps run in the reference's order (x offset outer, y offset inner) with
// its roundings, so sparse results are the same bits as one pixel per thread.
// Bound by the FMA and shared-load issue.  The whole call on GB300: sparse
// 32x1024^2 float32, k = 9, 1288 -> 185 us; dense 24x501x723 half, k = 13,
// 3562 -> 129 us (one pixel per thread before, with a global load, two 64-bit
// reflections and a double weight per tap).  Blocks of 64 x 32 pixels took 192
// and 135 us: more of a block waits at its barriers.
constexpr int kTileX = 32, kTileY = 32, kTileRows = 8;
constexpr int kTileThreads = kTileX * kTileY / kTileRows, kTileWarps = kTileThreads / 32;
constexpr int kTileSmem = 96 * 1024;

template <int OT, bool SPARSE>
struct Accumulate
{
    using T = float;
};
template <bool SPARSE>
struct Accumulate<TH_FLOAT64, SPARSE>
{
    using T = double;
};
template <>
struct Accumulate<TH_FLOAT16, true>
{
    using T = __half; // every operation rounds to half
};

__device__ __forceinline__ float tap(float w, float v, float acc)
{
    return __fmaf_rn(w, v, acc);
}
__device__ __forceinline__ double tap(double w, double v, double acc)
{
    return __fma_rn(w, v, acc);
}
// c10::Half multiplies and adds in float and rounds each result to half; the
// half instructions round the exact result once, which is the same number (a
// product of halves is exact in float, and float's 24 bits are at least
// 2 * 11 + 2, so rounding a sum twice changes nothing).
__device__ __forceinline__ __half tap(__half w, __half v, __half acc)
{
    return __hadd_rn(acc, __hmul_rn(w, v));
}

// as_out with the accumulation's type.
template <int DT, int OT, typename A>
__device__ __forceinline__ A tile_value(const void* img, int64_t i)
{
    if constexpr (OT == TH_FLOAT64)
        return load_f64<DT>(img, i);
    else if constexpr (OT == TH_FLOAT32)
        return load_f32<DT>(img, i);
    else if constexpr (sizeof(A) == 2)
        return __float2half_rn(load_f32<DT>(img, i));
    else
        return round_half(load_f32<DT>(img, i));
}

// The tile and its halo; a thread's loads are issued kLoadAhead at a time.
constexpr int kLoadAhead = 8;

template <int DT, int OT, typename A, bool INNER>
__device__ __forceinline__ void load_tile_part(const void* __restrict__ img, A* tile, const BlurGeom& g, int64_t base, int64_t y0, int64_t x0, int r)
{
    const int sx = kTileX + 2 * r, n = sx * (kTileY + 2 * r);
    const int step_y = kTileThreads / sx, step_x = kTileThreads - step_y * sx;
    int ly = threadIdx.x / sx, lx = threadIdx.x - ly * sx;
    const int64_t corner = base + (y0 - r) * g.W + x0 - r;
    const int W = static_cast<int>(g.W); // INNER: ly * W + lx from the corner, rows of less than 2^31 elements
    for (int i = threadIdx.x; i < n; i += kTileThreads * kLoadAhead)
    {
        A v[kLoadAhead];
#pragma unroll
        for (int u = 0; u < kLoadAhead; ++u)
        {
            if (i + kTileThreads * u < n)
            {
                int64_t at;
                if constexpr (INNER)
                    at = corner + static_cast<int64_t>(ly) * W + lx;
                else
                    at = base + reflect(y0 - r + ly, g.H) * g.W + reflect(x0 - r + lx, g.W);
                v[u] = tile_value<DT, OT, A>(img, at);
            }
            lx += step_x;
            ly += step_y;
            if (lx >= sx)
            {
                lx -= sx;
                ++ly;
            }
        }
#pragma unroll
        for (int u = 0; u < kLoadAhead; ++u)
            if (i + kTileThreads * u < n)
                tile[i + kTileThreads * u] = v[u];
    }
}

template <int DT, int OT, typename A>
__device__ __forceinline__ void load_tile(const void* __restrict__ img, A* tile, const BlurGeom& g, int64_t base, int64_t y0, int64_t x0, int r)
{
    if (x0 >= r && y0 >= r && x0 + kTileX + r <= g.W && y0 + kTileY + r <= g.H && g.W < (int64_t{ 1 } << 31))
        load_tile_part<DT, OT, A, true>(img, tile, g, base, y0, x0, r);
    else
        load_tile_part<DT, OT, A, false>(img, tile, g, base, y0, x0, r);
}

// Row stride of the weights in shared memory: rows of 16-byte multiples, read four at a time.
__host__ __device__ __forceinline__ int weight_stride(int k)
{
    return (k + 3) / 4 * 4;
}

template <typename A>
struct __align__(4 * sizeof(A)) Four
{
    A v[4];
};

// Convolves block blk of the images (SPARSE: its pixels in active tiles).
template <int OT, bool SPARSE, typename A>
__device__ __forceinline__ void blur_block(const void* __restrict__ img,
                                           int idt,
                                           void* __restrict__ out,
                                           const BlurGeom& g,
                                           const uint8_t* __restrict__ tiles,
                                           const A* w,
                                           A* tile,
                                           uint8_t* act,
                                           double norm,
                                           uint32_t blk,
                                           uint32_t nbx,
                                           uint32_t nby)
{
    const int tid = threadIdx.x, k = g.k, r = k / 2, ws = weight_stride(k);
    const int sx = kTileX + 2 * r;
    const uint32_t rest = blk / nbx, ib = rest / nby;
    const int64_t x0 = static_cast<int64_t>(blk - rest * nbx) * kTileX, b = ib,
                  y0 = static_cast<int64_t>(rest - ib * nby) * kTileY;
    const int64_t base = b * g.H * g.W;
    const int ts = static_cast<int>(g.ts);
    int ntx = 0, ox = 0, oy = 0; // the block's tiles along x, and its first pixel inside its first tile
    if constexpr (SPARSE)
    {
        const int64_t xl = x0 + kTileX < g.W ? x0 + kTileX - 1 : g.W - 1, yl = y0 + kTileY < g.H ? y0 + kTileY - 1 : g.H - 1;
        const int64_t tx0 = x0 / ts, ty0 = y0 / ts;
        ox = static_cast<int>(x0 - tx0 * ts);
        oy = static_cast<int>(y0 - ty0 * ts);
        ntx = static_cast<int>(xl / ts - tx0) + 1;
        const int nty = static_cast<int>(yl / ts - ty0) + 1;
        // the flags of the block's tiles and of those around them
        const int rx = ntx + 2;
        for (int t = tid; t < rx * (nty + 2); t += kTileThreads)
        {
            const int64_t yy = ty0 - 1 + t / rx, xx = tx0 - 1 + t % rx;
            act[t] = yy >= 0 && yy < g.TH && xx >= 0 && xx < g.TW ? tiles[(b * g.TH + yy) * g.TW + xx] : 0;
        }
    }
    dispatch_device(idt, [&]<int DT>() { load_tile<DT, OT, A>(img, tile, g, base, y0, x0, r); });
    __syncthreads();

    const int cx = tid & (kTileX - 1), cy = (tid / kTileX) * kTileRows; // first pixel of the thread's column
    const int64_t x = x0 + cx;
    uint32_t on = 0;
    if constexpr (SPARSE)
    {
        if (x < g.W)
        {
            const int tx = (ox + cx) / ts, rx = ntx + 2;
            int last = -1;
            bool near = false;
#pragma unroll
            for (int j = 0; j < kTileRows; ++j)
            {
                const int ty = (oy + cy + j) / ts;
                if (ty != last)
                {
                    const uint8_t* a = act + ty * rx + tx; // the tile up and to the left
                    near = (a[0] | a[1] | a[2] | a[rx] | a[rx + 1] | a[rx + 2] | a[2 * rx] | a[2 * rx + 1] | a[2 * rx + 2]) != 0;
                    last = ty;
                }
                if (y0 + cy + j < g.H && near)
                    on |= 1u << j;
            }
        }
    }
    else
        on = x < g.W ? 0xffu : 0u;
    A acc[kTileRows];
#pragma unroll
    for (int j = 0; j < kTileRows; ++j)
        acc[j] = A(0.f);
    if (__any_sync(0xffffffffu, on != 0))
    {
        for (int dx = 0; dx < k; ++dx)
        {
            // a sliding window of the column in two halves that change roles
            // every eight taps, so no value moves between registers
            const A* col = tile + cy * sx + cx + dx;
            const A* wd = w + dx * ws;
            A lo[kTileRows], hi[kTileRows];
#pragma unroll
            for (int j = 0; j < kTileRows; ++j)
                lo[j] = col[j * sx];
            auto taps = [&]<int U>(const A(&from)[kTileRows], A(&next)[kTileRows]) {
                col += kTileRows * sx;
#pragma unroll
                for (int u = 0; u < (U < kTileRows ? U - 1 : U); ++u)
                    next[u] = col[u * sx];
#pragma unroll
                for (int u = 0; u < U; u += 4)
                {
                    const Four<A> wt = *reinterpret_cast<const Four<A>*>(wd + u);
#pragma unroll
                    for (int i = 0; i < 4 && u + i < U; ++i)
                    {
#pragma unroll
                        for (int j = 0; j < kTileRows; ++j)
                        {
                            const int at = j + u + i;
                            acc[j] = tap(wt.v[i], at < kTileRows ? from[at < kTileRows ? at : 0] : next[at < kTileRows ? 0 : at - kTileRows], acc[j]);
                        }
                    }
                }
                wd += U;
            };
            auto rest = [&](const A(&from)[kTileRows], A(&next)[kTileRows]) {
                // k is odd
                const int left = k & 7;
                if (left == 1)
                    taps.template operator()<1>(from, next);
                else if (left == 3)
                    taps.template operator()<3>(from, next);
                else if (left == 5)
                    taps.template operator()<5>(from, next);
                else
                    taps.template operator()<7>(from, next);
            };
            int eights = k >> 3;
            for (; eights >= 2; eights -= 2)
            {
                taps.template operator()<8>(lo, hi);
                taps.template operator()<8>(hi, lo);
            }
            if (eights)
            {
                taps.template operator()<8>(lo, hi);
                rest(hi, lo);
            }
            else
                rest(lo, hi);
        }
    }
    if (x >= g.W)
        return;
#pragma unroll
    for (int j = 0; j < kTileRows; ++j)
    {
        const int64_t y = y0 + cy + j;
        if (y >= g.H)
            return;
        const int64_t i = base + y * g.W + x;
        if constexpr (sizeof(A) == 2)
        {
            if ((on >> j) & 1u)
                static_cast<__half*>(out)[i] = __float2half_rn(__fdiv_rn(__half2float(acc[j]), static_cast<float>(norm)));
        }
        else
        {
            A res = acc[j];
            if constexpr (SPARSE)
            {
                if constexpr (OT == TH_FLOAT64)
                    res = __ddiv_rn(res, norm);
                else
                    res = __fdiv_rn(res, static_cast<float>(norm));
                if (!((on >> j) & 1u))
                    continue; // the first pass copied it
            }
            store_out<OT>(out, i, static_cast<double>(res));
        }
    }
}

// Whether block blk has a pixel in an active tile (a warp's lanes look at the
// flags of its tiles and of one more around them).
__device__ __forceinline__ bool block_active(const BlurGeom& g, const uint8_t* __restrict__ tiles, uint32_t blk, uint32_t nbx, uint32_t nby)
{
    const uint32_t rest = blk / nbx, ib = rest / nby;
    const int64_t x0 = static_cast<int64_t>(blk - rest * nbx) * kTileX, y0 = static_cast<int64_t>(rest - ib * nby) * kTileY;
    const int64_t xl = x0 + kTileX < g.W ? x0 + kTileX - 1 : g.W - 1, yl = y0 + kTileY < g.H ? y0 + kTileY - 1 : g.H - 1;
    const int64_t ts = g.ts;
    const int64_t tx0 = x0 / ts > 0 ? x0 / ts - 1 : 0, ty0 = y0 / ts > 0 ? y0 / ts - 1 : 0;
    const int64_t tx1 = xl / ts + 1 < g.TW ? xl / ts + 1 : g.TW - 1, ty1 = yl / ts + 1 < g.TH ? yl / ts + 1 : g.TH - 1;
    const uint8_t* p = tiles + (ib * g.TH + ty0) * g.TW + tx0;
    const int nx = static_cast<int>(tx1 - tx0) + 1, n = nx * (static_cast<int>(ty1 - ty0) + 1);
    bool any = false;
#pragma unroll 4
    for (int t = threadIdx.x & 31; t < n; t += 32)
        any |= p[t / nx * g.TW + t % nx] != 0;
    return __any_sync(0xffffffffu, any);
}

// One block of output pixels at a time: dense block blockIdx.x; sparse, a
// block takes tickets, each for four blocks of pixels that lie far apart (few
// of them are active at once), looks at their flags with a warp each and
// convolves the active ones.  (A block per block of pixels, and a fixed share
// of the image per block, waited for the slowest: 147 and 171 us for
// 32x1024^2, k = 9, against 132 us.)
template <int OT, bool SPARSE>
__global__ void __launch_bounds__(kTileThreads, 6) blur_tile_kernel(const void* __restrict__ img,
                                                        int idt,
                                                        void* __restrict__ out,
                                                        BlurGeom g,
                                                        const uint8_t* __restrict__ tiles,
                                                        const double* __restrict__ wtab,
                                                        const double* __restrict__ norm_ptr,
                                                        uint32_t nblocks,
                                                        uint32_t* __restrict__ ticket)
{
    using A = typename Accumulate<OT, SPARSE>::T;
    extern __shared__ __align__(32) unsigned char blur_smem[];
    __shared__ uint32_t s_ticket, s_active;
    const int tid = threadIdx.x, k = g.k, r = k / 2;
    const int sx = kTileX + 2 * r, sy = kTileY + 2 * r, ws = weight_stride(k);
    A* w = reinterpret_cast<A*>(blur_smem);
    A* tile = w + k * ws;
    uint8_t* act = reinterpret_cast<uint8_t*>(tile + sx * sy);
    const uint32_t nbx = static_cast<uint32_t>((g.W + kTileX - 1) / kTileX), nby = static_cast<uint32_t>((g.H + kTileY - 1) / kTileY);
    for (int t = tid; t < k * k; t += kTileThreads)
    {
        const int at = t / k * ws + t % k;
        if constexpr (sizeof(A) == 2)
            w[at] = __float2half_rn(static_cast<float>(wtab[t]));
        else
            w[at] = static_cast<A>(wtab[t]);
    }
    const double norm = *norm_ptr;
    if constexpr (!SPARSE)
        blur_block<OT, SPARSE>(img, idt, out, g, tiles, w, tile, act, norm, blockIdx.x, nbx, nby);
    else
    {
        const uint32_t tickets = (nblocks + kTileWarps - 1) / kTileWarps;
        for (uint32_t done = 0; done <= tickets; ++done) // ends when the tickets do
        {
            __syncthreads();
            if (tid == 0)
            {
                s_ticket = atomicAdd(ticket, 1u);
                s_active = 0;
            }
            __syncthreads();
            const uint32_t t = s_ticket;
            if (t >= tickets)
                break;
            const uint32_t mine = t + (tid >> 5) * tickets;
            if (mine < nblocks && block_active(g, tiles, mine, nbx, nby) && (tid & 31) == 0)
                atomicOr(&s_active, 1u << (tid >> 5));
            __syncthreads();
            for (uint32_t left = s_active; left; left &= left - 1)
            {
                blur_block<OT, SPARSE>(img, idt, out, g, tiles, w, tile, act, norm, t + (__ffs(left) - 1) * tickets, nbx, nby);
                __syncthreads();
            }
        }
    }
}

// Shared memory of a block, 0 where the kernel is too wide for it (a block per
// SM would be left, or none): those take blur_kernel.
template <int OT, bool SPARSE>
size_t tile_smem(int k, int64_t ts)
{
    const int64_t r = k / 2;
    int64_t bytes = (int64_t{ k } * weight_stride(k) + (kTileX + 2 * r) * (kTileY + 2 * r)) *
                    static_cast<int64_t>(sizeof(typename Accumulate<OT, SPARSE>::T));
    if (SPARSE)
        bytes += (kTileX / ts + 4) * (kTileY / ts + 4);
    return bytes <= kTileSmem ? static_cast<size_t>(bytes) : 0;
}

template <int OT, bool SPARSE>
bool launch_tiles(const void* images, int idt, void* out, const BlurGeom& g, const uint8_t* tiles, const double* wtab, const double* norm, uint32_t* ticket, cudaStream_t s)
{
    const size_t smem = tile_smem<OT, SPARSE>(g.k, g.ts);
    const int64_t blocks = ((g.W + kTileX - 1) / kTileX) * ((g.H + kTileY - 1) / kTileY) * g.B;
    if (smem == 0 || blocks >= (int64_t{ 1 } << 31))
        return false;
    auto kernel = blur_tile_kernel<OT, SPARSE>;
    if (smem > 48 * 1024)
        TH_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmem));
    const unsigned grid = SPARSE ? static_cast<unsigned>(std::min<int64_t>(blocks, 6 * sm_count())) : static_cast<unsigned>(blocks);
    kernel<<<grid, kTileThreads, smem, s>>>(images, idt, out, g, tiles, wtab, norm, static_cast<uint32_t>(blocks), ticket);
    TH_LAUNCH_CHECK();
    return true;
}

template <int DT, int OT>
__global__ void __launch_bounds__(256) convert_kernel(const void* __restrict__ img, void* __restrict__ out, int64_t n)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        store_out<OT>(out, i, as_out<DT, OT>(img, i));
}

template <class F>
void dispatch_out(int odt, F&& f)
{
    switch (odt)
    {
    case TH_FLOAT16:
        f.template operator()<TH_FLOAT16>();
        break;
    case TH_FLOAT32:
        f.template operator()<TH_FLOAT32>();
        break;
    default:
        f.template operator()<TH_FLOAT64>();
        break;
    }
}

} // namespace

int64_t blur_tile_bytes(int64_t B, int64_t H, int64_t W, int kernel_size)
{
    const int64_t ts = kernel_size / 2;
    if (ts < 1)
        return 0;
    // tile table, padding and a ticket (16 bytes), the weight table (k*k doubles) and its sum
    return B * (H / ts + 1) * (W / ts + 1) + 16 + 8 * (static_cast<int64_t>(kernel_size) * kernel_size + 1);
}

void launch_gaussian_blur(const void* images,
                          int idt,
                          int64_t B,
                          int64_t H,
                          int64_t W,
                          int kernel_size,
                          float sigma,
                          bool sparse,
                          void* out,
                          int odt,
                          uint8_t* scratch,
                          cudaStream_t s)
{
    const int64_t n = B * H * W;
    if (n == 0)
        return;
    const int grid = grid_for(n, 256);
    if (kernel_size == 1)
    {
        dispatch_image_dtype(idt, [&]<int DT>() {
            dispatch_out(odt, [&]<int OT>() { convert_kernel<DT, OT><<<grid, 256, 0, s>>>(images, out, n); });
        });
        TH_LAUNCH_CHECK();
        return;
    }
    BlurGeom g;
    g.B = B;
    g.H = H;
    g.W = W;
    g.k = kernel_size;
    g.ts = kernel_size / 2;
    g.TH = H / g.ts + 1;
    g.TW = W / g.ts + 1;
    const int64_t tile_bytes = B * g.TH * g.TW;
    uint8_t* tiles = scratch;
    const int64_t woff = (tile_bytes + 15) / 16 * 16;
    double* wtab = reinterpret_cast<double*>(scratch + woff);
    double* norm = wtab + static_cast<int64_t>(kernel_size) * kernel_size;
    const int64_t zero_bytes = sparse ? woff : 0;
    // The second pass's ticket: four bytes of the padding before the weights,
    // or, where that is shorter, of what it leaves of its 16 bytes at the end
    // (blur_tile_bytes).
    uint32_t* ticket = woff - tile_bytes >= 4 ? reinterpret_cast<uint32_t*>(scratch + woff - 4)
                                              : reinterpret_cast<uint32_t*>(norm + 1);
    const unsigned zero_blocks = static_cast<unsigned>(grid_for((zero_bytes + 15) / 16, 256 * 4));
    dispatch_out(odt, [&]<int OT>() {
        weights_kernel<OT><<<1 + (sparse ? zero_blocks : 0u), 256, 0, s>>>(kernel_size, sigma, !sparse, wtab, norm,
                                                                            reinterpret_cast<uint4*>(tiles), zero_bytes,
                                                                            sparse ? ticket : nullptr);
    });
    TH_LAUNCH_CHECK();
    if (sparse)
    {
        auto edges = [&]<int DT, int V>() {
            const int64_t units = B * ((H + kEdgeRows - 1) / kEdgeRows) * ((W + 32 * V - 1) / (32 * V));
            const unsigned egrid = static_cast<unsigned>(std::min<int64_t>((units + 7) / 8, 64LL * sm_count()));
            edge_tiles_kernel<DT, V><<<egrid, 256, 0, s>>>(images, out, odt, B, H, W, g.ts, g.TH, g.TW, tiles);
        };
        const bool aligned = (reinterpret_cast<uintptr_t>(images) | reinterpret_cast<uintptr_t>(out)) % 16 == 0;
        if (aligned && idt == odt && odt == TH_FLOAT16 && W % 8 == 0)
            edges.template operator()<TH_FLOAT16, 8>();
        else if (aligned && idt == odt && odt == TH_FLOAT32 && W % 4 == 0)
            edges.template operator()<TH_FLOAT32, 4>();
        else if (aligned && idt == odt && odt == TH_FLOAT64 && W % 2 == 0)
            edges.template operator()<TH_FLOAT64, 2>();
        else
            dispatch_image_dtype(idt, [&]<int DT>() { edges.template operator()<DT, 1>(); });
        TH_LAUNCH_CHECK();
    }
    bool done = false;
    dispatch_out(odt, [&]<int OT>() {
        done = sparse ? launch_tiles<OT, true>(images, idt, out, g, tiles, wtab, norm, ticket, s)
                      : launch_tiles<OT, false>(images, idt, out, g, tiles, wtab, norm, nullptr, s);
    });
    if (done)
        return;
    // kernels too wide for a block's shared memory: one pixel per thread
    dispatch_image_dtype(idt, [&]<int DT>() {
        dispatch_out(odt, [&]<int OT>() {
            if (sparse)
                blur_kernel<DT, OT, true><<<grid, 256, 0, s>>>(images, out, g, tiles, wtab, norm);
            else
                blur_kernel<DT, OT, false><<<grid, 256, 0, s>>>(images, out, g, tiles, wtab, norm);
        });
    });
    TH_LAUNCH_CHECK();
}

} // namespace th
