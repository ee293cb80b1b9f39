// Integral images (summed-area tables) of the masks, one per view.
//
// The reference builds them with torch::cumsum over H and then over W in
// float32 (visual_hull_cuda.cu:76-90).  torch scans a non-innermost dimension
// one element at a time from 0, so every SAT value is the float result of that
// fixed sequence of additions.
//
// Two implementations give that exact table:
//
// * 0/1 masks (the usual case) with H*W <= 2^24: every partial sum is an
//   integer below 2^24 + 1, so float32 addition is exact in any order.
//   sat_bits_kernel reads the masks once and keeps one bit per pixel, 32 rows
//   of a column to a word; sat_bands_kernel writes the table once, each block
//   a band of 32 rows: a column's sum at a row is the ones in the bands above
//   (popcounts) and the set bits so far, a row of the table the prefix sum of
//   those.  DRAM traffic: the masks read once and the table written once; the
//   words (a 32nd of the pixels) stay in L2.  Bound by that traffic.  No block
//   waits for another.  (A single kernel that staged bands in shared memory
//   and took the rows above them by decoupled look-back kept one to three
//   blocks on an SM: 64x2048^2 float32 1315 -> 362 us, 32x1024^2 125 -> 69,
//   6x128^2 14.2 -> 10.2.)
// * anything else (blurred masks, very large images): the two sequential
//   passes below, which perform exactly torch's additions in torch's order,
//   so the table is bit-identical for any mask values.  They also run, gated
//   on the device, after the bit passes when those found a value other than 0
//   or 1: they recompute the whole table then.
//
// Column pass: one thread per (view, column) walks down the column; a warp
// covers 32 adjacent columns, so each step is one coalesced 128-byte row read.
// Row pass: one warp per 32 rows walks across them through 32x33 shared
// tiles (coalesced loads and stores, one lane per row scanning its 32 values).
// HBM traffic: read masks + write columns + read columns + write SAT.

#include <cstring>

#include "th_common.cuh"
#include "th_internal.h"

namespace th
{

namespace
{

// rows of a column in flight per thread and half: the columns of a request are
// few threads, each a serial chain (24x512^2: 28.5 us with 16, 23.1 with 32)
constexpr int kColUnroll = 32;

// Column pass.  Also flags (nonbinary != nullptr) whether any mask value,
// as float, is neither 0 nor 1: binary masks make every SAT value an exact
// integer, which the carve's view skipping relies on.
template <int DT>
__global__ void __launch_bounds__(256) sat_columns_kernel(const void* __restrict__ masks,
                                                          float* __restrict__ out,
                                                          int64_t B,
                                                          int64_t H,
                                                          int64_t W,
                                                          unsigned int* __restrict__ nonbinary,
                                                          const unsigned int* __restrict__ gate)
{
    // gate: run only when the bit passes could not be used (see the file comment)
    if (gate && *gate == 0u)
        return;
    const int64_t col = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (col >= B * W)
        return;
    const int64_t b = col / W, x = col - b * W;
    const int64_t base = b * H * W + x;
    float acc = 0.f;
    bool nb = false;
    int64_t y = 0;
    // two chunks of rows in flight: the next chunk's loads are issued before
    // the current one is summed (a thread walks its column sequentially)
    const int64_t full = H - H % kColUnroll;
    float v[kColUnroll];
    if (full > 0)
    {
#pragma unroll
        for (int k = 0; k < kColUnroll; ++k)
            v[k] = load_f32<DT>(masks, base + k * W);
    }
    for (; y < full; y += kColUnroll)
    {
        float nx[kColUnroll];
        if (y + kColUnroll < full)
        {
#pragma unroll
            for (int k = 0; k < kColUnroll; ++k)
                nx[k] = load_f32<DT>(masks, base + (y + kColUnroll + k) * W);
        }
#pragma unroll
        for (int k = 0; k < kColUnroll; ++k)
        {
            nb |= (v[k] != 0.f) & (v[k] != 1.f);
            acc = __fadd_rn(acc, v[k]);
            out[base + (y + k) * W] = acc;
        }
#pragma unroll
        for (int k = 0; k < kColUnroll; ++k)
            v[k] = nx[k];
    }
    for (; y < H; ++y)
    {
        const float v = load_f32<DT>(masks, base + y * W);
        nb |= (v != 0.f) & (v != 1.f);
        acc = __fadd_rn(acc, v);
        out[base + y * W] = acc;
    }
    if (nb && nonbinary)
        atomicOr(nonbinary, 1u);
}

constexpr int kRowWarps = 4;

// Row pass: a warp owns 32 rows and walks across them in 32-column tiles
// through shared memory (coalesced loads and stores, a lane per row for the
// sums).  The next tile's loads are in flight while the current one is summed,
// and a row's 32 values leave shared memory before its chain of additions
// starts, so that only those wait for each other (24x512^2: 34.8 -> 13.5 us).
__global__ void __launch_bounds__(32 * kRowWarps) sat_rows_kernel(float* __restrict__ data, int64_t rows, int64_t W,
                                                                  const unsigned int* __restrict__ gate)
{
    if (gate && *gate == 0u)
        return;
    __shared__ float tile[kRowWarps][32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t row0 = (static_cast<int64_t>(blockIdx.x) * kRowWarps + warp) * 32;
    if (row0 >= rows)
        return;
    const int nrows = static_cast<int>(rows - row0 < 32 ? rows - row0 : 32);
    float(*t)[33] = tile[warp];
    float* at = data + row0 * W + lane; // the lane's column of the first tile
    float ahead[32];
    auto load = [&](int64_t x0) {
#pragma unroll
        for (int r = 0; r < 32; ++r)
            ahead[r] = r < nrows && x0 + lane < W ? at[r * W + x0] : 0.f;
    };
    load(0);
    float carry = 0.f;
    for (int64_t x0 = 0; x0 < W; x0 += 32)
    {
#pragma unroll
        for (int r = 0; r < 32; ++r)
            t[r][lane] = ahead[r];
        if (x0 + 32 < W)
            load(x0 + 32);
        __syncwarp();
        // the sums past the row's end are not stored
        float v[32];
#pragma unroll
        for (int c = 0; c < 32; ++c)
            v[c] = t[lane][c];
#pragma unroll
        for (int c = 0; c < 32; ++c)
        {
            carry = __fadd_rn(carry, v[c]);
            t[lane][c] = carry;
        }
        __syncwarp();
        if (x0 + lane < W)
        {
#pragma unroll
            for (int r = 0; r < 32; ++r)
                if (r < nrows)
                    at[r * W + x0] = t[r][lane];
        }
        __syncwarp();
    }
}

// ---- 0/1 masks ------------------------------------------------------------

constexpr int kBandRows = 32; // rows to a word
// The bands above a block's are counted by the block itself up to this many
// (a word per column each), from a table of prefix counts beyond: the launch
// for the table costs few views more than the counting up to about 48 bands,
// whose work grows with the square.  Integral images, counted against the
// table: 4x1024^2 (32 bands) 45.8 us against 48.2, 64x1024^2 133.3 against
// 129.8; 1x1536^2 (48) 53.6 against 54.0, 28x1536^2 142 against 136; 1x2048^2
// (64) 65 against 61, 16x2048^2 159 against 144; 4x4096^2 237 against 162.
constexpr int kCountedBands = 32;
constexpr int kCountedWidth = 8192; // columns whose counts fit the block's shared memory

struct SatBits
{
    uint32_t* words;  // [B][bands][pitch]: bit r of column x: pixel (32 band + r, x) is 1
    uint32_t* counts; // [B][bands][pitch]: ones of column x in the bands above (unless counted)
    int64_t H, W, bands, pitch;
    bool counted;
};

SatBits bits_shape(int64_t B, int64_t H, int64_t W)
{
    SatBits s{};
    s.H = H;
    s.W = W;
    s.bands = (H + kBandRows - 1) / kBandRows;
    s.pitch = (W + 3) / 4 * 4;
    s.counted = s.bands <= kCountedBands && W <= kCountedWidth;
    return s;
}

// The bit words.  A thread owns V columns (16 bytes where the rows allow it,
// else one) of a band and issues eight rows' loads at a time.
template <int DT, int V>
__global__ void __launch_bounds__(256) sat_bits_kernel(const void* __restrict__ masks, SatBits p, int64_t B, unsigned int* __restrict__ nonbinary)
{
    using T = typename Elem<DT>::T;
    const int64_t per_band = (p.W + V - 1) / V;
    const int64_t n = B * p.bands * per_band;
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    bool nb = false;
    if (t < n)
    {
        const int64_t vb = t / per_band, x = (t - vb * per_band) * V;
        const int64_t b = vb / p.bands, band = vb - b * p.bands;
        const int rows = static_cast<int>(p.H - band * kBandRows < kBandRows ? p.H - band * kBandRows : kBandRows);
        const T* src = static_cast<const T*>(masks) + (b * p.H + band * kBandRows) * p.W + x;
        uint32_t w[V];
#pragma unroll
        for (int i = 0; i < V; ++i)
            w[i] = 0;
        constexpr int kAhead = 8;
        for (int r0 = 0; r0 < rows; r0 += kAhead)
        {
            T v[kAhead][V];
#pragma unroll
            for (int r = 0; r < kAhead; ++r)
            {
                if (r0 + r < rows)
                {
                    if constexpr (V > 1)
                    {
                        const uint4 u = __ldcs(reinterpret_cast<const uint4*>(src + static_cast<int64_t>(r0 + r) * p.W));
                        memcpy(v[r], &u, sizeof(u));
                    }
                    else
                        v[r][0] = src[static_cast<int64_t>(r0 + r) * p.W];
                }
            }
#pragma unroll
            for (int r = 0; r < kAhead; ++r)
            {
                if (r0 + r < rows)
                {
#pragma unroll
                    for (int i = 0; i < V; ++i)
                    {
                        const float f = load_f32<DT>(&v[r][i], 0);
                        nb |= (f != 0.f) & (f != 1.f);
                        w[i] |= f == 1.f ? 1u << (r0 + r) : 0u;
                    }
                }
            }
        }
        uint32_t* out = p.words + vb * p.pitch + x;
        if constexpr (V >= 4)
        {
#pragma unroll
            for (int i = 0; i < V; i += 4)
                *reinterpret_cast<uint4*>(out + i) = make_uint4(w[i], w[i + 1], w[i + 2], w[i + 3]);
        }
        else
        {
#pragma unroll
            for (int i = 0; i < V; ++i)
                out[i] = w[i];
        }
    }
    if (__syncthreads_or(nb) && threadIdx.x == 0)
        atomicOr(nonbinary, 1u);
}

// Ones above each band, a thread per column of a view.
__global__ void __launch_bounds__(128) sat_counts_kernel(SatBits p, int64_t B)
{
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= B * p.W)
        return;
    const int64_t b = t / p.W, x = t - b * p.W;
    const uint32_t* words = p.words + b * p.bands * p.pitch + x;
    uint32_t* counts = p.counts + b * p.bands * p.pitch + x;
    uint32_t sum = 0;
#pragma unroll 8
    for (int64_t i = 0; i < p.bands; ++i)
    {
        counts[i * p.pitch] = sum;
        sum += __popc(__ldg(words + i * p.pitch));
    }
}

// The table: a block per band, a warp per four rows, which share the words'
// loads and whose warp scans overlap; V columns per lane (4 where the table's
// rows are 16-byte aligned).
constexpr int kRowsPerWarp = 4;

template <int V>
__global__ void __launch_bounds__(32 * kBandRows / kRowsPerWarp) sat_bands_kernel(SatBits p, float* __restrict__ out)
{
    extern __shared__ uint32_t above_s[]; // counted: the columns' ones above the band
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t vb = blockIdx.x, b = vb / p.bands, band = vb - b * p.bands;
    const uint32_t* words = p.words + vb * p.pitch;
    const uint32_t* above = p.counts + vb * p.pitch;
    if (p.counted)
    {
        const uint32_t* first = p.words + b * p.bands * p.pitch;
        for (int64_t x = threadIdx.x; x < p.W; x += blockDim.x)
        {
            uint32_t sum = 0;
#pragma unroll 8
            for (int64_t i = 0; i < band; ++i)
                sum += __popc(__ldg(first + i * p.pitch + x));
            above_s[x] = sum;
        }
        __syncthreads();
    }
    const int r0 = warp * kRowsPerWarp;
    const int64_t y0 = band * kBandRows + r0;
    if (y0 >= p.H)
        return;
    const int rows = static_cast<int>(p.H - y0 < kRowsPerWarp ? p.H - y0 : kRowsPerWarp);
    float* dst = out + (b * p.H + y0) * p.W;
    const uint32_t low = (2u << r0) - 1u; // the rows up to the warp's first (r0 is at most 28)
    int32_t carry[kRowsPerWarp] = { 0, 0, 0, 0 };
    for (int64_t x0 = 0; x0 < p.W; x0 += 32 * V)
    {
        const int64_t x = x0 + lane * V;
        uint32_t w[V], col[V];
        // V > 1: W is a multiple of V; pitch rows start on 16 bytes
        const bool in = x < p.W;
        if constexpr (V == 4)
        {
            const uint4 u = in ? __ldg(reinterpret_cast<const uint4*>(words + x)) : make_uint4(0u, 0u, 0u, 0u);
            const uint4 a = !in ? make_uint4(0u, 0u, 0u, 0u)
                                : p.counted ? *reinterpret_cast<const uint4*>(above_s + x) : __ldg(reinterpret_cast<const uint4*>(above + x));
            w[0] = u.x, w[1] = u.y, w[2] = u.z, w[3] = u.w;
            col[0] = a.x, col[1] = a.y, col[2] = a.z, col[3] = a.w;
        }
        else
        {
            w[0] = in ? __ldg(words + x) : 0u;
            col[0] = !in ? 0u : p.counted ? above_s[x] : __ldg(above + x);
        }
#pragma unroll
        for (int i = 0; i < V; ++i)
            col[i] += __popc(w[i] & low);
#pragma unroll
        for (int r = 0; r < kRowsPerWarp; ++r)
        {
            if (r > 0)
            {
#pragma unroll
                for (int i = 0; i < V; ++i)
                    col[i] += (w[i] >> (r0 + r)) & 1u;
            }
            int32_t pre[V];
            pre[0] = static_cast<int32_t>(col[0]);
#pragma unroll
            for (int i = 1; i < V; ++i)
                pre[i] = pre[i - 1] + static_cast<int32_t>(col[i]);
            const int32_t incl = warp_inclusive_scan(pre[V - 1]);
            const int32_t base = carry[r] + incl - pre[V - 1];
            carry[r] += __shfl_sync(0xffffffffu, incl, 31);
            if (in && r < rows)
            {
                float* o = dst + r * p.W + x;
                if constexpr (V == 4)
                    *reinterpret_cast<float4*>(o) = make_float4(__int2float_rn(base + pre[0]), __int2float_rn(base + pre[1]),
                                                                __int2float_rn(base + pre[2]), __int2float_rn(base + pre[3]));
                else
                    *o = __int2float_rn(base + pre[0]);
            }
        }
    }
}

bool bits_apply(int64_t B, int64_t H, int64_t W, int dtype)
{
    return dtype >= TH_UINT8 && dtype <= TH_FLOAT64 && B > 0 && H > 0 && W > 0 && H * W <= (int64_t{ 1 } << 24) &&
           B * ((H + kBandRows - 1) / kBandRows) < (int64_t{ 1 } << 31);
}

} // namespace

int64_t sat_scratch_bytes(int64_t B, int64_t H, int64_t W, int dtype)
{
    if (!bits_apply(B, H, W, dtype))
        return 0;
    const SatBits bits = bits_shape(B, H, W);
    return (bits.counted ? 1 : 2) * 4 * B * bits.bands * bits.pitch;
}

void launch_integral_image(const void* masks,
                           int dtype,
                           int64_t B,
                           int64_t H,
                           int64_t W,
                           float* out,
                           cudaStream_t s,
                           unsigned int* nonbinary,
                           SatScratch scratch)
{
    if (B * H * W == 0)
        return;
    const unsigned int* gate = nullptr;
    if (bits_apply(B, H, W, dtype) && scratch.p && nonbinary)
    {
        SatBits bits = bits_shape(B, H, W);
        const int64_t n = B * bits.bands * bits.pitch;
        bits.words = static_cast<uint32_t*>(scratch.p);
        bits.counts = bits.words + (bits.counted ? 0 : n);
        const bool ok = dispatch_image_dtype(dtype, [&]<int DT>() {
            constexpr int V = 16 / static_cast<int>(sizeof(typename Elem<DT>::T));
            const bool vec = reinterpret_cast<uintptr_t>(masks) % 16 == 0 && W % V == 0;
            const int64_t threads = B * bits.bands * ((W + (vec ? V : 1) - 1) / (vec ? V : 1));
            const unsigned grid = static_cast<unsigned>((threads + 255) / 256);
            if (vec)
                sat_bits_kernel<DT, V><<<grid, 256, 0, s>>>(masks, bits, B, nonbinary);
            else
                sat_bits_kernel<DT, 1><<<grid, 256, 0, s>>>(masks, bits, B, nonbinary);
        });
        if (!ok)
            throw CudaError{ cudaErrorInvalidValue, "integral image: unsupported mask dtype" };
        TH_LAUNCH_CHECK();
        if (!bits.counted)
        {
            sat_counts_kernel<<<static_cast<unsigned>((B * W + 127) / 128), 128, 0, s>>>(bits, B);
            TH_LAUNCH_CHECK();
        }
        const unsigned blocks = static_cast<unsigned>(B * bits.bands), threads = 32 * kBandRows / kRowsPerWarp;
        const size_t smem = bits.counted ? sizeof(uint32_t) * static_cast<size_t>(bits.pitch) : 0;
        if (reinterpret_cast<uintptr_t>(out) % 16 == 0 && W % 4 == 0)
            sat_bands_kernel<4><<<blocks, threads, smem, s>>>(bits, out);
        else
            sat_bands_kernel<1><<<blocks, threads, smem, s>>>(bits, out);
        TH_LAUNCH_CHECK();
        gate = nonbinary; // the exact passes below run only if the masks were not 0/1
    }
    const int64_t cols = B * W;
    const unsigned grid = static_cast<unsigned>((cols + 255) / 256);
    bool ok = dispatch_image_dtype(dtype, [&]<int DT>() {
        sat_columns_kernel<DT><<<grid, 256, 0, s>>>(masks, out, B, H, W, nonbinary, gate);
    });
    if (!ok)
        throw CudaError{ cudaErrorInvalidValue, "integral image: unsupported mask dtype" };
    TH_LAUNCH_CHECK();
    const int64_t rows = B * H;
    const unsigned grid_rows = static_cast<unsigned>((rows + 32 * kRowWarps - 1) / (32 * kRowWarps));
    sat_rows_kernel<<<grid_rows, 32 * kRowWarps, 0, s>>>(out, rows, W, gate);
    TH_LAUNCH_CHECK();
}

} // namespace th
