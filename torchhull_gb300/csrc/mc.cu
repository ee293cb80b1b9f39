// Public marching cubes over a dense volume or a coalesced sparse COO volume
// (torchhull marching_cubes: marching_cubes_cuda.cu:376-533 for dense
// volumes, :535-831 for sparse ones).
//
// The reference builds a triangle soup (one vertex per table entry of every
// active cell, cells ascending, table order inside a cell), keys each soup
// vertex by its edge id (ravel(lower end point) << 3 | direction, :99-112,
// direction 1 / 2 / 4 for x / y / z) and sorts the keys with unique_dim; the
// faces are the soup's inverse indices.  The unique vertices therefore come
// in edge-id order: by the ravel index of the lower end point, then by axis.
// Here that order is produced directly: every grid point carries three bits
// (its +x, +y, +z edge holds a vertex), prefix sums number the set bits, and a
// face looks up its vertex as the number of set bits before its edge; no sort
// runs.  Dense volumes, and sparse ones that are not too empty, do this on
// words of 32 points (th_words.cuh); a very sparse volume keeps its entries in
// a hash table.
//
// Which edges hold vertices: every cell's triangulation uses exactly the cell
// edges whose end points lie on different sides of the isolevel (a property
// of the table, checked by the tests).  In a dense volume with all sizes >= 2
// every edge belongs to some cell, so the bits follow from the values alone.
// In a sparse volume an edge counts only when a complete cell (all 8 corners
// present) holds it.
//
// Axes: x runs along the last volume dimension (W), y along H, z along the
// first (D).  The reference mixes D and W in its index arithmetic; for
// volumes with D == W (all of its tests) that mixing is invisible and the
// results here are identical.

#include <cstring>
#include <cuda_fp16.h>

#include "mc_tables.h"
#include "th_internal.h"
#include "th_mc.cuh"

namespace th
{
namespace
{

__device__ const uint8_t mc_count[256] = TH_MC_TRI_COUNT_INIT;
__device__ const uint8_t mc_edges[256][15] = TH_MC_TRI_EDGES_INIT;

constexpr unsigned long long kEmptyKey = ~0ull;

// value < isolevel, compared in the value's own type (:166-171, :210-213).
template <int DT>
__device__ __forceinline__ bool below(const void* v, int64_t i, float iso)
{
    if constexpr (DT == TH_FLOAT64)
        return static_cast<const double*>(v)[i] < static_cast<double>(iso);
    else
        return load_f32<DT>(v, i) < iso;
}

// interpolate_vertex (:72-97) on the edge from point (x, y, z) along axis,
// then the optional map to local coordinates: v * 2 / (size - 1) - 1 as two
// rounded torch operations (:524-531).
__device__ __forceinline__ void mc_vertex(const McPlan& p, int64_t x, int64_t y, int64_t z, int axis, float v1, float v2, float* out)
{
    const float eps = 1e-5f;
    const int64_t c1[3] = { x, y, z };
    float q[3];
    // the reference's check order: snap to p1, to p2, then to p1 again
    int snap = 0;
    if (fabsf(__fsub_rn(p.iso, v1)) < eps)
        snap = 1;
    else if (fabsf(__fsub_rn(p.iso, v2)) < eps)
        snap = 2;
    else if (fabsf(__fsub_rn(v1, v2)) < eps)
        snap = 1;
    const float t = snap ? 0.f : __fdiv_rn(__fsub_rn(p.iso, v1), __fsub_rn(v2, v1));
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        // exact float conversions by adds below 2^23 (the 64-bit integer
        // conversions run on GB300's FP64 pipe)
        const int64_t i1 = c1[a], i2 = c1[a] + (a == axis ? 1 : 0);
        const float f1 = i1 < 8388608 ? small_i2f(static_cast<int32_t>(i1)) : static_cast<float>(i1);
        const float f2 = i2 < 8388608 ? small_i2f(static_cast<int32_t>(i2)) : static_cast<float>(i2);
        q[a] = snap == 1 ? f1 : (snap == 2 ? f2 : lerp(f1, f2, t));
        out[a] = p.local ? __fsub_rn(__fmul_rn(q[a], p.scale[a]), 1.f) : q[a];
    }
}

// ---------------------------------------------------------------------------
// dense volumes

// Triangle corners << 32 | vertices of the whole mesh (more than 2^28 active
// cells, 15 corners each, are refused: no total that is used has wrapped).
struct WordTotal
{
    McCounters* ctr;
    __device__ void operator()(unsigned long long t, bool) const
    {
        ctr->soup = t >> 32;
        ctr->verts = t & 0xffffffffull;
    }
    __device__ void block() const {}
};

struct SoupTotal
{
    McCounters* ctr;
    __device__ void operator()(unsigned long long t) const
    {
        ctr->soup = t;
    }
};

struct VertTotal
{
    McCounters* ctr;
    __device__ void operator()(unsigned long long t) const
    {
        ctr->verts = t;
    }
};

// Rows of a volume in words: word k is in row k / wr (y + H * z).
struct VolumeWords
{
    McPlan p;

    __device__ int64_t words() const
    {
        return p.nwords;
    }
    __device__ int64_t counted() const
    {
        return p.own;
    }
    __device__ uint32_t word(uint32_t i) const
    {
        return i;
    }
    __device__ void tail() const {}
    __device__ uint32_t sign(uint32_t k) const
    {
        return __ldg(p.sign + k);
    }
    // Word k's place: w in its row, y and z.
    __device__ void place(uint32_t k, uint32_t& w, uint32_t& y, uint32_t& z) const
    {
        const uint32_t row = fast_div(p.div_wr, k);
        w = k - row * p.wr;
        z = fast_div(p.div_h, row);
        y = row - z * p.div_h.d;
    }
    __device__ WordRows rows(uint32_t k) const
    {
        uint32_t w, y, z;
        place(k, w, y, z);
        WordRows r;
        r.next = w + 1 < p.wr;
        const bool up = y + 1 < p.div_h.d, back = static_cast<int64_t>(z) + 1 < p.D;
        const uint32_t plane = p.wr * p.div_h.d;
        r.idx[0] = k;
        r.idx[1] = up ? k + p.wr : kNoWord;
        r.idx[2] = back ? k + plane : kNoWord;
        r.idx[3] = up && back ? k + p.wr + plane : kNoWord;
        return r;
    }
};

template <int DT>
struct DenseWords : VolumeWords
{
    __device__ bool empty(uint32_t) const
    {
        return false;
    }
    // every edge inside the volume belongs to some cell
    __device__ EdgeBits edges(uint32_t k, const WordRows& r, const uint32_t s[4], const uint32_t sh[4], uint32_t& cells) const
    {
        const int64_t points = p.W - static_cast<int64_t>(k - fast_div(p.div_wr, k) * p.wr) * 32; // at least 1
        const uint32_t in = points >= 32 ? 0xffffffffu : (1u << points) - 1u;
        const uint32_t start = points > 32 ? 0xffffffffu : (1u << (points - 1)) - 1u; // with a right neighbour
        cells = r.idx[3] != kNoWord ? start : 0u;
        return EdgeBits{ (s[0] ^ sh[0]) & start, r.idx[1] != kNoWord ? (s[0] ^ s[1]) & in : 0u,
                         r.idx[2] != kNoWord ? (s[0] ^ s[2]) & in : 0u };
    }
    __device__ int64_t point(uint32_t k, int b, int64_t& x, int64_t& y, int64_t& z) const
    {
        uint32_t w, yy, zz;
        place(k, w, yy, zz);
        x = static_cast<int64_t>(w) * 32 + b;
        y = yy;
        z = zz;
        return (y + z * p.H) * p.W + x;
    }
    __device__ void vertex(uint32_t k, int b, int axis, float out[3]) const
    {
        int64_t x, y, z;
        const int64_t q = point(k, b, x, y, z);
        const int64_t q2 = q + (axis == 0 ? 1 : (axis == 1 ? p.W : p.W * p.H));
        mc_vertex(p, x, y, z + p.z0, axis, load_f32<DT>(p.volume, q), load_f32<DT>(p.volume, q2), out);
    }
    __device__ void values_at(const WordRows& r, int b, unsigned long long* corner) const
    {
        int64_t x, y, z;
        const int64_t q = point(r.idx[0], b, x, y, z);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            corner[i] = static_cast<unsigned long long>(q + (i & 1) + (i >> 1 & 1) * p.W + (i >> 2) * (p.W * p.H));
    }
    __device__ void soup_vertex(uint32_t k, int b, int lo, int axis, unsigned long long h1, unsigned long long h2, float out[3]) const
    {
        int64_t x, y, z;
        point(k, b, x, y, z);
        mc_vertex(p, x + (lo & 1), y + (lo >> 1 & 1), z + p.z0 + (lo >> 2 & 1), axis,
                  load_f32<DT>(p.volume, static_cast<int64_t>(h1)), load_f32<DT>(p.volume, static_cast<int64_t>(h2)), out);
    }
};

// Sign words of a dense volume: the only pass over its values.  VEC (rows and
// volume on 16-byte boundaries): a lane loads 16 bytes, the 32 / V lanes of a
// word OR their bits by shuffles, a warp makes V words per load and issues
// kSignLoads of them first.  Else a point per lane and a ballot per word.  The
// index arithmetic per word bounds the scalar form: 400^3 float32 117 us
// against 47 us for the vector form (256 MB: 38 us at the copy rate).
constexpr int kSignLoads = 8;

template <int DT, bool VEC>
__global__ void __launch_bounds__(256) mc_sign_kernel(McPlan p)
{
    using T = typename Elem<DT>::T;
    constexpr int V = VEC ? 16 / static_cast<int>(sizeof(T)) : 1; // points per lane = words per load
    constexpr int kLanes = 32 / V;                                // lanes per word
    const int lane = threadIdx.x & 31, sub = lane % kLanes;
    const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    constexpr int kWords = kSignLoads * V;
    const int64_t groups = (p.nwords + kWords - 1) / kWords;
    const T* volume = static_cast<const T*>(p.volume);
    for (int64_t g = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; g < groups; g += nwarps)
    {
        T v[kSignLoads][V];
        uint32_t in = 0;
#pragma unroll
        for (int i = 0; i < kSignLoads; ++i)
        {
            const int64_t kk = g * kWords + i * V + lane / kLanes;
            const uint32_t k = static_cast<uint32_t>(kk < p.nwords ? kk : p.nwords - 1);
            const uint32_t row = fast_div(p.div_wr, k);
            const int64_t x = static_cast<int64_t>(k - row * p.wr) * 32 + sub * V;
            const T* src = volume + static_cast<int64_t>(row) * p.W + x;
            // VEC: W is a multiple of V, so the V points are in the row or none is
            if (x < p.W)
            {
                in |= 1u << i;
                if constexpr (VEC)
                {
                    const uint4 w = __ldcs(reinterpret_cast<const uint4*>(src));
                    memcpy(v[i], &w, sizeof(w));
                }
                else
                    v[i][0] = *src;
            }
        }
#pragma unroll
        for (int i = 0; i < kSignLoads; ++i)
        {
            uint32_t word = 0;
            if ((in >> i) & 1u)
            {
#pragma unroll
                for (int j = 0; j < V; ++j)
                    word |= below<DT>(&v[i][j], 0, p.iso) ? 1u << j : 0u;
            }
            if constexpr (VEC)
            {
                word <<= sub * V;
#pragma unroll
                for (int d = kLanes / 2; d > 0; d >>= 1)
                    word |= __shfl_xor_sync(0xffffffffu, word, d);
            }
            else
                word = __ballot_sync(0xffffffffu, word != 0u);
            const int64_t k = g * kWords + i * V + lane / kLanes;
            if (sub == 0 && k < p.nwords)
                p.sign[k] = word;
        }
    }
}

// ---------------------------------------------------------------------------
// sparse volumes: an open-addressing table from ravel id to entry index
// (the reference uses a stdgpu unordered_map, :729-751)

// MurmurHash3's 64-bit finalizer (fmix64).
__device__ __forceinline__ uint64_t mix64(uint64_t k)
{
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return k;
}

// Entry t's coordinates, or false when it lies outside the volume.
__device__ __forceinline__ bool entry_point(const McPlan& p, int64_t t, int64_t& x, int64_t& y, int64_t& z)
{
    const int64_t b = p.indices[t];
    z = p.indices[p.nnz + t];
    y = p.indices[2 * p.nnz + t];
    x = p.indices[3 * p.nnz + t];
    return b == 0 && 0 <= x && x < p.W && 0 <= y && y < p.H && 0 <= z && z < p.D;
}

__device__ __forceinline__ int32_t mc_find(const McPlan& p, unsigned long long key)
{
    uint64_t slot = mix64(key) & p.hmask;
    for (uint64_t k = 0; k <= p.hmask; ++k)
    {
        const unsigned long long kk = p.keys[slot];
        if (kk == key)
            return p.slots[slot];
        if (kk == kEmptyKey)
            return -1;
        slot = (slot + 1) & p.hmask;
    }
    return -1;
}

// hash_volume (:114-131): every entry's ravel id into the table; flags
// entries outside the volume and indices that are not strictly ascending.
__global__ void __launch_bounds__(256) mc_sparse_insert_kernel(McPlan p)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < p.nnz; t += stride)
    {
        int64_t x, y, z;
        if (!entry_point(p, t, x, y, z))
        {
            atomicOr(&p.ctr->flags, static_cast<unsigned int>(kMcBadIndex));
            continue;
        }
        const unsigned long long key = static_cast<unsigned long long>(x + p.W * (y + p.H * z));
        if (t > 0)
        {
            int64_t px, py, pz;
            if (entry_point(p, t - 1, px, py, pz) &&
                static_cast<unsigned long long>(px + p.W * (py + p.H * pz)) >= key)
                atomicOr(&p.ctr->flags, static_cast<unsigned int>(kMcUnsorted));
        }
        uint64_t slot = mix64(key) & p.hmask;
        for (uint64_t k = 0; k <= p.hmask; ++k)
        {
            const unsigned long long prev = atomicCAS(&p.keys[slot], kEmptyKey, key);
            if (prev == kEmptyKey || prev == key)
            {
                p.slots[slot] = static_cast<int32_t>(t);
                break;
            }
            slot = (slot + 1) & p.hmask;
        }
    }
}

// Entry indices of the 8 corners of the cell with base entry t at (x, y, z)
// (corner i = base + (i & 1, i >> 1 & 1, i >> 2 & 1)); false if one is absent.
__device__ __forceinline__ bool cell_entries(const McPlan& p, int64_t t, int64_t x, int64_t y, int64_t z, int32_t c[8])
{
    if (!(x + 1 < p.W && y + 1 < p.H && z + 1 < p.D))
        return false;
    const unsigned long long key = static_cast<unsigned long long>(x + p.W * (y + p.H * z));
    const unsigned long long WH = static_cast<unsigned long long>(p.W * p.H);
    c[0] = static_cast<int32_t>(t);
#pragma unroll
    for (int i = 1; i < 8; ++i)
    {
        c[i] = mc_find(p, key + (i & 1) + ((i >> 1) & 1) * static_cast<unsigned long long>(p.W) + ((i >> 2) & 1) * WH);
        if (c[i] < 0)
            return false;
    }
    return true;
}

// classify_voxels_sparse (:180-223) plus, with unique vertices, the marking of
// the cell's vertex edges on the entries of their lower end points.
template <int DT>
__global__ void __launch_bounds__(256) mc_sparse_classify_kernel(McPlan p)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < p.nnz; t += stride)
    {
        int64_t x, y, z;
        int32_t c[8];
        int code = 0;
        if (entry_point(p, t, x, y, z) && cell_entries(p, t, x, y, z, c))
        {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (below<DT>(p.values, c[i], p.iso))
                    code |= 1 << i;
            if (p.unique && mc_count[code] != 0)
            {
                // corner lo owns the edges along the axes where its bit is 0;
                // an edge is a vertex edge when its two ends differ in the code
#pragma unroll
                for (int lo = 0; lo < 8; ++lo)
                {
                    uint32_t bits = 0;
#pragma unroll
                    for (int a = 0; a < 3; ++a)
                        if (!((lo >> a) & 1) && (((code >> lo) ^ (code >> (lo | (1 << a)))) & 1))
                            bits |= 1u << a;
                    if (bits)
                        atomicOr(&p.used[c[lo]], bits);
                }
            }
        }
        p.codes[t] = static_cast<uint8_t>(code);
    }
}

// Sparse volumes in words: the entries are in row order, so an entry's index
// is its word's first entry plus the present points before it.
template <int DT>
struct SparseWords : VolumeWords
{
    __device__ bool empty(uint32_t k) const
    {
        return __ldg(p.present + k) == 0;
    }
    __device__ EdgeBits edges(uint32_t k, const WordRows& r, const uint32_t s[4], const uint32_t sh[4], uint32_t& cells) const
    {
        uint32_t w, y, z;
        place(k, w, y, z);
        const uint32_t plane = p.wr * p.div_h.d;
        const bool low[2] = { y > 0, z > 0 }, high[2] = { y + 1 < p.div_h.d, static_cast<int64_t>(z) + 1 < p.D };
        return masked_edges(
                [&](int dy, int dz) {
                    if ((dy < 0 && !low[0]) || (dy > 0 && !high[0]) || (dz < 0 && !low[1]) || (dz > 0 && !high[1]))
                        return make_uint2(0u, 0u);
                    const uint32_t* bits = p.present + (k + dy * p.wr + dz * plane);
                    return word_runs(w > 0 ? __ldg(bits - 1) : 0u, __ldg(bits), r.next ? __ldg(bits + 1) : 0u);
                },
                s, sh, cells);
    }
    __device__ uint32_t entry(uint32_t k, int b) const
    {
        return __ldg(p.rank + k) + static_cast<uint32_t>(__popc(__ldg(p.present + k) & ((1u << b) - 1u)));
    }
    __device__ void vertex(uint32_t k, int b, int axis, float out[3]) const
    {
        const WordRows r = rows(k);
        const uint32_t e1 = entry(k, b);
        // the edge's other end is an entry: a complete cell holds both
        const uint32_t e2 = axis == 0 ? e1 + 1 : entry(r.idx[axis], b);
        uint32_t w, y, z;
        place(k, w, y, z);
        mc_vertex(p, static_cast<int64_t>(w) * 32 + b, y, z, axis, load_f32<DT>(p.values, e1), load_f32<DT>(p.values, e2), out);
    }
    __device__ void values_at(const WordRows& r, int b, unsigned long long* corner) const
    {
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            const uint32_t e = entry(r.idx[q], b);
            corner[2 * q] = e;
            corner[2 * q + 1] = e + 1;
        }
    }
    __device__ void soup_vertex(uint32_t k, int b, int lo, int axis, unsigned long long h1, unsigned long long h2, float out[3]) const
    {
        uint32_t w, y, z;
        place(k, w, y, z);
        mc_vertex(p, static_cast<int64_t>(w) * 32 + b + (lo & 1), static_cast<int64_t>(y) + (lo >> 1 & 1),
                  static_cast<int64_t>(z) + (lo >> 2 & 1), axis, load_f32<DT>(p.values, static_cast<int64_t>(h1)), load_f32<DT>(p.values, static_cast<int64_t>(h2)), out);
    }
};

// The entries' presence and sign bits and each word's first entry; flags
// entries outside the volume and indices that are not strictly ascending.
// Entries of one word are neighbours, so a warp ORs each word's bits first.
template <int DT>
__global__ void __launch_bounds__(256) mc_sparse_words_kernel(McPlan p)
{
    const int lane = threadIdx.x & 31;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x - lane; t0 < p.nnz; t0 += stride)
    {
        const int64_t t = t0 + lane;
        const bool valid = t < p.nnz;
        int64_t x = 0, y = 0, z = 0;
        const bool in = valid && entry_point(p, t, x, y, z);
        if (valid && !in)
            atomicOr(&p.ctr->flags, static_cast<unsigned int>(kMcBadIndex));
        const uint32_t word = in ? static_cast<uint32_t>((y + p.H * z) * p.wr + (x >> 5)) : kNoWord;
        // the entry before: the left lane's, or read
        int64_t px = __shfl_up_sync(0xffffffffu, x, 1), py = __shfl_up_sync(0xffffffffu, y, 1), pz = __shfl_up_sync(0xffffffffu, z, 1);
        bool pin = __shfl_up_sync(0xffffffffu, in ? 1 : 0, 1) != 0;
        if (lane == 0)
            pin = valid && t > 0 && entry_point(p, t - 1, px, py, pz);
        uint32_t pword = kNoWord;
        if (in && pin)
        {
            pword = static_cast<uint32_t>((py + p.H * pz) * p.wr + (px >> 5));
            if (px + p.W * (py + p.H * pz) >= x + p.W * (y + p.H * z))
                atomicOr(&p.ctr->flags, static_cast<unsigned int>(kMcUnsorted));
        }
        if (in && pword != word)
            p.rank[word] = static_cast<uint32_t>(t);
        const uint32_t bit = in ? 1u << (x & 31) : 0u;
        const uint32_t low = in && below<DT>(p.values, t, p.iso) ? bit : 0u;
        const uint32_t peers = __match_any_sync(0xffffffffu, word);
        const uint32_t bits = __reduce_or_sync(peers, bit), lows = __reduce_or_sync(peers, low);
        if (in && lane == __ffs(peers) - 1)
        {
            atomicOr(p.present + word, bits);
            if (lows)
                atomicOr(p.sign + word, lows);
        }
    }
}

struct SparseSoupCount
{
    const uint8_t* codes;
    __device__ unsigned long long operator()(int64_t t) const
    {
        return static_cast<unsigned long long>(mc_count[codes[t]]);
    }
};

struct SparseVertCount
{
    const uint32_t* used;
    __device__ unsigned long long operator()(int64_t t) const
    {
        return static_cast<unsigned long long>(__popc(used[t]));
    }
};

struct SparseVertEmit
{
    unsigned long long* vbase;
    __device__ void operator()(int64_t t, unsigned long long off, unsigned long long) const
    {
        vbase[t] = off;
    }
};

// The unique vertices, in edge-id order (entries are in ravel order).
template <int DT>
__global__ void __launch_bounds__(256) mc_sparse_verts_kernel(McPlan p, float* __restrict__ verts)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    const unsigned long long step[3] = { 1ull, static_cast<unsigned long long>(p.W),
                                         static_cast<unsigned long long>(p.W * p.H) };
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < p.nnz; t += stride)
    {
        const uint32_t bits = p.used[t];
        if (!bits)
            continue;
        int64_t x, y, z;
        entry_point(p, t, x, y, z);
        const unsigned long long key = static_cast<unsigned long long>(x + p.W * (y + p.H * z));
        const float v1 = load_f32<DT>(p.values, t);
        unsigned long long r = p.vbase[t];
#pragma unroll
        for (int a = 0; a < 3; ++a)
        {
            if (!((bits >> a) & 1u))
                continue;
            // present: a complete cell holds this edge
            const int32_t t2 = mc_find(p, key + step[a]);
            const float v2 = t2 >= 0 ? load_f32<DT>(p.values, t2) : __int_as_float(0x7fffffff);
            mc_vertex(p, x, y, z, a, v1, v2, verts + 3 * r);
            ++r;
        }
    }
}

// Soup of one active entry (generate_faces_sparse :308-374).
template <int DT>
struct SparseCellEmit
{
    McPlan p;
    float* verts;
    int64_t* faces;
    __device__ void operator()(int64_t t, unsigned long long off, unsigned long long cnt) const
    {
        if (cnt == 0)
            return;
        int64_t x, y, z;
        int32_t c[8];
        entry_point(p, t, x, y, z);
        if (!cell_entries(p, t, x, y, z, c))
            return; // not reached: an entry with a count has all its corners
        const int code = p.codes[t];
        for (int j = 0; j < static_cast<int>(cnt); ++j)
        {
            const uint32_t e = mc_edges[code][j];
            const int lo = static_cast<int>(e & 7u), axis = static_cast<int>(e >> 3);
            const int64_t k = static_cast<int64_t>(off) + j;
            const int32_t c1 = c[lo];
            if (p.unique)
            {
                faces[k] = static_cast<int64_t>(p.vbase[c1] + __popc(p.used[c1] & ((1u << axis) - 1u)));
            }
            else
            {
                const int32_t c2 = c[lo | (1 << axis)];
                mc_vertex(p, x + (lo & 1), y + ((lo >> 1) & 1), z + ((lo >> 2) & 1), axis, load_f32<DT>(p.values, c1),
                          load_f32<DT>(p.values, c2), verts + 3 * k);
                faces[k] = k;
            }
        }
    }
};

template <class Src>
void words_count(const Src& src, bool number, cudaStream_t s)
{
    const McPlan& p = src.p;
    const int grid = words_grid(p.nwords);
    if (p.unique)
        words_count_kernel<Src, true><<<grid, kWordThreads, 0, s>>>(src, p.mesh, &p.ctr->scan_soup, &p.ctr->active, WordTotal{ p.ctr });
    else
        words_count_kernel<Src, false><<<grid, kWordThreads, 0, s>>>(src, p.mesh, &p.ctr->scan_soup, &p.ctr->active, WordTotal{ p.ctr });
    TH_LAUNCH_CHECK();
    if (!number)
        return;
    words_base_kernel<Src><<<grid, kWordThreads, 0, s>>>(src, p.mesh);
    TH_LAUNCH_CHECK();
}

template <class Src>
void words_emit(const Src& src, float* verts, int64_t* faces, cudaStream_t s)
{
    const McPlan& p = src.p;
    const int grid = words_export_grid(p.nwords);
    launch_words_export<Src, false>(src, p.mesh, p.unique, grid, verts, faces, s);
}

template <int DT>
void dense_signs(const McPlan& p, cudaStream_t s)
{
    constexpr int V = 16 / static_cast<int>(sizeof(typename Elem<DT>::T));
    if (reinterpret_cast<uintptr_t>(p.volume) % 16 == 0 && p.W % V == 0)
        mc_sign_kernel<DT, true><<<grid_for(p.nwords * 32 / (kSignLoads * V) + 32, 256), 256, 0, s>>>(p);
    else
        mc_sign_kernel<DT, false><<<grid_for(p.nwords * 32 / kSignLoads + 32, 256), 256, 0, s>>>(p);
    TH_LAUNCH_CHECK();
}

template <int DT>
void dense_count(const McPlan& p, cudaStream_t s)
{
    dense_signs<DT>(p, s);
    words_count(DenseWords<DT>{ { p } }, true, s);
}

// The numbering that the next slab goes on from: what comes before word p.own,
// or the total when there is no halo.
__global__ void __launch_bounds__(32) mc_slab_end_kernel(McPlan p)
{
    unsigned long long at = p.ctr->scan_soup.total;
    if (p.own < p.nwords)
    {
        const int64_t first = p.own & ~int64_t{ 31 };
        const uint32_t c = first + threadIdx.x < p.own ? p.mesh.cnt[first + threadIdx.x] : 0u;
        const uint2 base = p.mesh.chunk[first >> 5];
        at = (static_cast<unsigned long long>(base.y + __reduce_add_sync(0xffffffffu, c >> 8)) << 32) |
             (base.x + __reduce_add_sync(0xffffffffu, c & 0xffu));
    }
    if (threadIdx.x == 0)
    {
        *p.mesh.start = at;
        WordTotal{ p.ctr }(at, false);
    }
}

// Slab by slab: the counts, or (emit) the numbering again and the mesh.
template <int DT>
void dense_slabs(const McPlan& p, bool emit, float* verts, int64_t* faces, cudaStream_t s)
{
    TH_CUDA(cudaMemsetAsync(p.mesh.start, 0, sizeof(unsigned long long), s));
    for (int64_t z0 = 0; z0 < p.D; z0 += p.slab)
    {
        McPlan q = dense_slab(p, z0);
        dense_signs<DT>(q, s);
        if (!emit)
            q.nwords = q.own; // the halo is only looked at
        words_count(DenseWords<DT>{ { q } }, emit, s);
        mc_slab_end_kernel<<<1, 32, 0, s>>>(q);
        TH_LAUNCH_CHECK();
        q.nwords = q.own;
        if (emit)
            words_emit(DenseWords<DT>{ { q } }, verts, faces, s);
    }
}

template <int DT>
void sparse_count(const McPlan& p, cudaStream_t s)
{
    const int grid = grid_for(p.nnz, 256);
    if (p.words)
    {
        mc_sparse_words_kernel<DT><<<grid, 256, 0, s>>>(p);
        TH_LAUNCH_CHECK();
        words_count(SparseWords<DT>{ { p } }, true, s);
        return;
    }
    mc_sparse_insert_kernel<<<grid, 256, 0, s>>>(p);
    TH_LAUNCH_CHECK();
    mc_sparse_classify_kernel<DT><<<grid, 256, 0, s>>>(p);
    TH_LAUNCH_CHECK();
    run_scan_reduce(SparseSoupCount{ p.codes }, SoupTotal{ p.ctr }, Count{ nullptr, p.nnz }, p.nnz, p.tiles_soup,
                    &p.ctr->scan_soup, s);
    if (p.unique)
        run_scan(SparseVertCount{ p.used }, SparseVertEmit{ p.vbase }, VertTotal{ p.ctr }, Count{ nullptr, p.nnz },
                 p.nnz, p.tiles_verts, &p.ctr->scan_verts, s);
}

template <int DT>
void sparse_emit(const McPlan& p, float* verts, int64_t* faces, cudaStream_t s)
{
    if (p.words)
    {
        words_emit(SparseWords<DT>{ { p } }, verts, faces, s);
        return;
    }
    if (p.unique)
    {
        mc_sparse_verts_kernel<DT><<<grid_for(p.nnz, 256), 256, 0, s>>>(p, verts);
        TH_LAUNCH_CHECK();
    }
    run_scan_apply(SparseSoupCount{ p.codes }, SparseCellEmit<DT>{ p, verts, faces }, Count{ nullptr, p.nnz }, p.nnz,
                   p.tiles_soup, s);
}

template <class F>
void dispatch_value_dtype(int dt, F&& f)
{
    switch (dt)
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

McPlan dense_slab(const McPlan& p, int64_t z0)
{
    McPlan q = p;
    q.z0 = z0;
    const int64_t planes = p.D - z0 < p.slab ? p.D - z0 : p.slab, size = p.dtype == TH_FLOAT64 ? 8 : (p.dtype == TH_FLOAT32 ? 4 : 2);
    q.volume = static_cast<const unsigned char*>(p.volume) + z0 * p.H * p.W * size;
    q.D = p.D - z0 < planes + 2 ? p.D - z0 : planes + 2;
    q.nwords = q.D * p.H * p.wr;
    q.own = planes * p.H * p.wr;
    return q;
}

void launch_mc_count(const McPlan& p, cudaStream_t s)
{
    TH_CUDA(cudaMemsetAsync(p.ctr, 0, sizeof(McCounters), s));
    if (p.sparse)
    {
        if (p.nnz == 0)
            return;
        if (p.words)
            TH_CUDA(cudaMemsetAsync(p.present, 0, 2 * sizeof(uint32_t) * p.nwords, s)); // and the sign words after them
        else
        {
            TH_CUDA(cudaMemsetAsync(p.keys, 0xff, sizeof(unsigned long long) * (p.hmask + 1), s));
            if (p.unique)
                TH_CUDA(cudaMemsetAsync(p.used, 0, sizeof(uint32_t) * p.nnz, s));
        }
        dispatch_value_dtype(p.dtype, [&]<int DT>() { sparse_count<DT>(p, s); });
        return;
    }
    dispatch_value_dtype(p.dtype, [&]<int DT>() {
        if (p.slab < p.D)
            dense_slabs<DT>(p, false, nullptr, nullptr, s);
        else
            dense_count<DT>(p, s);
    });
}

void launch_mc_emit(const McPlan& p, float* verts, int64_t* faces, cudaStream_t s)
{
    if (p.sparse)
    {
        if (p.nnz == 0)
            return;
        dispatch_value_dtype(p.dtype, [&]<int DT>() { sparse_emit<DT>(p, verts, faces, s); });
        return;
    }
    dispatch_value_dtype(p.dtype, [&]<int DT>() {
        if (p.slab < p.D)
            dense_slabs<DT>(p, true, verts, faces, s);
        else
            words_emit(DenseWords<DT>{ { p } }, verts, faces, s);
    });
}

} // namespace th
