// Marching cubes over bit words: 32 consecutive grid points of a row per
// word, one bit each for "value below the isolevel".
//
// Everything a mesh needs follows from words of neighbouring rows with bit
// operations: the cells the surface passes through, their codes, and the edges
// that hold a vertex (its end points lie on different sides and a complete
// cell holds it).  So the work per grid point is a few instructions per 32
// points, and only the cells on the surface are handled one by one.
//
// 1. words_count: per word the vertex-edge bits along x, y and z, the active
//    cells' bits and the two counts (vertices, triangle corners); tile sums.
// 2. words_base: the counts' prefix sums: per word the index of its first
//    vertex, per 32 words the first vertex and triangle corner.
// 3. words_export: a warp takes 32 words and deals their
//    vertices, or their active cells and the cells' triangle corners, to its
//    lanes: an edge's vertex index is its word's base plus the set bits before it.
//
// Vertices come by the lower end point of their edge (in row order), then by
// axis; triangles by cell, then in table order.  A source (Src) says how words
// are found:
//   int64_t words() const             number of items: words in row order, at least
//                                     those with a present point
//   int64_t counted() const           items whose active cells are counted
//   uint32_t word(uint32_t i) const   the word of an item
//   void tail() const                 more work for the threads of the base pass
//   WordRows rows(uint32_t k) const   the words of the cells that start in word k
//   uint32_t sign(uint32_t k) const   below-isolevel bits of a word
//   bool empty(uint32_t k) const      none of the word's points is present
//   EdgeBits edges(k, rows, s, sh, cells) const   vertex edges and complete cells of a word
//   void vertex(k, bit, axis, out) const          the vertex of an edge
//   void values_at(rows, bit, corner) const       handles of a cell's eight values (soup)
//   void soup_vertex(k, bit, lo, axis, h1, h2, out) const
//
// All three passes are bound by the latency of short dependent load chains on
// words that stay in L2; the volume itself is read once, by the pass that
// makes the sign words.  A 400^3 float32 sphere on GB300: 691 -> 203 us a call
// (447 us of it were one thread per point, exchanging planes through shared
// memory), its band of 1.5 M entries 395 -> 207 us (eight hash lookups per
// entry before, twice).
#pragma once

#include <cstdint>

#include "mc_tables.h"
#include "th_common.cuh"

namespace th
{

constexpr uint32_t kNoWord = 0xffffffffu;
constexpr int kWordTile = 1024; // words per tile of the count and base passes
constexpr int kWordThreads = 256;

struct WordMesh
{
    uint32_t* cnt;   // per item: vertices | triangle corners << 8
    uint32_t* cells; // per item: cells the surface passes through
    uint4* edges;    // per word with vertices: x, y and z edge bits, index of the first vertex
    uint2* chunk;    // per 32 items: first vertex, first triangle corner
    unsigned long long* tiles; // per tile: triangle corners << 32 | vertices, then exclusive offsets
    unsigned long long* start; // triangle corners << 32 | vertices before the first word; nullptr: none
};

// The four rows of cell corners (row q: y + (q & 1), z + (q >> 1)) of the
// cells that start in a word: word indices, kNoWord where a row is absent.
struct WordRows
{
    uint32_t idx[4];
    bool next; // the word has a right neighbour in its row
};

struct EdgeBits
{
    uint32_t x, y, z;
};

struct WordTables
{
    uint8_t count[256];
    uint8_t edges[256][16];
};

namespace words_detail
{
__device__ const uint8_t tri_count[256] = TH_MC_TRI_COUNT_INIT;
__device__ const uint8_t tri_edges[256][15] = TH_MC_TRI_EDGES_INIT;
} // namespace words_detail

// Code of the cell at bit b from its rows' words and those shifted by one point.
__device__ __forceinline__ uint32_t cell_code(const uint32_t s[4], const uint32_t sh[4], int b)
{
    uint32_t code = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        code |= (((s[q] >> b) & 1u) << (2 * q)) | (((sh[q] >> b) & 1u) << (2 * q + 1));
    return code;
}

// The sign words of the four rows and the same shifted by one point.
template <class Src>
__device__ __forceinline__ void sign_rows(const Src& src, const WordRows& r, uint32_t s[4], uint32_t sh[4])
{
    uint32_t nx[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
        s[q] = r.idx[q] != kNoWord ? src.sign(r.idx[q]) : 0u;
        nx[q] = r.next && r.idx[q] != kNoWord ? src.sign(r.idx[q] + 1) : 0u;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
        sh[q] = (s[q] >> 1) | (nx[q] << 31);
}

// Vertex edges and complete cells of a word where not every grid point is
// present: an edge counts when a cell with all its eight corners holds it.
// Such cells are runs of two present points in four neighbouring rows.
// run(dy, dz): for the word in the row (y + dy, z + dz), bits x: the points b
// and b + 1 are present, bit 0 of y: the points -1 and 0 are; zero where there
// is no such row.
template <class Run>
__device__ __forceinline__ EdgeBits masked_edges(Run&& run, const uint32_t s[4], const uint32_t sh[4], uint32_t& cells)
{
    uint2 r[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            r[i][j] = run(i - 1, j - 1);
    // complete cells that start in the rows (y - 1 + i, z - 1 + j), and the points they hold in this word
    uint32_t cell[2][2], held[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
    {
#pragma unroll
        for (int j = 0; j < 2; ++j)
        {
            cell[i][j] = r[i][j].x & r[i + 1][j].x & r[i][j + 1].x & r[i + 1][j + 1].x;
            const uint32_t left = r[i][j].y & r[i + 1][j].y & r[i][j + 1].y & r[i + 1][j + 1].y;
            held[i][j] = cell[i][j] | (cell[i][j] << 1) | left;
        }
    }
    cells = cell[1][1];
    return EdgeBits{ (s[0] ^ sh[0]) & (cell[1][1] | cell[0][1] | cell[1][0] | cell[0][0]),
                     (s[0] ^ s[1]) & (held[1][1] | held[1][0]), (s[0] ^ s[2]) & (held[1][1] | held[0][1]) };
}

// A word's runs (masked_edges) from its bits and its neighbours' in the row.
__device__ __forceinline__ uint2 word_runs(uint32_t prev, uint32_t bits, uint32_t next)
{
    return make_uint2(bits & ((bits >> 1) | (next << 31)), (prev >> 31) & bits & 1u);
}

// Exclusive offsets from tile sums by the block that finishes last, like
// finish_tile_sums, eight sums per thread and round.  A round's triangle
// corners are below 2^32 (2048 tiles of 1024 words, 480 corners a word), and
// every vertex is some triangle's corner, so the packed total wraps exactly
// when there are 2^32 triangle corners or more; epi is told.
template <class EpiF>
__device__ __forceinline__ void finish_word_tiles(int64_t ntiles, unsigned long long* tiles, const unsigned long long* start, ScanState* state, EpiF epi)
{
    __threadfence();
    __shared__ bool is_last;
    if (threadIdx.x == 0)
        is_last = atomicAdd(&state->blocks_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!is_last)
        return;
    __threadfence();
    unsigned long long carry = start ? *start : 0ull;
    bool wrapped = false;
    for (int64_t base = 0; base < ntiles; base += 8 * kWordThreads)
    {
        const int64_t t0 = base + 8 * static_cast<int64_t>(threadIdx.x);
        unsigned long long v[8], s = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            v[i] = t0 + i < ntiles ? __ldcg(tiles + t0 + i) : 0ull;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            s += v[i];
        unsigned long long tot;
        unsigned long long off = carry + block_exclusive_scan(s, &tot);
#pragma unroll
        for (int i = 0; i < 8; ++i)
        {
            if (t0 + i < ntiles)
                tiles[t0 + i] = off;
            off += v[i];
        }
        wrapped |= carry + tot < carry;
        carry += tot;
    }
    if (threadIdx.x == 0)
    {
        state->total = carry;
        state->blocks_done = 0;
        epi(carry, wrapped);
    }
    epi.block();
}

// Pass 1.  A thread per word; most words see one side only and leave after the
// loads.  epi(total, wrapped) gets the triangle corners << 32 | vertices on one
// thread, then epi.block() runs on the same block.
template <class Src, bool UNIQUE, class EpiF>
__global__ void __launch_bounds__(kWordThreads) words_count_kernel(Src src, WordMesh m, ScanState* state, unsigned long long* active, EpiF epi)
{
    __shared__ uint8_t count[256];
    for (int i = threadIdx.x; i < 256; i += kWordThreads)
        count[i] = words_detail::tri_count[i];
    __syncthreads();
    const int64_t n = src.words(), counted = src.counted();
    const int64_t ntiles = (n + kWordTile - 1) / kWordTile;
    unsigned long long nactive = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
    {
        unsigned long long sum = 0;
        for (int t = 0; t < kWordTile / kWordThreads; ++t)
        {
            const int64_t kk = tile * kWordTile + t * kWordThreads + threadIdx.x;
            if (kk >= n)
                break;
            const uint32_t i = static_cast<uint32_t>(kk), k = src.word(i);
            uint32_t s[4], sh[4], some = 0, all = 0;
            WordRows r;
            if (!src.empty(k))
            {
                r = src.rows(k);
                sign_rows(src, r, s, sh);
                some = s[0] | s[1] | s[2] | s[3] | sh[0] | sh[1] | sh[2] | sh[3];
                all = s[0] & s[1] & s[2] & s[3] & sh[0] & sh[1] & sh[2] & sh[3];
            }
            if ((some & ~all) == 0)
            {
                m.cnt[i] = 0; // all points around the word lie on one side
                continue;
            }
            uint32_t cells = 0;
            const EdgeBits e = src.edges(k, r, s, sh, cells);
            cells &= some & ~all;
            uint32_t soup = 0;
            for (uint32_t left = cells; left; left &= left - 1)
                soup += count[cell_code(s, sh, __ffs(left) - 1)];
            uint32_t verts = 0;
            if (UNIQUE)
            {
                verts = __popc(e.x) + __popc(e.y) + __popc(e.z);
                if (verts)
                    m.edges[k] = make_uint4(e.x, e.y, e.z, 0u);
            }
            m.cnt[i] = verts | (soup << 8);
            if (cells)
                m.cells[i] = cells;
            sum += (static_cast<unsigned long long>(soup) << 32) | verts;
            nactive += kk < counted ? __popc(cells) : 0;
        }
        unsigned long long tot;
        block_exclusive_scan(sum, &tot);
        if (threadIdx.x == 0)
            m.tiles[tile] = tot;
    }
    if (active)
    {
        unsigned long long tot;
        block_exclusive_scan(nactive, &tot);
        if (threadIdx.x == 0 && tot)
            atomicAdd(active, tot);
    }
    finish_word_tiles(ntiles, m.tiles, m.start, state, epi);
}

// Pass 2: a warp numbers 4 chunks of 32 consecutive words of a tile.
template <class Src>
__global__ void __launch_bounds__(kWordThreads) words_base_kernel(Src src, WordMesh m)
{
    constexpr int kChunks = kWordTile / kWordThreads;
    __shared__ unsigned long long warp_tot[kWordThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t n = src.words();
    const int64_t ntiles = (n + kWordTile - 1) / kWordTile;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
    {
        const int64_t first = tile * kWordTile + w * (32 * kChunks);
        uint32_t c[kChunks];
        unsigned long long s = 0;
#pragma unroll
        for (int i = 0; i < kChunks; ++i)
        {
            const int64_t k = first + i * 32 + lane;
            c[i] = k < n ? m.cnt[k] : 0u;
            s += (static_cast<unsigned long long>(c[i] >> 8) << 32) | (c[i] & 0xffu);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
            s += __shfl_xor_sync(0xffffffffu, s, d);
        if (lane == 0)
            warp_tot[w] = s;
        __syncthreads();
        unsigned long long off = m.tiles[tile];
        for (int v = 0; v < w; ++v)
            off += warp_tot[v];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kChunks; ++i)
        {
            const int64_t k = first + i * 32 + lane;
            if (k - lane >= n)
                break;
            // a chunk's sums fit 16 bits each: 32 * 480 corners, 32 * 96 vertices
            const uint32_t mine = ((c[i] >> 8) << 16) | (c[i] & 0xffu);
            const uint32_t incl = warp_inclusive_scan(mine);
            if (lane == 0)
                m.chunk[k >> 5] = make_uint2(static_cast<uint32_t>(off), static_cast<uint32_t>(off >> 32));
            if (c[i] & 0xffu)
                m.edges[src.word(static_cast<uint32_t>(k))].w = static_cast<uint32_t>(off) + ((incl - mine) & 0xffffu);
            const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
            off += (static_cast<unsigned long long>(tot >> 16) << 32) | (tot & 0xffffu);
        }
    }
    src.tail();
}

// Index of the first vertex of the point at bit b of a word, and the point's
// three edge bits below it: id << 3 | bits.
__device__ __forceinline__ unsigned long long point_vertices(const uint4& g, int b)
{
    const uint32_t lt = (1u << b) - 1u;
    const uint32_t id = g.w + __popc(g.x & lt) + __popc(g.y & lt) + __popc(g.z & lt);
    const uint32_t bits = ((g.x >> b) & 1u) | (((g.y >> b) & 1u) << 1) | (((g.z >> b) & 1u) << 2);
    return (static_cast<unsigned long long>(id) << 3) | bits;
}

constexpr int kWordExportWarps = 8;

// The export passes take a chunk of 32 words per warp; a warp's chunks lie far
// apart, which spreads the surface over the warps (eight neighbouring chunks
// per warp took 46 + 80 us for the vertices and faces of a 400^3 sphere,
// against 26 + 50).  All that says what a chunk holds is loaded at
// once, whether or not it holds anything.

// Pass 3, the vertices, by block `block` of `blocks`.
template <class Src>
__device__ __forceinline__ void export_verts(const Src& src, const WordMesh& m, float* __restrict__ verts, uint32_t block, uint32_t blocks)
{
    const int lane = threadIdx.x & 31;
    const int64_t n = src.words(), nchunks = (n + 31) / 32;
    const int64_t nwarps = static_cast<int64_t>(blocks) * kWordExportWarps;
    for (int64_t c = static_cast<int64_t>(block) * kWordExportWarps + (threadIdx.x >> 5); c < nchunks; c += nwarps)
    {
        const uint32_t item = static_cast<uint32_t>(c * 32) + lane;
        const bool in = c * 32 + lane < n;
        const uint32_t base = __ldg(&m.chunk[c].x);
        const uint32_t vc = in ? __ldg(m.cnt + item) & 0xffu : 0u;
        const uint32_t k = in ? src.word(item) : 0u;
        if (!__any_sync(0xffffffffu, vc != 0))
            continue;
        const uint4 g = vc ? __ldg(m.edges + k) : make_uint4(0u, 0u, 0u, 0u);
        const int incl = warp_inclusive_scan(static_cast<int>(vc));
        const int excl = incl - static_cast<int>(vc);
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        for (int i0 = 0; i0 < total; i0 += 32)
        {
            const int i = i0 + lane;
            const int s = item_slot(excl, i);
            int j = i - __shfl_sync(0xffffffffu, excl, s);
            uint32_t ex = __shfl_sync(0xffffffffu, g.x, s), ey = __shfl_sync(0xffffffffu, g.y, s),
                     ez = __shfl_sync(0xffffffffu, g.z, s);
            const uint32_t ks = __shfl_sync(0xffffffffu, k, s);
            if (i < total)
            {
                // the point with j vertices before it in the word, then the axis
                int b = 0;
#pragma unroll
                for (int w = 16; w > 0; w >>= 1)
                {
                    const uint32_t low = (1u << w) - 1u;
                    const int before = __popc(ex & low) + __popc(ey & low) + __popc(ez & low);
                    if (j >= before)
                    {
                        j -= before;
                        b += w;
                        ex >>= w;
                        ey >>= w;
                        ez >>= w;
                    }
                }
                const uint32_t here = (ex & 1u) | ((ey & 1u) << 1) | ((ez & 1u) << 2);
                const int axis = j == 0 ? __ffs(here) - 1 : (j == 2 || here != 7u ? 31 - __clz(here) : 1);
                float v[3];
                src.vertex(ks, b, axis, v);
                float* out = verts + 3 * (static_cast<int64_t>(base) + i);
                out[0] = v[0];
                out[1] = v[1];
                out[2] = v[2];
            }
        }
    }
}

// Pass 3.  UNIQUE: the even blocks write vertices, the odd ones triangles (one
// launch, so that a small mesh does not wait for two).  FLIP: the second and
// third corner of every triangle change places.  Without UNIQUE every triangle
// corner is a vertex of its own, written with the triangles.
template <class Src, bool UNIQUE, bool FLIP>
__global__ void __launch_bounds__(32 * kWordExportWarps) words_export_kernel(Src src, WordMesh m, float* __restrict__ verts, int64_t* __restrict__ faces)
{
    if (UNIQUE && blockIdx.x % 2 == 0)
    {
        export_verts(src, m, verts, blockIdx.x / 2, gridDim.x / 2);
        return;
    }
    const uint32_t block = UNIQUE ? blockIdx.x / 2 : blockIdx.x, blocks = UNIQUE ? gridDim.x / 2 : gridDim.x;
    __shared__ WordTables tab;
    // per warp and cell of a round: its corners' vertices (point_vertices), or
    // where their values are (Src::values_at)
    __shared__ unsigned long long corner_all[kWordExportWarps][32][9];
    __shared__ uint32_t stage_all[kWordExportWarps][UNIQUE ? 32 * 15 : 1];
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
    {
        tab.count[i] = words_detail::tri_count[i];
#pragma unroll
        for (int j = 0; j < 15; ++j)
            tab.edges[i][j] = words_detail::tri_edges[i][j];
    }
    __syncthreads();
    unsigned long long(*corner)[9] = corner_all[threadIdx.x >> 5];
    uint32_t* stage = stage_all[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int64_t n = src.words(), nchunks = (n + 31) / 32;
    const int64_t nwarps = static_cast<int64_t>(blocks) * kWordExportWarps;
    for (int64_t c = static_cast<int64_t>(block) * kWordExportWarps + (threadIdx.x >> 5); c < nchunks; c += nwarps)
    {
        const uint32_t item = static_cast<uint32_t>(c * 32) + lane;
        const bool in = c * 32 + lane < n;
        const uint32_t base = __ldg(&m.chunk[c].y);
        const uint32_t cn = in ? __ldg(m.cnt + item) : 0u, cl = in ? __ldg(m.cells + item) : 0u;
        const uint32_t k = in ? src.word(item) : 0u;
        const uint32_t cells = (cn >> 8) ? cl : 0u;
        if (!__any_sync(0xffffffffu, cells != 0))
            continue;
        const int cc = __popc(cells);
        const int cincl = warp_inclusive_scan(cc);
        const int cexcl = cincl - cc;
        const int ctotal = __shfl_sync(0xffffffffu, cincl, 31);
        int64_t at = base;
        for (int i0 = 0; i0 < ctotal; i0 += 32)
        {
            const int i = i0 + lane;
            const int s = item_slot(cexcl, i);
            const int j = i - __shfl_sync(0xffffffffu, cexcl, s);
            const uint32_t cs = __shfl_sync(0xffffffffu, cells, s);
            const uint32_t ks = __shfl_sync(0xffffffffu, k, s);
            uint32_t code = 0;
            int b = 0;
            if (i < ctotal)
            {
                b = nth_set_bit(cs, j);
                const WordRows r = src.rows(ks);
                uint32_t sg[4], sh[4];
                uint4 g[4];
                sign_rows(src, r, sg, sh);
                if constexpr (UNIQUE)
                {
                    // a word without vertices holds no edge of this cell: its entry is not read below
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        g[q] = __ldg(m.edges + r.idx[q]);
                }
                code = cell_code(sg, sh, b);
                if constexpr (UNIQUE)
                {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                    {
                        corner[lane][2 * q] = point_vertices(g[q], b);
                        corner[lane][2 * q + 1] =
                                b < 31 ? point_vertices(g[q], b + 1) : point_vertices(__ldg(m.edges + r.idx[q] + 1), 0);
                    }
                }
                else
                    src.values_at(r, b, corner[lane]);
            }
            const int cnt = tab.count[code];
            const int incl = warp_inclusive_scan(cnt);
            const int excl = incl - cnt;
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            __syncwarp();
            if constexpr (UNIQUE)
            {
                // a lane per cell parks its triangles' vertices, then all lanes write them
                for (int j = 0; j < cnt; j += 3)
                {
#pragma unroll
                    for (int t = 0; t < 3; ++t)
                    {
                        const uint32_t ed = tab.edges[code][j + t];
                        const unsigned long long p = corner[lane][ed & 7u];
                        // FLIP: the triangle's second and third corner change places
                        stage[excl + j + (FLIP && t > 0 ? 3 - t : t)] =
                                static_cast<uint32_t>(p >> 3) + __popc(static_cast<uint32_t>(p) & ((1u << (ed >> 3)) - 1u));
                    }
                }
                __syncwarp();
                for (int e = lane; e < total; e += 32)
                    faces[at + e] = static_cast<int64_t>(stage[e]);
            }
            else
            {
                for (int e0 = 0; e0 < total; e0 += 32)
                {
                    const int e = e0 + lane;
                    const int es = item_slot(excl, e);
                    const int ej = e - __shfl_sync(0xffffffffu, excl, es);
                    const uint32_t ecode = __shfl_sync(0xffffffffu, code, es);
                    const uint32_t ek = __shfl_sync(0xffffffffu, ks, es);
                    const int eb = __shfl_sync(0xffffffffu, b, es);
                    if (e < total)
                    {
                        const uint32_t ed = tab.edges[ecode][ej];
                        const int lo = static_cast<int>(ed & 7u), axis = static_cast<int>(ed >> 3);
                        const int slot = e % 3;
                        float v[3];
                        src.soup_vertex(ek, eb, lo, axis, corner[es][lo], corner[es][lo | (1 << axis)], v);
                        float* out = verts + 3 * (at + e);
                        out[0] = v[0];
                        out[1] = v[1];
                        out[2] = v[2];
                        faces[at + e + (FLIP ? (slot == 0 ? 0 : 3 - 2 * slot) : 0)] = at + e;
                    }
                }
            }
            at += total;
            __syncwarp();
        }
    }
}

inline int64_t word_tiles(int64_t words)
{
    return (words + kWordTile - 1) / kWordTile;
}

// Grid of the vertex and face passes (words: an upper bound).
inline int words_export_grid(int64_t words)
{
    const int64_t blocks = (words + 32 * kWordExportWarps - 1) / (32 * kWordExportWarps), cap = 8LL * sm_count();
    return static_cast<int>(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

// Pass 3 on stream s; grid: words_export_grid.
template <class Src, bool FLIP>
inline void launch_words_export(const Src& src, const WordMesh& m, bool unique, int grid, float* verts, int64_t* faces, cudaStream_t s)
{
    if (unique)
        words_export_kernel<Src, true, FLIP><<<2 * grid, 32 * kWordExportWarps, 0, s>>>(src, m, verts, faces);
    else
        words_export_kernel<Src, false, FLIP><<<grid, 32 * kWordExportWarps, 0, s>>>(src, m, verts, faces);
    check_launch("mesh export");
    note_launches(1);
}

// Grid of the count and base passes (words: an upper bound).
inline int words_grid(int64_t words)
{
    const int64_t tiles = word_tiles(words), cap = 8LL * sm_count();
    return static_cast<int>(tiles < 1 ? 1 : (tiles < cap ? tiles : cap));
}

} // namespace th
