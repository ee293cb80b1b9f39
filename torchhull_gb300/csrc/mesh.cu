// Leaf corners, hull field and sparse marching cubes.
//
// Corner set.  The reference turns the leaf cells into 8 corner ids each, then
// radix-sorts and uniques them (visual_hull_cuda.cu:770-825).  Here each leaf
// sets its corners in a bitmap over the (2^L+1)^3 grid, laid out row by row
// (x fastest, one row = WR 64-bit words) so that the set bits in memory order
// are the ids already ascending and unique.  A second bitmap flags the rows
// that hold any bit.  rows_kernel lists those rows and counts their corners,
// corners_kernel copies their words into a compact array (32 points a word),
// with the rank of each word's first corner, and writes the sorted list; it
// clears the bitmaps behind it.  "Index of corner v in the sorted list" is one
// word load, one rank load and a popcount: this replaces the hash map the
// reference builds for its marching cubes (marching_cubes_cuda.cu:66-70,
// :133-144).
//
// Hull field.  A corner's value is the product of the bilinear mask samples of
// all views in ascending view order, the order in which the reference's
// per-view launches (visual_hull_cuda.cu:827-888) multiply them.  The field
// also sets the corner's bit in the sign words when its value is below 0.5.
//
// Marching cubes.  A corner g is a cell when all 8 cube corners are present
// (marching_cubes_cuda.cu:180-223).  Cells, codes and vertex edges come from
// the presence and sign words by bit operations (th_words.cuh); the vertices
// are numbered in (corner, axis) order, which is exactly the reference's
// vertex order after torch::unique_dim over the edge ids (ravel(p1) << 3 |
// 1 << axis), (:99-112, :674-693), without a sort.  Faces are emitted per cell
// in ascending corner order and table order, as the reference's soup is.

#include <algorithm>

#include "th_hull.cuh"
#include "th_internal.h"

namespace th
{

namespace
{

// Level 0: the root is the only leaf (deeper leaves are marked by the carve).
__global__ void mark_root_kernel(HullPlan p)
{
    if (threadIdx.x == 0)
        mark_cell_corners(p.bitmap, p.rowbits, p.R, p.WR, 0, 0, 0);
}

// The corners of the leaves, the refined children of the level L-1 cells, from
// their child masks (HullPlan::mark_apart).  256 consecutive cells are close
// together and share most of their corners' words, so a block collects the
// words' bits in a table in shared memory and writes each word once: atomics
// of neighbouring cells on one word of the bitmap queued behind each other
// (headline scene: 147 to 171 us, this 103).
__global__ void __launch_bounds__(256) mark_corners_kernel(HullPlan p)
{
    __shared__ MarkTable table;
    const int tid = threadIdx.x, li = p.level - 1;
    const int64_t n = p.ctr->level_count[li];
    const int64_t* parents = p.nodes + p.ctr->level_off[li];
    const uint32_t R = static_cast<uint32_t>(p.R), wr = p.wr, low = (1u << li) - 1u;
    uint32_t* bitmap = reinterpret_cast<uint32_t*>(p.bitmap);
    for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * 256; t0 < n; t0 += static_cast<int64_t>(gridDim.x) * 256)
    {
        const int64_t t = t0 + tid;
        const uint32_t m = t < n ? p.child_masks[t] : 0u;
        const int64_t idx = t < n ? parents[t] : 0;
        for (int i = tid; i < kMarkSlots; i += 256)
        {
            table.key[i] = kNoWord;
            table.bits[i] = 0;
        }
        __syncthreads();
        if (m)
        {
            const uint32_t x = 2 * (static_cast<uint32_t>(idx) & low), y = 2 * (static_cast<uint32_t>(idx >> li) & low),
                           z = 2 * static_cast<uint32_t>(idx >> (2 * li));
            const uint32_t first = (y + z * R) * wr + (x >> 5);
            const int b = static_cast<int>(x & 31); // even: bit 30 is the last, one bit into the next word
#pragma unroll
            for (int q = 0; q < 9; ++q)
            {
                uint32_t xb = 0; // lattice x bits 0..2 of the row (y + q % 3, z + q / 3)
#pragma unroll
                for (int c = 0; c < 8; ++c)
                {
                    const int cx = c & 1, cy = (c >> 1) & 1, cz = c >> 2, dy = q % 3, dz = q / 3;
                    if ((dy == cy || dy == cy + 1) && (dz == cz || dz == cz + 1) && ((m >> c) & 1u))
                        xb |= 3u << cx;
                }
                if (!xb)
                    continue;
                const uint32_t w = first + (q % 3 + q / 3 * R) * wr;
                const uint32_t lo = xb << b, hi = b > 29 ? xb >> (32 - b) : 0u;
                if (lo && !mark_word(table, w, lo))
                {
                    atomicOr(bitmap + w, lo);
                    const uint32_t row = w / wr;
                    atomicOr(p.rowbits + (row >> 5), 1u << (row & 31));
                }
                if (hi && !mark_word(table, w + 1, hi))
                {
                    atomicOr(bitmap + w + 1, hi);
                    const uint32_t row = w / wr;
                    atomicOr(p.rowbits + (row >> 5), 1u << (row & 31));
                }
            }
        }
        __syncthreads();
        for (int i = tid; i < kMarkSlots; i += 256)
        {
            const uint32_t w = table.key[i];
            if (w == kNoWord)
                continue;
            atomicOr(bitmap + w, table.bits[i]);
            const uint32_t row = fast_div(p.div_wr, w), rb = 1u << (row & 31);
            if (!(__ldcg(p.rowbits + (row >> 5)) & rb))
                atomicOr(p.rowbits + (row >> 5), rb);
        }
        __syncthreads();
    }
}

// Sum of v over the block, to every thread.
__device__ __forceinline__ unsigned long long block_sum(unsigned long long v)
{
    unsigned long long total;
    block_exclusive_scan(v, &total);
    return total;
}

// Touched rows, their slots and their corner counts.  A block owns
// kRowBlock words of row flags; the rows before it are counted from the flags
// themselves (a few thousand words at the usual levels, read 16 bytes at a
// time), so no pass or wait comes in between.  Headline scene (32 x 1024^2,
// level 9, 13 M corners) on GB300: 10 us, where two scan passes over the flags
// took 40 and a pass for the corner counts 14.  The flags read so grow 16-fold
// per level, so from kCountRowBlocks blocks on (levels 11 and 12)
// row_counts_kernel counts the blocks' flags first (HullPlan::block_rows).  All
// passes over the corners of a thin rod: level 11 102 -> 55 us, level 12 936 ->
// 99; level 10, with 1027 blocks, takes 39 us either way.
__global__ void __launch_bounds__(256) row_counts_kernel(HullPlan p)
{
    const int64_t nwords = (p.R * p.R + 31) / 32;
    const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; // a warp per block of rows_kernel
    const uint32_t n = __reduce_add_sync(0xffffffffu, i < nwords ? __popc(p.rowbits[i]) : 0u);
    if ((threadIdx.x & 31) == 0 && i < nwords)
        p.block_rows[i / kRowBlock] = n;
}

__global__ void __launch_bounds__(256) rows_kernel(HullPlan p)
{
    __shared__ uint32_t base[kRowBlock];
    __shared__ unsigned long long s_before, s_corners;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t nwords = (p.R * p.R + 31) / 32;
    const int64_t first = static_cast<int64_t>(blockIdx.x) * kRowBlock;
    unsigned long long before = 0;
    if (p.block_rows)
    {
        for (uint32_t i = tid; i < blockIdx.x; i += 256)
            before += p.block_rows[i];
    }
    else
    {
        // first is a multiple of 4 and the buffer is 256-byte aligned
        for (int64_t i = tid; i < first / 4; i += 256)
        {
            const uint4 w = reinterpret_cast<const uint4*>(p.rowbits)[i];
            before += __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
        }
    }
    before = block_sum(before);
    if (warp == 0)
    {
        const uint32_t w = first + lane < nwords ? p.rowbits[first + lane] : 0u;
        const uint32_t incl = warp_inclusive_scan(static_cast<uint32_t>(__popc(w)));
        base[lane] = incl - __popc(w);
        if (lane == 31)
        {
            s_before = before + incl;
            s_corners = 0;
        }
    }
    __syncthreads();
    if (tid == 0 && first + kRowBlock >= nwords)
    {
        DevCounters* c = p.ctr;
        const int64_t rows = static_cast<int64_t>(s_before);
        c->rows = rows;
        if (rows * p.wr > p.word_cap)
            c->overflow |= kOverflowWords;
        const int L = p.level;
        if (L > 0)
        {
            // the last level's count, with the checks of the levels before it
            const int64_t start = c->level_off[L];
            int64_t n = static_cast<int64_t>(c->leaves);
            if (c->level_count[L - 1] > p.parent_cap)
                c->overflow |= kOverflowParents;
            if (start + n > p.node_cap)
            {
                c->overflow |= kOverflowNodes;
                n = 0;
            }
            c->level_count[L] = n;
            c->level_off[L + 1] = start + n;
        }
    }
    unsigned long long corners = 0; // lane 0's: of the warp
    for (int i = warp; i < kRowBlock; i += 8)
    {
        const uint32_t w = first + i < nwords ? p.rowbits[first + i] : 0u;
        if (w == 0)
            continue;
        const bool on = (w >> lane) & 1u;
        const uint32_t slot = static_cast<uint32_t>(before) + base[i] + __popc(w & ((1u << lane) - 1u));
        uint32_t cnt = 0, used = 0;
        if (on)
        {
            const int64_t row = (first + i) * 32 + lane;
            const uint2* bits = reinterpret_cast<const uint2*>(p.bitmap + row * p.WR);
#pragma unroll 4
            for (int64_t j = 0; j < p.WR; ++j)
            {
                const uint2 b = bits[j];
                cnt += __popc(b.x) + __popc(b.y);
                used += (b.x != 0 ? 1u : 0u) + (b.y != 0 ? 1u : 0u);
            }
            p.rows[slot] = static_cast<uint32_t>(row);
            p.row_slot[row] = slot;
            p.row_cnt[slot] = make_uint2(cnt, used);
        }
        // the slots of a word lie in at most two groups of 256
        const uint32_t g0 = __shfl_sync(0xffffffffu, slot, __ffs(w) - 1) >> 8;
        const bool second = (slot >> 8) != g0;
        const uint32_t c0 = __reduce_add_sync(0xffffffffu, second ? 0u : cnt), c1 = __reduce_add_sync(0xffffffffu, second ? cnt : 0u);
        const uint32_t u0 = __reduce_add_sync(0xffffffffu, second ? 0u : used), u1 = __reduce_add_sync(0xffffffffu, second ? used : 0u);
        if (lane == 0)
        {
            atomicAdd(&p.coarse[g0].x, c0);
            atomicAdd(&p.coarse[g0].y, u0);
            if (c1)
            {
                atomicAdd(&p.coarse[g0 + 1].x, c1);
                atomicAdd(&p.coarse[g0 + 1].y, u1);
            }
            corners += c0 + c1;
        }
    }
    if (corners)
        atomicAdd(&s_corners, corners);
    __syncthreads();
    if (tid == 0 && s_corners)
        atomicAdd(&p.ctr->row_corners, s_corners);
}

// The sorted corner list and the rows' words.  A block takes a contiguous
// range of slots, so what comes before it is summed once, 256 rows at a time; a
// warp takes as many rows as its lanes have 64-bit words for (three at level
// 9): presence, runs and ranks, the list of words with corners, then per word
// a lane per point.  The words of the bitmap and the row flags are cleared
// behind it.  Issue-bound: headline scene 151 -> 97 us (a warp searched the
// word of every corner before, and the bitmap was cleared by another pass).
constexpr int kRowGroup = 256; // rows whose places a block works out together

__global__ void __launch_bounds__(256) corners_kernel(HullPlan p)
{
    __shared__ uint2 before[kRowGroup]; // corners and words before each of the group's rows
    __shared__ uint32_t row_s[kRowGroup], yz_s[kRowGroup];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t rows = p.ctr->rows;
    const uint32_t wr = p.wr, R = static_cast<uint32_t>(p.R);
    const int WR = static_cast<int>(p.WR);
    const int64_t nflags = (p.R * p.R + 31) / 32;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + tid; i < nflags; i += static_cast<int64_t>(gridDim.x) * 256)
        p.rowbits[i] = 0;
    const int64_t groups = (rows + 31) / 32;
    const int64_t per = (groups + gridDim.x - 1) / gridDim.x;
    const int64_t s0 = per * blockIdx.x * 32;
    const int64_t s1 = s0 + per * 32 < rows ? s0 + per * 32 : rows;
    if (s0 >= rows)
        return;
    if (p.ctr->row_corners >> 32)
    {
        if (s0 == 0 && tid == 0)
            p.ctr->overflow |= kOverflowIndices; // corners and words stay 0: nothing after this has any to look at
        return;
    }
    // corners and words below 2^32: summed packed
    unsigned long long sum = 0;
    auto add = [&](uint2 c) { sum += (static_cast<unsigned long long>(c.y) << 32) | c.x; };
    for (int64_t i = tid; i < s0 / 256; i += 256)
        add(p.coarse[i]);
    for (int64_t i = (s0 & ~int64_t{ 255 }) + tid; i < s0; i += 256)
        add(p.row_cnt[i]);
    sum = block_sum(sum);
    uint32_t corners = static_cast<uint32_t>(sum), words = static_cast<uint32_t>(sum >> 32);
    // rows per warp and step
    const int G = WR <= 32 ? 32 / WR : 1;
    const int sub = WR <= 32 ? lane / WR : 0, first = WR <= 32 ? sub * WR : 0;
    for (int64_t g = s0; g < s1; g += kRowGroup)
    {
        const int nrows = static_cast<int>(s1 - g < kRowGroup ? s1 - g : kRowGroup);
        __syncthreads();
        unsigned long long mine_sum = 0, group_sum;
        if (tid < nrows)
        {
            const uint2 c = p.row_cnt[g + tid];
            mine_sum = (static_cast<unsigned long long>(c.y) << 32) | c.x;
        }
        const unsigned long long ahead = block_exclusive_scan(mine_sum, &group_sum);
        before[tid] = make_uint2(static_cast<uint32_t>(ahead), static_cast<uint32_t>(ahead >> 32));
        // the rows around each row: 3 * (dy + 1) + dz + 1
        for (int i = tid; i < nrows * 9; i += 256)
        {
            const int r = i / 9, q = i - 9 * r, dy = q / 3 - 1, dz = q - 3 * (q / 3) - 1;
            const uint32_t row = p.rows[g + r];
            const uint32_t z = fast_div(p.div_r, row), y = row - z * R;
            uint32_t near = kNoWord;
            if (q == 4)
            {
                near = y | (z << 16);
                row_s[r] = row;
                yz_s[r] = near;
            }
            else if ((dy >= 0 || y > 0) && (dy <= 0 || y + 1 < R) && (dz >= 0 || z > 0) && (dz <= 0 || z + 1 < R))
            {
                // the slot of a row that is not touched is stale: out of range, or another row's
                const uint32_t other = row + dy + dz * R, os = p.row_slot[other];
                if (os < static_cast<uint32_t>(rows) && p.rows[os] == other)
                    near = os;
            }
            p.row_place[g + r].near[q] = near;
        }
        __syncthreads();
        for (int i0 = warp * G; i0 < nrows; i0 += 8 * G)
        {
            const int i = i0 + sub;
            const bool mine = sub < G && i < nrows;
            const uint32_t row = mine ? row_s[i] : 0u, yz = mine ? yz_s[i] : 0u;
            uint32_t at = mine ? corners + before[i].x : 0u, wat = mine ? words + before[i].y : 0u;
            uint32_t last = 0; // the last 32 points of the words before (WR > 32)
            for (int w0 = 0; w0 < WR; w0 += 32)
            {
                const int w = w0 + lane - first;
                const bool on = mine && w < WR;
                uint2* src = reinterpret_cast<uint2*>(p.bitmap + static_cast<int64_t>(row) * WR + w);
                const uint2 b = on ? *src : make_uint2(0u, 0u);
                uint32_t after = on && lane == 31 && w + 1 < WR ? src[1].x : 0u;
                uint32_t prev = __shfl_up_sync(0xffffffffu, b.y, 1);
                const uint32_t down = __shfl_down_sync(0xffffffffu, b.x, 1);
                if (w == w0)
                    prev = last;
                const uint32_t next = lane == 31 ? after : (w + 1 < WR ? down : 0u);
                last = __shfl_sync(0xffffffffu, b.y, 31);
                if (b.x | b.y)
                    *src = make_uint2(0u, 0u);
                // ranks inside the row: inclusive scans over the warp less what lies before the row's first lane
                const uint32_t cnt = __popc(b.x) + __popc(b.y), used = (b.x != 0 ? 1u : 0u) + (b.y != 0 ? 1u : 0u);
                const uint32_t incl = warp_inclusive_scan((used << 16) | cnt); // 64 * 32 corners at most
                const uint32_t excl = incl - ((used << 16) | cnt);
                const uint32_t start = __shfl_sync(0xffffffffu, excl, first & 31);
                const uint32_t rank = at + ((excl - start) & 0xffffu), wrank = wat + ((excl - start) >> 16);
                const int64_t k = (g + i) * wr + 2 * w;
                if (on && k + 1 < p.word_cap)
                {
                    *reinterpret_cast<uint2*>(p.present + k) = b;
                    *reinterpret_cast<uint2*>(p.rank + k) = make_uint2(rank, rank + __popc(b.x));
                    *reinterpret_cast<uint2*>(p.sign + k) = make_uint2(0u, 0u);
                    const uint2 lo = word_runs(prev, b.x, b.y), hi = word_runs(b.x, b.y, next);
                    *reinterpret_cast<uint4*>(p.runs + k) = make_uint4(lo.x, lo.y, hi.x, hi.y);
                    if (b.x)
                        p.word_list[wrank] = static_cast<uint32_t>(k);
                    if (b.y)
                        p.word_list[wrank + (b.x != 0 ? 1u : 0u)] = static_cast<uint32_t>(k) + 1;
                }
                for (uint32_t todo = __ballot_sync(0xffffffffu, cnt != 0); todo; todo &= todo - 1)
                {
                    const int j = __ffs(todo) - 1;
                    const uint32_t bx = __shfl_sync(0xffffffffu, b.x, j), by = __shfl_sync(0xffffffffu, b.y, j);
                    const uint32_t r = __shfl_sync(0xffffffffu, rank, j), ryz = __shfl_sync(0xffffffffu, yz, j);
                    const int x = __shfl_sync(0xffffffffu, w, j) * 64 + lane;
                    const int64_t id = pack_corner(x, ryz & 0xffffu, ryz >> 16);
                    const uint32_t lt = (1u << lane) - 1u;
                    const uint32_t o0 = r + __popc(bx & lt), o1 = r + __popc(bx) + __popc(by & lt);
                    if (((bx >> lane) & 1u) && o0 < p.corner_cap)
                        p.corners[o0] = id;
                    if (((by >> lane) & 1u) && o1 < p.corner_cap)
                        p.corners[o1] = id + 32;
                }
                if (WR > 32)
                {
                    const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
                    at += all & 0xffffu;
                    wat += all >> 16;
                }
            }
        }
        corners += static_cast<uint32_t>(group_sum);
        words += static_cast<uint32_t>(group_sum >> 32);
    }
    if (s1 == rows && tid == 0)
    {
        const bool over = static_cast<int64_t>(corners) > p.corner_cap;
        if (over)
            p.ctr->overflow |= kOverflowCorners;
        // an overflowing request is run again: nothing after this looks at its corners
        const bool none = over || (p.ctr->overflow & kOverflowWords);
        p.ctr->corners = none ? 0 : corners;
        p.ctr->words = none ? 0 : words;
    }
}

template <int DT>
__device__ __forceinline__ float mask_sample(const HullPlan& p, const void* masks, int64_t b, int64_t y, int64_t x, float pad)
{
    // 0 <= y < H and 0 <= x < W, as unsigned compares
    return (static_cast<uint64_t>(y) < static_cast<uint64_t>(p.H) && static_cast<uint64_t>(x) < static_cast<uint64_t>(p.W))
                   ? load_f32<DT>(masks, (b * p.H + y) * p.W + x)
                   : pad;
}

// Factor of view b for the corner at world point (wx, wy, wz): the bilinear
// mask sample (image_utils.h:162-214), or exactly 1 when partial mode skips
// the view (x * 1 == x, so multiplying by it equals skipping it).
//
// The reference converts the rounded pixel to int64.  Near the image the
// rounding and the conversion are done exactly with float adds (the
// conversion instructions run on narrow pipes, the 64-bit ones on GB300's
// FP64 pipe); far from it (|coordinate| >= 2^22, or NaN) the saturating int32
// conversion stands in: the in-image tests decide identically, and where its
// value differs from the int64 one (|coordinate| >= 2^31) all four samples
// are padding, for which the interpolation gives the same result (0, 1 or
// NaN) for either weight.
template <int DT, bool PARTIAL>
__device__ __forceinline__ float view_factor(const HullPlan& p, const void* masks, int64_t b, const float4 (&rows)[3], float wx, float wy, float wz, float Hf, float Wf)
{
    float px, py;
    to_pixel_rows(rows[0], rows[1], rows[2], wx, wy, wz, p.opengl, Hf, Wf, px, py);
    const float pad = PARTIAL ? 1.f : 0.f;
    if constexpr (PARTIAL)
    {
        // 1 <= round(q) < size - 1 (half away from zero) exactly when 0.5 <= q < size - 1.5
        if (!(px >= 0.5f && px < __fsub_rn(Wf, 1.5f) && py >= 0.5f && py < __fsub_rn(Hf, 1.5f)))
            return 1.f;
        // In frame q - 0.5 is exact and >= 0, so round(q - 0.5) = floor(q), in
        // [0, size - 2]; q + 2^23 rounded down is 2^23 + floor(q) (the floats
        // in [2^23, 2^24) are the integers).
        const float sy = __fadd_rd(py, kTwo23), sx = __fadd_rd(px, kTwo23);
        const int64_t y0 = __float_as_int(sy) - kTwo23Bits, x0 = __float_as_int(sx) - kTwo23Bits;
        // all-ones footprint: exactly 1 (the weights below are in [0, 1])
        if (p.field_ones)
        {
            const uint32_t word = __ldg(p.ones + (b * p.H + y0) * p.WW + (x0 >> 5));
            if ((word >> (x0 & 31)) & 1u)
                return 1.f;
        }
        const int64_t i = (b * p.H + y0) * p.W + x0;
        const float v00 = load_f32<DT>(masks, i);
        const float v01 = load_f32<DT>(masks, i + 1);
        const float v10 = load_f32<DT>(masks, i + p.W);
        const float v11 = load_f32<DT>(masks, i + p.W + 1);
        return bilerp(v00, v10, v01, v11, __fsub_rn(py, __fsub_rn(sy, kTwo23)), __fsub_rn(px, __fsub_rn(sx, kTwo23)));
    }
    Snapped ry, rx;
    if (!round_small(__fadd_rn(py, -0.5f), ry))
    {
        ry.i = __float2int_rz(roundf(__fadd_rn(py, -0.5f)));
        ry.f = __int2float_rn(ry.i);
    }
    if (!round_small(__fadd_rn(px, -0.5f), rx))
    {
        rx.i = __float2int_rz(roundf(__fadd_rn(px, -0.5f)));
        rx.f = __int2float_rn(rx.i);
    }
    const int64_t y0 = ry.i, x0 = rx.i;
    // All-ones footprint: the sample is exactly 1.  The weights q - round(q
    // - 0.5) lie in [0, 1] whenever the footprint starts inside the image
    // (q - 0.5 is exact for q >= 0.5; below, a start of 0 means q in (0,
    // 0.5)), except for q = NaN, whose sample is NaN.
    if (p.field_ones && static_cast<uint64_t>(y0) < static_cast<uint64_t>(p.H) &&
        static_cast<uint64_t>(x0) < static_cast<uint64_t>(p.W) && px == px && py == py)
    {
        const uint32_t word = __ldg(p.ones + (b * p.H + y0) * p.WW + (x0 >> 5));
        if ((word >> (x0 & 31)) & 1u)
            return 1.f;
    }
    const float v00 = mask_sample<DT>(p, masks, b, y0, x0, pad);
    const float v10 = mask_sample<DT>(p, masks, b, y0 + 1, x0, pad);
    const float v01 = mask_sample<DT>(p, masks, b, y0, x0 + 1, pad);
    const float v11 = mask_sample<DT>(p, masks, b, y0 + 1, x0 + 1, pad);
    const float ty = __fsub_rn(py, ry.f);
    const float tx = __fsub_rn(px, rx.f);
    return bilerp(v00, v10, v01, v11, ty, tx);
}

// The all-ones footprint bitmap of the masks (HullPlan::ones).  A warp owns
// 32 columns of a band of kOnesBand rows of one view: it loads the band's
// rows and the row below at once (the last lane also the column after the
// chunk), then per row a lane tests its column, takes its right neighbour's
// result by a shuffle, and a ballot gives the row's "this column and the next
// are 1" bits; a footprint word is the AND of two consecutive rows' bits.
// Each mask row is read once, plus one row per band of 8.  Columns x = W-1 and the
// last row have no 2x2 footprint and get 0.
constexpr int kOnesBand = 8;

template <int DT>
__global__ void __launch_bounds__(256) ones_kernel(HullPlan p)
{
    const void* masks = p.rq->masks;
    const int64_t H = p.H, W = p.W, WW = p.WW;
    const int64_t bands = (H + kOnesBand - 1) / kOnesBand;
    const int64_t units = p.B * bands * WW;
    const int lane = threadIdx.x & 31;
    const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t u = warp; u < units; u += nwarps)
    {
        // chunk fastest: neighbouring warps read neighbouring segments of a row
        const int64_t chunk = u % WW, vb = u / WW;
        const int64_t band = vb % bands, b = vb / bands;
        const int64_t y0 = band * kOnesBand;
        const int64_t x = chunk * 32 + lane;
        const int64_t view = b * H;
        float own[kOnesBand + 1], right[kOnesBand + 1];
#pragma unroll
        for (int i = 0; i <= kOnesBand; ++i)
        {
            const bool row = y0 + i < H;
            own[i] = row && x < W ? load_f32<DT>(masks, (view + y0 + i) * W + x) : 0.f;
            right[i] = row && lane == 31 && x + 1 < W ? load_f32<DT>(masks, (view + y0 + i) * W + x + 1) : 0.f;
        }
        uint32_t prev = 0;
#pragma unroll
        for (int i = 0; i <= kOnesBand; ++i)
        {
            const bool one = own[i] == 1.f;
            bool next = __shfl_down_sync(0xffffffffu, one, 1);
            if (lane == 31)
                next = right[i] == 1.f;
            const uint32_t pair = __ballot_sync(0xffffffffu, one && next);
            if (i > 0 && lane == 0 && y0 + i - 1 < H)
                p.ones[(view + y0 + i - 1) * WW + chunk] = prev & pair;
            prev = pair;
        }
    }
}

// Sets the bits of the corners below the isolevel in the sign words.  A warp's
// corners are neighbours in the list, so most of them share a few words: one
// atomic per word and warp.
__device__ __forceinline__ void mark_sign(const HullPlan& p, bool valid, int64_t gx, int64_t gy, int64_t gz, float value)
{
    uint32_t k = kNoWord;
    if (valid)
    {
        const uint32_t row = static_cast<uint32_t>(gy) + static_cast<uint32_t>(gz) * static_cast<uint32_t>(p.R);
        k = __ldg(p.row_slot + row) * p.wr + static_cast<uint32_t>(gx >> 5);
    }
    const bool low = valid && value < 0.5f;
    if (!__any_sync(0xffffffffu, low))
        return;
    const uint32_t peers = __match_any_sync(0xffffffffu, k);
    const uint32_t bits = __reduce_or_sync(peers, low ? 1u << (gx & 31) : 0u);
    if (bits && static_cast<int>(threadIdx.x & 31) == __ffs(peers) - 1)
        atomicOr(p.sign + k, bits);
}

// Adds the block's evaluated (corner, view) pairs to the request's counter.
__device__ __forceinline__ void count_items(const HullPlan& p, unsigned long long items)
{
    const unsigned long long total = block_sum(items);
    if (threadIdx.x == 0 && total)
        atomicAdd(&p.ctr->field_items, total);
}

// accumulate_hull_counts_{full,partial} (visual_hull_cuda.cu:419-520): the
// views [b0, b1) multiplied into each corner's running product in ascending
// view order (b0 == 0 starts it at 1).  Views go in chunks of kFieldViews, one
// launch each, so that all resident threads read the masks of the same few
// views and those stay in L2; the product is the same sequence of roundings.
constexpr int64_t kFieldViews = 16;

template <int DT, bool PARTIAL>
__global__ void __launch_bounds__(256) field_kernel(HullPlan p, int64_t b0, int64_t b1)
{
    // the projection rows of the chunk's views, read from shared memory by
    // every (corner, view) pair instead of twelve global loads each
    __shared__ float4 rows[kFieldViews][3];
    const int nv = static_cast<int>(b1 - b0);
    for (int i = threadIdx.x; i < 3 * nv; i += blockDim.x)
    {
        const int v = i / 3, r = i - 3 * (i / 3);
        const int row = r < 2 ? r : (p.opengl ? 3 : 2);
        rows[v][r] = *reinterpret_cast<const float4*>(p.tf + 16 * (b0 + v) + 4 * row);
    }
    __syncthreads();
    const int64_t n = p.ctr->corners;
    const int64_t R = p.R;
    const float inv_rc = __fdiv_rn(1.f, static_cast<float>(R - 1)); // exact: a power of two
    const float Hf = small_i2f(static_cast<int32_t>(p.H)), Wf = small_i2f(static_cast<int32_t>(p.W));
    const float cx = p.rq->corner[0], cy = p.rq->corner[1], cz = p.rq->corner[2], length = p.rq->length;
    const void* masks = p.rq->masks;
    const int lane = threadIdx.x & 31;
    const bool final = b1 >= p.B;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    unsigned long long items = 0;
    for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x - lane; t0 < n; t0 += stride)
    {
        const int64_t t = t0 + lane;
        const bool valid = t < n;
        int64_t gx = 0, gy = 0, gz = 0;
        float value = 1.f;
        if (valid)
        {
            unpack_corner(p.corners[t], gx, gy, gz);
            // c + v/r * L fused (visual_hull_cuda.cu:444-448); v/r == v * (1/r) exactly
            // corner coordinates are at most 2^12
            const float wx = __fmaf_rn(__fmul_rn(small_i2f(static_cast<int32_t>(gx)), inv_rc), length, cx);
            const float wy = __fmaf_rn(__fmul_rn(small_i2f(static_cast<int32_t>(gy)), inv_rc), length, cy);
            const float wz = __fmaf_rn(__fmul_rn(small_i2f(static_cast<int32_t>(gz)), inv_rc), length, cz);
            if (b0 > 0)
                value = p.values[t];
            items += nv;
#pragma unroll 4
            for (int v = 0; v < nv; ++v)
                value = __fmul_rn(value, view_factor<DT, PARTIAL>(p, masks, b0 + v, rows[v], wx, wy, wz, Hf, Wf));
            p.values[t] = value;
        }
        if (final)
            mark_sign(p, valid, gx, gy, gz, value);
    }
    count_items(p, items);
}

// Views of mask word `word` whose factor at a corner is exactly 1: the OR of the cell-mask
// entries of the level L-1 cells whose lattice holds the corner (x >> 1, and
// also (x - 1) >> 1 for an even x > 0, per axis; cells beyond the grid and
// cells that are no node hold 0).
__device__ __forceinline__ uint32_t corner_view_mask(const HullPlan& p, int word, int64_t gx, int64_t gy, int64_t gz)
{
    // a plane of the table has at most 2^27 cells
    const uint32_t li = p.level - 1, r = 1u << li;
    const uint32_t x0 = static_cast<uint32_t>(gx) >> 1, y0 = static_cast<uint32_t>(gy) >> 1, z0 = static_cast<uint32_t>(gz) >> 1;
    const bool x_low = !(gx & 1) && gx > 0, y_low = !(gy & 1) && gy > 0, z_low = !(gz & 1) && gz > 0;
    const bool x_in = x0 < r, y_in = y0 < r, z_in = z0 < r;
    const uint32_t* c = p.cell_masks + (static_cast<int64_t>(word) << (3 * li)) + (x0 + (y0 << li) + (z0 << (2 * li)));
    // up to eight cells, a fixed pattern of predicated loads (issued together)
    uint32_t m = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
        const bool use = ((q & 1) ? y_low : y_in) && ((q >> 1) ? z_low : z_in);
        const uint32_t* row = c - ((q & 1) ? int64_t{ 1 } << li : 0) - ((q >> 1) ? int64_t{ 1 } << (2 * li) : 0);
        if (use && x_in)
            m |= __ldg(row);
        if (use && x_low)
            m |= __ldg(row - 1);
    }
    return m;
}

constexpr int kMaskedWarps = 8;

// The field with the cell masks, for the views [b0, b1) (at most 32): the
// views of a corner's mask are left out of its product (x * 1 == x); the
// remaining (corner, view) items of a warp's 32 corners are dealt out to its
// lanes, the factors parked in shared memory, and each lane multiplies its
// corner's factors in ascending view order, the reference's order.  A warp
// whose corners skip nothing walks the views directly, one corner per lane.
template <int DT, bool PARTIAL>
__global__ void __launch_bounds__(32 * kMaskedWarps) field_masked_kernel(HullPlan p, int64_t b0, int64_t b1)
{
    __shared__ float4 rows[32][3];
    // a warp's items: their corner (lane) << 8 | view, then their factors
    __shared__ float fac_all[kMaskedWarps][32 * 32];
    const int nv = static_cast<int>(b1 - b0);
    for (int i = threadIdx.x; i < 3 * nv; i += blockDim.x)
    {
        const int v = i / 3, r = i - 3 * (i / 3);
        const int row = r < 2 ? r : (p.opengl ? 3 : 2);
        rows[v][r] = *reinterpret_cast<const float4*>(p.tf + 16 * (b0 + v) + 4 * row);
    }
    __syncthreads();
    float* fac = fac_all[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int64_t n = p.ctr->corners;
    const float inv_rc = __fdiv_rn(1.f, static_cast<float>(p.R - 1)); // exact: a power of two
    const float Hf = small_i2f(static_cast<int32_t>(p.H)), Wf = small_i2f(static_cast<int32_t>(p.W));
    const float cx = p.rq->corner[0], cy = p.rq->corner[1], cz = p.rq->corner[2], length = p.rq->length;
    const void* masks = p.rq->masks;
    const uint32_t vb = nv >= 32 ? 0xffffffffu : ((1u << nv) - 1u);
    const bool final = b1 >= p.B;
    unsigned long long items = 0; // lane 0's: of the warp
    const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t base = warp * 32; base < n; base += nwarps * 32)
    {
        const int64_t t = base + lane;
        const bool valid = t < n;
        float wx = 0.f, wy = 0.f, wz = 0.f, value = 1.f;
        int64_t gx = 0, gy = 0, gz = 0;
        uint32_t skip = 0;
        if (valid)
        {
            unpack_corner(p.corners[t], gx, gy, gz);
            // c + v/r * L fused (visual_hull_cuda.cu:444-448), as in field_kernel
            wx = __fmaf_rn(__fmul_rn(small_i2f(static_cast<int32_t>(gx)), inv_rc), length, cx);
            wy = __fmaf_rn(__fmul_rn(small_i2f(static_cast<int32_t>(gy)), inv_rc), length, cy);
            wz = __fmaf_rn(__fmul_rn(small_i2f(static_cast<int32_t>(gz)), inv_rc), length, cz);
            if (b0 < 32 * p.mask_words)
                skip = corner_view_mask(p, static_cast<int>(b0 >> 5), gx, gy, gz) & vb;
            if (b0 > 0)
                value = p.values[t];
        }
        if (!__any_sync(0xffffffffu, skip != 0))
        {
            const unsigned nvalid = __popc(__ballot_sync(0xffffffffu, valid));
            items += static_cast<unsigned long long>(nvalid) * nv;
            if (valid)
            {
#pragma unroll 4
                for (int v = 0; v < nv; ++v)
                    value = __fmul_rn(value, view_factor<DT, PARTIAL>(p, masks, b0 + v, rows[v], wx, wy, wz, Hf, Wf));
            }
        }
        else
        {
            const uint32_t active = valid ? (vb & ~skip) : 0u;
            const int count = __popc(active);
            const int incl = warp_inclusive_scan(count);
            const int excl = incl - count;
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            items += static_cast<unsigned long long>(total);
            // each lane lists its corner's items, then the items go to the lanes
            // in turn (finding an item's corner and view by searching the
            // lanes' offsets and masks cost half as much as its factor)
            int at = excl;
            for (uint32_t m = active; m; m &= m - 1)
                fac[at++] = __int_as_float((lane << 8) | (__ffs(m) - 1));
            __syncwarp();
            for (int k0 = 0; k0 < total; k0 += 32)
            {
                const int k = k0 + lane;
                const uint32_t item = k < total ? __float_as_uint(fac[k]) : 0u;
                const int s = static_cast<int>(item >> 8);
                const float sx = __shfl_sync(0xffffffffu, wx, s);
                const float sy = __shfl_sync(0xffffffffu, wy, s);
                const float sz = __shfl_sync(0xffffffffu, wz, s);
                if (k < total)
                {
                    const int v = static_cast<int>(item & 0xffu);
                    fac[k] = view_factor<DT, PARTIAL>(p, masks, b0 + v, rows[v], sx, sy, sz, Hf, Wf);
                }
            }
            __syncwarp();
            for (int j = 0; j < count; ++j)
                value = __fmul_rn(value, fac[excl + j]);
            __syncwarp();
        }
        if (valid)
            p.values[t] = value;
        if (final)
            mark_sign(p, valid, gx, gy, gz, value);
    }
    count_items(p, lane == 0 ? items : 0);
}

// interpolate_vertex (marching_cubes_cuda.cu:72-97) followed by the world
// transform of to_global_coordinates (visual_hull_cuda.cu:916-939).
__device__ __forceinline__ void edge_vertex(const HullPlan& p,
                                            uint32_t x1,
                                            uint32_t y1,
                                            uint32_t z1,
                                            int axis,
                                            float v1,
                                            float v2,
                                            float scale,
                                            float* out)
{
    const float iso = 0.5f, eps = 1e-5f;
    // 1: snap to p1, 2: snap to p2, 0: interpolate (the reference's check order)
    int snap = 0;
    if (fabsf(__fsub_rn(iso, v1)) < eps)
        snap = 1;
    else if (fabsf(__fsub_rn(iso, v2)) < eps)
        snap = 2;
    else if (fabsf(__fsub_rn(v1, v2)) < eps)
        snap = 1;
    const float t = __fdiv_rn(__fsub_rn(iso, v1), __fsub_rn(v2, v1)); // unused after a snap
    // grid coordinates are below 2^13: exact float conversions by adds (the
    // 64-bit integer conversions run on GB300's FP64 pipe)
    const float f1[3] = { small_i2f(static_cast<int32_t>(x1)), small_i2f(static_cast<int32_t>(y1)), small_i2f(static_cast<int32_t>(z1)) };
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        const float f2 = a == axis ? __fadd_rn(f1[a], 1.f) : f1[a];
        const float q = snap == 1 ? f1[a] : (snap == 2 ? f2 : lerp(f1[a], f2, t));
        out[a] = __fmaf_rn(scale, q, p.corner[a]);
    }
}

// The corner grid's words (th_words.cuh): those of the touched rows.
struct HullWords
{
    HullPlan p;
    float scale;

    __device__ int64_t words() const
    {
        return p.ctr->words;
    }
    __device__ int64_t counted() const
    {
        return 0; // not asked for
    }
    __device__ uint32_t word(uint32_t i) const
    {
        return __ldg(p.word_list + i);
    }
    // After the field: its cell-mask table is left clear for the next request.
    __device__ void tail() const
    {
        if (!p.cell_masks)
            return;
        const int li = p.level - 1;
        const int64_t n = p.ctr->level_count[li], off = p.ctr->level_off[li], stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
        for (int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; k < n; k += stride)
            for (int w = 0; w < p.mask_words; ++w)
                p.cell_masks[(static_cast<int64_t>(w) << (3 * li)) + p.nodes[off + k]] = 0;
    }
    __device__ bool empty(uint32_t) const
    {
        return false; // listed words have corners
    }
    __device__ uint32_t sign(uint32_t k) const
    {
        return __ldg(p.sign + k);
    }
    __device__ WordRows rows(uint32_t k) const
    {
        const uint32_t slot = fast_div(p.div_wr, k), w = k - slot * p.wr;
        const uint32_t* near = p.row_place[slot].near;
        const uint32_t up = __ldg(near + 7), back = __ldg(near + 5), both = __ldg(near + 8);
        WordRows r;
        r.next = w + 1 < p.wr;
        r.idx[0] = k;
        r.idx[1] = up != kNoWord ? up * p.wr + w : kNoWord;
        r.idx[2] = back != kNoWord ? back * p.wr + w : kNoWord;
        r.idx[3] = both != kNoWord ? both * p.wr + w : kNoWord;
        return r;
    }
    __device__ EdgeBits edges(uint32_t k, const WordRows&, const uint32_t s[4], const uint32_t sh[4], uint32_t& cells) const
    {
        const uint32_t slot = fast_div(p.div_wr, k), w = k - slot * p.wr;
        const uint4* place = reinterpret_cast<const uint4*>(p.row_place + slot);
        const uint4 n0 = __ldg(place), n1 = __ldg(place + 1);
        const uint32_t near[9] = { n0.x, n0.y, n0.z, n0.w, slot, n1.y, n1.z, n1.w, __ldg(p.row_place[slot].near + 8) };
        return masked_edges(
                [&](int dy, int dz) {
                    const uint32_t n = near[3 * (dy + 1) + dz + 1];
                    return n != kNoWord ? __ldg(p.runs + (n * p.wr + w)) : make_uint2(0u, 0u);
                },
                s, sh, cells);
    }
    __device__ uint32_t entry(uint32_t k, int b) const
    {
        return __ldg(p.rank + k) + static_cast<uint32_t>(__popc(__ldg(p.present + k) & ((1u << b) - 1u)));
    }
    __device__ void vertex(uint32_t k, int b, int axis, float out[3]) const
    {
        const uint32_t slot = fast_div(p.div_wr, k), w = k - slot * p.wr;
        const uint32_t* near = p.row_place[slot].near;
        const uint32_t yz = __ldg(near + 4);
        const uint32_t e1 = entry(k, b);
        // the edge's other end is a corner: a complete cell holds both
        const uint32_t e2 = axis == 0 ? e1 + 1 : entry(__ldg(near + (axis == 1 ? 7 : 5)) * p.wr + w, b);
        edge_vertex(p, w * 32 + b, yz & 0xffffu, yz >> 16, axis, __ldg(p.values + e1), __ldg(p.values + e2), scale, out);
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
        const uint32_t slot = fast_div(p.div_wr, k), w = k - slot * p.wr;
        const uint32_t yz = __ldg(p.row_place[slot].near + 4);
        edge_vertex(p, w * 32 + b + (lo & 1), (yz & 0xffffu) + (lo >> 1 & 1), (yz >> 16) + (lo >> 2 & 1), axis,
                    __ldg(p.values + h1), __ldg(p.values + h2), scale, out);
    }
};

// The last counters of a request; the block that writes them then copies all
// of them to the host.
struct MeshTotal
{
    DevCounters* ctr;
    DevCounters* host;
    __device__ void operator()(unsigned long long total, bool wrapped) const
    {
        if (wrapped)
            ctr->overflow |= kOverflowIndices;
        ctr->soup = static_cast<int64_t>(total >> 32);
        ctr->verts = static_cast<int64_t>(total & 0xffffffffull);
    }
    __device__ void block() const
    {
        __syncthreads();
        for (int i = threadIdx.x; i < static_cast<int>(sizeof(DevCounters) / 8); i += blockDim.x)
            reinterpret_cast<volatile unsigned long long*>(host)[i] = reinterpret_cast<const volatile unsigned long long*>(ctr)[i];
    }
};

HullWords hull_words(const HullPlan& p)
{
    return HullWords{ p, p.length / static_cast<float>(int64_t{ 1 } << p.level) };
}

} // namespace

void launch_corners(const HullPlan& p, cudaStream_t s)
{
    if (p.level == 0)
    {
        mark_root_kernel<<<1, 32, 0, s>>>(p);
        TH_LAUNCH_CHECK();
    }
    else if (p.mark_apart)
    {
        mark_corners_kernel<<<grid_for(p.node_cap, 256), 256, 0, s>>>(p);
        TH_LAUNCH_CHECK();
    }
    launch_rank_corners(p, s);
}

void launch_rank_corners(const HullPlan& p, cudaStream_t s)
{
    const int64_t row_words = (p.R * p.R + 31) / 32;
    if (p.block_rows)
    {
        row_counts_kernel<<<static_cast<unsigned>((row_words + 255) / 256), 256, 0, s>>>(p);
        TH_LAUNCH_CHECK();
    }
    rows_kernel<<<static_cast<unsigned>((row_words + kRowBlock - 1) / kRowBlock), 256, 0, s>>>(p);
    TH_LAUNCH_CHECK();
    corners_kernel<<<grid_for(p.R * p.R, 32), 256, 0, s>>>(p);
    TH_LAUNCH_CHECK();
}

void launch_field(const HullPlan& p, cudaStream_t s)
{
    if (p.field_ones)
    {
        bool ok = dispatch_image_dtype(p.masks_dtype, [&]<int DT>() {
            const int64_t units = p.B * ((p.H + kOnesBand - 1) / kOnesBand) * p.WW;
            ones_kernel<DT><<<grid_for(units * 32, 256), 256, 0, s>>>(p);
        });
        if (!ok)
            throw CudaError{ cudaErrorInvalidValue, "hull field: unsupported mask dtype" };
        TH_LAUNCH_CHECK();
    }
    if (p.cell_masks)
    {
        const int grid = grid_for(p.corner_cap, 32 * kMaskedWarps);
        // at least one launch, so that B == 0 still writes the empty product 1
        for (int64_t b0 = 0; b0 == 0 || b0 < p.B; b0 += 32)
        {
            const int64_t b1 = b0 + 32 < p.B ? b0 + 32 : p.B;
            bool ok = dispatch_image_dtype(p.masks_dtype, [&]<int DT>() {
                if (p.partial)
                    field_masked_kernel<DT, true><<<grid, 32 * kMaskedWarps, 0, s>>>(p, b0, b1);
                else
                    field_masked_kernel<DT, false><<<grid, 32 * kMaskedWarps, 0, s>>>(p, b0, b1);
            });
            if (!ok)
                throw CudaError{ cudaErrorInvalidValue, "hull field: unsupported mask dtype" };
            TH_LAUNCH_CHECK();
        }
        return;
    }
    const int grid = grid_for(p.corner_cap, 256);
    // at least one launch, so that B == 0 still writes the empty product 1
    for (int64_t b0 = 0; b0 == 0 || b0 < p.B; b0 += kFieldViews)
    {
        const int64_t b1 = b0 + kFieldViews < p.B ? b0 + kFieldViews : p.B;
        bool ok = dispatch_image_dtype(p.masks_dtype, [&]<int DT>() {
            if (p.partial)
                field_kernel<DT, true><<<grid, 256, 0, s>>>(p, b0, b1);
            else
                field_kernel<DT, false><<<grid, 256, 0, s>>>(p, b0, b1);
        });
        if (!ok)
            throw CudaError{ cudaErrorInvalidValue, "hull field: unsupported mask dtype" };
        TH_LAUNCH_CHECK();
    }
}

void launch_marching_cubes(const HullPlan& p, cudaStream_t s)
{
    const HullWords src = hull_words(p);
    const int grid = words_grid(std::min(p.word_cap, p.R * p.R * static_cast<int64_t>(p.wr)));
    if (p.unique)
        words_count_kernel<HullWords, true><<<grid, kWordThreads, 0, s>>>(src, p.mesh, &p.ctr->scan, nullptr, MeshTotal{ p.ctr, p.host_ctr });
    else
        words_count_kernel<HullWords, false><<<grid, kWordThreads, 0, s>>>(src, p.mesh, &p.ctr->scan, nullptr, MeshTotal{ p.ctr, p.host_ctr });
    TH_LAUNCH_CHECK();
    words_base_kernel<HullWords><<<grid, kWordThreads, 0, s>>>(src, p.mesh);
    TH_LAUNCH_CHECK();
}

void launch_export(const HullPlan& p, int64_t words, float* verts, int64_t* faces, cudaStream_t s)
{
    const HullWords src = hull_words(p);
    const int grid = words_export_grid(words);
    launch_words_export<HullWords, true>(src, p.mesh, p.unique, grid, verts, faces, s);
}

namespace
{

template <bool COO>
__global__ void __launch_bounds__(256) export_field_kernel(HullPlan p, int64_t n, int64_t* __restrict__ indices, float* __restrict__ values)
{
    const int64_t R = p.R;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < n; t += stride)
    {
        int64_t x, y, z;
        unpack_corner(p.corners[t], x, y, z);
        if constexpr (COO)
        {
            indices[t] = 0;
            indices[n + t] = z;
            indices[2 * n + t] = y;
            indices[3 * n + t] = x;
        }
        else
            indices[t] = x + y * R + z * R * R;
        // coalescing sums a point's values from 0, so no value of the tensor is -0 (a
        // product of negative mask samples can be)
        values[t] = COO ? __fadd_rn(p.values[t], 0.f) : p.values[t];
    }
}

} // namespace

void launch_export_field(const HullPlan& p, int64_t n, int64_t* indices, float* values, cudaStream_t s)
{
    if (n <= 0)
        return;
    export_field_kernel<false><<<grid_for(n, 256), 256, 0, s>>>(p, n, indices, values);
    TH_LAUNCH_CHECK();
}

void launch_export_field_coo(const HullPlan& p, int64_t n, int64_t* indices, float* values, cudaStream_t s)
{
    if (n <= 0)
        return;
    export_field_kernel<true><<<grid_for(n, 256), 256, 0, s>>>(p, n, indices, values);
    TH_LAUNCH_CHECK();
}

} // namespace th
