// Octree carving: the first levels in one launch, then one launch pair per
// level (classify, then compact), the last level without the second.
//
// Reference: classify_children_full / _partial (visual_hull_cuda.cu:168-417)
// run one thread per child and project each of the child's 8 corners for
// every view; the level loop (:633-751) compacts the flags with cub and reads
// the count back to the host.
//
// Lattice.  For one parent and one view, a lane walks the parent's 3x3x3
// lattice of child corners plane by plane (z).  The nested fmas of the
// projection fma(a0,x,fma(a1,y,fma(a2,z,a3))) are evaluated innermost-first,
// so the z and (y,z) partial sums are shared between lattice points without
// changing a single rounding; each plane is reduced to the pixel boxes of its
// four 2x2 point cells, and the four children between two consecutive planes
// take the union of their two cells: 27 projections where the reference makes
// 64.  Per child the per-view outcomes combine by OR (empty in any view,
// partial in any view, fully inside some frame), so any split of the views
// across lanes, OR-reduced, gives the reference's decision exactly.
//
// Two kernels share that per-(parent, view) routine:
//  * views over lanes: a group of LANES lanes owns one parent, lane = view;
//    coherent and best while every view must be evaluated;
//  * (parent, view) items: a warp takes a chunk of parents, lists the views
//    each parent still needs (below) and deals the items out to its lanes;
//    results are merged in the parent's slot by shared atomics.  Best when
//    many views are skipped.
// The host picks one per level (autotuned by measuring both).
//
// View skipping (binary masks).  When a child's pixel box grown by two pixels
// lies inside the image and holds only ones, every descendant of the child is
// "object" in that view: the descendants' corners project into the child's
// box up to rounding errors far below a pixel, so their rounded boxes stay
// within one pixel of the child's, their boxes grown by one pixel stay inside
// the grown box, every pixel there is 1, and "object" contributes nothing to
// the decision.  The child records the view in its skip mask, its children
// inherit the mask, and the item kernel never evaluates the view for any of
// them.  In partial mode a skipped view must also report "fully inside" at the
// last level, so the rule also requires every corner of the child to round at
// least two pixels inside the frame.  All corners must be in front of the
// camera for any of this.
//
// Out-of-frame views (partial masks).  A child box more than two pixels
// outside the image (box_out) can change nothing for any descendant; the view
// goes into the child's out mask, is inherited and skipped the same way.
//
// Conversions: the reference converts the rounded pixel coordinates to int64
// (glm::i64vec2).  On GB300 64-bit float<->int conversions run on the FP64
// pipe, which made them the bottleneck, so the kernels convert to int32 with
// saturation instead.  Every use of those values is a clamp to [0, size-1] or
// an in-image test, whose outcome is the same for the int64 and the saturated
// int32 value (including +-inf and NaN).  The one exception is partial mode's
// unclamped box area; a child whose rounded box leaves the int32 range takes
// the exact int64 path for that view.
//
// The 8 child flags of a parent become one byte; children_kernel writes the
// refined children (and their masks) in the reference's stable order (parent
// order, then child index) and stores the level's size on the device for the
// next one.

#include <algorithm>
#include <cfloat>
#include <cooperative_groups.h>
#include <cstddef>

#include "th_classify.cuh"
#include "th_hull.cuh"
#include "th_internal.h"

namespace th
{

namespace
{

#ifndef TH_CARVE_WARPS
#define TH_CARVE_WARPS 8
#endif
constexpr int kWarps = TH_CARVE_WARPS; // warps per block of the classify kernels
#ifndef TH_CARVE_MIN_BLOCKS
#define TH_CARVE_MIN_BLOCKS 2
#endif
// resident blocks per SM the classify kernels' register budget is cut for
constexpr int kMinBlocks = TH_CARVE_MIN_BLOCKS;
constexpr int kGridPerSm = 16; // blocks of the item kernel's grid per SM

template <int DT>
__device__ __forceinline__ float transform_value(const void* tf, int64_t i)
{
    return load_f32<DT>(tf, i);
}

__global__ void __launch_bounds__(256) begin_kernel(HullPlan p, const void* tf, int tf_dtype, const ReqConsts* host_rq, ReqConsts* rq, float* out, unsigned int* flags, bool clear_flags)
{
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = t; i < p.B * 16; i += stride)
        out[i] = tf_dtype == TH_FLOAT32 ? transform_value<TH_FLOAT32>(tf, i)
                 : tf_dtype == TH_FLOAT64 ? transform_value<TH_FLOAT64>(tf, i) : transform_value<TH_FLOAT16>(tf, i);
    // the counters: level 0 is the root, level 1 starts behind it
    constexpr int64_t kWords = sizeof(DevCounters) / 8;
    constexpr int64_t kCount0 = offsetof(DevCounters, level_count) / 8, kOff1 = offsetof(DevCounters, level_off) / 8 + 1;
    auto* ctr = reinterpret_cast<unsigned long long*>(p.ctr);
    for (int64_t i = t; i < kWords; i += stride)
        ctr[i] = i == kCount0 || i == kOff1 ? 1ull : 0ull;
    for (int64_t i = t; i < p.R * p.R / 256 + 2; i += stride)
        p.coarse[i] = make_uint2(0u, 0u);
    if (t < 4)
        p.carve_sums[t & 1][t >> 1] = 0;
    if (t == 0)
    {
        p.nodes[0] = 0;
        for (int w = 0; w < p.mask_words; ++w)
        {
            p.node_skip[w * p.node_cap] = 0;
            p.node_out[w * p.node_cap] = 0;
        }
        *rq = *host_rq;
        if (clear_flags)
            *flags = 0;
    }
}

// Per-level constants shared by both kernels.
struct LevelInfo
{
    int64_t n;
    const int64_t* parents;
    const uint32_t* parent_skip;
    const uint32_t* parent_out;
    float inv_rc;
    bool last;
    bool skips;       // binary masks: skip masks are valid and may be produced
    bool produce;     // compute the children's skip masks (the next level consumes them)
    bool skip_inside; // partial mode: the skip rule also wants the corners in frame
    bool produce_out; // compute the children's out-of-frame masks (partial; the next level consumes them)
    int skip_grow;    // margin of the children's skip rule: 1 when their children are leaves, else 2
};

__device__ __forceinline__ LevelInfo level_info(const HullPlan& p, int li, bool partial)
{
    LevelInfo L;
    const DevCounters* ctr = p.ctr;
    L.n = ctr->level_count[li];
    const int64_t off = ctr->level_off[li];
    L.parents = p.nodes + off;
    L.parent_skip = p.node_skip + off;
    L.parent_out = p.node_out + off;
    L.inv_rc = __int_as_float((127 - (li + 1)) << 23); // 2^-(li + 1), exact
    L.last = (li == p.level - 1);
    L.skips = p.skip_ok && (*p.nonbinary == 0);
    // the children are parents of the next level, which uses the item kernel
    L.produce = L.skips && (li + 1 < p.level) && p.carve_variant[li + 1] == 1;
    L.skip_inside = partial;
    L.produce_out = partial && (li + 1 < p.level) && p.carve_variant[li + 1] == 1;
    L.skip_grow = li + 2 == p.level ? 1 : 2;
    return L;
}

// The refined children of a warp's parents (base: its first parent; valid
// lanes hold parent pi and cell idx): their mask is kept; before the last
// level their number goes into the level's sums of 1024 parents, for the
// compaction; at the last level they are the leaves, which are counted into
// leaves and, unless that is left to another launch, marked at once (the leaf
// list itself is written only when its candidates are exported).
__device__ __forceinline__ void finish_parents(const HullPlan& p, const LevelInfo& L, int li, int64_t base, bool valid, int64_t pi, int64_t idx, uint32_t empty, uint32_t refine, uint32_t inside, bool partial, uint32_t& leaves)
{
    uint32_t mask = 0;
    if (valid)
    {
        mask = refine & ~empty;
        if (partial && L.last)
            mask &= inside;
        p.child_masks[pi] = static_cast<uint8_t>(mask);
    }
    if (L.last)
    {
        leaves += __popc(mask);
        if (mask && !p.mark_apart)
        {
            const int64_t r = int64_t{ 1 } << li;
            mark_children_corners(p.bitmap, p.rowbits, p.R, p.WR, 2 * (idx & (r - 1)), 2 * ((idx >> li) & (r - 1)),
                                  2 * (idx >> (2 * li)), mask);
        }
        return;
    }
    // a warp's parents lie in at most two groups
    const int64_t g0 = base >> 10;
    const uint32_t cnt = __popc(mask);
    const bool second = valid && (pi >> 10) != g0;
    const uint32_t a = __reduce_add_sync(0xffffffffu, second ? 0u : cnt), b = __reduce_add_sync(0xffffffffu, second ? cnt : 0u);
    if ((threadIdx.x & 31) == 0)
    {
        if (a)
            atomicAdd(p.carve_sums[li & 1] + g0, a);
        if (b)
            atomicAdd(p.carve_sums[li & 1] + g0 + 1, b);
    }
}

// Adds the block's evaluated (parent, view) items (lane 0's) and leaves (every
// lane's) to the request's counters.
__device__ __forceinline__ void count_carved(const HullPlan& p, int li, uint32_t items, uint32_t leaves)
{
    __shared__ unsigned long long sums[2];
    if (threadIdx.x < 2)
        sums[threadIdx.x] = 0;
    __syncthreads();
    leaves = __reduce_add_sync(0xffffffffu, leaves);
    if ((threadIdx.x & 31) == 0)
    {
        if (items)
            atomicAdd(&sums[0], static_cast<unsigned long long>(items));
        if (leaves)
            atomicAdd(&sums[1], static_cast<unsigned long long>(leaves));
    }
    __syncthreads();
    if (threadIdx.x < 2 && sums[threadIdx.x])
        atomicAdd(threadIdx.x == 0 ? &p.ctr->items[li] : &p.ctr->leaves, sums[threadIdx.x]);
}

// Views over lanes: a group of LANES lanes owns one parent.
template <int LANES, bool PARTIAL, bool OPENGL>
__global__ void __launch_bounds__(32 * kWarps, kMinBlocks) classify_views_kernel(HullPlan p, int li)
{
    constexpr int G = 32 / LANES;
    const LevelInfo L = level_info(p, li, PARTIAL);
    const int lane = threadIdx.x & 31;
    const int sub = lane % LANES, grp = lane / LANES;
    const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    // skip masks can come out of a ballot only when lane == view (of a word)
    const bool produce = L.produce && LANES == 32;
    const bool produce_out = L.produce_out && LANES == 32;
    uint32_t items = 0, leaves = 0; // a warp's items of one level: below 2^32
    for (int64_t base = warp * G; base < L.n; base += nwarps * G)
    {
        const int64_t pi = base + grp;
        const bool valid = pi < L.n;
        items += static_cast<uint32_t>(p.B * (L.n - base < G ? L.n - base : G));
        uint32_t empty = 0, refine = 0, inside = 0;
        float wx[3], wy[3], wz[3];
        const int64_t idx = valid ? L.parents[pi] : 0;
        if (valid)
            lattice_world(p.rq->corner, p.rq->length, idx, li, L.inv_rc, wx, wy, wz);
        const ViewSource src = make_view_source(p.tf, p.sat, p.H, p.W);
        const bool keep = LANES == 32 && pi < p.parent_cap && !L.last; // the children's masks are kept
        for (int64_t b0 = 0; b0 < p.B; b0 += LANES)
        {
            const int64_t b = b0 + sub;
            uint32_t skip = 0, outb = 0;
            if (valid && b < p.B)
            {
                const bool word = b < 32 * kMaxMaskWords;
                const ItemResult r = classify_item(PARTIAL, OPENGL, src, b, wx, wy, wz, produce && word, L.skip_inside,
                                                                    produce_out && word, L.skip_grow, L.last);
                empty |= r.empty;
                refine |= r.refine;
                inside |= r.inside;
                skip = r.skip;
                outb = r.out;
            }
            const int64_t w = b0 / 32;
            if (keep && w < p.mask_words)
            {
                // one parent per warp: lane c writes the masks of child c
                uint32_t cskip = 0, cout = 0;
                if (produce || produce_out)
                {
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                    {
                        const uint32_t sk = __ballot_sync(0xffffffffu, (skip >> c) & 1u), ou = __ballot_sync(0xffffffffu, (outb >> c) & 1u);
                        if (lane == c)
                        {
                            cskip = sk;
                            cout = ou;
                        }
                    }
                    // the children inherit the parent's skip views (all descendants are object there)
                    if (produce)
                        cskip |= L.parent_skip[w * p.node_cap + pi];
                }
                if (lane < 8)
                {
                    p.child_skip[w * p.parent_cap * 8 + pi * 8 + lane] = cskip;
                    p.child_out[w * p.parent_cap * 8 + pi * 8 + lane] = cout;
                }
            }
        }
#pragma unroll
        for (int off = LANES / 2; off > 0; off >>= 1)
        {
            empty |= __shfl_xor_sync(0xffffffffu, empty, off);
            refine |= __shfl_xor_sync(0xffffffffu, refine, off);
            inside |= __shfl_xor_sync(0xffffffffu, inside, off);
        }
        finish_parents(p, L, li, base, valid && sub == 0, pi, idx, empty, refine, inside, PARTIAL, leaves);
        if (LANES < 32 && valid && sub == 0 && pi < p.parent_cap && !L.last)
        {
#pragma unroll
            for (int c = 0; c < 8; ++c)
            {
                p.child_skip[pi * 8 + c] = 0u; // at most 16 views: one mask word
                p.child_out[pi * 8 + c] = 0u;
            }
        }
    }
    count_carved(p, li, lane == 0 ? items : 0, leaves);
}

// (parent, view) items: a warp deals the unskipped views of a chunk of parents
// out to its lanes, or, with POOL, a block those of its warps' chunks to all
// its threads.  The pool evens out the chunks and fills the lanes, but its
// warps wait for the slowest three times a chunk.  At the last level, whose
// items hand no masks on, that is less than it gives (32x1024^2, level 8: 625
// -> 536 us; 64x2048^2, level 9: 455 -> 382; 13x437x611, level 6: 85 -> 79);
// above it is more (level 7 of the first 378 -> 470, level 8 of the second
// 367 -> 454).
template <bool PARTIAL, bool OPENGL, int MW, bool POOL>
__global__ void __launch_bounds__(32 * kWarps, kMinBlocks) classify_items_kernel(HullPlan p, int li)
{
    __shared__ WarpSlots<MW> slots_all[kWarps];
    constexpr int kPool = POOL ? 32 * kWarps : 1;
    __shared__ int64_t parent_id[kPool];
    __shared__ uint32_t parent_done[MW][kPool]; // views that are no items
    __shared__ int first_item[kPool], warp_items[kWarps];
    const int wi = threadIdx.x >> 5;
    WarpSlots<MW>& ws = slots_all[wi];
    const LevelInfo L = level_info(p, li, PARTIAL);
    const int lane = threadIdx.x & 31;
    const int B = static_cast<int>(p.B);
    // Parents per chunk: a chunk for each of 16 blocks per SM where that
    // leaves at least eight parents (their items must fill 32 lanes), else for
    // half as many, at most one parent per lane.  Two blocks fit an SM; the
    // others start as those end, which evens out what parents cost, and the
    // warps of a block take neighbouring chunks, whose integral-image reads
    // meet in L1.  (Headline scene, levels 7 and 8: 433 and 656 us with 8
    // blocks per SM, 376 and 625 so, 512 and 673 with resident blocks only;
    // chunks handed out by a counter scattered the reads: 64x2048^2, level 8,
    // 599 us against 360.)
    const int64_t share = static_cast<int64_t>(kGridPerSm) * kWarps * p.sms;
    const int64_t fine = (L.n + share - 1) / share, coarse = (2 * L.n + share - 1) / share;
    const int64_t per = fine >= 8 ? fine : (coarse < 8 ? coarse : 8);
    const int ppw = static_cast<int>(per < 1 ? 1 : (per > 32 ? 32 : per));
    uint32_t items = 0, leaves = 0; // a warp's items of one level: below 2^32

    for (int64_t first = static_cast<int64_t>(blockIdx.x) * kWarps * ppw; first < L.n; first += static_cast<int64_t>(gridDim.x) * kWarps * ppw)
    {
        const int64_t base = first + wi * ppw;
        const int64_t pi = base + lane;
        const bool valid = lane < ppw && pi < L.n;
        const int64_t idx = valid ? L.parents[pi] : 0;
        // skipped views, and those that see the parent out of the frame for good (partial mode)
        uint32_t skipm[MW], outm[MW], all[MW], skipped = 0;
        int count = valid ? B : 0;
#pragma unroll
        for (int w = 0; w < MW; ++w)
        {
            const uint32_t vb = view_bits(B, w);
            skipm[w] = (valid && L.skips) ? (L.parent_skip[w * p.node_cap + pi] & vb) : 0u;
            outm[w] = (valid && PARTIAL) ? (L.parent_out[w * p.node_cap + pi] & vb) : 0u;
            all[w] = skipm[w] | outm[w];
            skipped |= skipm[w];
            count -= __popc(all[w]);
        }
        // a skipped view before the last level (partial mode) is one where
        // every child is fully inside the frame
        ws.clear(lane, (PARTIAL && L.last && skipped) ? 0xffu : 0u, outm);
        const int incl = warp_inclusive_scan(count);
        const int sum = __shfl_sync(0xffffffffu, incl, 31);
        items += static_cast<uint32_t>(sum);
        if constexpr (POOL)
        {
            if (lane == 31)
                warp_items[wi] = sum;
            parent_id[threadIdx.x] = idx;
#pragma unroll
            for (int w = 0; w < MW; ++w)
                parent_done[w][threadIdx.x] = all[w];
            __syncthreads();
            int before = 0, total = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w)
            {
                const int n = warp_items[w];
                before += w < wi ? n : 0;
                total += n;
            }
            first_item[threadIdx.x] = before + incl - count;
            __syncthreads();
            for (int k = threadIdx.x; k < total; k += 32 * kWarps)
            {
                // the last parent whose first item is not past k
                int s = 0;
#pragma unroll
                for (int step = 16 * kWarps; step > 0; step >>= 1)
                    s += first_item[s + step] <= k ? step : 0;
                uint32_t alls[MW];
#pragma unroll
                for (int w = 0; w < MW; ++w)
                    alls[w] = parent_done[w][s];
                const int b = item_view<MW>(B, alls, k - first_item[s]);
                float wx[3], wy[3], wz[3];
                lattice_world(p.rq->corner, p.rq->length, parent_id[s], li, L.inv_rc, wx, wy, wz);
                const ViewSource src = make_view_source(p.tf, p.sat, p.H, p.W);
                merge_item<MW>(slots_all[s >> 5], s & 31, b,
                               classify_item(PARTIAL, OPENGL, src, b, wx, wy, wz, L.produce && b < 32 * MW, L.skip_inside,
                                             L.produce_out && b < 32 * MW, L.skip_grow, L.last));
            }
            __syncthreads();
        }
        else
        {
            const int excl = incl - count;
            __syncwarp();
            for (int k0 = 0; k0 < sum; k0 += 32)
            {
                const int k = k0 + lane;
                const int s = item_slot(excl, k);
                const int es = __shfl_sync(0xffffffffu, excl, s);
                uint32_t alls[MW];
#pragma unroll
                for (int w = 0; w < MW; ++w)
                    alls[w] = __shfl_sync(0xffffffffu, all[w], s);
                const int64_t is = __shfl_sync(0xffffffffu, idx, s);
                if (k < sum)
                {
                    const int b = item_view<MW>(B, alls, k - es);
                    float wx[3], wy[3], wz[3];
                    lattice_world(p.rq->corner, p.rq->length, is, li, L.inv_rc, wx, wy, wz);
                    const ViewSource src = make_view_source(p.tf, p.sat, p.H, p.W);
                    merge_item<MW>(ws, s, b,
                                   classify_item(PARTIAL, OPENGL, src, b, wx, wy, wz, L.produce && b < 32 * MW, L.skip_inside,
                                                                  L.produce_out && b < 32 * MW, L.skip_grow, L.last));
                }
            }
            __syncwarp();
        }
        finish_parents(p, L, li, base, valid, pi, idx, ws.empty[lane], ws.refine[lane], ws.inside[lane], PARTIAL, leaves);
        if (valid && pi < p.parent_cap && !L.last)
        {
#pragma unroll
            for (int w = 0; w < MW; ++w)
            {
                uint32_t* cs = p.child_skip + w * p.parent_cap * 8 + pi * 8;
                uint32_t* co = p.child_out + w * p.parent_cap * 8 + pi * 8;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                {
                    cs[c] = L.produce ? (ws.cskip[w][lane][c] | skipm[w]) : 0u;
                    co[c] = L.produce_out ? (ws.cout[w][lane][c] | ws.cout_all[w][lane]) : 0u;
                }
            }
        }
        __syncwarp();
    }
    count_carved(p, li, lane == 0 ? items : 0, leaves);
}

struct ChildCount
{
    const uint8_t* masks;
    __device__ unsigned long long operator()(int64_t i) const
    {
        return static_cast<unsigned long long>(__popc(masks[i]));
    }
};

// The leaves, without view masks: nothing reads those.
struct ChildEmit
{
    HullPlan p;
    int li;
    __device__ void operator()(int64_t i, unsigned long long off, unsigned long long cnt) const
    {
        if (cnt == 0)
            return;
        const DevCounters* c = p.ctr;
        const int64_t mask = (int64_t{ 1 } << li) - 1;
        // Read-only loads: this launch writes only the next level's slots
        // (from level_off[li + 1] on), never this level's nodes or the
        // parents' child masks, so the loads of one chunk of items need not
        // wait for the stores of the previous one.
        const int64_t idx = __ldg(p.nodes + c->level_off[li] + i);
        const int64_t gx = 2 * (idx & mask), gy = 2 * ((idx >> li) & mask), gz = 2 * (idx >> (2 * li));
        const int sh = li + 1; // children ravel at resolution 2^(li+1)
        const uint32_t m = __ldg(p.child_masks + i);
        int64_t out = c->level_off[li + 1] + static_cast<int64_t>(off);
#pragma unroll
        for (int k = 0; k < 8; ++k)
        {
            if (m >> k & 1u)
            {
                if (out < p.node_cap)
                    p.nodes[out] = (gx + (k & 1)) | ((gy + (k >> 1 & 1)) << sh) | ((gz + (k >> 2 & 1)) << (2 * sh));
                ++out;
            }
        }
    }
};

struct ChildEpilogue
{
    DevCounters* ctr;
    int li;
    int64_t node_cap;
    int64_t parent_cap;
    __device__ void operator()(unsigned long long total) const
    {
        const int64_t start = ctr->level_off[li + 1];
        int64_t n = static_cast<int64_t>(total);
        if (ctr->level_count[li] > parent_cap)
            ctr->overflow |= kOverflowParents; // skip masks were dropped for the excess
        if (start + n > node_cap)
        {
            ctr->overflow |= kOverflowNodes;
            n = 0; // stop the octree here; the host retries with a larger pool
        }
        ctr->level_count[li + 1] = n;
        ctr->level_off[li + 2] = start + n;
    }
};

// Compaction of a level: the refined children of its cells, in cell order,
// with their masks, and (the children of level L-2) their entries of the
// field's cell-mask table.  A block takes a contiguous range of parents; the
// children before it are the sums of 1024 parents that the classify kernels
// left, and the masks since.  A parent per thread (a scan pass that gave a
// thread eight parents in turn took 12 to 28 us at any size, and another launch
// for the sums 4 to 6, and one for the table 20; this takes 7 us at 4096
// parents, 52 at the 1.7 M children of the headline scene's level 8).
__global__ void __launch_bounds__(256) children_kernel(HullPlan p, int li)
{
    const DevCounters* c = p.ctr;
    const int tid = threadIdx.x;
    const int64_t n = c->level_count[li], start = c->level_off[li], next = c->level_off[li + 1];
    const uint32_t* sums = p.carve_sums[li & 1];
    // the next level's sums start at zero
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + tid; i < (8 * n < p.node_cap ? 8 * n : p.node_cap) / 1024 + 2; i += static_cast<int64_t>(gridDim.x) * 256)
        p.carve_sums[(li + 1) & 1][i] = 0;
    const int64_t tiles = (n + 255) / 256, per = (tiles + gridDim.x - 1) / gridDim.x;
    const int64_t t0 = per * blockIdx.x, t1 = t0 + per < tiles ? t0 + per : tiles;
    if (t0 >= tiles && (blockIdx.x > 0 || n > 0))
        return;
    unsigned long long before = 0, total;
    for (int64_t i = tid; i < t0 / 4; i += 256)
        before += sums[i];
    for (int64_t i = t0 / 4 * 1024 + tid; i < t0 * 256; i += 256)
        before += __popc(p.child_masks[i]);
    block_exclusive_scan(before, &total);
    int64_t base = next + static_cast<int64_t>(total);
    const int sh = li + 1; // children ravel at resolution 2^(li+1)
    const int64_t low = (int64_t{ 1 } << li) - 1;
    const bool cells = p.cell_masks && li + 2 == p.level;
    for (int64_t tile = t0; tile < t1; ++tile)
    {
        const int64_t i = tile * 256 + tid;
        const uint32_t m = i < n ? p.child_masks[i] : 0u;
        uint32_t sum;
        int64_t out = base + block_exclusive_scan(static_cast<uint32_t>(__popc(m)), &sum);
        base += sum;
        if (!m)
            continue;
        const int64_t idx = __ldg(p.nodes + start + i);
        const int64_t gx = 2 * (idx & low), gy = 2 * ((idx >> li) & low), gz = 2 * (idx >> (2 * li));
        const bool masks = i < p.parent_cap;
#pragma unroll
        for (int k = 0; k < 8; ++k)
        {
            if (!((m >> k) & 1u))
                continue;
            if (out < p.node_cap)
            {
                const int64_t child = (gx + (k & 1)) | ((gy + (k >> 1 & 1)) << sh) | ((gz + (k >> 2 & 1)) << (2 * sh));
                p.nodes[out] = child;
                for (int w = 0; w < p.mask_words; ++w)
                {
                    const int64_t at = w * p.parent_cap * 8 + i * 8 + k;
                    const uint32_t skip = masks ? __ldg(p.child_skip + at) : 0u, gone = masks ? __ldg(p.child_out + at) : 0u;
                    p.node_skip[w * p.node_cap + out] = skip;
                    p.node_out[w * p.node_cap + out] = gone;
                    if (cells)
                        p.cell_masks[(static_cast<int64_t>(w) << (3 * sh)) + child] = skip | gone;
                }
            }
            ++out;
        }
    }
    if (t1 == tiles && tid == 0)
        ChildEpilogue{ p.ctr, li, p.node_cap, p.parent_cap }(static_cast<unsigned long long>(base - next));
}

// The first levels in one launch: at most 1, 8 and 64 parents, too few for the
// GPU, so a launch per step would be all latency (the classify, sum and
// compaction launches of three levels took 47 to 58 us; this takes 15 us
// for 8 views, 24 for 32).  A cluster of blocks deals (child, view) tasks to
// its lanes, eight times as many as (parent, view) items; the outcomes are
// OR-ed into the first block's shared memory, and every block lists the next
// level's cells for itself.  The first block writes the lists out.  No view is
// ruled out here: the masks begin with the children of the level kTopLevels.
constexpr int kTopLevels = 3;
constexpr int kTopCells = 1 + 8 + 64 + 512; // cells of the levels 0 to 3
constexpr int kTopBlocks = 8, kTopThreads = 512;

struct TopShared
{
    uint32_t empty[73], refine[73]; // per parent of the levels 0 to 2
    int32_t node[kTopCells];
};

template <bool PARTIAL, bool OPENGL>
__global__ void __cluster_dims__(kTopBlocks, 1, 1) __launch_bounds__(kTopThreads) carve_top_kernel(HullPlan p, int levels)
{
    namespace cg = cooperative_groups;
    __shared__ TopShared sh;
    cg::cluster_group cluster = cg::this_cluster();
    TopShared& first = *cluster.map_shared_rank(&sh, 0);
    const int tid = threadIdx.x, rank = static_cast<int>(cluster.block_rank());
    const int B = static_cast<int>(p.B);
    const ViewSource src = make_view_source(p.tf, p.sat, p.H, p.W);
    for (int i = tid; i < static_cast<int>(sizeof(TopShared) / 4); i += kTopThreads)
        reinterpret_cast<uint32_t*>(&sh)[i] = 0;
    cluster.sync();
    int n = 1, off = 0;     // cells of the level and their place in the lists
    int64_t start = 0;      // the same in the node pool
    for (int li = 0; li < levels && n > 0; ++li)
    {
        const float inv_rc = __int_as_float((127 - (li + 1)) << 23);
        const int64_t tasks = static_cast<int64_t>(n) * 8 * B;
        uint32_t items = 0;
        for (int64_t t = rank * kTopThreads + tid; t < tasks; t += kTopBlocks * kTopThreads)
        {
            const int c = static_cast<int>(t & 7), q = static_cast<int>(t >> 3);
            const int b = q / n, pi = off + (q - b * n);
            items += c == 0 ? 1u : 0u;
            float wx[3], wy[3], wz[3];
            lattice_world(p.rq->corner, p.rq->length, sh.node[pi], li, inv_rc, wx, wy, wz);
            const int dx = c & 1, dy = (c >> 1) & 1, dz = c >> 2;
            const float cx[2] = { dx ? wx[1] : wx[0], dx ? wx[2] : wx[1] };
            const float cy[2] = { dy ? wy[1] : wy[0], dy ? wy[2] : wy[1] };
            const float cz[2] = { dz ? wz[1] : wz[0], dz ? wz[2] : wz[1] };
            const uint32_t cls = classify_child(PARTIAL, OPENGL, src, b, cx, cy, cz);
            if (cls == kEmpty)
                atomicOr(&first.empty[pi], 1u << c);
            else if (cls == kRefine)
                atomicOr(&first.refine[pi], 1u << c);
        }
        items = __reduce_add_sync(0xffffffffu, items);
        if ((tid & 31) == 0 && items)
            atomicAdd(&p.ctr->items[li], static_cast<unsigned long long>(items));
        cluster.sync();
        // every block lists the children; the first one also writes them out
        uint32_t mask = 0, total;
        if (tid < n)
            mask = first.refine[off + tid] & ~first.empty[off + tid];
        uint32_t at = block_exclusive_scan(static_cast<uint32_t>(__popc(mask)), &total);
        const int noff = off + n;
        const int64_t nstart = start + n;
        const int s = li + 1;
        for (; mask; mask &= mask - 1)
        {
            const int c = __ffs(mask) - 1, pi = off + tid;
            const int idx = sh.node[pi], low = (1 << li) - 1;
            const int child = (2 * (idx & low) + (c & 1)) | ((2 * ((idx >> li) & low) + (c >> 1 & 1)) << s) |
                              ((2 * (idx >> (2 * li)) + (c >> 2)) << (2 * s));
            sh.node[noff + at] = child;
            if (rank == 0)
            {
                p.nodes[nstart + at] = child;
                for (int w = 0; w < p.mask_words; ++w)
                {
                    p.node_skip[w * p.node_cap + nstart + at] = 0;
                    p.node_out[w * p.node_cap + nstart + at] = 0;
                }
            }
            ++at;
        }
        if (rank == 0 && tid == 0)
        {
            p.ctr->level_count[li + 1] = total;
            p.ctr->level_off[li + 2] = nstart + total;
        }
        off = noff;
        start = nstart;
        n = static_cast<int>(total);
        __syncthreads();
    }
    cluster.sync(); // the first block's shared memory is read until here
}

template <bool PARTIAL, bool OPENGL>
void launch_classify(const HullPlan& p, int li, int64_t max_parents, cudaStream_t s)
{
    const int threads = 32 * kWarps;
    if (p.carve_variant[li] == 1)
    {
        // about one lane per (parent, view) item when the level is small
        const int grid = static_cast<int>(std::min<int64_t>((max_parents * p.B + threads - 1) / threads, static_cast<int64_t>(kGridPerSm) * p.sms));
        const bool pool = li + 1 == p.level;
        if (p.mask_words == 1)
            (pool ? classify_items_kernel<PARTIAL, OPENGL, 1, true> : classify_items_kernel<PARTIAL, OPENGL, 1, false>)<<<grid, threads, 0, s>>>(p, li);
        else
            (pool ? classify_items_kernel<PARTIAL, OPENGL, kMaxMaskWords, true>
                  : classify_items_kernel<PARTIAL, OPENGL, kMaxMaskWords, false>)<<<grid, threads, 0, s>>>(p, li);
        return;
    }
    const int grid = grid_for(max_parents * 32, threads);
    if (p.B <= 4)
        classify_views_kernel<4, PARTIAL, OPENGL><<<grid, threads, 0, s>>>(p, li);
    else if (p.B <= 8)
        classify_views_kernel<8, PARTIAL, OPENGL><<<grid, threads, 0, s>>>(p, li);
    else if (p.B <= 16)
        classify_views_kernel<16, PARTIAL, OPENGL><<<grid, threads, 0, s>>>(p, li);
    else
        classify_views_kernel<32, PARTIAL, OPENGL><<<grid, threads, 0, s>>>(p, li);
}

} // namespace

int grid_for(int64_t work_items, int threads)
{
    const int64_t blocks = (work_items + threads - 1) / threads;
    const int64_t cap = 8LL * sm_count();
    return static_cast<int>(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

void launch_begin(const HullPlan& p, const void* tf, int tf_dtype, const ReqConsts* host_rq, unsigned int* flags, bool clear_flags, cudaStream_t s)
{
    const int64_t items = std::max<int64_t>(p.B * 16, p.R * p.R / 256 + 2);
    begin_kernel<<<grid_for(items, 256), 256, 0, s>>>(p, tf, tf_dtype, host_rq, const_cast<ReqConsts*>(p.rq), const_cast<float*>(p.tf),
                                                      flags, clear_flags);
    TH_LAUNCH_CHECK();
}

// The last level marks corners, which the top kernel does not.
int top_levels(int level)
{
    return level - 1 < kTopLevels ? (level > 1 ? level - 1 : 0) : kTopLevels;
}

void launch_top(const HullPlan& p, cudaStream_t s)
{
    const int levels = top_levels(p.level);
    if (levels == 0)
        return;
    if (p.partial)
    {
        if (p.opengl)
            carve_top_kernel<true, true><<<kTopBlocks, kTopThreads, 0, s>>>(p, levels);
        else
            carve_top_kernel<true, false><<<kTopBlocks, kTopThreads, 0, s>>>(p, levels);
    }
    else
    {
        if (p.opengl)
            carve_top_kernel<false, true><<<kTopBlocks, kTopThreads, 0, s>>>(p, levels);
        else
            carve_top_kernel<false, false><<<kTopBlocks, kTopThreads, 0, s>>>(p, levels);
    }
    TH_LAUNCH_CHECK();
}

void launch_carve_level(const HullPlan& p, int li, cudaStream_t s)
{
    // Upper bound of the parents at level li, for the grid size only.
    const int64_t bound = li < 10 ? (int64_t{ 1 } << (3 * li)) : p.node_cap;
    const int64_t max_parents = bound < p.node_cap ? bound : p.node_cap;
    if (p.partial)
    {
        if (p.opengl)
            launch_classify<true, true>(p, li, max_parents, s);
        else
            launch_classify<true, false>(p, li, max_parents, s);
    }
    else
    {
        if (p.opengl)
            launch_classify<false, true>(p, li, max_parents, s);
        else
            launch_classify<false, false>(p, li, max_parents, s);
    }
    TH_LAUNCH_CHECK();
    // The leaves are not written out: the last level counted them (rows_kernel
    // closes the count), their corners are marked from the child masks, and the leaf list is emitted
    // only when the candidates of the last level are exported.
    if (li + 1 == p.level)
        return;
    children_kernel<<<grid_for(max_parents, 256), 256, 0, s>>>(p, li);
    TH_LAUNCH_CHECK();
}

void launch_emit_leaves(const HullPlan& p, cudaStream_t s)
{
    const int li = p.level - 1;
    if (li < 0)
        return;
    const int64_t bound = li < 10 ? (int64_t{ 1 } << (3 * li)) : p.node_cap;
    const int64_t max_parents = bound < p.node_cap ? bound : p.node_cap;
    run_scan(ChildCount{ p.child_masks }, ChildEmit{ p, li }, NoEpilogue{}, Count{ &p.ctr->level_count[li], 0 },
             max_parents, p.tile_sums, &p.ctr->scan, s);
}

} // namespace th
