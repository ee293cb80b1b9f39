// Per-(parent, view) routine of the carve kernels: the 3x3x3 lattice of a
// parent projected into one view and the classification of its eight children
// (see carve.cu for the design).
#pragma once

#include <cfloat>

#include "th_common.cuh"

namespace th
{

struct Box
{
    float minx, miny, maxx, maxy;
};

__device__ __forceinline__ Box merge(const Box& a, const Box& b)
{
    return Box{ fminf(a.minx, b.minx), fminf(a.miny, b.miny), fmaxf(a.maxx, b.maxx), fmaxf(a.maxy, b.maxy) };
}

// Saturating float -> int32 (NaN to a value outside every image).
__device__ __forceinline__ int32_t f2i32(float f)
{
    return __float2int_rz(f);
}

__device__ __forceinline__ bool fits_i32(float f)
{
    return f > -2147483648.0f && f < 2147483648.0f;
}

__device__ __forceinline__ float box_sum(const float* __restrict__ sat_b, int32_t W, int32_t x0, int32_t y0, int32_t x1, int32_t y1)
{
    // sample_zeros_padding at the four corners (image_utils.h:84-97); inputs are
    // clamped to the image, so only the -1 row/column can leave it.
    const float* row_hi = sat_b + static_cast<int64_t>(y1) * W;
    const float* row_lo = sat_b + static_cast<int64_t>(y0 - 1) * W;
    const float i11 = row_hi[x1];
    const float i10 = x0 > 0 ? row_hi[x0 - 1] : 0.f;
    const float i01 = y0 > 0 ? row_lo[x1] : 0.f;
    const float i00 = (x0 > 0 && y0 > 0) ? row_lo[x0 - 1] : 0.f;
    return __fsub_rn(__fsub_rn(__fadd_rn(i11, i00), i10), i01);
}

enum ViewClass : uint32_t
{
    kNone = 0,
    kEmpty = 1,
    kRefine = 2,
    kObject = 3,
};

struct ViewResult
{
    uint32_t cls;
    bool skip; // the child's children may skip this view
};

// One child in one view from its pixel box (visual_hull_cuda.cu:236-285 and
// :365-410).  The box starts the reference's min/max from +-FLT_MAX.
// want_skip: evaluate the skip rule (the caller checked corners in front and,
// if needed, two pixels inside).  1 <= H, W < 2^23; Hf, Wf the same as floats.
__device__ __forceinline__ ViewResult classify_view(bool PARTIAL, const float* __restrict__ sat_b, int32_t H, int32_t W, float Hf, float Wf, Box bb, bool want_skip, int grow = 2)
{
    const float margin = 0.5f - 0.1f; // isolevel - epsilon (visual_hull_cuda.cu:259-267)
    bb.minx = fminf(FLT_MAX, bb.minx);
    bb.miny = fminf(FLT_MAX, bb.miny);
    bb.maxx = fmaxf(-FLT_MAX, bb.maxx);
    bb.maxy = fmaxf(-FLT_MAX, bb.maxy);
    const float vminx = __fadd_rn(bb.minx, -0.5f);
    const float vminy = __fadd_rn(bb.miny, -0.5f);
    const float vmaxx = __fadd_rn(bb.maxx, 0.5f);
    const float vmaxy = __fadd_rn(bb.maxy, 0.5f);
    // the rounded corners clamped to the image
    const Snapped x0 = round_clamp(vminx, __fsub_rn(Wf, 1.f));
    const Snapped y0 = round_clamp(vminy, __fsub_rn(Hf, 1.f));
    const Snapped x1 = round_clamp(vmaxx, __fsub_rn(Wf, 1.f));
    const Snapped y1 = round_clamp(vmaxy, __fsub_rn(Hf, 1.f));
    // every rounded corner inside the image (the clamps were no-ops): round(v)
    // is in [0, size - 1] exactly when v is in (-0.5, size - 0.5)
    const float hx = __fsub_rn(Wf, 0.5f), hy = __fsub_rn(Hf, 0.5f);
    // (min <= max, so the two outer tests say it all; a box without a point
    // without NaN is FLT_MAX to -FLT_MAX, which neither test passes)
    const bool framed = vminx > -0.5f && vmaxx < hx && vminy > -0.5f && vmaxy < hy && vminx < hx && vminy < hy;
    if (PARTIAL && !framed && vminx > -4194304.f && vmaxx < 4194304.f && vminy > -4194304.f && vmaxy < 4194304.f &&
        vminx < 4194304.f && vminy < 4194304.f)
    {
        // Not "whole": with |v| < 2^22 the rounded box spans at least 2
        // pixels per axis (v_max - v_min >= 1 and round(v + 1) >= round(v) + 1),
        // so on an axis that leaves the image the clamp shortens it and the
        // clamped area is below the unclamped one.  Neither empty nor object
        // then, and the sum is not needed.
        ViewResult res{ kNone, false };
        if (y1.i - y0.i > 1 && x1.i - x0.i > 1)
            res.cls = kRefine;
        return res;
    }
    const float sum = box_sum(sat_b, W, x0.i, y0.i, x1.i, y1.i);
    // float(area) of the int64 area: a product of two exact integers, rounded once
    const float area_f = __fmul_rn(__fadd_rn(__fsub_rn(y1.f, y0.f), 1.f), __fadd_rn(__fsub_rn(x1.f, x0.f), 1.f));
    bool whole = true;
    if (PARTIAL && !framed)
    {
        // full_area_bb (:377) from the unclamped rounded box, int64 arithmetic
        // wrapping like the device's; exact int64 values when int32 cannot hold them.
        const float fminx = roundf(vminx), fminy = roundf(vminy);
        const float fmaxx = roundf(vmaxx), fmaxy = roundf(vmaxy);
        int64_t rminx, rminy, rmaxx, rmaxy;
        if (fits_i32(fminx) && fits_i32(fminy) && fits_i32(fmaxx) && fits_i32(fmaxy))
        {
            rminx = f2i32(fminx);
            rminy = f2i32(fminy);
            rmaxx = f2i32(fmaxx);
            rmaxy = f2i32(fmaxy);
        }
        else
        {
            rminx = f2i64(fminx);
            rminy = f2i64(fminy);
            rmaxx = f2i64(fmaxx);
            rmaxy = f2i64(fmaxy);
        }
        const int64_t area = static_cast<int64_t>(y1.i - y0.i + 1) * static_cast<int64_t>(x1.i - x0.i + 1);
        const uint64_t fy = static_cast<uint64_t>(rmaxy) - static_cast<uint64_t>(rminy) + 1u;
        const uint64_t fx = static_cast<uint64_t>(rmaxx) - static_cast<uint64_t>(rminx) + 1u;
        whole = (static_cast<uint64_t>(area) == fy * fx);
    }
    ViewResult res{ kNone, false };
    if (sum <= 0.f + margin && whole)
        res.cls = kEmpty;
    else if (sum >= __fsub_rn(area_f, margin) && whole)
        res.cls = kObject;
    else if (!PARTIAL || (y1.i - y0.i > 1 && x1.i - x0.i > 1))
        res.cls = kRefine;
    if (want_skip && res.cls == kObject && framed && x0.i >= grow && y0.i >= grow && x1.i <= W - 1 - grow &&
        y1.i <= H - 1 - grow && x0.i <= x1.i && y0.i <= y1.i)
    {
        // the box grown by `grow` pixels is inside the image: all ones there?
        const int32_t gx0 = x0.i - grow, gy0 = y0.i - grow, gx1 = x1.i + grow, gy1 = y1.i + grow;
        const float grown = box_sum(sat_b, W, gx0, gy0, gx1, gy1);
        const float g2 = grow == 1 ? 3.f : 5.f; // 2 * grow + 1
        res.skip = grown == __fmul_rn(__fadd_rn(__fsub_rn(y1.f, y0.f), g2), __fadd_rn(__fsub_rn(x1.f, x0.f), g2));
    }
    return res;
}

#ifndef TH_CARVE_ROLL_Z
#define TH_CARVE_ROLL_Z 1
#endif

struct ItemResult
{
    uint32_t empty, refine, inside, skip; // 8-bit child masks
    uint32_t out;                         // children out of the frame for good (partial mode, want_out)
};

// Partial mode: a child box (from corners all in front of the camera) more
// than 2 pixels outside the image on one side, with every coordinate below
// 2^21 in magnitude.  Every descendant's corners project into this box up to
// rounding errors far below a pixel, so every descendant's box leaves the
// frame on that side too: never whole, a clamped extent of one pixel there
// (not refined), no corner in frame (not inside).  Such a view contributes
// nothing to any descendant and is skipped below.
__device__ __forceinline__ bool box_out(const Box& bb, float Hf, float Wf)
{
    const float lim = 2097152.f;
    return (bb.maxx < -2.f || bb.minx > __fadd_rn(Wf, 1.f) || bb.maxy < -2.f || bb.miny > __fadd_rn(Hf, 1.f)) &&
           fabsf(bb.minx) < lim && fabsf(bb.maxx) < lim && fabsf(bb.miny) < lim && fabsf(bb.maxy) < lim;
}

// View masks hold at most this many words of 32 views (HullPlan::mask_words):
// the kernels keep a word per plane in registers and the pools grow by 0.5 to 1
// GB with each.  Views past the masks are evaluated for every cell: calls of n
// views of 512^2, level 8, take 325 us at 32, 475 at 64 (4.7 us a view more), 534
// at 72, 740 at 96 and 946 at 128 (7.4 a view).
constexpr int kMaxMaskWords = 2;

inline int mask_words_for(int64_t views)
{
    return views > 32 ? kMaxMaskWords : 1;
}

// The views of mask word w that a request with B views has.
__device__ __forceinline__ uint32_t view_bits(int B, int w)
{
    const int n = B - 32 * w;
    return n >= 32 ? 0xffffffffu : (n > 0 ? (1u << n) - 1u : 0u);
}

// Shared-memory accumulators of one warp's chunk of parents (one slot each).
template <int MW>
struct WarpSlots
{
    uint32_t empty[32], refine[32], inside[32];
    uint32_t cskip[MW][32][8];
    // out-of-frame view masks of the children: per child, and for all 8
    uint32_t cout[MW][32][8], cout_all[MW][32];

    __device__ __forceinline__ void clear(int lane, uint32_t inside_views, const uint32_t (&outm)[MW])
    {
        empty[lane] = 0;
        refine[lane] = 0;
        inside[lane] = inside_views;
#pragma unroll
        for (int w = 0; w < MW; ++w)
        {
#pragma unroll
            for (int c = 0; c < 8; ++c)
            {
                cskip[w][lane][c] = 0;
                cout[w][lane][c] = 0;
            }
            // the children inherit the parent's out-of-frame views
            cout_all[w][lane] = outm[w];
        }
    }
};

// View of item j of a parent: its j-th view that is not in all (later views
// than the masks hold come last).
template <int MW>
__device__ __forceinline__ int item_view(int B, const uint32_t (&all)[MW], int j)
{
#pragma unroll
    for (int w = 0; w < MW; ++w)
    {
        const uint32_t active = view_bits(B, w) & ~all[w];
        const int n = __popc(active);
        if (j < n)
            return 32 * w + nth_set_bit(active, j);
        j -= n;
    }
    return 32 * MW + j;
}

// World coordinates of the lattice of the cell idx (ravelled at resolution
// 2^li): c + v/r * L with the product fused (visual_hull_cuda.cu:206-213);
// v/r == v * (1/r) exactly (r = 2^k).
__device__ __forceinline__ void lattice_world(const float corner[3],
                                              float length,
                                              int64_t idx,
                                              int li,
                                              float inv_rc,
                                              float wx[3],
                                              float wy[3],
                                              float wz[3])
{
    const int64_t mask = (int64_t{ 1 } << li) - 1;
    const int32_t gx = static_cast<int32_t>(idx & mask), gy = static_cast<int32_t>((idx >> li) & mask),
                  gz = static_cast<int32_t>(idx >> (2 * li));
#pragma unroll
    for (int d = 0; d < 3; ++d)
    {
        // lattice coordinates below 2^(li + 1) <= 2^14
        wx[d] = __fmaf_rn(__fmul_rn(small_i2f(2 * gx + d), inv_rc), length, corner[0]);
        wy[d] = __fmaf_rn(__fmul_rn(small_i2f(2 * gy + d), inv_rc), length, corner[1]);
        wz[d] = __fmaf_rn(__fmul_rn(small_i2f(2 * gz + d), inv_rc), length, corner[2]);
    }
}

// The per-view data an item reads.
struct ViewSource
{
    const float* tf;  // [B,16] float32 transforms
    const float* sat; // [B,H,W] integral images
    int64_t H, W;     // below 2^23
    float Hf, Wf;     // H, W as floats
};

__device__ __forceinline__ ViewSource make_view_source(const float* tf, const float* sat, int64_t H, int64_t W)
{
    return ViewSource{ tf, sat, H, W, small_i2f(static_cast<int32_t>(H)), small_i2f(static_cast<int32_t>(W)) };
}

// One (parent, view) item: the parent's lattice projected into view b.
// want_skip: compute the children's skip bits; skip_inside: the skip rule also
// needs the child's corners two pixels inside the frame; want_out (partial
// mode): compute the children's out-of-frame bits (box_out); grow: the skip
// rule's margin in pixels, 2 for masks inherited by all descendants, 1 for the
// children whose own children are leaves (one level below them, and the
// field's bilinear footprints of the leaves' corners, stay within one pixel);
// want_inside (partial mode): compute the children's "fully inside" bits (only
// the last level uses them).
//
// "Every corner rounds into the frame" (a pixel coordinate q passes when
// 0.5 <= q < size - 1.5, NaN fails) is tested on the child's box: for corners
// without NaN it holds for all eight exactly when it holds for the box's
// minimum and maximum, so the box test plus a NaN bit per lattice point gives
// the per-corner answer (fminf/fmaxf leave NaN out of the box).
// The modes are arguments (constants where a kernel is built for one); this
// form is a function of its own, for it is rarely wanted.
static __device__ __noinline__ ItemResult classify_item_general(bool PARTIAL,
                                                         bool OPENGL,
                                                         ViewSource p,
                                                         int64_t b,
                                                         float3 x3,
                                                         float3 y3,
                                                         float3 z3,
                                                         bool want_skip,
                                                         bool skip_inside,
                                                         bool want_out,
                                                         int grow,
                                                         bool want_inside)
{
    const float wx[3] = { x3.x, x3.y, x3.z }, wy[3] = { y3.x, y3.y, y3.z }, wz[3] = { z3.x, z3.y, z3.z };
    const int32_t H = static_cast<int32_t>(p.H), W = static_cast<int32_t>(p.W);
    const float Hf = p.Hf, Wf = p.Wf;
    const float* m = p.tf + 16 * b;
    // rows x, y and the divisor row (w for OpenGL, z for OpenCV)
    const float4 rx = *reinterpret_cast<const float4*>(m);
    const float4 ry = *reinterpret_cast<const float4*>(m + 4);
    const float4 rd = *reinterpret_cast<const float4*>(m + (OPENGL ? 12 : 8));
    const float* sat_b = p.sat + b * p.H * p.W;
    const float in_hx = __fsub_rn(Wf, 1.5f), in_hy = __fsub_rn(Hf, 1.5f);
    const float in2_hx = __fsub_rn(Wf, 2.5f), in2_hy = __fsub_rn(Hf, 2.5f);
    ItemResult out{ 0, 0, 0, 0, 0 };
    want_out = PARTIAL && want_out;
    want_inside = PARTIAL && want_inside;
    const bool want_in2 = PARTIAL && want_skip && skip_inside;
    const bool want_nan = want_inside || want_in2;
    Box prev[4];
    uint32_t prev_nan = 0, prev_front = 0;
    // Rolled (the default), the plane loop keeps one copy of the plane's code,
    // a third of the unrolled footprint: 9-11 % faster carve levels on GB300
    // (fewer instruction-fetch stalls); unrolled, it schedules across planes.
#if TH_CARVE_ROLL_Z
#pragma unroll 1
#else
#pragma unroll
#endif
    for (int z = 0; z < 3; ++z)
    {
        const float wzz = z == 0 ? wz[0] : (z == 1 ? wz[1] : wz[2]);
        const float tzx = __fmaf_rn(rx.z, wzz, rx.w);
        const float tzy = __fmaf_rn(ry.z, wzz, ry.w);
        const float tzd = __fmaf_rn(rd.z, wzz, rd.w);
        float px[9], py[9];
        uint32_t nan9 = 0, front9 = 0;
#pragma unroll
        for (int y = 0; y < 3; ++y)
        {
            const float tyx = __fmaf_rn(rx.y, wy[y], tzx);
            const float tyy = __fmaf_rn(ry.y, wy[y], tzy);
            const float tyd = __fmaf_rn(rd.y, wy[y], tzd);
#pragma unroll
            for (int x = 0; x < 3; ++x)
            {
                const int k = x + 3 * y;
                const float cx = __fmaf_rn(rx.x, wx[x], tyx);
                const float cy = __fmaf_rn(ry.x, wx[x], tyy);
                const float cd = __fmaf_rn(rd.x, wx[x], tyd);
                const float nx = __fdiv_rn(cx, cd);
                const float ny = __fdiv_rn(cy, cd);
                if (OPENGL)
                {
                    // (n + 1) * size / 2 - 0.5 (image_utils.h:67-71); /2 == *0.5 exactly
                    px[k] = __fsub_rn(__fmul_rn(__fmul_rn(__fadd_rn(nx, 1.f), Wf), 0.5f), 0.5f);
                    py[k] = __fsub_rn(__fmul_rn(__fmul_rn(__fadd_rn(ny, 1.f), Hf), 0.5f), 0.5f);
                }
                else
                {
                    px[k] = __fsub_rn(nx, 0.5f);
                    py[k] = __fsub_rn(ny, 0.5f);
                }
                if ((want_skip || want_out) && cd > 0.f)
                    front9 |= 1u << k;
                if (want_nan && !(px[k] == px[k] && py[k] == py[k]))
                    nan9 |= 1u << k;
            }
        }
        Box cur[4];
        uint32_t cur_nan = 0, cur_front = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c)
        {
            const int cx = c & 1, cy = c >> 1;
            const int k0 = cx + 3 * cy, k1 = k0 + 1, k2 = k0 + 3, k3 = k0 + 4;
            cur[c] = Box{ fminf(fminf(px[k0], px[k1]), fminf(px[k2], px[k3])),
                          fminf(fminf(py[k0], py[k1]), fminf(py[k2], py[k3])),
                          fmaxf(fmaxf(px[k0], px[k1]), fmaxf(px[k2], px[k3])),
                          fmaxf(fmaxf(py[k0], py[k1]), fmaxf(py[k2], py[k3])) };
            const uint32_t need = (1u << k0) | (1u << k1) | (1u << k2) | (1u << k3);
            if (nan9 & need)
                cur_nan |= 1u << c;
            if ((front9 & need) == need)
                cur_front |= 1u << c;
        }
        if (z > 0)
        {
#pragma unroll
            for (int c = 0; c < 4; ++c)
            {
                const uint32_t cbit = 1u << c;
                const uint32_t bit = 1u << (c + 4 * (z - 1));
                const bool front = (prev_front & cur_front & cbit) != 0;
                const bool nan = ((prev_nan | cur_nan) & cbit) != 0;
                const Box cb = merge(prev[c], cur[c]);
                // 1 <= round(q) < size - 1 (round half away from zero) exactly
                // when 0.5 <= q < size - 1.5; two pixels in: 1.5 <= q < size - 2.5
                const bool in2 = want_in2 && !nan && cb.minx >= 1.5f && cb.maxx < in2_hx && cb.miny >= 1.5f &&
                                 cb.maxy < in2_hy;
                const ViewResult r = classify_view(PARTIAL, sat_b, H, W, Hf, Wf, cb,
                                                            want_skip && front && (!skip_inside || in2), grow);
                if (want_out && front && box_out(cb, Hf, Wf))
                    out.out |= bit;
                if (r.cls == kEmpty)
                    out.empty |= bit;
                else if (r.cls == kRefine)
                    out.refine |= bit;
                if (r.skip)
                    out.skip |= bit;
                if (want_inside && !nan && cb.minx >= 0.5f && cb.maxx < in_hx && cb.miny >= 0.5f &&
                    cb.maxy < in_hy)
                    out.inside |= bit;
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
            prev[c] = cur[c];
        prev_nan = cur_nan;
        prev_front = cur_front;
    }
    return out;
}

// Smallest and largest value of fma(m.x, x, fma(m.y, y, fma(m.z, z, m.w))) over
// a lattice with ascending coordinates: each fma is monotone in its factors,
// roundings included, so they are values at corners.
__device__ __forceinline__ float lattice_bound(const float4& m, const float wx[3], const float wy[3], const float wz[3], bool high)
{
    const float x = (m.x >= 0.f) == high ? wx[2] : wx[0], y = (m.y >= 0.f) == high ? wy[2] : wy[0],
                z = (m.z >= 0.f) == high ? wz[2] : wz[0];
    return __fmaf_rn(m.x, x, __fmaf_rn(m.y, y, __fmaf_rn(m.z, z, m.w)));
}

// A pixel coordinate from a quotient (image_utils.h:62-82).  Monotone, so the
// smallest and largest of several are those of the smallest and largest
// quotient.
__device__ __forceinline__ float pixel_of(bool OPENGL, float n, float size)
{
    if (OPENGL)
        // (n + 1) * size / 2 - 0.5; /2 == *0.5 exactly
        return __fsub_rn(__fmul_rn(__fmul_rn(__fadd_rn(n, 1.f), size), 0.5f), 0.5f);
    return __fsub_rn(n, 0.5f);
}

// One (parent, view) item: the parent's lattice projected into view b (see
// classify_item_general, whose outcome this gives).  The usual item sees the
// whole lattice in front of the camera and in the range of fast_divide: no
// point needs its own front or NaN test, the quotients of a point share a
// reciprocal, and the pixel mapping is left to the boxes of the children.
// The level 8 of the headline scene executes 343 M warp instructions
// this way, 450 M in the general form.
__device__ __forceinline__ ItemResult classify_item(bool PARTIAL,
                                                    bool OPENGL,
                                                    const ViewSource& p,
                                                    int64_t b,
                                                    const float wx[3],
                                                    const float wy[3],
                                                    const float wz[3],
                                                    bool want_skip,
                                                    bool skip_inside,
                                                    bool want_out = false,
                                                    int grow = 2,
                                                    bool want_inside = true)
{
    const float* m = p.tf + 16 * b;
    // rows x, y and the divisor row (w for OpenGL, z for OpenCV)
    const float4 rx = *reinterpret_cast<const float4*>(m);
    const float4 ry = *reinterpret_cast<const float4*>(m + 4);
    const float4 rd = *reinterpret_cast<const float4*>(m + (OPENGL ? 12 : 8));
    constexpr float kLow = kDivideLow, kHigh = kDivideHigh;
    const bool usual = lattice_bound(rd, wx, wy, wz, false) >= kLow && lattice_bound(rd, wx, wy, wz, true) <= kHigh &&
                       lattice_bound(rx, wx, wy, wz, false) >= -kHigh && lattice_bound(rx, wx, wy, wz, true) <= kHigh &&
                       lattice_bound(ry, wx, wy, wz, false) >= -kHigh && lattice_bound(ry, wx, wy, wz, true) <= kHigh;
    if (!usual)
        return classify_item_general(PARTIAL, OPENGL, p, b, make_float3(wx[0], wx[1], wx[2]), make_float3(wy[0], wy[1], wy[2]),
                                                      make_float3(wz[0], wz[1], wz[2]), want_skip, skip_inside, want_out, grow,
                                                      want_inside);
    want_out = PARTIAL && want_out;
    want_inside = PARTIAL && want_inside;
    const bool want_in2 = PARTIAL && skip_inside;
    const int32_t H = static_cast<int32_t>(p.H), W = static_cast<int32_t>(p.W);
    const float Hf = p.Hf, Wf = p.Wf;
    const float* sat_b = p.sat + b * p.H * p.W;
    ItemResult out{ 0, 0, 0, 0, 0 };
    Box prev[4]; // in quotients
#pragma unroll 1
    for (int z = 0; z < 3; ++z)
    {
        const float wzz = z == 0 ? wz[0] : (z == 1 ? wz[1] : wz[2]);
        const float tzx = __fmaf_rn(rx.z, wzz, rx.w), tzy = __fmaf_rn(ry.z, wzz, ry.w), tzd = __fmaf_rn(rd.z, wzz, rd.w);
        Box row[2], cur[4]; // the pairs of points of a row, the cells of the plane
#pragma unroll
        for (int y = 0; y < 3; ++y)
        {
            const float tyx = __fmaf_rn(rx.y, wy[y], tzx), tyy = __fmaf_rn(ry.y, wy[y], tzy), tyd = __fmaf_rn(rd.y, wy[y], tzd);
            float nx[3], ny[3];
#pragma unroll
            for (int x = 0; x < 3; ++x)
            {
                const float cd = __fmaf_rn(rd.x, wx[x], tyd);
                const float rec = fast_reciprocal(cd);
                nx[x] = fast_divide(__fmaf_rn(rx.x, wx[x], tyx), cd, rec);
                ny[x] = fast_divide(__fmaf_rn(ry.x, wx[x], tyy), cd, rec);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
            {
                const Box pair{ fminf(nx[i], nx[i + 1]), fminf(ny[i], ny[i + 1]), fmaxf(nx[i], nx[i + 1]), fmaxf(ny[i], ny[i + 1]) };
                if (y > 0)
                    cur[i + 2 * (y - 1)] = merge(row[i], pair);
                row[i] = pair;
            }
        }
        if (z > 0)
        {
#pragma unroll
            for (int c = 0; c < 4; ++c)
            {
                const uint32_t bit = 1u << (c + 4 * (z - 1));
                const Box nb = merge(prev[c], cur[c]);
                const Box cb{ pixel_of(OPENGL, nb.minx, Wf), pixel_of(OPENGL, nb.miny, Hf), pixel_of(OPENGL, nb.maxx, Wf),
                              pixel_of(OPENGL, nb.maxy, Hf) };
                // two pixels in: 1.5 <= q < size - 2.5; in the frame: 0.5 <= q < size - 1.5 (classify_item_general)
                const bool in2 = !want_in2 || (cb.minx >= 1.5f && cb.maxx < __fsub_rn(Wf, 2.5f) && cb.miny >= 1.5f &&
                                               cb.maxy < __fsub_rn(Hf, 2.5f));
                const ViewResult r = classify_view(PARTIAL, sat_b, H, W, Hf, Wf, cb, want_skip && in2, grow);
                if (want_out && box_out(cb, Hf, Wf))
                    out.out |= bit;
                if (r.cls == kEmpty)
                    out.empty |= bit;
                else if (r.cls == kRefine)
                    out.refine |= bit;
                if (r.skip)
                    out.skip |= bit;
                if (want_inside && cb.minx >= 0.5f && cb.maxx < __fsub_rn(Wf, 1.5f) && cb.miny >= 0.5f &&
                    cb.maxy < __fsub_rn(Hf, 1.5f))
                    out.inside |= bit;
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
            prev[c] = cur[c];
    }
    return out;
}

// ViewClass of one child of a parent in view b (the top levels, where a lane per
// child is wanted for latency): classify_item's outcome for that child alone, from
// the same operations on its eight corners.
__device__ __forceinline__ uint32_t classify_child(bool PARTIAL,
                                                   bool OPENGL,
                                                   const ViewSource& p,
                                                   int64_t b,
                                                   const float wx[2],
                                                   const float wy[2],
                                                   const float wz[2])
{
    const float* m = p.tf + 16 * b;
    const float4 rx = *reinterpret_cast<const float4*>(m);
    const float4 ry = *reinterpret_cast<const float4*>(m + 4);
    const float4 rd = *reinterpret_cast<const float4*>(m + (OPENGL ? 12 : 8));
    float px[8], py[8];
#pragma unroll
    for (int z = 0; z < 2; ++z)
    {
        const float tzx = __fmaf_rn(rx.z, wz[z], rx.w), tzy = __fmaf_rn(ry.z, wz[z], ry.w), tzd = __fmaf_rn(rd.z, wz[z], rd.w);
#pragma unroll
        for (int y = 0; y < 2; ++y)
        {
            const float tyx = __fmaf_rn(rx.y, wy[y], tzx), tyy = __fmaf_rn(ry.y, wy[y], tzy), tyd = __fmaf_rn(rd.y, wy[y], tzd);
#pragma unroll
            for (int x = 0; x < 2; ++x)
            {
                const int k = x + 2 * y + 4 * z;
                const float cx = __fmaf_rn(rx.x, wx[x], tyx), cy = __fmaf_rn(ry.x, wx[x], tyy), cd = __fmaf_rn(rd.x, wx[x], tyd);
                float nx, ny;
                divide_pair(cx, cy, cd, nx, ny);
                px[k] = pixel_of(OPENGL, nx, p.Wf);
                py[k] = pixel_of(OPENGL, ny, p.Hf);
            }
        }
    }
    Box bb{ px[0], py[0], px[0], py[0] };
#pragma unroll
    for (int k = 1; k < 8; ++k)
        bb = merge(bb, Box{ px[k], py[k], px[k], py[k] });
    return classify_view(PARTIAL, p.sat + b * p.H * p.W, static_cast<int32_t>(p.H), static_cast<int32_t>(p.W), p.Hf, p.Wf, bb, false).cls;
}

// Merges an item's outcome into its slot: one shared atomic per non-zero word
// (a slot's items sit in neighbouring lanes, so conflicts are short).
template <int MW>
__device__ __forceinline__ void merge_item(WarpSlots<MW>& ws, int s, int b, const ItemResult& res)
{
    if (b < 32 * MW)
    {
        const int w = b >> 5;
        const uint32_t bit = 1u << (b & 31);
        if (res.out == 0xffu)
            atomicOr(&ws.cout_all[w][s], bit);
        else
            for (uint32_t o = res.out; o; o &= o - 1)
                atomicOr(&ws.cout[w][s][__ffs(o) - 1], bit);
        for (uint32_t m = res.skip; m; m &= m - 1)
            atomicOr(&ws.cskip[w][s][__ffs(m) - 1], bit);
    }
    if (res.empty)
        atomicOr(&ws.empty[s], res.empty);
    if (res.refine)
        atomicOr(&ws.refine[s], res.refine);
    if (res.inside)
        atomicOr(&ws.inside[s], res.inside);
}

} // namespace th
