// Device-side state of one visual-hull request and the launch entry points of
// its stages (carve.cu, mesh.cu).  Every count lives in device memory, so the
// stages chain on one stream with no host round trip; kernels are grid-stride
// loops sized from the SM count that read their item count on the device.
#pragma once

#include <cstdint>

#include "th_common.cuh"
#include "th_words.cuh"

namespace th
{

enum OverflowBits : int64_t
{
    kOverflowNodes = 1,
    kOverflowCorners = 2,
    kOverflowIndices = 4, // more corners, or triangle corners, than 32 bits number: refused
    kOverflowParents = 8,
    kOverflowWords = 16,
};

// From this level on the corners of the leaves are marked by a launch of their
// own: the last classify kernel keeps 16 warps on an SM, few for the waits on
// the bitmap when there are many leaves, while a small request feels the
// launch.  Whole calls, apart against in that kernel: level 6 24x512^2 193 us
// against 185; level 7 230 against 237, 32x1024^2 partial 473 against 480; level
// 8 308 against 318, 815 against 814; level 9 508 against 521, 1961 against
// 1975; level 7 could go either way.  (Before that kernel shared its items between a block's warps, level 9
// took 906 us against 625 + 103 for the two.)
constexpr int kMarkApartLevel = 8;

constexpr int kRowBlock = 32;           // words of row flags a block of rows_kernel owns
constexpr int64_t kCountRowBlocks = 2048; // blocks from which their flags are counted first

struct DevCounters
{
    int64_t level_count[kMaxLevel + 2]; // cells of level i (level 0: the root)
    int64_t level_off[kMaxLevel + 3];   // start of level i in the node pool
    int64_t rows;                       // bitmap rows holding at least one corner
    int64_t corners;                    // unique leaf corners (the sparse field)
    int64_t words;                      // words of 32 points with a corner
    int64_t soup;                       // soup vertices, 3 per face
    int64_t verts;                      // unique mesh vertices
    int64_t overflow;                   // OverflowBits
    int64_t row_words;                  // words of the row-occupancy bitmap
    unsigned long long leaves;          // refined children of the last level
    unsigned long long row_corners;     // corners of the touched rows (corners: once they are known to fit)
    unsigned long long items[kMaxLevel];  // (parent, view) items the carve evaluated per parent level
    unsigned long long field_items;       // (corner, view) pairs the field evaluated
    ScanState scan;
};

// The inputs that differ between requests of one shape, read by the carve
// and field kernels from device memory (written before each run), so that a
// captured graph of the pipeline serves every request of that shape.
struct ReqConsts
{
    float corner[3];
    float length;
    const void* masks;
};

// A touched row and the slots of its eight neighbours, kNoWord where one is not
// touched: near[3 * (dy + 1) + dz + 1] without the middle one, which is yz.
struct RowPlace
{
    uint32_t near[9]; // [4]: y | z << 16
    uint32_t pad[3];
};

// Per-request constants and buffers, passed to kernels by value.
struct HullPlan
{
    // inputs
    const void* masks;
    int masks_dtype;
    int64_t B, H, W;
    const float* tf;  // [B,16] float32
    const float* sat; // [B,H,W]
    bool opengl, partial, unique;
    float corner[3];
    float length;
    int level;
    int sms;         // SMs of the device
    bool mark_apart; // the last level's corners are marked by a launch of their own
    // octree node pool: all levels back to back
    int64_t* nodes;
    int64_t node_cap;
    uint8_t* child_masks; // one byte per parent of the current level
    uint32_t* carve_sums[2]; // children of 1024 parents each, of even and of odd levels
    unsigned long long* tile_sums;
    // View skipping (binary masks only).  node_skip[k] has bit b set when view
    // b need not be evaluated for any descendant of node k: the box of node k
    // or of one of its ancestors, grown by two pixels, lies inside the image
    // and holds only ones, so every descendant is "object" there (and, in
    // partial mode, fully inside the frame).  child_skip holds the same masks
    // for the 8 children of each parent of the current level.
    // All masks have mask_words planes of 32 views each (plane w: views 32 w
    // to 32 w + 31); later views have no bit and are always evaluated.
    int mask_words;       // 1 or 2
    uint32_t* node_skip;  // [mask_words][node_cap]
    uint32_t* child_skip; // [mask_words][parent_cap * 8]
    // Out-of-frame views (partial mode): node_out[k] has bit b when node k's
    // box in view b lies more than 2 pixels outside the image (box_out); no
    // descendant's item in view b can change anything, so the item kernel
    // skips it and the children inherit the bit.  child_out: the same for
    // the 8 children of each parent of the current level.
    uint32_t* node_out;   // [mask_words][node_cap]
    uint32_t* child_out;  // [mask_words][parent_cap * 8]
    int64_t parent_cap;
    // carve kernel per parent level: 0 = views over lanes, 1 = (parent, view) items
    uint8_t carve_variant[kMaxLevel];
    const unsigned int* nonbinary; // set by the SAT pass when a mask value is not 0/1
    bool skip_ok;                  // exact integer SAT sums (H * W < 2^24)
    // All-ones footprints: bit x of word (b*H + y)*WW + x/32 is set when the
    // mask values of view b at (x, y), (x+1, y), (x, y+1) and (x+1, y+1) are
    // all exactly 1 (as floats).  A bilinear sample whose footprint is such a
    // 2x2 block is exactly 1 (lerp(1, 1, t) == 1 for every t in [0, 1.25],
    // checked exhaustively), so the field skips the four mask reads.
    bool field_ones;
    uint32_t* ones; // [B*H*WW]
    int64_t WW;
    // Field masks: the skip and out-of-frame views of the cells of the last
    // carve level (the parents of the leaves) hold for all their descendants,
    // so for every mesh corner that is one of their lattice points the field
    // factor of those views is exactly 1 (a footprint of four ones with
    // weights in [0, 1], or a point out of the frame).  cell_masks is a dense
    // table over the cells of level L-1, scattered before the field and
    // cleared after it (nullptr: no table, every pair is evaluated).
    uint32_t* cell_masks; // [mask_words][8^(L-1)]
    // corner grid: R^3 points, one bit each, rows of WR 64-bit words (x fastest)
    int64_t R, WR;
    uint64_t* bitmap;     // [R*R*WR]
    uint32_t* rowbits;    // [ceil(R*R/32)] touched-row flags
    // Touched rows, ascending, and the words of 32 points of those rows only:
    // word k = slot * wr + w holds the points x = 32 w.. of row rows[slot].
    uint32_t* block_rows; // touched rows of each block of rows_kernel, counted first (nullptr: by the blocks themselves)
    uint32_t* rows;       // [R*R]
    uint32_t* row_slot;   // [R*R] slot of a touched row (others: stale)
    RowPlace* row_place;  // [R*R] a slot's row and the rows around it
    uint2* row_cnt;       // [R*R] corners and words with a corner of a slot's row
    uint2* coarse;        // [R*R / 256 + 2] the same of 256 slots
    uint32_t wr;          // 2 * WR
    FastDiv div_wr, div_r; // by wr and by R
    int64_t word_cap;
    uint32_t* present;    // [word_cap] corner bits
    uint2* runs;          // [word_cap] word_runs of the corner bits
    uint32_t* rank;       // [word_cap] corners before the word
    uint32_t* sign;       // [word_cap] bits: field value below 0.5
    uint32_t* word_list;  // [word_cap] the words with a corner, ascending
    WordMesh mesh;
    // sparse field, by corner rank
    int64_t* corners;
    float* values;
    int64_t corner_cap;
    DevCounters* ctr;
    DevCounters* host_ctr; // mapped host memory the finished counters are written to
    const ReqConsts* rq; // corner, length and masks of the running request (device)
};

// Corner ids inside the pipeline: x | y << 21 | z << 42 (grid points < 2^21
// per axis).  Ascending packed ids are ascending ravelled ids x + y*R + z*R*R,
// and decoding needs shifts instead of 64-bit divisions by R.
__device__ __forceinline__ int64_t pack_corner(int64_t x, int64_t y, int64_t z)
{
    return x | (y << 21) | (z << 42);
}

__device__ __forceinline__ void unpack_corner(int64_t v, int64_t& x, int64_t& y, int64_t& z)
{
    x = v & 0x1FFFFF;
    y = (v >> 21) & 0x1FFFFF;
    z = v >> 42;
}

// Everything a request starts from, in one launch: its transforms as float32,
// its ReqConsts (host_rq: device address of mapped host memory), cleared
// counters, the root cell and (clear_flags) the 0/1 flag of its masks.
void launch_begin(const HullPlan& p, const void* tf, int tf_dtype, const ReqConsts* host_rq, unsigned int* flags, bool clear_flags, cudaStream_t s);
// Levels launch_top carves in one launch (the first levels of the octree).
int top_levels(int level);
void launch_top(const HullPlan& p, cudaStream_t s);
// Sparse field export: ravelled ids (x + y*R + z*R*R) and values.
void launch_export_field(const HullPlan& p, int64_t n, int64_t* indices, float* values, cudaStream_t s);
// The same with the indices of a sparse tensor: four rows of n (0, z, y, x).
void launch_export_field_coo(const HullPlan& p, int64_t n, int64_t* indices, float* values, cudaStream_t s);
void launch_carve_level(const HullPlan& p, int level_index, cudaStream_t s);
// The leaf list (level L) from the last level's child masks; the carve itself
// only counts the leaves.
void launch_emit_leaves(const HullPlan& p, cudaStream_t s);
void launch_corners(const HullPlan& p, cudaStream_t s);
// The part of launch_corners after the bitmap is set: touched rows, sorted
// unique corners and the rows' words.  Leaves the bitmap and the row flags
// clear for the next request.
void launch_rank_corners(const HullPlan& p, cudaStream_t s);

// Sets the 8 corner bits of a leaf cell (x, y, z) at resolution 2^L in a
// corner bitmap of R points per axis and WR words per row.
__device__ __forceinline__ void mark_cell_corners(uint64_t* bitmap, uint32_t* rowbits, int64_t R, int64_t WR,
                                                  int64_t x, int64_t y, int64_t z)
{
    const int b = static_cast<int>(x & 63);
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
        const int64_t row = (y + (q & 1)) + (z + (q >> 1)) * R;
        const int64_t w = row * WR + (x >> 6);
        const uint64_t bits0 = (b < 63) ? (3ull << b) : (1ull << 63);
        if ((bitmap[w] & bits0) != bits0)
            atomicOr(reinterpret_cast<unsigned long long*>(bitmap + w), static_cast<unsigned long long>(bits0));
        if (b == 63 && !(bitmap[w + 1] & 1ull))
            atomicOr(reinterpret_cast<unsigned long long*>(bitmap + w + 1), 1ull);
        const uint32_t rb = 1u << (row & 31);
        if (!(rowbits[row >> 5] & rb))
            atomicOr(rowbits + (row >> 5), rb);
    }
}
// Sets the corner bits of the refined children (child mask m) of a cell whose
// lattice starts at (x, y, z) at resolution 2^L: per lattice row (y + dy,
// z + dz) one OR of the x bits its children cover, instead of four words per
// child (neighbouring children share 27 of their 64 corners).  Most bits are
// set already by a neighbour: the nine words are read first, together, and
// only what is missing is written (a row whose bits are all set has its flag
// from whoever set them).
__device__ __forceinline__ void mark_children_corners(uint64_t* bitmap, uint32_t* rowbits, int64_t R, int64_t WR,
                                                      int64_t x, int64_t y, int64_t z, uint32_t m)
{
    const uint32_t wx = static_cast<uint32_t>(x >> 6);
    const int b = static_cast<int>(x & 63);
    uint32_t xb[9]; // lattice x bits 0..2 of the rows
    uint64_t have[9];
    uint64_t* const first = bitmap + (y + z * R) * WR + wx;
#pragma unroll
    for (int q = 0; q < 9; ++q)
    {
        const int dy = q % 3, dz = q / 3;
        xb[q] = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c)
        {
            const int cx = c & 1, cy = (c >> 1) & 1, cz = c >> 2;
            if ((dy == cy || dy == cy + 1) && (dz == cz || dz == cz + 1) && ((m >> c) & 1u))
                xb[q] |= 3u << cx;
        }
        have[q] = xb[q] ? __ldcg(first + (dy + dz * R) * WR) : 0ull;
    }
#pragma unroll
    for (int q = 0; q < 9; ++q)
    {
        const uint64_t lo = static_cast<uint64_t>(xb[q]) << b;
        const bool spill = b > 61 && (xb[q] >> (64 - b)) != 0; // into the next word
        if ((have[q] & lo) == lo && !spill)
            continue;
        const int64_t row = (y + q % 3) + (z + q / 3) * R;
        uint64_t* w = first + (q % 3 + q / 3 * R) * WR;
        if (lo)
            atomicOr(reinterpret_cast<unsigned long long*>(w), static_cast<unsigned long long>(lo));
        if (spill)
            atomicOr(reinterpret_cast<unsigned long long*>(w + 1), static_cast<unsigned long long>(xb[q] >> (64 - b)));
        const uint32_t rb = 1u << (row & 31);
        if (!(__ldcg(rowbits + (row >> 5)) & rb))
            atomicOr(rowbits + (row >> 5), rb);
    }
}

// mark_children_corners into a block's table of bitmap words (kMarkSlots
// entries, keys kNoWord when free): false when the table is full.
constexpr int kMarkSlots = 2048;

struct MarkTable
{
    uint32_t key[kMarkSlots]; // word of 32 points of the bitmap
    uint32_t bits[kMarkSlots];
};

__device__ __forceinline__ bool mark_word(MarkTable& t, uint32_t word, uint32_t bits)
{
    uint32_t slot = (word * 2654435761u) >> 21; // Knuth's multiplicative hash, 11 bits
    for (int k = 0; k < 64; ++k)
    {
        const uint32_t had = atomicCAS(&t.key[slot], kNoWord, word);
        if (had == kNoWord || had == word)
        {
            if ((*static_cast<volatile uint32_t*>(&t.bits[slot]) & bits) != bits)
                atomicOr(&t.bits[slot], bits);
            return true;
        }
        slot = (slot + 1) % kMarkSlots;
    }
    return false;
}

void launch_field(const HullPlan& p, cudaStream_t s);
void launch_marching_cubes(const HullPlan& p, cudaStream_t s);
// words: the request's DevCounters::words (read back with the counts).
void launch_export(const HullPlan& p, int64_t words, float* verts, int64_t* faces, cudaStream_t s);

} // namespace th
