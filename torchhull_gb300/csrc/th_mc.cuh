// Device-side plan of one public marching-cubes request and the launch entry
// points of its two phases (mc.cu).
#pragma once

#include <cstdint>

#include "th_common.cuh"
#include "th_words.cuh"

namespace th
{

enum McFlags : unsigned int
{
    kMcBadIndex = 1, // a sparse index outside the volume (or a batch index other than 0)
    kMcUnsorted = 2, // sparse indices not strictly ascending (not a coalesced tensor)
};

struct McCounters
{
    unsigned long long soup;   // soup vertices, 3 per face
    unsigned long long verts;  // unique vertices
    unsigned long long active; // active cells (dense volumes)
    unsigned int flags;       // McFlags
    unsigned int pad;
    ScanState scan_soup;
    ScanState scan_verts;
};

struct McPlan
{
    int dtype; // TH_FLOAT16, TH_FLOAT32 or TH_FLOAT64
    bool sparse, unique, local;
    int64_t D, H, W;       // volume sizes along z, y, x
    float iso;
    float scale[3];        // 2 / (size - 1) along x, y, z
    const void* volume;    // dense: [D, H, W], x fastest
    const int64_t* indices; // sparse: [4, nnz] rows (0, z, y, x)
    const void* values;     // sparse: [nnz]
    int64_t nnz;
    // Bit words (th_words.cuh): rows of wr words, one bit per grid point; dense
    // volumes, and sparse ones whose words are few enough for their entries.
    bool words;
    int64_t nwords;
    // A dense volume that would need too much scratch goes slab by slab of
    // `slab` planes, through the same kernels: a plan of a slab (dense_slab) has the
    // volume and D of its planes, z0 its first plane, and `own` words that are
    // no halo.  The slab's numbering goes on from mesh.start.
    int64_t slab, z0, own;
    uint32_t wr;
    FastDiv div_wr, div_h;    // by wr and by H
    uint32_t* sign;           // bit: below the isolevel
    uint32_t* present;        // sparse: bit: the volume has an entry
    uint32_t* rank;           // sparse: first entry of a word that has any
    WordMesh mesh;
    // sparse volumes with few entries for their size
    unsigned long long* keys; // open-addressing table of ravel ids
    int32_t* slots;           // entry index of each key
    uint64_t hmask;           // table capacity - 1 (a power of two minus one)
    uint8_t* codes;           // cell code of each entry; 0: no cell
    uint32_t* used;           // unique: vertex edge bits of each entry
    unsigned long long* vbase; // unique: first vertex of each entry
    unsigned long long* tiles_soup;
    unsigned long long* tiles_verts;
    McCounters* ctr;
};

// Scan tiles a scan over n items needs.
inline int64_t mc_scan_tiles(int64_t n)
{
    return (n + kScanTile - 1) / kScanTile;
}

// Slab `z0` of the dense volume of plan p: its own planes, and behind them the
// one whose vertices its last cells use, with the one that gives those their
// z edges.
McPlan dense_slab(const McPlan& p, int64_t z0);
// Phase 1: the soup and vertex counts (ctr) and the vertex numbering.
void launch_mc_count(const McPlan& p, cudaStream_t s);
// Phase 2: vertices [verts, 3] and faces [soup / 3, 3] into caller buffers.
void launch_mc_emit(const McPlan& p, float* verts, int64_t* faces, cudaStream_t s);

} // namespace th
