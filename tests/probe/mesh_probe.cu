// Test-only probe of the mesh stages (mesh.cu) at sizes that no test scene reaches.
#include "../../torchhull_gb300/csrc/mesh.cu"

namespace th
{

void note_launches(int) {}

void check_launch(const char*) {}

int sm_count()
{
    return 148;
}

int grid_for(int64_t work_items, int threads)
{
    const int64_t blocks = (work_items + threads - 1) / threads;
    return static_cast<int>(blocks < 1 ? 1 : (blocks < 8 * 148 ? blocks : 8 * 148));
}

} // namespace th

using namespace th;

// Corners of a bitmap of level `level` whose touched rows are flagged; no room
// for words.  Returns a CUDA error; result: overflow bits, corners.
extern "C" int corners_probe(int level, uint64_t* bitmap, uint32_t* rowbits, uint32_t* rows, uint32_t* row_slot, RowPlace* row_place, uint2* row_cnt, int64_t* corners, int64_t corner_cap, void* counters, int64_t* result)
{
    HullPlan p{};
    p.level = level;
    p.R = (int64_t{ 1 } << level) + 1;
    p.WR = (p.R + 63) / 64;
    p.wr = static_cast<uint32_t>(2 * p.WR);
    p.div_wr = make_fastdiv(p.wr);
    p.div_r = make_fastdiv(static_cast<uint32_t>(p.R));
    p.node_cap = p.parent_cap = int64_t{ 1 } << 40;
    p.bitmap = bitmap;
    p.rowbits = rowbits;
    p.rows = rows;
    p.row_slot = row_slot;
    p.row_place = row_place;
    p.row_cnt = row_cnt;
    p.corners = corners;
    p.corner_cap = corner_cap;
    p.ctr = static_cast<DevCounters*>(counters);
    p.coarse = reinterpret_cast<uint2*>(p.ctr + 1);
    launch_rank_corners(p, nullptr);
    DevCounters c;
    const cudaError_t e = cudaMemcpy(&c, p.ctr, sizeof(c), cudaMemcpyDeviceToHost);
    result[0] = c.overflow;
    result[1] = c.corners;
    return e;
}

extern "C" int64_t counters_bytes(int level)
{
    const int64_t R = (int64_t{ 1 } << level) + 1;
    return sizeof(DevCounters) + sizeof(uint2) * (R * R / 256 + 2);
}

namespace th
{
namespace
{

// n words around which every cell has four triangles (the corners of a cell
// lie on alternating sides) but the last of a word, and no vertices.
struct Checkers
{
    int64_t n;
    __device__ int64_t words() const { return n; }
    __device__ int64_t counted() const { return 0; }
    __device__ uint32_t word(uint32_t i) const { return i; }
    __device__ bool empty(uint32_t) const { return false; }
    __device__ uint32_t sign(uint32_t i) const { return (i & 3u) == 0 || (i & 3u) == 3 ? 0x55555555u : 0xaaaaaaaau; }
    __device__ WordRows rows(uint32_t k) const { return WordRows{ { 4 * k, 4 * k + 1, 4 * k + 2, 4 * k + 3 }, false }; }
    __device__ EdgeBits edges(uint32_t, const WordRows&, const uint32_t*, const uint32_t*, uint32_t& cells) const
    {
        cells = 0x7fffffffu;
        return EdgeBits{ 0u, 0u, 0u };
    }
};

} // namespace
} // namespace th

// Triangle corners of such words; result: overflow bits, corners.
extern "C" int triangles_probe(int64_t words, uint32_t* cnt, uint32_t* cells, unsigned long long* tiles, void* counters, int64_t* result)
{
    DevCounters* ctr = static_cast<DevCounters*>(counters);
    const WordMesh mesh{ cnt, cells, nullptr, nullptr, tiles, nullptr };
    words_count_kernel<Checkers, true><<<words_grid(words), kWordThreads>>>(Checkers{ words }, mesh, &ctr->scan, nullptr, MeshTotal{ ctr, ctr + 1 });
    DevCounters c;
    const cudaError_t e = cudaMemcpy(&c, ctr + 1, sizeof(c), cudaMemcpyDeviceToHost);
    result[0] = c.overflow;
    result[1] = c.soup;
    return e;
}
