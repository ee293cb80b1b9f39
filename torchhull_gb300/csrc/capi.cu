// C ABI: contexts with resident device pools, request orchestration and
// argument validation with the reference's error behaviour.
//
// One request enqueues every stage on the caller's stream and reads back one
// small counter block at the end (the reference synchronises after every
// kernel and reads counts back per level, visual_hull_cuda.cu:742, :820 and
// marching_cubes_cuda.cu:600-634).  Pools only grow: a request whose octree or
// corner set outgrows them is detected on the device, the pools grow fourfold
// and the request runs again, so repeated requests of similar size never allocate.

#include <algorithm>
#include <array>
#include <atomic>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include <sstream>

#include "th_classify.cuh"
#include "th_hull.cuh"
#include "th_internal.h"
#include "th_mc.cuh"

namespace th
{

namespace
{
std::atomic<int64_t> g_launches{ 0 };
}

// Kernels enqueued while this thread captures a graph are counted when the
// graph is replayed, not when captured.
thread_local bool t_capturing = false;
thread_local int64_t t_captured = 0;

void note_launches(int n)
{
    if (t_capturing)
        t_captured += n;
    else
        g_launches.fetch_add(n, std::memory_order_relaxed);
}

void check_launch(const char* what)
{
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        throw CudaError{ e, std::string("kernel launch: ") + what };
}

int sm_count()
{
    static int cache[64] = { 0 };
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
        return 148;
    if (cache[dev] == 0)
    {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
            n = 148;
        cache[dev] = n;
    }
    return cache[dev];
}

namespace
{

// Small host <-> device transfers (request constants in, counters out) run
// as a one-block kernel over mapped pinned host memory instead of
// cudaMemcpyAsync: a copy engine may be busy with a caller's bulk copy on
// another stream (a previous mesh going out, the next request's masks coming
// in), and a small copy queued behind it would stall the whole pipeline.
__global__ void small_copy_kernel(const unsigned char* __restrict__ src, unsigned char* __restrict__ dst, int64_t n)
{
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
        dst[i] = src[i];
    __threadfence_system();
}

__global__ void zero_kernel(unsigned char* __restrict__ p, int64_t n)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        p[i] = 0;
}

// dst and src are device addresses (device memory, or mapped host memory's device address).
void small_copy(void* dst, const void* src, size_t bytes, cudaStream_t st)
{
    small_copy_kernel<<<1, 256, 0, st>>>(static_cast<const unsigned char*>(src), static_cast<unsigned char*>(dst),
                                          static_cast<int64_t>(bytes));
    TH_LAUNCH_CHECK();
}

// Pinned host memory for count objects of T, mapped into the device's address space.
template <typename T>
void alloc_mapped(T** host, T** dev, size_t count = 1)
{
    void* h = nullptr;
    TH_CUDA(cudaHostAlloc(&h, sizeof(T) * count, cudaHostAllocMapped));
    void* d = nullptr;
    const cudaError_t e = cudaHostGetDevicePointer(&d, h, 0);
    if (e != cudaSuccess)
    {
        cudaFreeHost(h);
        throw CudaError{ e, "cudaHostGetDevicePointer" };
    }
    *host = static_cast<T*>(h);
    *dev = static_cast<T*>(d);
}

}  // namespace

void launch_zero(void* p, size_t bytes, cudaStream_t s)
{
    if (bytes == 0)
        return;
    const int64_t n = static_cast<int64_t>(bytes);
    const unsigned grid = static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, 64));
    zero_kernel<<<grid, 256, 0, s>>>(static_cast<unsigned char*>(p), n);
    TH_LAUNCH_CHECK();
}

namespace
{

struct DevBuf
{
    void* p = nullptr;
    size_t bytes = 0;

    // Returns true when fresh memory was allocated (contents undefined).  What
    // uses the memory it replaces must be queued on st, or on a stream that st
    // waits for: a batch's requests share the pool of their stream, and one that
    // needs more is prepared while those before it still run.
    bool ensure(size_t need, cudaStream_t st)
    {
        if (need <= bytes && p)
            return false;
        if (p)
        {
            TH_CUDA(cudaStreamSynchronize(st));
            TH_CUDA(cudaFree(p));
        }
        p = nullptr;
        bytes = 0;
        size_t sz = std::max<size_t>(need, 256);
        TH_CUDA(cudaMalloc(&p, sz));
        bytes = sz;
        return true;
    }
    void release()
    {
        if (p)
            cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    template <typename T>
    T* as() const
    {
        return static_cast<T*>(p);
    }
};

struct ArgError
{
    th_status status;
    std::string msg;
};

const char* dtype_name(int d)
{
    static const char* names[] = { "Bool", "Byte", "Char", "Short", "Int", "Long", "Half", "Float", "Double", "BFloat16" };
    return (d >= 0 && d <= 9) ? names[d] : "Unknown";
}

bool is_image_dtype(int d)
{
    return d >= TH_UINT8 && d <= TH_FLOAT64;
}

// What a request needs while it runs and not afterwards: the octree, the corner
// bitmap and the field's cell-mask table (both clear between requests), sums.
// The requests of a batch that follow each other on a stream share one.
struct WorkPool
{
    DevBuf nodes, node_skip, node_out, child_masks, child_skip, child_out, carve_sums, tile_sums, cell_masks, bitmap, rowbits;
    int64_t node_cap = 0, parent_cap = 0;
    bool unfinished = false; // a run was cut short: the bitmaps and the cell masks may hold bits

    std::vector<const DevBuf*> buffers() const
    {
        return { &nodes, &node_skip, &node_out, &child_masks, &child_skip, &child_out, &carve_sums, &tile_sums, &cell_masks,
                 &bitmap, &rowbits };
    }
    void release()
    {
        for (const DevBuf* b : buffers())
            const_cast<DevBuf*>(b)->release();
    }
};

// Pools and the state of the last request of one context.
struct HullSlot
{
    WorkPool work; // plain requests; a batch's slots use its streams' pools
    DevBuf tf, sat, ones, rows, row_slot, row_cnt, row_place, present, runs, word_list, rank, sign, word_cnt, word_cells, word_edges,
            word_chunk, corners, values, counters, flags, sat_scratch;
    int64_t corner_cap = 0, word_cap = 0;
    HullPlan plan{};
    DevCounters* host = nullptr; // pinned, mapped copy of the counters
    DevCounters* host_d = nullptr; // its device address
    DevBuf rq;                   // ReqConsts of the running request (device)
    ReqConsts* host_rq = nullptr; // pinned, mapped source of rq
    ReqConsts* host_rq_d = nullptr; // its device address
    th_hull_info info{};
    bool has_result = false;
    cudaEvent_t done = nullptr; // the last export that read the buffers
    bool exported = false;      // one was queued since the last request waited for it

    // Captured pipelines, keyed by the plan with the per-request fields cleared.
    struct Graph
    {
        HullPlan key;
        cudaGraphExec_t exec = nullptr;
        int64_t kernels = 0;
    };
    std::vector<Graph> graphs;
    cudaStream_t capture_stream = nullptr; // capture only (graphs launch on the caller's stream)

    void drop_graphs()
    {
        for (auto& g : graphs)
            if (g.exec)
                cudaGraphExecDestroy(g.exec);
        graphs.clear();
    }

    std::vector<const DevBuf*> buffers() const
    {
        std::vector<const DevBuf*> all = { &tf, &sat, &ones, &rows, &row_slot, &row_cnt, &row_place, &present, &runs, &word_list,
                                           &rank, &sign, &word_cnt, &word_cells, &word_edges, &word_chunk, &corners, &values,
                                           &counters, &flags, &sat_scratch, &rq };
        for (const DevBuf* b : work.buffers())
            all.push_back(b);
        return all;
    }

    void release()
    {
        drop_graphs();
        for (const DevBuf* b : buffers())
            const_cast<DevBuf*>(b)->release();
        if (host)
            cudaFreeHost(host);
        host = nullptr;
        host_d = nullptr;
        if (host_rq)
            cudaFreeHost(host_rq);
        host_rq = nullptr;
        host_rq_d = nullptr;
        if (capture_stream)
            cudaStreamDestroy(capture_stream);
        capture_stream = nullptr;
        if (done)
            cudaEventDestroy(done);
        done = nullptr;
    }
};

} // namespace
} // namespace th

namespace th
{
namespace
{

// CUDA events between the stages of one request (th_context_set_profiling).
struct StageEvents
{
    static constexpr int kCount = TH_MAX_LEVEL + 6;
    cudaEvent_t ev[kCount] = {};
    bool ready = false;

    void create()
    {
        if (ready)
            return;
        for (auto& e : ev)
            TH_CUDA(cudaEventCreate(&e));
        ready = true;
    }
    void destroy()
    {
        if (!ready)
            return;
        for (auto& e : ev)
            cudaEventDestroy(e);
        ready = false;
    }
    void record(int i, cudaStream_t s)
    {
        TH_CUDA(cudaEventRecord(ev[i], s));
    }
    float between(int a, int b) const
    {
        float ms = 0.f;
        TH_CUDA(cudaEventElapsedTime(&ms, ev[a], ev[b]));
        return ms;
    }
};

} // namespace
} // namespace th

namespace th
{
namespace
{

// Request signature for the carve-kernel autotuner.
using TuneKey = std::array<int64_t, 8>;
using CarveVariants = std::array<uint8_t, kMaxLevel>;

TuneKey tune_key(const th_hull_args* a)
{
    return { a->batch, a->height, a->width, a->level, a->masks_partial, a->transforms_opengl, a->masks_dtype, 0 };
}

CarveVariants views_everywhere()
{
    CarveVariants v{};
    return v;
}

// Work items from level 4 on (levels below have at most 8^3 parents).
CarveVariants items_from_level4()
{
    CarveVariants v{};
    for (int i = 4; i < kMaxLevel; ++i)
        v[i] = 1;
    return v;
}

} // namespace
} // namespace th

namespace th
{
namespace
{

// Shared state of the batched form: the streams its requests run on, with a
// work pool each.
struct BatchState
{
    std::vector<WorkPool> pools;
    std::vector<cudaStream_t> streams;
    std::vector<cudaEvent_t> joins;
    cudaEvent_t fork = nullptr;

    void release()
    {
        for (auto& w : pools)
            w.release();
        for (auto s : streams)
            cudaStreamDestroy(s);
        for (auto e : joins)
            cudaEventDestroy(e);
        if (fork)
            cudaEventDestroy(fork);
        pools.clear();
        streams.clear();
        joins.clear();
        fork = nullptr;
    }
};

} // namespace
} // namespace th

namespace th
{
namespace
{

// Pools and the last result of the public marching cubes.
struct McSlot
{
    DevBuf bits, rank, edges, cnt, cells, chunk, start, keys, slots, codes, used, vbase, tiles_soup, tiles_verts, ctr;
    McCounters* host = nullptr; // pinned, mapped copy of the counters
    McCounters* host_d = nullptr; // its device address
    McPlan plan{};
    th_mc_info info{};
    bool has_result = false;
    cudaEvent_t done = nullptr; // the last export that read the buffers
    bool exported = false;      // one was queued since the last call waited for it

    std::vector<const DevBuf*> buffers() const
    {
        return { &bits, &rank, &edges, &cnt, &cells, &chunk, &start, &keys, &slots, &codes, &used, &vbase, &tiles_soup,
                 &tiles_verts, &ctr };
    }

    void release()
    {
        for (const DevBuf* b : buffers())
            const_cast<DevBuf*>(b)->release();
        if (host)
            cudaFreeHost(host);
        host = nullptr;
        if (done)
            cudaEventDestroy(done);
        done = nullptr;
    }
};

} // namespace
} // namespace th

namespace th
{
namespace
{

bool in_capture(cudaStream_t st)
{
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    TH_CUDA(cudaStreamIsCapturing(st, &status));
    return status != cudaStreamCaptureStatusNone;
}

// Runs launch(), the kernels of an export of slot s on st, and records s.done
// behind them for the next request.  Exports of one result may be on several streams: each
// waits for the one before, as some use scratch (the leaf list, the words of a
// volume in slabs), and so the last event stands for them all.  An export
// recorded into a caller's graph is not ordered here: its event could not be
// waited on outside the graph.
template <class Slot, class F>
void export_on(Slot& s, cudaStream_t st, F&& launch)
{
    if (in_capture(st))
        return launch();
    if (s.exported)
        TH_CUDA(cudaStreamWaitEvent(st, s.done, 0));
    s.exported = true;
    try
    {
        launch();
    }
    catch (...)
    {
        cudaEventRecord(s.done, st); // what is queued
        throw;
    }
    TH_CUDA(cudaEventRecord(s.done, st));
}

// Scratch of the calls that a caller records into a graph.  The graph's
// kernels keep the addresses they were recorded with, for as long as the graph
// or anything instantiated from it lives, and run in no order with the calls
// outside it.  So each recorded call has a block of its own, which the graph
// holds through a CUDA user object; when that is gone, the block is for the
// next recording.  Blocks have power-of-two sizes and are freed with the
// context: there are as many as were held at one time.
class GraphScratch
{
public:
    // A block of at least `bytes`, held by the graph that st is capturing.
    void* take(cudaStream_t st, size_t bytes)
    {
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        cudaGraph_t graph = nullptr;
        TH_CUDA(cudaStreamGetCaptureInfo(st, &status, nullptr, &graph));
        if (status != cudaStreamCaptureStatusActive)
            throw CudaError{ cudaErrorStreamCaptureInvalidated, "scratch of a recorded call" };
        size_t size = 256;
        while (size < bytes)
            size *= 2;
        void* p = nullptr;
        {
            std::lock_guard<std::mutex> g(blocks_->lock);
            for (Block& b : blocks_->all)
            {
                if (!b.held && b.size == size)
                {
                    b.held = true;
                    p = b.p;
                    break;
                }
            }
        }
        if (!p)
        {
            // an allocation is no part of the graph: allowed in the relaxed mode
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            TH_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
            const cudaError_t e = cudaMalloc(&p, size);
            cudaThreadExchangeStreamCaptureMode(&mode);
            TH_CUDA(e);
            std::lock_guard<std::mutex> g(blocks_->lock);
            blocks_->all.push_back(Block{ p, size, true });
        }
        Lease* lease = new Lease{ blocks_, p };
        cudaUserObject_t held = nullptr;
        const cudaError_t e = cudaUserObjectCreate(&held, lease, &GraphScratch::end, 1, cudaUserObjectNoDestructorSync);
        if (e != cudaSuccess)
        {
            end(lease);
            throw CudaError{ e, "cudaUserObjectCreate" };
        }
        const cudaError_t r = cudaGraphRetainUserObject(graph, held, 1, cudaGraphUserObjectMove);
        if (r != cudaSuccess)
        {
            cudaUserObjectRelease(held, 1);
            throw CudaError{ r, "cudaGraphRetainUserObject" };
        }
        return p;
    }
    int64_t bytes() const
    {
        std::lock_guard<std::mutex> g(blocks_->lock);
        int64_t total = 0;
        for (const Block& b : blocks_->all)
            total += static_cast<int64_t>(b.size);
        return total;
    }
    // Frees all blocks: graphs recorded with the context are not replayed after it.
    void release()
    {
        std::lock_guard<std::mutex> g(blocks_->lock);
        for (Block& b : blocks_->all)
            cudaFree(b.p);
        blocks_->all.clear();
    }

private:
    struct Block
    {
        void* p;
        size_t size;
        bool held;
    };
    struct Blocks
    {
        std::mutex lock;
        std::vector<Block> all;
    };
    struct Lease
    {
        std::shared_ptr<Blocks> blocks; // a graph may outlive the context
        void* p;
    };
    static void CUDART_CB end(void* data)
    {
        std::unique_ptr<Lease> lease(static_cast<Lease*>(data));
        std::lock_guard<std::mutex> g(lease->blocks->lock);
        for (Block& b : lease->blocks->all)
            if (b.p == lease->p)
                b.held = false;
    }

    std::shared_ptr<Blocks> blocks_ = std::make_shared<Blocks>();
};

} // namespace
} // namespace th

struct th_context
{
    int device = 0;
    std::string error;
    th::HullSlot hull;
    std::vector<th::HullSlot> batch;
    th::BatchState bstate;
    th::DevBuf blur_scratch;
    th::DevBuf blurred; // masks blurred by th_visual_hull_blurred
    cudaEvent_t blur_done = nullptr; // the last blur that used blur_scratch
    th::DevBuf sat_aux; // th_integral_image: its 0/1 flag word, then the bit passes' scratch
    cudaEvent_t sat_aux_done = nullptr; // the last th_integral_image that used sat_aux
    th::GraphScratch graph_scratch; // the same for blurs and integral images recorded into a caller's graph
    th::McSlot mc;
    bool profiling = false;
    th::StageEvents events;
    th_stage_times times{};
    int carve_mode = 0; // TH_OPTION_CARVE_KERNEL
    bool graphs = true;  // TH_OPTION_GRAPHS
    bool batch_route = false; // TH_OPTION_BATCH_ROUTE
    bool field_ones = true;   // TH_OPTION_FIELD_ONES
    bool field_masks = true;  // TH_OPTION_FIELD_MASKS
    bool sat_single_pass = true; // TH_OPTION_SAT_SINGLE_PASS
    std::map<th::TuneKey, th::CarveVariants> carve_tuned;
    cudaEvent_t tune_ev[2] = { nullptr, nullptr };
};

namespace th
{
namespace
{

int64_t pool_bytes(const th_context* ctx)
{
    auto sum = [](const HullSlot& s) {
        int64_t b = 0;
        for (const DevBuf* d : s.buffers())
            b += static_cast<int64_t>(d->bytes);
        return b;
    };
    int64_t total = sum(ctx->hull) + static_cast<int64_t>(ctx->blur_scratch.bytes) +
                    static_cast<int64_t>(ctx->blurred.bytes) + static_cast<int64_t>(ctx->sat_aux.bytes) +
                    ctx->graph_scratch.bytes();
    for (const DevBuf* d : ctx->mc.buffers())
        total += static_cast<int64_t>(d->bytes);
    for (const auto& s : ctx->batch)
        total += sum(s);
    for (const auto& w : ctx->bstate.pools)
        for (const DevBuf* d : w.buffers())
            total += static_cast<int64_t>(d->bytes);
    return total;
}

void validate(const th_hull_args* a)
{
    if (!a)
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "args is NULL" };
    // visual_hull_cuda.cu:591-613
    if (a->batch < 0 || a->height < 0 || a->width < 0)
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "Check failed: masks sizes must be non-negative" };
    if (a->level < 0)
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "Check failed: level >= 0 (" + std::to_string(a->level) + " vs. 0)" };
    if (a->level > TH_MAX_LEVEL)
        throw ArgError{ TH_ERR_INVALID_ARGUMENT,
                        "level " + std::to_string(a->level) + " exceeds the supported maximum " +
                                std::to_string(TH_MAX_LEVEL) };
    if (!(a->cube_length > 0.f))
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "Check failed: cube_length > 0.f" };
    // AT_DISPATCH_FLOATING_TYPES_AND_HALF over transforms (:646) and
    // AT_DISPATCH_ALL_TYPES_AND(Half) over masks (:832)
    if (!(a->transforms_dtype == TH_FLOAT16 || a->transforms_dtype == TH_FLOAT32 || a->transforms_dtype == TH_FLOAT64))
        throw ArgError{ TH_ERR_UNSUPPORTED_DTYPE,
                        std::string("\"classify_children\" not implemented for '") + dtype_name(a->transforms_dtype) +
                                "'" };
    if (!is_image_dtype(a->masks_dtype))
        throw ArgError{ TH_ERR_UNSUPPORTED_DTYPE,
                        std::string("\"accumulate_hull_counts\" not implemented for '") + dtype_name(a->masks_dtype) +
                                "'" };
    if (a->batch * a->height * a->width > 0 && (!a->masks || !a->transforms))
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "masks or transforms pointer is NULL" };
    // Flagged/Unique/stdgpu use 32-bit indices (visual_hull_cuda.cu:716, :798)
    if (a->batch * a->height * a->width >= (int64_t{ 1 } << 40))
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "masks too large" };
    // pixel indices are carried exactly in float mantissas by the carve
    if (a->height >= (int64_t{ 1 } << 23) || a->width >= (int64_t{ 1 } << 23))
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "mask height and width must be below 2^23" };
}

int64_t max_nodes(int level)
{
    // sum over levels of 8^i, the most the octree can hold
    int64_t s = 0;
    for (int i = 0; i <= level && i <= 12; ++i)
        s += int64_t{ 1 } << (3 * i);
    return s;
}

// Bytes of the counters and the row groups' corner counts (HullPlan::coarse).
size_t counter_bytes(int64_t R)
{
    return sizeof(DevCounters) + sizeof(uint2) * static_cast<size_t>(R * R / 256 + 2);
}

// Sizes the pools of slot s for request a and fills its plan.
// Work happens in pool w.  batch_slot: one of many, which starts smaller.
void prepare(HullSlot& s, WorkPool& w, const th_hull_args* a, cudaStream_t st, bool field_ones, bool field_masks, bool batch_slot = false)
{
    const int L = a->level;
    const int64_t B = a->batch, H = a->height, W = a->width;
    const int64_t R = (int64_t{ 1 } << L) + 1;
    const int64_t WR = (R + 63) / 64;
    // Every request starts from at least the capacity its level could need up
    // to 16 M nodes and corners (about 0.5 GB; a level-9 hull of 32 megapixel
    // views fits without a rerun), whatever smaller requests the context
    // served before; beyond that the pools grow x4 per rerun.  Batch slots
    // start at 4 M corners.
    w.node_cap = std::max<int64_t>(w.node_cap, std::min<int64_t>(max_nodes(L), int64_t{ 1 } << 24));
    w.parent_cap = std::max<int64_t>(w.parent_cap, std::min<int64_t>(max_nodes(L), int64_t{ 1 } << 22));
    s.corner_cap = std::max<int64_t>(s.corner_cap, std::min<int64_t>(R * R * R, int64_t{ 1 } << (batch_slot ? 22 : 24)));
    const int64_t node_cap = std::min<int64_t>(w.node_cap, max_nodes(L));
    const int64_t corner_cap = std::min<int64_t>(s.corner_cap, R * R * R);
    const int64_t parent_cap = std::min<int64_t>(w.parent_cap, node_cap);
    // words of 32 points of the touched rows: all rows up to 32 M words (level
    // 9: 4.7 M), more on demand; a batch slot starts at 8 M
    const int64_t all_words = R * R * 2 * WR;
    s.word_cap = std::max<int64_t>(s.word_cap, std::min<int64_t>(all_words, int64_t{ 1 } << (batch_slot ? 23 : 25)));
    const int64_t word_cap = std::min<int64_t>(s.word_cap, all_words);
    const int mask_words = mask_words_for(B);

    s.tf.ensure(sizeof(float) * std::max<int64_t>(B, 1) * 16, st);
    s.sat.ensure(sizeof(float) * std::max<int64_t>(B * H * W, 1), st);
    const int64_t sat_scratch = sat_scratch_bytes(B, H, W, a->masks_dtype);
    if (sat_scratch > 0)
        s.sat_scratch.ensure(static_cast<size_t>(sat_scratch), st);
    const int64_t WW = (W + 31) / 32;
    // the field's cell-mask table of level L-1 (up to 2^27 cells, 512 MB:
    // level 10) skips most pairs; the all-ones bitmap only pays without it
    const bool cell_masks = field_masks && L >= 1 && 3 * (L - 1) <= 27 &&
                            (a->masks_partial != 0 || (B > 0 && H > 0 && W > 0 && H * W <= (int64_t{ 1 } << 23)));
    field_ones = field_ones && !cell_masks;
    if (field_ones)
        s.ones.ensure(sizeof(uint32_t) * std::max<int64_t>(B * H * WW, 1), st);
    w.nodes.ensure(sizeof(int64_t) * node_cap, st);
    w.node_skip.ensure(sizeof(uint32_t) * mask_words * node_cap, st);
    w.node_out.ensure(sizeof(uint32_t) * mask_words * node_cap, st);
    w.child_masks.ensure(node_cap, st);
    w.child_skip.ensure(sizeof(uint32_t) * 8 * mask_words * parent_cap, st);
    w.child_out.ensure(sizeof(uint32_t) * 8 * mask_words * parent_cap, st);
    s.flags.ensure(sizeof(unsigned int) * 4, st);
    const int64_t rwords = (R * R + 31) / 32;
    const int64_t row_blocks = (rwords + kRowBlock - 1) / kRowBlock;
    w.tile_sums.ensure(sizeof(unsigned long long) *
                       std::max<int64_t>({ (node_cap + kScanTile - 1) / kScanTile, word_tiles(word_cap), row_blocks }), st);
    w.carve_sums.ensure(2 * sizeof(uint32_t) * (node_cap / 1024 + 4), st);
    const int64_t words = R * R * WR;
    if (w.bitmap.ensure(sizeof(uint64_t) * words, st))
        TH_CUDA(cudaMemsetAsync(w.bitmap.p, 0, w.bitmap.bytes, st));
    if (w.rowbits.ensure(sizeof(uint32_t) * rwords, st))
        TH_CUDA(cudaMemsetAsync(w.rowbits.p, 0, w.rowbits.bytes, st));
    if (w.unfinished)
    {
        for (const DevBuf* b : { &w.bitmap, &w.rowbits, &w.cell_masks })
            if (b->p)
                TH_CUDA(cudaMemsetAsync(b->p, 0, b->bytes, st));
        w.unfinished = false;
    }
    s.rows.ensure(sizeof(uint32_t) * R * R, st);
    s.row_slot.ensure(sizeof(uint32_t) * R * R, st);
    s.row_cnt.ensure(sizeof(uint2) * R * R, st);
    s.row_place.ensure(sizeof(RowPlace) * R * R, st);
    s.present.ensure(sizeof(uint32_t) * word_cap, st);
    s.word_list.ensure(sizeof(uint32_t) * word_cap, st);
    s.runs.ensure(sizeof(uint2) * word_cap, st);
    s.rank.ensure(sizeof(uint32_t) * word_cap, st);
    s.sign.ensure(sizeof(uint32_t) * word_cap, st);
    s.word_cnt.ensure(sizeof(uint32_t) * word_cap, st);
    s.word_cells.ensure(sizeof(uint32_t) * word_cap, st);
    s.word_edges.ensure(sizeof(uint4) * word_cap, st);
    s.word_chunk.ensure(sizeof(uint2) * ((word_cap + 31) / 32), st);
    s.corners.ensure(sizeof(int64_t) * corner_cap, st);
    s.values.ensure(sizeof(float) * corner_cap, st);
    // the counters and, behind them, the corners of 256 rows each: cleared together
    s.counters.ensure(counter_bytes(R), st);
    if (!s.host)
        alloc_mapped(&s.host, &s.host_d);
    if (!s.done)
        TH_CUDA(cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming));

    HullPlan& p = s.plan;
    std::memset(&p, 0, sizeof(HullPlan)); // zero padding too: plans are compared bytewise
    p.masks = a->masks;
    p.masks_dtype = a->masks_dtype;
    p.B = B;
    p.H = H;
    p.W = W;
    p.tf = s.tf.as<float>();
    p.sat = s.sat.as<float>();
    p.opengl = a->transforms_opengl != 0;
    p.partial = a->masks_partial != 0;
    p.unique = a->unique_verts != 0;
    p.corner[0] = a->cube_corner_bfl[0];
    p.corner[1] = a->cube_corner_bfl[1];
    p.corner[2] = a->cube_corner_bfl[2];
    p.length = a->cube_length;
    p.level = L;
    p.mark_apart = L >= kMarkApartLevel;
    p.sms = sm_count();
    p.nodes = w.nodes.as<int64_t>();
    p.node_cap = node_cap;
    p.child_masks = w.child_masks.as<uint8_t>();
    p.tile_sums = w.tile_sums.as<unsigned long long>();
    p.carve_sums[0] = w.carve_sums.as<uint32_t>();
    p.carve_sums[1] = p.carve_sums[0] + node_cap / 1024 + 4;
    p.mask_words = mask_words;
    p.node_skip = w.node_skip.as<uint32_t>();
    p.child_skip = w.child_skip.as<uint32_t>();
    p.node_out = w.node_out.as<uint32_t>();
    p.child_out = w.child_out.as<uint32_t>();
    p.parent_cap = parent_cap;
    p.nonbinary = s.flags.as<unsigned int>();
    // exact integer box sums need every SAT sum of two entries below 2^24
    p.skip_ok = B > 0 && H > 0 && W > 0 && H * W <= (int64_t{ 1 } << 23);
    p.field_ones = field_ones && B > 0 && H > 0 && W > 0;
    p.cell_masks = nullptr;
    if (cell_masks)
    {
        if (w.cell_masks.ensure(sizeof(uint32_t) * mask_words * (int64_t{ 1 } << (3 * (L - 1))), st))
            TH_CUDA(cudaMemsetAsync(w.cell_masks.p, 0, w.cell_masks.bytes, st));
        p.cell_masks = w.cell_masks.as<uint32_t>();
    }
    p.ones = field_ones ? s.ones.as<uint32_t>() : nullptr;
    p.WW = WW;
    p.R = R;
    p.WR = WR;
    p.bitmap = w.bitmap.as<uint64_t>();
    p.rowbits = w.rowbits.as<uint32_t>();
    p.block_rows = row_blocks >= kCountRowBlocks ? w.tile_sums.as<uint32_t>() : nullptr; // free until the mesh passes
    p.rows = s.rows.as<uint32_t>();
    p.row_slot = s.row_slot.as<uint32_t>();
    p.row_cnt = s.row_cnt.as<uint2>();
    p.coarse = reinterpret_cast<uint2*>(s.counters.as<DevCounters>() + 1);
    p.wr = static_cast<uint32_t>(2 * WR);
    p.div_wr = make_fastdiv(p.wr);
    p.div_r = make_fastdiv(static_cast<uint32_t>(R));
    p.word_cap = word_cap;
    p.row_place = s.row_place.as<RowPlace>();
    p.present = s.present.as<uint32_t>();
    p.runs = s.runs.as<uint2>();
    p.word_list = s.word_list.as<uint32_t>();
    p.rank = s.rank.as<uint32_t>();
    p.sign = s.sign.as<uint32_t>();
    p.mesh = WordMesh{ s.word_cnt.as<uint32_t>(), s.word_cells.as<uint32_t>(), s.word_edges.as<uint4>(),
                       s.word_chunk.as<uint2>(), w.tile_sums.as<unsigned long long>(), nullptr };
    p.corners = s.corners.as<int64_t>();
    p.values = s.values.as<float>();
    p.corner_cap = corner_cap;
    p.ctr = s.counters.as<DevCounters>();
    p.host_ctr = s.host_d;
    // the per-request inputs the carve and field kernels read from the device
    s.rq.ensure(sizeof(ReqConsts), st);
    if (!s.host_rq)
        alloc_mapped(&s.host_rq, &s.host_rq_d);
    *s.host_rq = ReqConsts{ { p.corner[0], p.corner[1], p.corner[2] }, p.length, p.masks };
    p.rq = s.rq.as<ReqConsts>();
}

void fill_info(const HullSlot& s, th_hull_info* info)
{
    const DevCounters& c = *s.host;
    th_hull_info out{};
    const HullPlan& p = s.plan;
    // candidates_octree: levels up to and including the first empty one
    int n = 1;
    out.level_sizes[0] = c.level_count[0];
    for (int i = 1; i <= p.level; ++i)
    {
        out.level_sizes[i] = c.level_count[i];
        n = i + 1;
        if (c.level_count[i] == 0)
            break;
    }
    out.num_levels = n;
    const bool empty = c.level_count[p.level] == 0;
    out.num_corners = empty ? 0 : c.corners;
    if (empty || c.soup == 0)
    {
        out.num_verts = 0;
        out.num_faces = 0;
    }
    else
    {
        out.num_verts = p.unique ? c.verts : c.soup;
        out.num_faces = c.soup / 3;
    }
    *info = out;
}

// Everything of a run after the integral image: octree levels, corners,
// field, marching cubes and the read-back of the counters (stream-ordered
// only, so that it can be captured as a graph).
void enqueue_core(th_context* ctx, HullSlot& s, cudaStream_t st, StageEvents* ev, bool tune)
{
    const HullPlan& p = s.plan;
    const int L = p.level;
    // With an empty image every child is empty in the first view (the
    // reference samples zeros everywhere), so the octree stops at the root;
    // without views nothing is refined either.  Skip the carve in both cases.
    const bool carve = p.B > 0 && p.H > 0 && p.W > 0;
    if (tune)
        TH_CUDA(cudaEventRecord(ctx->tune_ev[0], st));
    const int top = carve ? top_levels(p.level) : 0;
    if (carve)
        launch_top(p, st);
    for (int li = 0; li < p.level; ++li)
    {
        if (carve && li >= top)
            launch_carve_level(p, li, st);
        if (ev)
            ev->record(2 + li, st);
    }
    if (tune)
        TH_CUDA(cudaEventRecord(ctx->tune_ev[1], st));
    if (ev)
        ev->record(L + 2, st);
    launch_corners(p, st);
    if (ev)
        ev->record(L + 3, st);
    launch_field(p, st);
    if (ev)
        ev->record(L + 4, st);
    launch_marching_cubes(p, st);
    if (ev)
        ev->record(L + 5, st);
}

// enqueue_core as a graph: captured once per plan (the per-request corner,
// length and masks come through p.rq, uploaded by prepare), replayed after.
void replay_core(HullSlot& s, cudaStream_t st)
{
    HullPlan key;
    std::memcpy(&key, &s.plan, sizeof(HullPlan));
    key.masks = nullptr;
    key.corner[0] = key.corner[1] = key.corner[2] = 0.f;
    key.length = 0.f;
    HullSlot::Graph* g = nullptr;
    for (auto& e : s.graphs)
        if (std::memcmp(&e.key, &key, sizeof(HullPlan)) == 0)
            g = &e;
    if (!g)
    {
        if (s.graphs.size() >= 8)
            s.drop_graphs();
        // captured on a private stream (the caller's may be the legacy
        // default stream, which cannot capture); nothing runs while capturing
        if (!s.capture_stream)
            TH_CUDA(cudaStreamCreateWithFlags(&s.capture_stream, cudaStreamNonBlocking));
        const cudaStream_t cs = s.capture_stream;
        cudaGraph_t graph = nullptr;
        TH_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
        t_capturing = true;
        t_captured = 0;
        try
        {
            enqueue_core(nullptr, s, cs, nullptr, false);
        }
        catch (...)
        {
            t_capturing = false;
            cudaStreamEndCapture(cs, &graph);
            if (graph)
                cudaGraphDestroy(graph);
            throw;
        }
        t_capturing = false;
        TH_CUDA(cudaStreamEndCapture(cs, &graph));
        cudaGraphExec_t exec = nullptr;
        const cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        TH_CUDA(e);
        s.graphs.push_back(HullSlot::Graph{ key, exec, t_captured });
        g = &s.graphs.back();
    }
    TH_CUDA(cudaGraphLaunch(g->exec, st));
    note_launches(static_cast<int>(g->kernels));
}

// What no larger pool helps against.  The request's pool is left unfinished then.
void refuse_overflow(int64_t overflow)
{
    if (overflow & kOverflowIndices)
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "visual hull: 2^32 or more corners of leaf cells or of triangles" };
}

// One complete run of a request with the given carve kernels.  carve_ms
// (optional) receives the time of the carve stage, for the autotuner.
void run_hull_once(th_context* ctx,
                   HullSlot& s,
                   const th_hull_args* a,
                   cudaStream_t st,
                   StageEvents* ev,
                   const CarveVariants& variants,
                   float* carve_ms)
{
    if (s.done)
        TH_CUDA(cudaStreamWaitEvent(st, s.done, 0)); // the last request's exports read the pools
    s.exported = false;
    s.has_result = false;
    const int L = a->level;
    for (int attempt = 0; attempt < 8; ++attempt)
    {
        prepare(s, s.work, a, st, ctx->field_ones, ctx->field_masks);
        for (int i = 0; i < kMaxLevel; ++i)
            s.plan.carve_variant[i] = variants[i];
        const HullPlan& p = s.plan;
        s.work.unfinished = true;
        if (attempt == 0)
        {
            if (ev)
                ev->record(0, st);
            launch_begin(p, a->transforms, a->transforms_dtype, s.host_rq_d, s.flags.as<unsigned int>(), true, st);
            launch_integral_image(a->masks, a->masks_dtype, a->batch, a->height, a->width, s.sat.as<float>(), st,
                                  s.flags.as<unsigned int>(),
                                  ctx->sat_single_pass ? SatScratch{ s.sat_scratch.p } : SatScratch{});
            if (ev)
                ev->record(1, st);
        }
        else
            launch_begin(p, a->transforms, a->transforms_dtype, s.host_rq_d, s.flags.as<unsigned int>(), false, st);
        if (ctx->graphs && !ev && !carve_ms)
            replay_core(s, st);
        else
            enqueue_core(ctx, s, st, ev, carve_ms != nullptr);
        TH_CUDA(cudaStreamSynchronize(st));
        const int64_t ovf = s.host->overflow;
        refuse_overflow(ovf);
        s.work.unfinished = false;
        // A level wider than the skip-mask scratch only loses view skipping
        // for its excess parents (results are unchanged): keep the result and
        // grow the scratch for the next request.
        if (ovf & kOverflowParents)
            s.work.parent_cap *= 4;
        if ((ovf & ~int64_t{ kOverflowParents }) == 0)
            break;
        if (ovf & kOverflowNodes)
        {
            s.work.node_cap *= 4;
            s.work.unfinished = true; // cells past the pool's end are not cleared from the cell masks
        }
        if (ovf & kOverflowCorners)
            s.corner_cap *= 4;
        if (ovf & kOverflowWords)
            s.word_cap *= 4;
        if (attempt == 7)
        {
            const DevCounters& c = *s.host;
            std::string counts;
            for (int i = 0; i <= L; ++i)
                counts += (i ? "," : "") + std::to_string(c.level_count[i]);
            throw ArgError{ TH_ERR_OUT_OF_MEMORY,
                            "visual hull pools could not be grown enough (overflow " + std::to_string(ovf) +
                                    ", level counts " + counts + ", corners " + std::to_string(c.corners) + ", rows " +
                                    std::to_string(c.rows) + ", node cap " + std::to_string(p.node_cap) +
                                    ", corner cap " + std::to_string(p.corner_cap) + ")" };
        }
    }
    fill_info(s, &s.info);
    s.has_result = true;
    if (ev)
    {
        th_stage_times t{};
        t.levels = L;
        t.integral_image_ms = ev->between(0, 1);
        for (int li = 0; li < L; ++li)
            t.carve_ms[li] = ev->between(1 + li, 2 + li);
        t.corners_ms = ev->between(L + 2, L + 3);
        t.field_ms = ev->between(L + 3, L + 4);
        t.marching_cubes_ms = ev->between(L + 4, L + 5);
        t.total_ms = ev->between(0, L + 5);
        for (int li = 0; li < L; ++li)
            t.carve_items[li] = static_cast<int64_t>(s.host->items[li]);
        t.field_items = static_cast<int64_t>(s.host->field_items);
        ctx->times = t;
    }
    if (carve_ms)
        TH_CUDA(cudaEventElapsedTime(carve_ms, ctx->tune_ev[0], ctx->tune_ev[1]));
}

// Runs request a on slot s.  With the autotuner on, the first request of a
// signature runs with both carve kernels (the results are identical) and the
// faster choice is kept for later requests of that signature.
void run_hull(th_context* ctx, HullSlot& s, const th_hull_args* a, cudaStream_t st, StageEvents* ev)
{
    validate(a);
    if (ctx->carve_mode == 1)
        return run_hull_once(ctx, s, a, st, ev, views_everywhere(), nullptr);
    if (ctx->carve_mode == 2)
        return run_hull_once(ctx, s, a, st, ev, items_from_level4(), nullptr);
    const TuneKey key = tune_key(a);
    auto it = ctx->carve_tuned.find(key);
    if (it != ctx->carve_tuned.end())
        return run_hull_once(ctx, s, a, st, ev, it->second, nullptr);
    if (a->level <= 4)
    {
        ctx->carve_tuned[key] = views_everywhere(); // both choices coincide
        return run_hull_once(ctx, s, a, st, ev, views_everywhere(), nullptr);
    }
    for (auto& e : ctx->tune_ev)
        if (!e)
            TH_CUDA(cudaEventCreate(&e));
    float t_views = 0.f, t_items = 0.f;
    run_hull_once(ctx, s, a, st, nullptr, views_everywhere(), &t_views);
    run_hull_once(ctx, s, a, st, ev, items_from_level4(), &t_items);
    ctx->carve_tuned[key] = (t_items < t_views) ? items_from_level4() : views_everywhere();
}

// Batched form: the requests' pipelines side by side on up to eight streams,
// the ones with most work first, with a single wait at the end.  (One
// persistent cooperative kernel over all octrees, before, took 3.8 ms for the
// carve of 16 mixed requests alone, whose neighbouring cells it scattered over
// the SMs: 7393 -> 5611 us with the faster stages around it, 4495 so.)
void run_batch(th_context* ctx, const th_hull_args* args, int32_t n, cudaStream_t st, th_hull_info* infos)
{
    for (int32_t r = 0; r < n; ++r)
        validate(&args[r]);
    if (n == 0)
        return;
    BatchState& bs = ctx->bstate;
    if (static_cast<int32_t>(ctx->batch.size()) < n)
        ctx->batch.resize(n);
    const int nstreams = std::min<int32_t>(n, 8);
    while (static_cast<int>(bs.streams.size()) < nstreams)
    {
        cudaStream_t s = nullptr;
        cudaEvent_t e = nullptr;
        TH_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        TH_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        bs.streams.push_back(s);
        bs.joins.push_back(e);
    }
    if (static_cast<int>(bs.pools.size()) < nstreams)
        bs.pools.resize(nstreams);
    if (!bs.fork)
        TH_CUDA(cudaEventCreateWithFlags(&bs.fork, cudaEventDisableTiming));
    for (int32_t r = 0; r < n; ++r)
    {
        HullSlot& s = ctx->batch[r];
        if (s.done)
            TH_CUDA(cudaStreamWaitEvent(st, s.done, 0)); // the last batch's exports read the pools
        s.exported = false;
        s.has_result = false;
    }
    std::vector<int32_t> order(n);
    std::iota(order.begin(), order.end(), 0);
    auto work = [&](int32_t r) { return static_cast<double>(args[r].batch) * static_cast<double>(int64_t{ 1 } << (2 * args[r].level)); };
    std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) { return work(x) > work(y); });
    for (int attempt = 0; attempt < 8; ++attempt)
    {
        TH_CUDA(cudaEventRecord(bs.fork, st));
        for (int i = 0; i < nstreams; ++i)
            TH_CUDA(cudaStreamWaitEvent(bs.streams[i], bs.fork, 0));
        // until the wait below, no pool is known to be clear
        auto unfinished = [&](bool u) {
            for (int i = 0; i < nstreams; ++i)
                bs.pools[i].unfinished = u;
        };
        try
        {
            for (int32_t k = 0; k < n; ++k)
            {
                const int32_t r = order[k];
                const th_hull_args* a = &args[r];
                HullSlot& s = ctx->batch[r];
                WorkPool& w = bs.pools[k % nstreams];
                const cudaStream_t sr = bs.streams[k % nstreams];
                prepare(s, w, a, sr, ctx->field_ones, ctx->field_masks, true);
                const auto tuned = ctx->carve_tuned.find(tune_key(a));
                const CarveVariants variants = ctx->carve_mode == 1 ? views_everywhere()
                                               : ctx->carve_mode == 2 || tuned == ctx->carve_tuned.end() ? items_from_level4()
                                                                                                         : tuned->second;
                for (int i = 0; i < kMaxLevel; ++i)
                    s.plan.carve_variant[i] = variants[i];
                launch_begin(s.plan, a->transforms, a->transforms_dtype, s.host_rq_d, s.flags.as<unsigned int>(), attempt == 0, sr);
                if (attempt == 0)
                    launch_integral_image(a->masks, a->masks_dtype, a->batch, a->height, a->width, s.sat.as<float>(), sr,
                                          s.flags.as<unsigned int>(),
                                          ctx->sat_single_pass ? SatScratch{ s.sat_scratch.p } : SatScratch{});
                enqueue_core(ctx, s, sr, nullptr, false);
            }
        }
        catch (...)
        {
            // what is queued reads the callers' masks and the slots' buffers
            for (int i = 0; i < nstreams; ++i)
                cudaStreamSynchronize(bs.streams[i]);
            unfinished(true);
            throw;
        }
        unfinished(true);
        for (int i = 0; i < nstreams; ++i)
        {
            TH_CUDA(cudaEventRecord(bs.joins[i], bs.streams[i]));
            TH_CUDA(cudaStreamWaitEvent(st, bs.joins[i], 0));
        }
        TH_CUDA(cudaStreamSynchronize(st));
        unfinished(false);
        for (int32_t r = 0; r < n; ++r)
        {
            if (ctx->batch[r].host->overflow & kOverflowIndices)
                unfinished(true);
            refuse_overflow(ctx->batch[r].host->overflow);
        }
        bool retry = false;
        for (int32_t k = 0; k < n; ++k)
        {
            HullSlot& s = ctx->batch[order[k]];
            WorkPool& w = bs.pools[k % nstreams];
            const int64_t ovf = s.host->overflow;
            // as for a plain request: only view skipping was lost
            if (ovf & kOverflowParents)
                w.parent_cap = std::max(w.parent_cap, 4 * s.plan.parent_cap);
            if (ovf & kOverflowNodes)
            {
                w.node_cap = std::max(w.node_cap, 4 * s.plan.node_cap);
                // cells past the pool's end are not cleared from the cell
                // masks, which later requests of the stream read: all run again
                w.unfinished = true;
            }
            if (ovf & kOverflowCorners)
                s.corner_cap *= 4;
            if (ovf & kOverflowWords)
                s.word_cap *= 4;
            retry = retry || (ovf & ~int64_t{ kOverflowParents }) != 0;
        }
        if (!retry)
            break;
        if (attempt == 7)
            throw ArgError{ TH_ERR_OUT_OF_MEMORY, "batch pools could not be grown enough" };
    }
    for (int32_t r = 0; r < n; ++r)
    {
        HullSlot& s = ctx->batch[r];
        const DevCounters& c = *s.host;
        th_hull_info info{};
        info.num_corners = c.corners;
        info.num_levels = 0; // per-level candidates are not kept by the batched form
        if (c.soup > 0)
        {
            info.num_verts = s.plan.unique ? c.verts : c.soup;
            info.num_faces = c.soup / 3;
        }
        s.info = info;
        s.has_result = true;
        infos[r] = info;
    }
}

// With routing on, a request whose octree alone fills the GPU (level >= 8
// and at least 16 M mask pixels) runs by itself, as th_visual_hull does, and
// the others side by side.  Off by default: a batch's requests run through the
// same pipeline on its streams, where the small ones fill the large ones' gaps.
// Results are identical either way.
bool fills_gpu(const th_hull_args& a)
{
    return a.level >= 8 && a.batch * a.height * a.width >= (int64_t{ 1 } << 24);
}

void run_batch_routed(th_context* ctx, const th_hull_args* args, int32_t n, cudaStream_t st, th_hull_info* infos)
{
    for (int32_t r = 0; r < n; ++r)
        validate(&args[r]);
    std::vector<int32_t> shared, solo;
    for (int32_t r = 0; r < n; ++r)
        (ctx->batch_route && fills_gpu(args[r]) ? solo : shared).push_back(r);
    if (static_cast<int32_t>(ctx->batch.size()) < n)
        ctx->batch.resize(n);
    if (!shared.empty())
    {
        std::vector<th_hull_args> sub(shared.size());
        std::vector<th_hull_info> sub_infos(shared.size());
        for (size_t j = 0; j < shared.size(); ++j)
            sub[j] = args[shared[j]];
        run_batch(ctx, sub.data(), static_cast<int32_t>(sub.size()), st, sub_infos.data());
        // results of shared[j] sit in slot j <= shared[j]: move them into place,
        // last first, so no placed result is moved again
        for (size_t j = shared.size(); j-- > 0;)
        {
            std::swap(ctx->batch[j], ctx->batch[shared[j]]);
            infos[shared[j]] = sub_infos[j];
        }
    }
    for (int32_t r : solo)
    {
        run_hull(ctx, ctx->batch[r], &args[r], st, nullptr);
        infos[r] = ctx->batch[r].info;
    }
}

th_status fail(th_context* ctx, th_status st, const std::string& msg)
{
    if (ctx)
        ctx->error = msg;
    return st;
}

template <class F>
th_status guarded(th_context* ctx, F&& f)
{
    if (!ctx)
        return TH_ERR_INVALID_ARGUMENT;
    ctx->error.clear();
    try
    {
        TH_CUDA(cudaSetDevice(ctx->device));
        f();
        return TH_OK;
    }
    catch (const ArgError& e)
    {
        return fail(ctx, e.status, e.msg);
    }
    catch (const CudaError& e)
    {
        cudaGetLastError(); // reported here: the next launch's check, ours or the caller's, must not find it again
        const th_status st = (e.code == cudaErrorMemoryAllocation) ? TH_ERR_OUT_OF_MEMORY : TH_ERR_CUDA;
        return fail(ctx, st, std::string(cudaGetErrorString(e.code)) + " (" + e.where + ")");
    }
    catch (const std::exception& e)
    {
        return fail(ctx, TH_ERR_CUDA, e.what());
    }
}

} // namespace
} // namespace th

namespace th
{
namespace
{

// gaussian_blur_cuda.cu:294-305 and :79-81, in the reference's order.
void check_blur_args(int32_t images_dtype, int32_t kernel_size, float sigma, int32_t out_dtype)
{
    if (kernel_size <= 0)
        throw ArgError{ TH_ERR_INVALID_ARGUMENT,
                        "Check failed: kernel_size > 0 (" + std::to_string(kernel_size) + " vs. 0)" };
    if (kernel_size % 2 != 1)
        throw ArgError{ TH_ERR_INVALID_ARGUMENT,
                        "Check failed: kernel_size % 2 == 1 (" + std::to_string(kernel_size % 2) + " vs. 1)" };
    if (!(sigma > 0.f))
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "Check failed: sigma > 0.f" };
    if (!(out_dtype == TH_FLOAT16 || out_dtype == TH_FLOAT32 || out_dtype == TH_FLOAT64))
    {
        if (out_dtype == TH_BFLOAT16)
            throw ArgError{ TH_ERR_UNSUPPORTED_DTYPE, "\"tile_convolution_kernel\" not implemented for 'BFloat16'" };
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "Check failed: torch::isFloatingType(dtype_result) == true" };
    }
    if (!is_image_dtype(images_dtype))
        throw ArgError{ TH_ERR_UNSUPPORTED_DTYPE,
                        std::string("\"edge_kernel\" not implemented for '") + dtype_name(images_dtype) + "'" };
}

// Runs launch(scratch) on st with scratch of at least `bytes`.  Calls on
// different streams share the context's buffer: each waits for the one before.
// A call that is recorded into a caller's graph takes a block of its own.
template <class F>
void with_scratch(th_context* ctx, DevBuf& buf, cudaEvent_t& done, size_t bytes, cudaStream_t st, F&& launch)
{
    if (bytes == 0)
        return launch(nullptr);
    if (in_capture(st))
        return launch(ctx->graph_scratch.take(st, bytes));
    if (done)
        TH_CUDA(cudaStreamWaitEvent(st, done, 0));
    else
        TH_CUDA(cudaEventCreateWithFlags(&done, cudaEventDisableTiming));
    buf.ensure(bytes, st);
    launch(buf.p);
    TH_CUDA(cudaEventRecord(done, st));
}

// Element size of a float dtype code.
size_t float_size(int32_t dt)
{
    return dt == TH_FLOAT64 ? 8 : (dt == TH_FLOAT32 ? 4 : 2);
}

std::string float_text(float v)
{
    std::ostringstream os;
    os << v;
    return os.str();
}

// Argument checks of marching_cubes_cuda_{dense,sparse} (:382-385, :758-764,
// :789-795) that reach the C ABI; the tensor-layout checks live in the torch layer.
void run_mc(McSlot& s, const th_mc_args* a, cudaStream_t st)
{
    s.has_result = false;
    if (!a)
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "args is NULL" };
    if (a->depth < 0 || a->height < 0 || a->width < 0 || a->nnz < 0)
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "volume sizes must be non-negative" };
    if (!(a->isolevel >= 0.f))
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "Check failed: isolevel >= 0 (" + float_text(a->isolevel) + " vs. 0)" };
    const char* kernel = a->sparse ? "classify_voxels_sparse" : "classify_voxels_dense";
    if (!(a->dtype == TH_FLOAT16 || a->dtype == TH_FLOAT32 || a->dtype == TH_FLOAT64))
        throw ArgError{ TH_ERR_UNSUPPORTED_DTYPE,
                        std::string("\"") + kernel + "\" not implemented for '" + dtype_name(a->dtype) + "'" };
    const int64_t D = a->depth, H = a->height, W = a->width;
    McPlan p{};
    p.dtype = a->dtype;
    p.sparse = a->sparse != 0;
    p.unique = a->unique_verts != 0;
    p.local = a->return_local_coords != 0;
    p.D = D;
    p.H = H;
    p.W = W;
    p.iso = a->isolevel;
    // 2.f / static_cast<float>(size - 1) (:515-517), x along W
    p.scale[0] = 2.f / static_cast<float>(W - 1);
    p.scale[1] = 2.f / static_cast<float>(H - 1);
    p.scale[2] = 2.f / static_cast<float>(D - 1);
    if (p.sparse)
    {
        if (a->nnz >= (int64_t{ 1 } << 31))
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "sparse volumes hold fewer than 2^31 values" };
        if (a->nnz > 0 && (!a->indices || !a->values))
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "indices or values pointer is NULL" };
        p.indices = a->indices;
        p.values = a->values;
        p.nnz = a->nnz;
    }
    else
    {
        // the dense driver sizes its cell arrays (D-1)(H-1)(W-1) and reads the
        // last scan entry back (:392-397, :421-423)
        const int64_t cells = (D - 1) * (H - 1) * (W - 1);
        if (D < 1 || H < 1 || W < 1)
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "Trying to create tensor with negative dimension " +
                                                             std::to_string(cells) + ": [" + std::to_string(cells) + "]" };
        if (cells == 0)
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "index -1 is out of bounds for dimension 0 with size 0" };
        if (!a->volume)
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "volume pointer is NULL" };
        p.volume = a->volume;
    }
    // Rows of 32-point words.  A sparse volume takes them when they are at
    // most kWordsPerEntry per entry (and always below kFewWords).  The line
    // bounds the scratch, not the time: a word takes 40 bytes where an entry's
    // table takes 60, and words are faster well past it (512^3, calls with words
    // against the table: one word per entry 415 us against 1313, 8 190 against
    // 265, 16 162 against 214, 64 132 against 187).
    constexpr int64_t kWordsPerEntry = 8, kFewWords = int64_t{ 1 } << 18;
    p.wr = 0;
    if (W > 0 && H > 0 && D > 0)
    {
        const int64_t wr = (W + 31) / 32;
        bool fits = H < (int64_t{ 1 } << 32) / wr && D < (int64_t{ 1 } << 32) / (wr * H); // word indices below 2^32
        p.nwords = fits ? wr * H * D : 0;
        p.slab = D;
        if (!p.sparse && H < (int64_t{ 1 } << 32) / wr)
        {
            // A word takes 28 bytes of scratch, however few points its row has:
            // slabs keep it below 1.75 bytes a point (what rows of 16 points and
            // more need), or 3.8 GB where that is less.  A slab's words are
            // counted twice, now and for the export (12000 x 12000 x 3 float32,
            // two slabs: 16.4 ms; 11100 x 12000 x 3 at once: 8.2).
            const int64_t plane = wr * H;
            const int64_t most = std::min<int64_t>(std::max<int64_t>(int64_t{ 1 } << 27, D * H * W / 16), (int64_t{ 1 } << 32) - 1);
            if (!fits || p.nwords > most)
            {
                p.slab = std::max<int64_t>(most / plane - 2, 1);
                p.nwords = std::min<int64_t>(p.slab + 2, D) * plane; // of the largest slab
                fits = p.nwords < (int64_t{ 1 } << 32);
            }
        }
        p.own = p.nwords;
        // fewer than 2^28 entries: packed counts, like the active cells of a dense volume below
        p.words = fits && (!p.sparse || (p.nnz < (int64_t{ 1 } << 28) &&
                                         (p.nwords <= kFewWords || p.nwords / kWordsPerEntry <= p.nnz)));
        if (!p.sparse && !fits)
            throw ArgError{ TH_ERR_OUT_OF_MEMORY, "marching cubes: the volume has too many rows of 32 points" };
    }
    if (p.words)
    {
        p.wr = static_cast<uint32_t>((W + 31) / 32);
        p.div_wr = make_fastdiv(p.wr);
        p.div_h = make_fastdiv(static_cast<uint32_t>(H));
    }

    // the last mesh may still be read from the buffers on another stream
    if (s.done)
        TH_CUDA(cudaStreamWaitEvent(st, s.done, 0));
    else
        TH_CUDA(cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming));
    s.exported = false;
    if (!s.host)
        alloc_mapped(&s.host, &s.host_d);
    s.ctr.ensure(sizeof(McCounters), st);
    p.ctr = s.ctr.as<McCounters>();
    if (p.words && !(p.sparse && p.nnz == 0))
    {
        const size_t n = static_cast<size_t>(p.nwords);
        s.bits.ensure(sizeof(uint32_t) * n * (p.sparse ? 2 : 1), st);
        p.sign = s.bits.as<uint32_t>() + (p.sparse ? n : 0);
        if (p.sparse)
        {
            s.rank.ensure(sizeof(uint32_t) * n, st);
            p.present = s.bits.as<uint32_t>();
            p.rank = s.rank.as<uint32_t>();
        }
        s.cnt.ensure(sizeof(uint32_t) * n, st);
        s.cells.ensure(sizeof(uint32_t) * n, st);
        s.chunk.ensure(sizeof(uint2) * ((n + 31) / 32), st);
        s.tiles_soup.ensure(sizeof(unsigned long long) * word_tiles(p.nwords), st);
        if (p.unique)
            s.edges.ensure(sizeof(uint4) * n, st);
        p.mesh = WordMesh{ s.cnt.as<uint32_t>(), s.cells.as<uint32_t>(), s.edges.as<uint4>(), s.chunk.as<uint2>(),
                           s.tiles_soup.as<unsigned long long>(), nullptr };
        if (p.slab < D)
        {
            s.start.ensure(sizeof(unsigned long long), st);
            p.mesh.start = s.start.as<unsigned long long>();
        }
    }
    else if (p.sparse)
    {
        const int64_t n = p.nnz;
        uint64_t cap = 64;
        while (cap < 2 * static_cast<uint64_t>(n))
            cap <<= 1;
        s.keys.ensure(sizeof(unsigned long long) * cap, st);
        s.slots.ensure(sizeof(int32_t) * cap, st);
        s.codes.ensure(static_cast<size_t>(n), st);
        s.tiles_soup.ensure(sizeof(unsigned long long) * mc_scan_tiles(n), st);
        p.keys = s.keys.as<unsigned long long>();
        p.slots = s.slots.as<int32_t>();
        p.hmask = cap - 1;
        p.codes = s.codes.as<uint8_t>();
        p.tiles_soup = s.tiles_soup.as<unsigned long long>();
        if (p.unique)
        {
            s.used.ensure(sizeof(uint32_t) * n, st);
            s.vbase.ensure(sizeof(unsigned long long) * n, st);
            s.tiles_verts.ensure(sizeof(unsigned long long) * mc_scan_tiles(n), st);
            p.used = s.used.as<uint32_t>();
            p.vbase = s.vbase.as<unsigned long long>();
            p.tiles_verts = s.tiles_verts.as<unsigned long long>();
        }
    }

    try
    {
        launch_mc_count(p, st);
        small_copy(s.host_d, p.ctr, sizeof(McCounters), st);
        TH_CUDA(cudaStreamSynchronize(st));
    }
    catch (...)
    {
        // what is queued writes the buffers, which the next call may use on another stream
        cudaStreamSynchronize(st);
        throw;
    }
    const McCounters& c = *s.host;
    if (c.flags & kMcBadIndex)
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "sparse volume indices lie outside the volume" };
    if (c.flags & kMcUnsorted)
        throw ArgError{ TH_ERR_INVALID_ARGUMENT,
                        "sparse volume indices must be coalesced (strictly ascending in (z, y, x))" };
    // the counts are summed packed (corners << 32 | vertices): both below 2^32
    if (!p.sparse && c.active >= (1ull << 28))
        throw ArgError{ TH_ERR_INVALID_ARGUMENT, "marching cubes: more than 2^28 active cells" };
    s.plan = p;
    s.info.num_faces = static_cast<int64_t>(c.soup / 3);
    s.info.num_verts = static_cast<int64_t>(p.unique ? c.verts : c.soup);
    s.has_result = true;
}

} // namespace
} // namespace th

using namespace th;

extern "C" {

th_status th_context_create(int32_t device, th_context** out)
{
    if (!out)
        return TH_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0)
        return TH_ERR_NO_DEVICE;
    if (device < 0 || device >= n)
        return TH_ERR_INVALID_ARGUMENT;
    auto* ctx = new th_context;
    ctx->device = device;
    *out = ctx;
    return TH_OK;
}

void th_context_destroy(th_context* ctx)
{
    if (!ctx)
        return;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(ctx->device);
    cudaDeviceSynchronize();
    ctx->hull.release();
    for (auto& s : ctx->batch)
        s.release();
    ctx->blur_scratch.release();
    ctx->blurred.release();
    ctx->sat_aux.release();
    ctx->graph_scratch.release();
    if (ctx->sat_aux_done)
        cudaEventDestroy(ctx->sat_aux_done);
    if (ctx->blur_done)
        cudaEventDestroy(ctx->blur_done);
    ctx->mc.release();
    ctx->bstate.release();
    ctx->events.destroy();
    for (auto& e : ctx->tune_ev)
        if (e)
            cudaEventDestroy(e);
    cudaSetDevice(prev);
    delete ctx;
}

const char* th_context_error(const th_context* ctx)
{
    return ctx ? ctx->error.c_str() : "";
}

const char* th_status_string(th_status status)
{
    switch (status)
    {
    case TH_OK:
        return "ok";
    case TH_ERR_INVALID_ARGUMENT:
        return "invalid argument";
    case TH_ERR_UNSUPPORTED_DTYPE:
        return "unsupported dtype";
    case TH_ERR_CUDA:
        return "CUDA error";
    case TH_ERR_OUT_OF_MEMORY:
        return "out of memory";
    case TH_ERR_STATE:
        return "invalid call order";
    case TH_ERR_NO_DEVICE:
        return "no CUDA device";
    }
    return "unknown status";
}

int64_t th_context_device_bytes(const th_context* ctx)
{
    return ctx ? pool_bytes(ctx) : 0;
}

th_status th_context_set_option(th_context* ctx, int32_t option, int64_t value)
{
    return guarded(ctx, [&] {
        if (option == TH_OPTION_CARVE_KERNEL && value >= 0 && value <= 2)
            ctx->carve_mode = static_cast<int>(value);
        else if (option == TH_OPTION_GRAPHS && (value == 0 || value == 1))
            ctx->graphs = value != 0;
        else if (option == TH_OPTION_BATCH_ROUTE && (value == 0 || value == 1))
            ctx->batch_route = value != 0;
        else if (option == TH_OPTION_FIELD_ONES && (value == 0 || value == 1))
            ctx->field_ones = value != 0;
        else if (option == TH_OPTION_FIELD_MASKS && (value == 0 || value == 1))
            ctx->field_masks = value != 0;
        else if (option == TH_OPTION_SAT_SINGLE_PASS && (value == 0 || value == 1))
            ctx->sat_single_pass = value != 0;
        else
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "unknown option or value" };
    });
}

th_status th_context_set_profiling(th_context* ctx, int32_t enable)
{
    return guarded(ctx, [&] {
        if (enable)
            ctx->events.create();
        ctx->profiling = enable != 0;
    });
}

th_status th_context_stage_times(const th_context* ctx, th_stage_times* out)
{
    if (!ctx || !out)
        return TH_ERR_INVALID_ARGUMENT;
    *out = ctx->times;
    return TH_OK;
}

int64_t th_launch_count(void)
{
    return g_launches.load(std::memory_order_relaxed);
}

namespace th
{
namespace
{

// 16-byte words, then the tail bytes.  Reads of host memory are latency
// bound: each thread keeps kCopyUnroll independent 16-byte loads in flight.
constexpr int kCopyUnroll = 8;

__global__ void __launch_bounds__(256) sm_copy_kernel(const unsigned char* __restrict__ src,
                                                      unsigned char* __restrict__ dst,
                                                      int64_t n,
                                                      int vec)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    const int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    int64_t done = 0;
    if (vec)
    {
        const int64_t nv = n / 16;
        const uint4* s4 = reinterpret_cast<const uint4*>(src);
        uint4* d4 = reinterpret_cast<uint4*>(dst);
        int64_t i = t0;
        for (; i + (kCopyUnroll - 1) * stride < nv; i += kCopyUnroll * stride)
        {
            uint4 r[kCopyUnroll];
#pragma unroll
            for (int k = 0; k < kCopyUnroll; ++k)
                r[k] = s4[i + k * stride];
#pragma unroll
            for (int k = 0; k < kCopyUnroll; ++k)
                d4[i + k * stride] = r[k];
        }
        for (; i < nv; i += stride)
            d4[i] = s4[i];
        done = nv * 16;
    }
    for (int64_t i = done + t0; i < n; i += stride)
        dst[i] = src[i];
}

// The device address of a copy operand for a kernel on the current device:
// its own device memory and managed memory as they are, pinned host memory
// through its mapping (host = true); nullptr for another device's memory and
// for host memory the device cannot address.
const void* device_address(const void* p, bool& host)
{
    host = false;
    cudaPointerAttributes a{};
    int current = -1;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess || cudaGetDevice(&current) != cudaSuccess)
    {
        cudaGetLastError();
        return nullptr;
    }
    if (a.type == cudaMemoryTypeManaged)
        return p;
    if (a.type == cudaMemoryTypeDevice)
        return a.device == current ? p : nullptr;
    if (a.type == cudaMemoryTypeHost)
    {
        host = true;
        return a.devicePointer;
    }
    return nullptr;
}

} // namespace
} // namespace th

th_status th_copy(void* dst, const void* src, int64_t bytes, void* stream)
{
    if (bytes < 0 || ((!dst || !src) && bytes > 0))
        return TH_ERR_INVALID_ARGUMENT;
    if (bytes == 0)
        return TH_OK;
    bool src_host = false, dst_host = false;
    const void* s = th::device_address(src, src_host);
    void* d = const_cast<void*>(th::device_address(dst, dst_host));
    if (!s || !d)
        return TH_ERR_INVALID_ARGUMENT;
    const int vec = (reinterpret_cast<uintptr_t>(d) % 16 == 0) && (reinterpret_cast<uintptr_t>(s) % 16 == 0);
    // A copy to or from host memory runs beside the hull kernels on a few
    // blocks: on GB300 eight blocks read host memory at ~130 GB/s and six
    // write it at ~190 GB/s (the link's rate), while a grid over all SMs
    // slows the concurrent hulls.  Device-to-device copies take every SM.
    const int grid = src_host ? 8 : dst_host ? 6 : 2 * th::sm_count();
    th::sm_copy_kernel<<<static_cast<unsigned>(grid), 256, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const unsigned char*>(s), static_cast<unsigned char*>(d), bytes, vec);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError() == cudaSuccess ? TH_OK : TH_ERR_CUDA;
}

th_status th_visual_hull(th_context* ctx, const th_hull_args* args, void* stream, th_hull_info* info)
{
    return guarded(ctx, [&] {
        run_hull(ctx, ctx->hull, args, static_cast<cudaStream_t>(stream), ctx->profiling ? &ctx->events : nullptr);
        if (info)
            *info = ctx->hull.info;
    });
}

th_status th_visual_hull_blurred(th_context* ctx,
                                 const th_hull_args* args,
                                 int32_t kernel_size,
                                 float sigma,
                                 void* stream,
                                 th_hull_info* info)
{
    return guarded(ctx, [&] {
        if (!args)
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "args is NULL" };
        // gaussian_blur(masks, kernel_size, sigma) first: its checks come first
        check_blur_args(args->masks_dtype, kernel_size, sigma, args->masks_dtype);
        validate(args);
        auto st = static_cast<cudaStream_t>(stream);
        th_hull_args a = *args;
        const int64_t n = args->batch * args->height * args->width;
        if (n > 0)
        {
            ctx->blurred.ensure(float_size(args->masks_dtype) * static_cast<size_t>(n), st);
            const int64_t bytes = blur_tile_bytes(args->batch, args->height, args->width, kernel_size);
            with_scratch(ctx, ctx->blur_scratch, ctx->blur_done, static_cast<size_t>(bytes), st, [&](void* scratch) {
                launch_gaussian_blur(args->masks, args->masks_dtype, args->batch, args->height, args->width, kernel_size,
                                     sigma, true, ctx->blurred.p, args->masks_dtype, static_cast<uint8_t*>(scratch), st);
            });
            a.masks = ctx->blurred.p;
        }
        run_hull(ctx, ctx->hull, &a, st, ctx->profiling ? &ctx->events : nullptr);
        if (info)
            *info = ctx->hull.info;
    });
}

th_status th_visual_hull_export(th_context* ctx, float* verts, int64_t* faces, void* stream)
{
    return guarded(ctx, [&] {
        HullSlot& s = ctx->hull;
        if (!s.has_result)
            throw ArgError{ TH_ERR_STATE, "th_visual_hull_export called without a successful th_visual_hull" };
        auto st = static_cast<cudaStream_t>(stream);
        if (s.info.num_faces > 0)
        {
            if (!verts || !faces)
                throw ArgError{ TH_ERR_INVALID_ARGUMENT, "verts or faces pointer is NULL" };
            export_on(s, st, [&] { launch_export(s.plan, s.host->words, verts, faces, st); });
        }
    });
}

th_status th_visual_hull_export_candidates(th_context* ctx, int32_t level, int64_t* dst, void* stream)
{
    return guarded(ctx, [&] {
        HullSlot& s = ctx->hull;
        if (!s.has_result)
            throw ArgError{ TH_ERR_STATE, "export called without a successful th_visual_hull" };
        if (level < 0 || level >= s.info.num_levels)
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "candidate level out of range" };
        const int64_t n = s.info.level_sizes[level];
        if (n > 0)
        {
            if (!dst)
                throw ArgError{ TH_ERR_INVALID_ARGUMENT, "dst is NULL" };
            const cudaStream_t st = static_cast<cudaStream_t>(stream);
            export_on(s, st, [&] {
                // the leaves are written out on demand
                if (level == s.plan.level)
                    launch_emit_leaves(s.plan, st);
                TH_CUDA(cudaMemcpyAsync(dst, s.plan.nodes + s.host->level_off[level], sizeof(int64_t) * n,
                                        cudaMemcpyDeviceToDevice, st));
            });
        }
    });
}

th_status th_visual_hull_export_field(th_context* ctx, int64_t* indices, float* values, void* stream)
{
    return guarded(ctx, [&] {
        HullSlot& s = ctx->hull;
        if (!s.has_result)
            throw ArgError{ TH_ERR_STATE, "export called without a successful th_visual_hull" };
        const int64_t n = s.info.num_corners;
        auto st = static_cast<cudaStream_t>(stream);
        if (n > 0)
        {
            if (!indices || !values)
                throw ArgError{ TH_ERR_INVALID_ARGUMENT, "indices or values pointer is NULL" };
            export_on(s, st, [&] { launch_export_field(s.plan, n, indices, values, st); });
        }
    });
}

th_status th_visual_hull_export_field_coo(th_context* ctx, int64_t* indices, float* values, void* stream)
{
    return guarded(ctx, [&] {
        HullSlot& s = ctx->hull;
        if (!s.has_result)
            throw ArgError{ TH_ERR_STATE, "export called without a successful th_visual_hull" };
        const int64_t n = s.info.num_corners;
        auto st = static_cast<cudaStream_t>(stream);
        if (n > 0)
        {
            if (!indices || !values)
                throw ArgError{ TH_ERR_INVALID_ARGUMENT, "indices or values pointer is NULL" };
            export_on(s, st, [&] { launch_export_field_coo(s.plan, n, indices, values, st); });
        }
    });
}

th_status th_gaussian_blur(th_context* ctx,
                           const void* images,
                           int32_t images_dtype,
                           int64_t batch,
                           int64_t height,
                           int64_t width,
                           int32_t kernel_size,
                           float sigma,
                           int32_t sparse,
                           void* out,
                           int32_t out_dtype,
                           void* stream)
{
    return guarded(ctx, [&] {
        check_blur_args(images_dtype, kernel_size, sigma, out_dtype);
        if (batch < 0 || height < 0 || width < 0)
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "image sizes must be non-negative" };
        const int64_t n = batch * height * width;
        if (n == 0)
            return;
        if (!images || !out)
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "images or out pointer is NULL" };
        const int64_t bytes = blur_tile_bytes(batch, height, width, kernel_size);
        const cudaStream_t st = static_cast<cudaStream_t>(stream);
        with_scratch(ctx, ctx->blur_scratch, ctx->blur_done, static_cast<size_t>(bytes), st, [&](void* scratch) {
            launch_gaussian_blur(images, images_dtype, batch, height, width, kernel_size, sigma, sparse != 0, out, out_dtype,
                                 static_cast<uint8_t*>(scratch), st);
        });
    });
}

th_status th_integral_image(th_context* ctx,
                            const void* masks,
                            int32_t masks_dtype,
                            int64_t batch,
                            int64_t height,
                            int64_t width,
                            float* out,
                            void* stream)
{
    return guarded(ctx, [&] {
        if (!is_image_dtype(masks_dtype))
            throw ArgError{ TH_ERR_UNSUPPORTED_DTYPE,
                            std::string("integral image not implemented for '") + dtype_name(masks_dtype) + "'" };
        if (batch < 0 || height < 0 || width < 0)
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "mask sizes must be non-negative" };
        if (batch * height * width == 0)
            return;
        if (!masks || !out)
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "masks or out pointer is NULL" };
        const cudaStream_t st = static_cast<cudaStream_t>(stream);
        const int64_t sb = ctx->sat_single_pass ? sat_scratch_bytes(batch, height, width, masks_dtype) : 0;
        constexpr int64_t kFlagBytes = 256;
        with_scratch(ctx, ctx->sat_aux, ctx->sat_aux_done, sb > 0 ? static_cast<size_t>(kFlagBytes + sb) : 0, st, [&](void* scratch) {
            unsigned int* flag = static_cast<unsigned int*>(scratch);
            SatScratch sc{};
            if (flag)
            {
                launch_zero(flag, sizeof(unsigned int), st);
                sc = SatScratch{ static_cast<unsigned char*>(scratch) + kFlagBytes };
            }
            launch_integral_image(masks, masks_dtype, batch, height, width, out, st, flag, sc);
        });
    });
}

th_status th_marching_cubes(th_context* ctx, const th_mc_args* args, void* stream, th_mc_info* info)
{
    return guarded(ctx, [&] {
        run_mc(ctx->mc, args, static_cast<cudaStream_t>(stream));
        if (info)
            *info = ctx->mc.info;
    });
}

th_status th_marching_cubes_export(th_context* ctx, float* verts, int64_t* faces, void* stream)
{
    return guarded(ctx, [&] {
        McSlot& s = ctx->mc;
        if (!s.has_result)
            throw ArgError{ TH_ERR_STATE, "th_marching_cubes_export called without a successful th_marching_cubes" };
        if (s.info.num_faces > 0)
        {
            if (!verts || !faces)
                throw ArgError{ TH_ERR_INVALID_ARGUMENT, "verts or faces pointer is NULL" };
            const cudaStream_t st = static_cast<cudaStream_t>(stream);
            export_on(s, st, [&] { launch_mc_emit(s.plan, verts, faces, st); });
        }
    });
}

th_status th_candidate_wireframe(th_context* ctx,
                                 const int64_t* candidates,
                                 int64_t n,
                                 int32_t level_index,
                                 const float cube_corner_bfl[3],
                                 float cube_length,
                                 float* verts,
                                 int64_t* edges,
                                 void* stream)
{
    return guarded(ctx, [&] {
        if (n < 0 || level_index < 0 || level_index > 20 || !cube_corner_bfl)
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "invalid wireframe arguments" };
        if (n > 0 && (!candidates || !verts || !edges))
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "candidates, verts or edges pointer is NULL" };
        launch_wireframe(candidates, n, level_index, cube_corner_bfl, cube_length, verts, edges,
                         static_cast<cudaStream_t>(stream));
    });
}

th_status th_store_curve_network(th_context* ctx,
                                 const char* filename,
                                 const float* verts,
                                 int64_t nv,
                                 const int64_t* edges,
                                 int64_t ne,
                                 int32_t verbose)
{
    // host only: no device is needed, ctx (may be NULL) only receives the message
    if (ctx)
        ctx->error.clear();
    if (!filename || nv < 0 || ne < 0 || (nv > 0 && !verts) || (ne > 0 && !edges))
        return fail(ctx, TH_ERR_INVALID_ARGUMENT, "invalid curve network arguments");
    const std::string name(filename);
    try
    {
        if (!store_curve_network(name, verts, nv, edges, ne, verbose != 0))
            return fail(ctx, TH_ERR_INVALID_ARGUMENT,
                        "No implementation for file extension \"" + file_extension(name) + "\".");
    }
    catch (const std::exception& e)
    {
        return fail(ctx, TH_ERR_INVALID_ARGUMENT, e.what());
    }
    return TH_OK;
}

th_status th_visual_hull_batch(th_context* ctx, const th_hull_args* args, int32_t n, void* stream, th_hull_info* infos)
{
    return guarded(ctx, [&] {
        if (n < 0 || (n > 0 && (!args || !infos)))
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "invalid batch arguments" };
        run_batch_routed(ctx, args, n, static_cast<cudaStream_t>(stream), infos);
    });
}

th_status th_visual_hull_batch_export(th_context* ctx, int32_t index, float* verts, int64_t* faces, void* stream)
{
    return guarded(ctx, [&] {
        if (index < 0 || index >= static_cast<int32_t>(ctx->batch.size()) || !ctx->batch[index].has_result)
            throw ArgError{ TH_ERR_STATE, "no batched result at this index" };
        HullSlot& s = ctx->batch[index];
        auto st = static_cast<cudaStream_t>(stream);
        if (s.info.num_faces > 0)
        {
            if (!verts || !faces)
                throw ArgError{ TH_ERR_INVALID_ARGUMENT, "verts or faces pointer is NULL" };
            export_on(s, st, [&] { launch_export(s.plan, s.host->words, verts, faces, st); });
        }
    });
}

th_status th_visual_hull_batch_export_all(th_context* ctx, int32_t n, float* const* verts, int64_t* const* faces,
                                          void* stream)
{
    return guarded(ctx, [&] {
        if (n < 0 || n > static_cast<int32_t>(ctx->batch.size()))
            throw ArgError{ TH_ERR_STATE, "no batched result for that many requests" };
        if (n > 0 && (!verts || !faces))
            throw ArgError{ TH_ERR_INVALID_ARGUMENT, "verts or faces array is NULL" };
        for (int32_t i = 0; i < n; ++i)
        {
            if (!ctx->batch[i].has_result)
                throw ArgError{ TH_ERR_STATE, "no batched result at this index" };
            if (ctx->batch[i].info.num_faces > 0 && (!verts[i] || !faces[i]))
                throw ArgError{ TH_ERR_INVALID_ARGUMENT, "verts or faces pointer is NULL" };
        }
        auto st = static_cast<cudaStream_t>(stream);
        BatchState& bs = ctx->bstate;
        const int ns = std::min<int>(n, static_cast<int>(bs.streams.size()));
        const bool recorded = in_capture(st); // export_on
        if (!recorded)
            for (int32_t i = 0; i < n; ++i)
            {
                if (ctx->batch[i].exported)
                    TH_CUDA(cudaStreamWaitEvent(st, ctx->batch[i].done, 0));
                ctx->batch[i].exported = true;
            }
        if (ns > 1)
        {
            // the exports side by side on the batch's streams, joined back into st
            TH_CUDA(cudaEventRecord(bs.fork, st));
            for (int i = 0; i < ns; ++i)
                TH_CUDA(cudaStreamWaitEvent(bs.streams[i], bs.fork, 0));
        }
        for (int32_t i = 0; i < n; ++i)
        {
            HullSlot& s = ctx->batch[i];
            if (s.info.num_faces > 0)
                launch_export(s.plan, s.host->words, verts[i], faces[i], ns > 1 ? bs.streams[i % ns] : st);
        }
        if (ns > 1)
        {
            for (int i = 0; i < ns; ++i)
            {
                TH_CUDA(cudaEventRecord(bs.joins[i], bs.streams[i]));
                TH_CUDA(cudaStreamWaitEvent(st, bs.joins[i], 0));
            }
        }
        if (!recorded)
            for (int32_t i = 0; i < n; ++i)
                TH_CUDA(cudaEventRecord(ctx->batch[i].done, st));
    });
}

} // extern "C"
