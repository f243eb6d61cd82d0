// topology.cu — resident flow topology: inflow count, upstream masks, downstream levels, statistics.
//
// Reference counterparts (ALG/ = source/framework/algorithm/include/lue/framework/algorithm/):
//   inflow count per cell ............ ALG/detail/inflow_count.hpp:9-351 plus the partition input
//                                      cells of ALG/definition/inflow_count.hpp:97-577; on one device
//                                      the whole raster is one domain, so the count is taken over all
//                                      eight neighbours directly (the public inflow_count<uint8> result,
//                                      ALG/definition/inflow_count.hpp:665-726)
//   D8 decoding ...................... ALG/detail/flow_direction.hpp:11-112
#include <cstring>
#include <new>
#include <string>

#include "topology.cuh"
#include "walk.cuh"
#include "window.cuh"

namespace lue_gb300 {

thread_local std::string g_last_error;
static std::atomic<unsigned long long> g_launches{0};

void count_launches(int n) { g_launches.fetch_add((unsigned long long)n, std::memory_order_relaxed); }

void set_error(const std::string& msg) { g_last_error = msg; }

int fail(int status, const std::string& msg)
{
    g_last_error = msg;
    return status;
}

int cuda_status(cudaError_t err, const char* what)
{
    if (err == cudaSuccess) return LUE_GPU_OK;
    if (err == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return fail(LUE_GPU_ENOMEM, std::string(what) + ": " + cudaGetErrorString(err));
    }
    return fail(LUE_GPU_ECUDA, std::string(what) + ": " + cudaGetErrorString(err));
}

// For each cell, which neighbours drain into it; value_policies marks no-data cells with 255
// (ALG/policy/mark_no_data_by_value.hpp).  3 bytes a cell: bound by memory on large rasters and by its latency at
// 2048^2, where nine loads and an index division per cell (k_count_upmask) took 23 us, and this 13.5 us.
template <bool EDGE>
__device__ __forceinline__ void count_window(const uint8_t* __restrict__ fd, int64_t rows, int64_t cols, bool value_policies,
                                             uint8_t* __restrict__ count, uint8_t* __restrict__ upmask)
{
    const WindowAt<EDGE> w(rows, cols);
    if (w.idle()) return;
    unsigned f[kWindowRows + 2], mask[kWindowRows + 2];
    w.load(f, fd, (unsigned)kNoData);
#pragma unroll
    for (int j = 0; j < kWindowRows + 2; ++j) {
        const unsigned west = __shfl_up_sync(0xffffffffu, f[j], 1), east = __shfl_down_sync(0xffffffffu, f[j], 1);
        if (j + 1 <= kWindowRows) mask[j + 1] = (west == 3u ? 1u : 0u) | (f[j] == 2u ? 2u : 0u) | (east == 1u ? 4u : 0u);
        if (j >= 1 && j <= kWindowRows) mask[j] |= (west == 6u ? 8u : 0u) | (east == 4u ? 16u : 0u);
        if (j >= 2) {
            const unsigned m = mask[j - 1] | (west == 9u ? 32u : 0u) | (f[j] == 8u ? 64u : 0u) | (east == 7u ? 128u : 0u);
            if (upmask) w.store(upmask, j - 2, (uint8_t)m);
            w.store(count, j - 2, (uint8_t)(value_policies && f[j - 1] == kNoData ? kNoData : __popc(m)));
        }
    }
}
__global__ void __launch_bounds__(kWindowThreads)
    k_count_window(const uint8_t* __restrict__ fd, int64_t rows, int64_t cols, int value_policies, uint8_t* count,
                   uint8_t* upmask)
{
    if (window_inside(rows, cols)) count_window<false>(fd, rows, cols, value_policies, count, upmask);
    else count_window<true>(fd, rows, cols, value_policies, count, upmask);
}

// The same without windows, for rasters with more rows than a grid of windows holds.
__global__ void __launch_bounds__(256)
    k_count_upmask(const uint8_t* __restrict__ fd, int64_t rows, int64_t cols, int value_policies,
                   uint8_t* __restrict__ count, uint8_t* __restrict__ upmask)
{
    const int64_t n = rows * cols;
    for (int64_t i = grid_stride_begin(); i < n; i += grid_stride()) {
        int64_t r = i / cols, c = i - r * cols;
        uint8_t code = __ldg(fd + i);
        unsigned mask = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            int64_t rn = r + nb_dr(k), cn = c + nb_dc(k);
            if (rn >= 0 && rn < rows && cn >= 0 && cn < cols && __ldg(fd + rn * cols + cn) == nb_inflow_code(k))
                mask |= 1u << k;
        }
        if (upmask) upmask[i] = (uint8_t)mask;
        count[i] = (value_policies && code == kNoData) ? kNoData : (uint8_t)__popc(mask);
    }
}

struct LevelVisitor {
    const uint8_t* upmask;
    int32_t* level;
    int64_t cols;
    __device__ void enter(int64_t c)
    {
        unsigned m = __ldg(upmask + c);
        int32_t lv = -1;
        while (m) {
            int k = __ffs(m) - 1;
            m &= m - 1;
            int32_t u = load_cg(level + c + nb_dr(k) * cols + nb_dc(k));
            lv = u > lv ? u : lv;
        }
        level[c] = lv + 1;
    }
    __device__ void no_data(int64_t) {}
};

static void launch_count(const uint8_t* fd, int64_t rows, int64_t cols, int value_policies, uint8_t* count, uint8_t* upmask,
                         cudaStream_t stream)
{
    dim3 grid;
    unsigned threads = 0;
    if (window_grid(rows, cols, grid, threads))
        k_count_window<<<grid, threads, 0, stream>>>(fd, rows, cols, value_policies, count, upmask);
    else
        k_count_upmask<<<grid_for(rows * cols, 256), 256, 0, stream>>>(fd, rows, cols, value_policies, count, upmask);
}

__global__ void k_fill_i32(int32_t* p, int64_t n, int32_t v)
{
    for (int64_t i = grid_stride_begin(); i < n; i += grid_stride()) p[i] = v;
}

// stats: [valid, ridge, outlet, sink, cycle, max_level]
__global__ void __launch_bounds__(256)
    k_stats(const uint8_t* fd, const uint8_t* count, const int32_t* level, int64_t rows, int64_t cols,
            unsigned long long* stats)
{
    const int64_t n = rows * cols;
    unsigned long long v = 0, ridge = 0, outlet = 0, sink = 0, cycle = 0;
    int maxl = 0;
    for (int64_t i = grid_stride_begin(); i < n; i += grid_stride()) {
        uint8_t code = fd[i];
        if (code == kNoData) continue;
        ++v;
        if (count[i] == 0) ++ridge;
        int dr, dc;
        if (!d8_offset(code, dr, dc)) {
            ++sink;
        } else {
            int64_t r = i / cols + dr, c = i % cols + dc;
            if (r < 0 || r >= rows || c < 0 || c >= cols) ++outlet;
        }
        if (level[i] < 0) ++cycle;
        else if (level[i] > maxl) maxl = level[i];
    }
    for (int off = 16; off > 0; off >>= 1) {
        v += __shfl_down_sync(0xffffffffu, v, off);
        ridge += __shfl_down_sync(0xffffffffu, ridge, off);
        outlet += __shfl_down_sync(0xffffffffu, outlet, off);
        sink += __shfl_down_sync(0xffffffffu, sink, off);
        cycle += __shfl_down_sync(0xffffffffu, cycle, off);
        int o = __shfl_down_sync(0xffffffffu, maxl, off);
        maxl = o > maxl ? o : maxl;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(stats + 0, v);
        atomicAdd(stats + 1, ridge);
        atomicAdd(stats + 2, outlet);
        atomicAdd(stats + 3, sink);
        atomicAdd(stats + 4, cycle);
        atomicMax(stats + 5, (unsigned long long)maxl);
    }
}

// The handle's stage_flow_error word (with core->stage_mutex held).  Pinned memory takes 110 us to allocate and 160 us
// to release, more than a small raster's build: only handles that can come to run a stage engine launch have one.
// A call that is being captured cannot allocate it, so it is there before: from the build of the stage structures on,
// for the handle that builds them, and from a clone on for both handles (either may then use what the other built).
int stage_flag(lue_gpu_topology* t)
{
    if (t->stage_flow_error) return LUE_GPU_OK;
    int* flag = nullptr;
    if (int rc = cuda_status(cudaHostAlloc(&flag, sizeof(int), cudaHostAllocDefault), "scratch flag")) return rc;
    *flag = 0;
    t->stage_flow_error = flag;
    return LUE_GPU_OK;
}

namespace {

struct ScratchPlan {
    size_t count, lo;
    TileScratchPlan tiles;
};

void plan_scratch(int64_t n, Arena& a, ScratchPlan* p)
{
    p->count = a.add(words_for(n) * 4);
    p->lo = a.add(n * (int64_t)sizeof(float));
}

void take_scratch(lue_gpu_topology* t, Arena& a, const ScratchPlan& p)
{
    t->work_count = a.at<uint32_t>(p.count);
    t->lo = a.at<float>(p.lo);
    t->scratch_bytes = (int64_t)a.bytes();
    if (t->core->tiles) tile_scratch_take(a, p.tiles, &t->tile_scratch);
}

}  // namespace

int allocate_scratch(lue_gpu_topology* t)
{
    Arena a;
    ScratchPlan p{};
    plan_scratch(t->core->n, a, &p);
    if (t->core->tiles) tile_scratch_plan(t->core->tiles->ntiles, t->core->tiles->nexit, a, &p.tiles);
    if (int rc = cuda_status(a.allocate(), "scratch")) return rc;
    t->arena = a.release();
    take_scratch(t, a, p);
    if (!t->core->tiles) return LUE_GPU_OK;
    if (int rc = tile_scratch_clear(a, p.tiles, nullptr)) return rc;
    return cuda_status(cudaStreamSynchronize(nullptr), "tile scratch");  // the calls' streams may not wait for it
}

// The first build of a topology, in two allocations (its own and the handle's scratch, in which the build's arrays lie
// too): cudaMalloc takes 35 us and cudaFree 30 to 60 us whatever the size, and with one of each for every array (45 and
// 35) they took half of the build of a 2048^2 raster.  With `tiles`, *done stays false, and nothing is kept, when
// the raster has more exits than the tile engine takes.  A raster with a flow cycle has its levels from the tiles too
// (with one 2 x 2 cycle at 256^2 / 2048^2 / 8192^2: 0.42 / 0.93 / 5.4 ms; by a walk over its cells after the attempt with
// tiles 1.5 / 9.6 / 54 ms), and keeps no tile structures.
static int build_topology(lue_gpu_topology* t, const uint8_t* flow_direction, bool tiles, cudaStream_t stream, bool* done,
                          unsigned long long* hstats)
{
    TopologyCore* core = t->core;
    const int64_t n = core->n, padded = words_for(n) * 4;
    int rc = 0;
    Arena a, s;
    TileCorePlan tile_plan{};
    ScratchPlan scratch{};
    const size_t fd = a.add(padded), count = a.add(padded), upmask = a.add(padded),
                 level = a.add(n * (int64_t)sizeof(int32_t));
    const size_t base = a.bytes();
    core->bytes = (int64_t)base;
    plan_scratch(n, s, &scratch);
    *done = false;
    if (tiles) {
        int64_t exits = 0;
        if ((rc = tile_exit_bound(flow_direction, core->rows, core->cols, stream, &exits))) return rc;
        if (tile_core_plan(core->rows, core->cols, exits, a, &tile_plan, s, &scratch.tiles)) return LUE_GPU_OK;
    }
    if ((rc = cuda_status(a.allocate(), "topology"))) return rc;
    if ((rc = cuda_status(s.allocate(), "scratch"))) return rc;
    core->fd = a.at<uint8_t>(fd);
    core->count = a.at<uint8_t>(count);
    core->upmask = a.at<uint8_t>(upmask);
    core->level = a.at<int32_t>(level);
    // the last word is padded with no-data
    if ((rc = cuda_status(cudaMemsetAsync(core->fd + padded - 4, kNoData, 4, stream), "memset"))) return rc;
    if ((rc = cuda_status(cudaMemcpyAsync(core->fd, flow_direction, n, cudaMemcpyDeviceToDevice, stream),
                          "copy flow direction")))
        return rc;
    if ((rc = cuda_status(cudaMemsetAsync(core->count + padded - 4, 0, 4, stream), "memset"))) return rc;
    launch_count(core->fd, core->rows, core->cols, 1, core->count, core->upmask, stream);
    if (tiles) {
        rc = tile_core_build(core, a, tile_plan, s, scratch.tiles, stream, hstats);
        if (rc) return rc == LUE_GPU_ECUDA || rc == LUE_GPU_ENOMEM ? rc : LUE_GPU_OK;
        core->bytes += (int64_t)tile_plan.bytes;
        Arena a0, s0;  // without the tiles: the same arrays come first in both
        if (!core->tiles) {
            ScratchPlan plain{};
            a0.add((int64_t)base);
            plan_scratch(n, s0, &plain);
            if (!cuda_status(a0.allocate(), "topology") && !cuda_status(s0.allocate(), "scratch")) {
                if ((rc = cuda_status(cudaMemcpyAsync(a0.at<char>(0), a.at<char>(0), base, cudaMemcpyDeviceToDevice, stream),
                                      "topology")) ||
                    (rc = cuda_status(cudaStreamSynchronize(stream), "topology")))
                    return rc;
                core->bytes = (int64_t)base;
                a.swap(a0);
                s.swap(s0);
                core->fd = a.at<uint8_t>(fd);
                core->count = a.at<uint8_t>(count);
                core->upmask = a.at<uint8_t>(upmask);
                core->level = a.at<int32_t>(level);
            }
        }
    } else {  // levels by a walk over the cells
        uint32_t* work = s.at<uint32_t>(scratch.count);
        unsigned long long* dstats = nullptr;
        Arena d;
        const size_t stats = d.add(6 * sizeof(unsigned long long));
        if ((rc = cuda_status(d.allocate(), "topology stats"))) return rc;
        dstats = d.at<unsigned long long>(stats);
        k_fill_i32<<<grid_for(n, 256), 256, 0, stream>>>(core->level, n, -1);
        if ((rc = cuda_status(cudaMemcpyAsync(work, core->count, padded, cudaMemcpyDeviceToDevice, stream), "reset counters")))
            return rc;
        WalkGrid g{core->fd, core->count, work, core->rows, core->cols, n};
        LevelVisitor v{core->upmask, core->level, core->cols};
        k_walk<<<grid_all(n, 256), 256, 0, stream>>>(g, v);
        if ((rc = cuda_status(cudaMemsetAsync(dstats, 0, d.bytes(), stream), "memset"))) return rc;
        k_stats<<<grid_for(n, 256), 256, 0, stream>>>(core->fd, core->count, core->level, core->rows, core->cols, dstats);
        if ((rc = cuda_status(cudaGetLastError(), "topology kernels"))) return rc;
        if ((rc = cuda_status(cudaMemcpyAsync(hstats, dstats, 6 * sizeof *hstats, cudaMemcpyDeviceToHost, stream), "stats")))
            return rc;
        if ((rc = cuda_status(cudaStreamSynchronize(stream), "topology_create"))) return rc;
    }
    take_scratch(t, s, scratch);
    core->arena = a.release();
    t->arena = s.release();
    *done = true;
    return LUE_GPU_OK;
}

static void free_core(TopologyCore* core)
{
    if (!core) return;
    cudaFree(core->arena);
    cudaFree(core->order);
    delete core->tiles;
    stage_core_free(core->stages);
    path_core_free(core->paths);
    delete core;
}

static void free_handle(lue_gpu_topology* t)
{
    if (!t) return;
    cudaFree(t->arena);
    cudaFree(t->history);
    cudaFree(t->planes);
    stage_buffers_free(t);
    path_buffers_free(t);
    cudaFreeHost(t->stage_flow_error);
    if (t->core && --t->core->refs == 0) free_core(t->core);
    delete t;
}

}  // namespace lue_gb300

using namespace lue_gb300;

extern "C" int lue_gpu_abi_version(void) { return LUE_GPU_ABI_VERSION; }

extern "C" unsigned long long lue_gpu_kernel_launches(void) { return g_launches.load(); }

extern "C" const char* lue_gpu_last_error(void) { return g_last_error.c_str(); }

extern "C" int lue_gpu_topology_create(const uint8_t* flow_direction, int64_t rows, int64_t cols,
                                       int64_t partition_rows, int64_t partition_cols, void* stream_,
                                       lue_gpu_topology** out)
{
    if (!out) return fail(LUE_GPU_EINVAL, "topology_create: NULL result pointer");
    *out = nullptr;
    if (!flow_direction) return fail(LUE_GPU_EINVAL, "topology_create: NULL flow direction");
    if (rows <= 0 || cols <= 0) return fail(LUE_GPU_EINVAL, "topology_create: array shape must not be empty");
    if (partition_rows <= 0 || partition_cols <= 0)
        return fail(LUE_GPU_EINVAL, "topology_create: partition shape must not be empty");
    if (partition_rows > rows || partition_cols > cols)
        return fail(LUE_GPU_EINVAL, "topology_create: partition shape must not exceed the array shape");
    if (rows > (int64_t(1) << 31) || cols > (int64_t(1) << 31) || rows * cols > (int64_t(1) << 40))
        return fail(LUE_GPU_ERANGE, "topology_create: array too large");
    cudaStream_t stream = (cudaStream_t)stream_;
    auto* core = new (std::nothrow) TopologyCore();
    auto* t = new (std::nothrow) lue_gpu_topology();
    if (!core || !t) {
        delete core;
        delete t;
        return fail(LUE_GPU_ENOMEM, "topology_create: host allocation");
    }
    t->core = core;
    core->rows = rows;
    core->cols = cols;
    core->prow = partition_rows;
    core->pcol = partition_cols;
    core->n = rows * cols;
    // the tiles need 32-bit cell indices; their build gives the levels and statistics
    bool done = false;
    unsigned long long hstats[6] = {0, 0, 0, 0, 0, 0};
    int rc = LUE_GPU_OK, tiles = LUE_GPU_OK;
    if (core->n < (int64_t(1) << 32)) {
        // without a grid or the memory for the tiles only rasters with cycles, which have none, are taken
        if (tile_rows_fit(rows)) {
            tiles = build_topology(t, flow_direction, true, stream, &done, hstats);
            if (tiles == LUE_GPU_ECUDA) rc = tiles;
        } else {
            tiles = LUE_GPU_ECUDA;
        }
    }
    if (!rc && !done) rc = build_topology(t, flow_direction, false, stream, &done, hstats);
    if (!rc && tiles && hstats[4] == 0) rc = fail(tiles, "topology_create: no memory or grid for the tile structures");
    if (rc) {
        free_handle(t);
        return rc;
    }
    core->stats.rows = rows;
    core->stats.cols = cols;
    core->stats.partition_rows = partition_rows;
    core->stats.partition_cols = partition_cols;
    core->stats.valid_cells = (int64_t)hstats[0];
    core->stats.ridge_cells = (int64_t)hstats[1];
    core->stats.outlet_cells = (int64_t)hstats[2];
    core->stats.sink_cells = (int64_t)hstats[3];
    core->stats.cycle_cells = (int64_t)hstats[4];
    core->stats.max_level = (int64_t)hstats[5];
    if (core->tiles) {
        core->stats.tile_exits = core->tiles->nexit;
        core->stats.exit_forest_depth = core->tiles->max_depth;
    }
    *out = t;
    return LUE_GPU_OK;
}

extern "C" int lue_gpu_topology_clone(const lue_gpu_topology* topology, lue_gpu_topology** clone)
{
    if (!topology || !clone) return fail(LUE_GPU_EINVAL, "topology_clone: NULL argument");
    *clone = nullptr;
    auto* t = new (std::nothrow) lue_gpu_topology();
    if (!t) return fail(LUE_GPU_ENOMEM, "topology_clone: host allocation");
    t->core = topology->core;
    t->core->refs++;
    int rc = allocate_scratch(t);
    if (!rc) {
        std::lock_guard<std::mutex> lock(t->core->stage_mutex);
        rc = stage_flag(t);
        if (!rc) rc = stage_flag(const_cast<lue_gpu_topology*>(topology));
    }
    if (rc) {
        free_handle(t);
        return rc;
    }
    *clone = t;
    return LUE_GPU_OK;
}

extern "C" int lue_gpu_topology_prepare(lue_gpu_topology* topology, void* stream)
{
    if (!topology) return fail(LUE_GPU_EINVAL, "topology_prepare: NULL topology");
    if (int rc = path_prepare(topology, (cudaStream_t)stream)) return rc;
    return stage_prepare(topology, (cudaStream_t)stream);
}

extern "C" int lue_gpu_topology_destroy(lue_gpu_topology* topology)
{
    if (!topology) return fail(LUE_GPU_EINVAL, "topology_destroy: NULL topology");
    free_handle(topology);
    return LUE_GPU_OK;
}

extern "C" int lue_gpu_topology_get_stats(const lue_gpu_topology* topology, lue_gpu_topology_stats* stats)
{
    if (!topology || !stats) return fail(LUE_GPU_EINVAL, "topology_stats: NULL argument");
    *stats = topology->core->stats;
    stats->device_bytes = topology->core->bytes + topology->scratch_bytes;
    return LUE_GPU_OK;
}

extern "C" int lue_gpu_inflow_count_u8(const lue_gpu_topology* topology, int value_policies, uint8_t* inflow_count,
                                       void* stream_)
{
    if (!topology || !inflow_count) return fail(LUE_GPU_EINVAL, "inflow_count: NULL argument");
    cudaStream_t stream = (cudaStream_t)stream_;
    const TopologyCore* core = topology->core;
    if (value_policies) {
        return cuda_status(
            cudaMemcpyAsync(inflow_count, core->count, core->n, cudaMemcpyDeviceToDevice, stream), "inflow_count");
    }
    launch_count(core->fd, core->rows, core->cols, 0, inflow_count, nullptr, stream);
    return cuda_status(cudaGetLastError(), "inflow_count");
}

extern "C" int lue_gpu_downstream_level_i32(const lue_gpu_topology* topology, int32_t* level, void* stream_)
{
    if (!topology || !level) return fail(LUE_GPU_EINVAL, "downstream_level: NULL argument");
    const TopologyCore* core = topology->core;
    return cuda_status(cudaMemcpyAsync(level, core->level, core->n * sizeof(int32_t), cudaMemcpyDeviceToDevice,
                                       (cudaStream_t)stream_),
                       "downstream_level");
}
