// path_route.cu — the path engine (see path_route.cuh): heavy-path layout of the flow forest, built once
// per raster, and accu_threshold / accu_fraction / accu_capacity / accu_trigger (float32) as one prefix scan
// per path level.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>

#include "route_walk_visitors.cuh"
#include "topology.cuh"

namespace lue_gb300 {

// ---------------------------------------------------------------------------------------------------
// Build
// ---------------------------------------------------------------------------------------------------

// Upstream-first walk: per cell the cells upstream of it (itself included), its heavy upstream neighbour
// (the one with most cells upstream, the first in neighbour order on ties; 8: none), the cells above it
// on its path, and its path level (the largest number of light edges on a flow path ending at it).
struct PathVisitor {
    const uint8_t* upmask;
    int32_t* size;
    int32_t* dtop;
    int32_t* plev;
    int32_t* heavy;
    int64_t cols;
    __device__ void enter(int64_t c)
    {
        const unsigned m = __ldg(upmask + c);
        int32_t sz = 1, best = -1;
        int hk = 8;
        for (unsigned mm = m; mm; mm &= mm - 1) {
            const int k = __ffs(mm) - 1;
            const int32_t s = load_cg(size + c + nb_dr(k) * cols + nb_dc(k));
            sz += s;
            if (s > best) {
                best = s;
                hk = k;
            }
        }
        int32_t lv = 0, dt = 0;
        for (unsigned mm = m; mm; mm &= mm - 1) {
            const int k = __ffs(mm) - 1;
            const int64_t u = c + nb_dr(k) * cols + nb_dc(k);
            const int32_t l = load_cg(plev + u);
            if (k == hk) {
                lv = max(lv, l);
                dt = load_cg(dtop + u) + 1;
            } else {
                lv = max(lv, l + 1);
            }
        }
        size[c] = sz;
        plev[c] = lv;
        dtop[c] = dt;
        heavy[c] = hk;
    }
    __device__ void no_data(int64_t) {}
};

// Neighbour slot k of a cell's upstream neighbour that drains into it with D8 code `code`.
__device__ __forceinline__ int inflow_slot(uint8_t code)
{
    switch (code) {
        case 3: return 0;
        case 2: return 1;
        case 1: return 2;
        case 6: return 3;
        case 4: return 4;
        case 9: return 5;
        case 8: return 6;
        case 7: return 7;
        default: return -1;
    }
}

// next[c]: the cell below c on its path (c itself at the bottom), -1 for no-data.
__global__ void k_path_next(const uint8_t* fd, const int32_t* heavy, int64_t rows, int64_t cols, int64_t n,
                            int32_t* next)
{
    for (int64_t c = grid_stride_begin(); c < n; c += grid_stride()) {
        const uint8_t code = __ldg(fd + c);
        if (code == kNoData) {
            next[c] = -1;
            continue;
        }
        const int64_t r = c / cols, col = c - r * cols;
        int64_t d = 0;
        int32_t v = (int32_t)c;
        if (downstream(code, r, col, rows, cols, d) && __ldg(fd + d) != kNoData && heavy[d] == inflow_slot(code))
            v = (int32_t)d;
        next[c] = v;
    }
}

// One round of pointer jumping: next[c] = next[next[c]] (in place: a value read from a cell that has
// already jumped this round is still a cell of the same path, at or above the bottom).
__global__ void k_path_jump(int32_t* next, int64_t n)
{
    for (int64_t c = grid_stride_begin(); c < n; c += grid_stride()) {
        const int32_t v = next[c];
        if (v >= 0) next[c] = next[v];
    }
}

constexpr int kPathMaxLevels = 254;
constexpr int kPathTile = 64;                            // paths are grouped by the 64 x 64 tile of their bottom
constexpr int kPathTileCells = kPathTile * kPathTile;

// key[c] = path level of c if c is the bottom of its path, else 255; stats: [0] largest level,
// [1] longest path, [2] cells whose next is not a bottom (must be 0), [3 + l] longest path of level l;
// cells[l]: cells of the paths of level l.
__global__ void __launch_bounds__(256) k_path_keys(const int32_t* next, const int32_t* plev, const int32_t* dtop,
                                                   int64_t n, uint8_t* key, int* stats, unsigned long long* cells)
{
    __shared__ unsigned s_cells[256];
    __shared__ int s_longest[256];
    s_cells[threadIdx.x] = 0;
    s_longest[threadIdx.x] = 0;
    __syncthreads();
    int lmax = -1, bad = 0;
    for (int64_t c = grid_stride_begin(); c < n; c += grid_stride()) {
        const int32_t v = next[c];
        uint8_t k = 255;
        if (v >= 0) {
            if (next[v] != v) ++bad;
            if (v == c) {
                const int l = min(plev[c], kPathMaxLevels), len = dtop[c] + 1;
                k = (uint8_t)l;
                lmax = max(lmax, l);
                atomicMax(&s_longest[l], len);
                atomicAdd(&s_cells[l], (unsigned)len);
            }
        }
        key[c] = k;
    }
    lmax = __reduce_max_sync(0xffffffffu, lmax);
    bad = __reduce_add_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        if (lmax >= 0) atomicMax(stats, lmax);
        if (bad) atomicAdd(stats + 2, bad);
    }
    __syncthreads();
    if (s_cells[threadIdx.x]) {
        atomicAdd(cells + threadIdx.x, (unsigned long long)s_cells[threadIdx.x]);
        atomicMax(stats + 3 + threadIdx.x, s_longest[threadIdx.x]);
        atomicMax(stats + 1, s_longest[threadIdx.x]);
    }
}

// Exclusive sum over a CTA of NT threads; ends with a block barrier.
template <int NT>
__device__ __forceinline__ long long block_excl_sum(long long v, long long* s_warp, long long& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long x = v;
    for (int d = 1; d < 32; d <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        long long w = lane < NT / 32 ? s_warp[lane] : 0;
        for (int d = 1; d < 32; d <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += y;
        }
        if (lane < NT / 32) s_warp[lane] = w;
    }
    __syncthreads();
    total = s_warp[NT / 32 - 1];
    const long long before = warp ? s_warp[warp - 1] : 0;
    __syncthreads();
    return before + x - v;
}

struct PathGeom {
    int64_t rows, cols, tcols, ntiles;
    __device__ __forceinline__ bool cell(int64_t tile, int loc, int64_t& c) const
    {
        const int64_t r = tile / tcols * kPathTile + loc / kPathTile, col = tile % tcols * kPathTile + loc % kPathTile;
        c = r * cols + col;
        return r < rows && col < cols;
    }
};

// Per tile and level: the cells of the paths whose bottom lies in the tile, counts[level * ntiles + tile].
__global__ void __launch_bounds__(256) k_paths_count(const uint8_t* key, const int32_t* dtop, PathGeom g, int levels,
                                                     int32_t* counts)
{
    __shared__ int s_cells[kPathMaxLevels + 1];
    for (int i = threadIdx.x; i < levels; i += 256) s_cells[i] = 0;
    __syncthreads();
    const int64_t tile = blockIdx.x;
    for (int i = threadIdx.x; i < kPathTileCells; i += 256) {
        int64_t c;
        if (g.cell(tile, i, c) && key[c] != 255) atomicAdd(&s_cells[key[c]], dtop[c] + 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < levels; i += 256) counts[i * g.ntiles + tile] = s_cells[i];
}

// counts -> the first position of each level's paths of each tile (a CTA per level; starts[level]: the level's
// first position).
__global__ void __launch_bounds__(1024) k_paths_scan(int32_t* counts, int64_t ntiles, const int32_t* starts)
{
    __shared__ long long s_warp[32];
    int32_t* x = counts + blockIdx.x * ntiles;
    const int64_t per = (ntiles + 1023) / 1024;
    const int64_t t0 = min(ntiles, (int64_t)threadIdx.x * per), t1 = min(ntiles, t0 + per);
    long long s = 0, total = 0;
    for (int64_t t = t0; t < t1; ++t) s += x[t];
    long long v = starts[blockIdx.x] + block_excl_sum<1024>(s, s_warp, total);
    for (int64_t t = t0; t < t1; ++t) {
        const int32_t y = x[t];
        x[t] = (int32_t)v;
        v += y;
    }
}

// Per tile: its paths sorted by level and cell, and with that their positions.  base[b]: first position of the
// path whose bottom is b.
__global__ void __launch_bounds__(256)
    k_paths_assign(const uint8_t* key, const int32_t* dtop, PathGeom g, const int32_t* counts, int32_t* base)
{
    __shared__ uint32_t s_key[kPathTileCells];
    __shared__ int s_pos[kPathMaxLevels + 1];
    __shared__ long long s_warp[8];
    __shared__ int s_n;
    const int64_t tile = blockIdx.x;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < kPathTileCells; i += 256) {
        int64_t c;
        if (g.cell(tile, i, c) && key[c] != 255) s_key[atomicAdd(&s_n, 1)] = ((unsigned)key[c] << 12) | (unsigned)i;
    }
    __syncthreads();
    const int n = s_n;
    int size = 256;
    while (size < n) size <<= 1;
    for (int i = n + threadIdx.x; i < size; i += 256) s_key[i] = 0xFFFFFFFFu;
    __syncthreads();
    for (int k = 2; k <= size; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < size; i += 256) {
                const int o = i ^ j;
                if (o > i) {
                    const uint32_t a = s_key[i], b = s_key[o];
                    if ((a > b) == ((i & k) == 0)) {
                        s_key[i] = b;
                        s_key[o] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
    const int per = size / 256, i0 = threadIdx.x * per;
    long long sum = 0, total = 0;
    for (int i = i0; i < min(n, i0 + per); ++i) {
        int64_t c;
        g.cell(tile, (int)(s_key[i] & 0xFFFu), c);
        sum += dtop[c] + 1;
    }
    const int before = (int)block_excl_sum<256>(sum, s_warp, total);
    int at = before;
    for (int i = i0; i < min(n, i0 + per); ++i) {
        int64_t c;
        g.cell(tile, (int)(s_key[i] & 0xFFFu), c);
        if (i == 0 || (s_key[i - 1] >> 12) != (s_key[i] >> 12)) s_pos[s_key[i] >> 12] = at;
        at += dtop[c] + 1;
    }
    __syncthreads();
    at = before;
    for (int i = i0; i < min(n, i0 + per); ++i) {
        int64_t c;
        g.cell(tile, (int)(s_key[i] & 0xFFFu), c);
        const unsigned l = s_key[i] >> 12;
        base[c] = counts[l * g.ntiles + tile] + at - s_pos[l];
        at += dtop[c] + 1;
    }
}

// order and the number of light upstream neighbours by position (order starts as all ones: no cell).  bad counts
// positions outside [0, npos) and positions written twice; the build then fails instead of handing on a wrong
// layout.
__global__ void k_path_place(const int32_t* next, const int32_t* base, const int32_t* dtop, const int32_t* heavy,
                             const uint8_t* upmask, int64_t n, int64_t npos, int64_t slot_base, int32_t* order,
                             uint8_t* light, int* bad)
{
    int nbad = 0;
    for (int64_t c = grid_stride_begin(); c < n; c += grid_stride()) {
        const int32_t b = next[c];
        if (b < 0) continue;
        const int32_t dt = dtop[c];
        const int64_t pos = (int64_t)base[b] + dt;
        if (pos < 0 || pos >= npos) {
            ++nbad;
            continue;
        }
        const int32_t old = atomicExch(order + pos, (int32_t)((uint32_t)c | (dt == 0 ? 0x80000000u : 0u)));
        if (old != -1) ++nbad;
        const int hk = heavy[c];
        const unsigned m = __ldg(upmask + c) & ~(hk < 8 ? 1u << hk : 0u);
        if (pos >= slot_base) light[pos - slot_base] = (uint8_t)__popc(m);
        else if (m) ++nbad;  // a cell of level 0 has no light inflow
    }
    if (nbad) atomicAdd(bad, nbad);
}

// Positions that no cell took.
__global__ void k_path_unwritten(const int32_t* order, int64_t npos, int* bad)
{
    int nbad = 0;
    for (int64_t i = grid_stride_begin(); i < npos; i += grid_stride()) nbad += order[i] == -1;
    if (nbad) atomicAdd(bad, nbad);
}

constexpr int kLightPer = 32;                  // positions per thread
constexpr int kLightBlock = 256 * kLightPer;   // positions per CTA

// slot_first = exclusive sums of the light neighbour counts: sums of blocks, their scan, the positions.
__global__ void __launch_bounds__(256) k_light_sums(const uint8_t* light, int64_t n, long long* bsum)
{
    __shared__ long long s_warp[8];
    const int64_t i0 = (int64_t)blockIdx.x * kLightBlock + (int64_t)threadIdx.x * kLightPer;
    long long s = 0;
    for (int64_t i = i0; i < min(n, i0 + kLightPer); ++i) s += light[i];
    long long total = 0;
    block_excl_sum<256>(s, s_warp, total);
    if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}
__global__ void __launch_bounds__(1024) k_light_scan(long long* bsum, int64_t nblk)
{
    __shared__ long long s_warp[32];
    const int64_t per = (nblk + 1023) / 1024;
    const int64_t b0 = min(nblk, (int64_t)threadIdx.x * per), b1 = min(nblk, b0 + per);
    long long s = 0;
    for (int64_t b = b0; b < b1; ++b) s += bsum[b];
    long long total = 0;
    long long x = block_excl_sum<1024>(s, s_warp, total);
    for (int64_t b = b0; b < b1; ++b) {
        const long long v = bsum[b];
        bsum[b] = x;
        x += v;
    }
    if (threadIdx.x == 0) bsum[nblk] = total;
}
__global__ void __launch_bounds__(256) k_light_apply(const uint8_t* light, int64_t n, const long long* bsum,
                                                     int64_t nblk, int32_t* first)
{
    __shared__ long long s_warp[8];
    const int64_t i0 = (int64_t)blockIdx.x * kLightBlock + (int64_t)threadIdx.x * kLightPer;
    long long s = 0;
    for (int64_t i = i0; i < min(n, i0 + kLightPer); ++i) s += light[i];
    long long total = 0;
    long long x = block_excl_sum<256>(s, s_warp, total) + bsum[blockIdx.x];
    for (int64_t i = i0; i < min(n, i0 + kLightPer); ++i) {
        first[i] = (int32_t)x;
        x += light[i];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) first[n] = (int32_t)bsum[nblk];
}

// The slot that takes each path's outflow, at the position of its bottom: that of the bottom among the light
// neighbours of the cell below.
__global__ void k_path_slots(const uint8_t* fd, const uint8_t* upmask, const uint8_t* key, const int32_t* next,
                             const int32_t* base, const int32_t* dtop, const int32_t* heavy,
                             const int32_t* slot_first, int64_t slot_base, int64_t rows, int64_t cols,
                             int32_t* path_slot, int* bad)
{
    for (int64_t c = grid_stride_begin(); c < rows * cols; c += grid_stride()) {
        if (key[c] == 255) continue;
        const uint8_t code = __ldg(fd + c);
        int32_t slot = -1;
        int64_t d = 0;
        if (downstream(code, c / cols, c % cols, rows, cols, d) && __ldg(fd + d) != kNoData) {
            const int64_t pos = (int64_t)base[next[d]] + dtop[d];
            const int k = inflow_slot(code), hk = heavy[d];
            const unsigned m = __ldg(upmask + d) & ~(hk < 8 ? 1u << hk : 0u);
            if (pos >= slot_base && k >= 0 && ((m >> k) & 1u))
                slot = slot_first[pos - slot_base] + __popc(m & ((1u << k) - 1u));
            else
                atomicAdd(bad, 1);
        }
        path_slot[base[c] + dtop[c]] = slot;
    }
}

// The first path top at or after position s (p1 if none), for every lane of a warp.
__device__ __forceinline__ int64_t next_top(const int32_t* order, int64_t s, int64_t p1)
{
    const int lane = threadIdx.x & 31;
    for (int64_t pos = s; pos < p1; pos += 32) {
        const unsigned m = __ballot_sync(0xffffffffu, pos + lane < p1 && __ldg(order + pos + lane) < 0);
        if (m) return pos + __ffs(m) - 1;
    }
    return p1;
}

// One warp per cut of a level's positions: every `step` positions, moved to the next path top.
__global__ void k_path_cuts(const int32_t* order, int64_t p0, int64_t p1, int64_t step, int64_t ncut, int32_t* cut)
{
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i > ncut) return;
    const int64_t at = i == 0 ? p0 : next_top(order, min(p0 + i * step, p1), p1);
    if ((threadIdx.x & 31) == 0) cut[i] = (int32_t)at;
}

// Position arrays are padded to whole 8-position chunks plus one chunk, for the vector loads of the
// per-call kernels.
static int64_t path_padded(int64_t npos) { return ((npos + 7) / 8 + 1) * 8; }

// Positions per thread of a level's scan.  Level 0: 4 from 2^20 positions on (2 and 8 were slower there).  The levels
// above wait for memory more than they compute (0.97 instructions per cycle with four positions a thread), and read
// their first slots with their inputs when two positions leave the registers for it: 2 from 2^18 positions on
// (accu_threshold at 8192^2 / 16384^2 in us: four positions 1963 / 6928, two 1803 / 6661, two and the shorter CTA
// ranges below 1735 / 6445; one: 1908 at 8192^2).  Small levels: 1, short chains of dependent loads per thread.
constexpr int64_t kPathSmallLevel = 1 << 20, kPathTinyLevel = 1 << 18;
static int path_per(int level, int64_t n)
{
    if (level > 0) return n < kPathTinyLevel ? 1 : 2;
    return n < kPathSmallLevel ? 1 : 4;
}

// A level scans without look-back when its longest path is at most this many positions.
static int path_free_longest(int per) { return per == 1 ? 2 * kPathThreads : 8 * kPathThreads; }

// Positions of a CTA's range in such a level, cut at path tops.  Level 0: two chunks less a sixteenth, as a range runs on
// to the next top (accu_threshold at 8192^2: 1.2 % faster than two whole chunks; one chunk leaves most ranges a second
// one that is nearly empty, 11.3 ms at 16384^2, and four lengthen the serial part of a CTA, 6.8 ms against 6.6).  Large
// levels above: one chunk, more CTAs to wait on memory at once (two: 6661 us).  Small levels, which cannot fill
// the GPU: half a chunk, so most ranges are one chunk and the launch is over sooner (accu_fraction at 2311 x 1501 119 ->
// 100 us, accu_trigger at 1500^2 161 -> 134 us; a quarter: 99 and 135).
static int64_t path_cut_step(int level, int64_t n)
{
    const int64_t T = (int64_t)kPathThreads * path_per(level, n);
    if (n < kPathTinyLevel) return T / 2;
    return level > 0 ? T : 2 * T - T / 16;
}

// From this many cells on, the two results of a rule are collected by position and spread over the raster by a kernel of
// its own (k_path_spread).  Below, the raster stays in L2, where partial writes cost little (accu_threshold 2048 x
// 2500: 183 us straight, 194 spread; 2600 x 2700: 247 and 241; 2900^2: 288 and 271; 4000 x 4100: 528 and 460; 8192^2:
// 1746 and 1415; 16384^2: 6461 and 4959).  accu has one result of 8 bytes, where it is slower at every size (8192^2: 1779
// and 1912).  LUE_GB300_PATH_SPREAD: another limit (test hook).
constexpr int64_t kPathSpreadCells = int64_t(1) << 23;
static int64_t path_spread_cells()
{
    const char* e = getenv("LUE_GB300_PATH_SPREAD");
    return e ? atoll(e) : kPathSpreadCells;
}

__global__ void k_path_at(const int32_t* order, int64_t npos, int32_t* at)
{
    for (int64_t i = grid_stride_begin(); i < npos; i += grid_stride()) at[order[i] & 0x7fffffff] = (int32_t)i;
}

void path_core_free(PathCore* pc)
{
    if (!pc) return;
    cudaFree(pc->at);
    cudaFree(pc->order);
    cudaFree(pc->path_slot);
    cudaFree(pc->slot_first);
    cudaFree(pc->cut);
    delete pc;
}

// The positions of the cells, built on the first call that spreads its results.  Without the memory for them the
// levels write straight to the raster.
static int path_at_build(const TopologyCore* core, PathCore* pc, cudaStream_t stream)
{
    const int64_t n = core->n;
    pc->at_decided = true;
    if (n < path_spread_cells()) return LUE_GPU_OK;
    int rc = cuda_status(cudaMalloc(&pc->at, n * sizeof(int32_t)), "path positions");
    if (rc) {
        pc->at = nullptr;
        return rc == LUE_GPU_ENOMEM ? LUE_GPU_OK : rc;
    }
    if ((rc = cuda_status(cudaMemsetAsync(pc->at, 0xFF, n * sizeof(int32_t), stream), "path positions"))) return rc;
    k_path_at<<<grid_for(pc->npos, 256), 256, 0, stream>>>(pc->order, pc->npos, pc->at);
    count_launches(1);
    if ((rc = cuda_status(cudaGetLastError(), "path positions"))) return rc;
    return cuda_status(cudaStreamSynchronize(stream), "path positions");  // the calls' streams may not wait for it
}

static bool capturing(cudaStream_t stream)
{
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(stream, &s) == cudaSuccess && s != cudaStreamCaptureStatusNone;
}

int path_core_build(const TopologyCore* core, uint32_t* work, cudaStream_t stream, PathCore** out)
{
    *out = nullptr;
    const int64_t n = core->n, rows = core->rows, cols = core->cols;
    // test hook: LUE_GB300_PATH_NO_MEMORY (layout or buffers: there is no memory for them)
    if (const char* e = getenv("LUE_GB300_PATH_NO_MEMORY"))
        if (e[0] == 'l') return fail(LUE_GPU_ENOMEM, "path topology: no memory (test hook)");
    // positions are 32-bit, and a CTA of the scan may look past the last one
    if (n >= (int64_t(1) << 31) - 65536) return fail(LUE_GPU_ERANGE, "path topology: about 2^31 cells or more");
    const int64_t npos = core->stats.valid_cells;
    auto* pc = new (std::nothrow) PathCore();
    if (!pc) return fail(LUE_GPU_ENOMEM, "path topology: host allocation");
    pc->npos = npos;
    const PathGeom g{rows, cols, (cols + kPathTile - 1) / kPathTile,
                     (cols + kPathTile - 1) / kPathTile * ((rows + kPathTile - 1) / kPathTile)};
    int32_t *size = nullptr, *dtop = nullptr, *plev = nullptr, *heavy = nullptr, *next = nullptr;
    uint8_t *key = nullptr, *light = nullptr;
    long long* bsum = nullptr;
    int32_t *counts = nullptr, *starts = nullptr;
    unsigned long long* cells = nullptr;
    int* stats = nullptr;
    constexpr int kStats = 3 + 256;
    int rc = LUE_GPU_OK, levels = 0, hstats[kStats] = {}, launches = 6;
    unsigned long long hcells[256] = {};
    std::vector<int32_t> hstart;
    int64_t ncuts = 0, nlight = 0, nblk = 0;
    const char* what = "path topology";
#define TRY(call) \
    if ((rc = cuda_status((call), what))) goto done
    TRY(cudaMalloc(&size, n * sizeof(int32_t)));
    TRY(cudaMalloc(&dtop, n * sizeof(int32_t)));
    TRY(cudaMalloc(&plev, n * sizeof(int32_t)));
    TRY(cudaMalloc(&heavy, n * sizeof(int32_t)));
    TRY(cudaMalloc(&next, n * sizeof(int32_t)));
    TRY(cudaMalloc(&key, n));
    TRY(cudaMalloc(&stats, kStats * sizeof(int)));
    TRY(cudaMalloc(&cells, sizeof hcells));
    TRY(cudaMalloc(&pc->order, path_padded(npos) * sizeof(int32_t)));
    // 1. sizes, heavy neighbours, cells above on the path, path levels
    k_fill_i32<<<grid_for(n, 256), 256, 0, stream>>>(heavy, n, 8);
    TRY(cudaMemcpyAsync(work, core->count, words_for(n) * 4, cudaMemcpyDeviceToDevice, stream));
    {
        WalkGrid wg{core->fd, core->count, work, rows, cols, n};
        PathVisitor v{core->upmask, size, dtop, plev, heavy, cols};
        k_walk<<<grid_all(n, 256), 256, 0, stream>>>(wg, v);
    }
    // 2. bottom of each cell's path: pointer jumping over the path links
    k_path_next<<<grid_for(n, 256), 256, 0, stream>>>(core->fd, heavy, rows, cols, n, next);
    {
        int rounds = 1;
        while ((int64_t(1) << rounds) < core->stats.max_level + 2) ++rounds;
        for (int i = 0; i <= rounds; ++i) k_path_jump<<<grid_for(n, 256), 256, 0, stream>>>(next, n);
        launches += rounds + 1;
    }
    // 3. levels
    TRY(cudaMemsetAsync(stats, 0, kStats * sizeof(int), stream));
    TRY(cudaMemsetAsync(cells, 0, sizeof hcells, stream));
    k_path_keys<<<grid_for(n, 256), 256, 0, stream>>>(next, plev, dtop, n, key, stats, cells);
    TRY(cudaMemcpyAsync(hstats, stats, sizeof hstats, cudaMemcpyDeviceToHost, stream));
    TRY(cudaMemcpyAsync(hcells, cells, sizeof hcells, cudaMemcpyDeviceToHost, stream));
    TRY(cudaStreamSynchronize(stream));
    if (hstats[2] != 0 || hstats[0] >= kPathMaxLevels) {
        rc = fail(LUE_GPU_ERANGE, "path topology: " + std::to_string(hstats[2]) + " cells without a bottom, " +
                                      std::to_string(hstats[0] + 1) + " levels");
        goto done;
    }
    levels = npos > 0 ? hstats[0] + 1 : 0;
    // 4. positions: levels in order, and the paths of a level tile by tile
    pc->levels.resize(levels);
    hstart.resize(levels + 1);
    for (int l = 0; l < levels; ++l) {
        PathLevel& v = pc->levels[l];
        if (hcells[l] > (unsigned long long)(npos - hstart[l])) {
            rc = fail(LUE_GPU_ERANGE, "path topology: more positions than cells");
            goto done;
        }
        v.p0 = hstart[l];
        v.p1 = hstart[l + 1] = (int32_t)(hstart[l] + (int64_t)hcells[l]);
        v.longest = hstats[3 + l];
        v.per = path_per(l, v.p1 - v.p0);
        v.cut0 = (int32_t)ncuts;
        v.ncut = (int32_t)((v.p1 - v.p0 + path_cut_step(l, v.p1 - v.p0) - 1) / path_cut_step(l, v.p1 - v.p0));
        ncuts += v.ncut + 1;
        pc->tiles = std::max<int64_t>(pc->tiles, (v.p1 - v.p0) / (kPathThreads * v.per) + 2);
    }
    if (hstart[levels] != npos) {
        rc = fail(LUE_GPU_ERANGE, "path topology: " + std::to_string(hstart[levels]) + " positions for " +
                                      std::to_string(npos) + " cells");
        goto done;
    }
    pc->slot_base = levels > 0 ? pc->levels[0].p1 : 0;
    nlight = npos - pc->slot_base;
    nblk = (nlight + kLightBlock - 1) / kLightBlock;
    TRY(cudaMalloc(&counts, std::max<int64_t>(1, levels * g.ntiles) * sizeof(int32_t)));
    TRY(cudaMalloc(&starts, (levels + 1) * sizeof(int32_t)));
    TRY(cudaMalloc(&pc->path_slot, std::max<int64_t>(1, npos) * sizeof(int32_t)));
    TRY(cudaMalloc(&pc->slot_first, (nlight + 1) * sizeof(int32_t)));
    TRY(cudaMalloc(&pc->cut, std::max<int64_t>(1, ncuts) * sizeof(int32_t)));
    TRY(cudaMalloc(&light, std::max<int64_t>(1, nlight)));
    TRY(cudaMalloc(&bsum, (nblk + 1) * sizeof(long long)));
    pc->bytes = path_padded(npos) * 4 + npos * 4 + (nlight + 1) * 4 + ncuts * 4;
    if (levels > 0) {
        int32_t* base = size;  // no longer needed
        TRY(cudaMemcpyAsync(starts, hstart.data(), (levels + 1) * sizeof(int32_t), cudaMemcpyHostToDevice, stream));
        k_paths_count<<<(unsigned)g.ntiles, 256, 0, stream>>>(key, dtop, g, levels, counts);
        k_paths_scan<<<(unsigned)levels, 1024, 0, stream>>>(counts, g.ntiles, starts);
        k_paths_assign<<<(unsigned)g.ntiles, 256, 0, stream>>>(key, dtop, g, counts, base);
        TRY(cudaMemsetAsync(pc->order, 0xFF, path_padded(npos) * sizeof(int32_t), stream));
        TRY(cudaMemsetAsync(stats + 2, 0, sizeof(int), stream));
        k_path_place<<<grid_for(n, 256), 256, 0, stream>>>(next, base, dtop, heavy, core->upmask, n, npos,
                                                          pc->slot_base, pc->order, light, stats + 2);
        k_path_unwritten<<<grid_for(npos, 256), 256, 0, stream>>>(pc->order, npos, stats + 2);
        // 5. slots
        if (nlight > 0) k_light_sums<<<(unsigned)nblk, 256, 0, stream>>>(light, nlight, bsum);
        k_light_scan<<<1, 1024, 0, stream>>>(bsum, nblk);
        if (nlight > 0) k_light_apply<<<(unsigned)nblk, 256, 0, stream>>>(light, nlight, bsum, nblk, pc->slot_first);
        k_path_slots<<<grid_for(n, 256), 256, 0, stream>>>(core->fd, core->upmask, key, next, base, dtop, heavy,
                                                          pc->slot_first, pc->slot_base, rows, cols, pc->path_slot,
                                                          stats + 2);
        // 6. CTA ranges of the scans
        for (int l = 0; l < levels; ++l) {
            const PathLevel& v = pc->levels[l];
            if (v.ncut > 0)
                k_path_cuts<<<(unsigned)(((v.ncut + 1) * 32 + 255) / 256), 256, 0, stream>>>(
                    pc->order, v.p0, v.p1, path_cut_step(l, v.p1 - v.p0), v.ncut, pc->cut + v.cut0);
        }
        launches += 8 + levels;
        long long hslots = 0;
        int bad = 0;
        TRY(cudaMemcpyAsync(&hslots, bsum + nblk, sizeof hslots, cudaMemcpyDeviceToHost, stream));
        TRY(cudaMemcpyAsync(&bad, stats + 2, sizeof(int), cudaMemcpyDeviceToHost, stream));
        TRY(cudaStreamSynchronize(stream));
        TRY(cudaGetLastError());
        pc->nslots = hslots;
        if (bad) {
            rc = fail(LUE_GPU_ERANGE, "path topology: inconsistent layout (" + std::to_string(bad) + " misplaced)");
            goto done;
        }
    }
    count_launches(launches);
    if (getenv("LUE_GB300_VERBOSE")) {
        fprintf(stderr, "path topology: %lld cells, %d levels, %lld slots, longest path %d cells; positions (longest path) "
                        "by level:",
                (long long)npos, levels, (long long)pc->nslots, hstats[1]);
        for (const PathLevel& v : pc->levels) fprintf(stderr, " %d (%d)", v.p1 - v.p0, v.longest);
        fprintf(stderr, "\n");
    }
done:
#undef TRY
    cudaFree(size);
    cudaFree(dtop);
    cudaFree(plev);
    cudaFree(heavy);
    cudaFree(next);
    cudaFree(key);
    cudaFree(light);
    cudaFree(bsum);
    cudaFree(counts);
    cudaFree(starts);
    cudaFree(cells);
    cudaFree(stats);
    if (rc) {
        path_core_free(pc);
        return rc;
    }
    *out = pc;
    return LUE_GPU_OK;
}

// ---------------------------------------------------------------------------------------------------
// Per call
// ---------------------------------------------------------------------------------------------------

// Kinds of maps, from a cell's inflow along its path to its outflow: x -> max(x + a, b) (threshold),
// x -> min(x + a, b) (capacity), x -> a * x + b (fraction), and x -> x + b where x >= a, else c (trigger).
//
// The trigger's maps compose into maps of the same form because every one of them is monotone on x >= 0 and c
// is its value at 0: m2 after m1, with c1 >= a2, passes everything on (x >= a1 gives x + b1 >= c1 >= a2):
// (a1, b1 + b2, c1 + b2); with c1 < a2 what m1 holds back stays held back: (max(a1, a2 - b1), b1 + b2, c2).
//
// On the stage engine accu_trigger was bound by its chain of rounds (1500^2: 1595 us a call); as a scan it
// takes 121 us.
constexpr int kMaxPlus = 0, kMinPlus = 1, kAffine = 2, kTrigger = 3, kSum = 4;

// a, b and c float-float.  flags bit 0: the map of a path's top cell, which ignores its input (its value is
// value()); bit 1: no-data (NaN) from the cell itself or from upstream.
template <int K>
struct PMap {
    float ah, al, bh, bl;
    int flags;
    __device__ FF value() const { return FF{bh, bl}; }
};
template <>
struct PMap<kTrigger> {
    float ah, al, bh, bl;
    int flags;
    float ch, cl;
    __device__ FF value() const { return FF{ch, cl}; }
};

// x -> x + b in float64 (accu); the value of a top cell's map is b.
template <>
struct PMap<kSum> {
    double b;
    int flags;
    __device__ double value() const { return b; }
};

template <int K>
__device__ __forceinline__ PMap<K> pm_identity()
{
    if constexpr (K == kSum) return PMap<K>{0.0, 0};
    else if constexpr (K == kAffine) return PMap<K>{1.0f, 0.0f, 0.0f, 0.0f, 0};
    else if constexpr (K == kTrigger) return PMap<K>{-INFINITY, 0.0f, 0.0f, 0.0f, 0, 0.0f, 0.0f};
    else return PMap<K>{0.0f, 0.0f, K == kMinPlus ? INFINITY : -INFINITY, 0.0f, 0};
}

// x + y for float-float values; a sum that is not finite is kept with lo = 0 (two_sum's error terms would
// turn an infinity into NaN).  Selects, no branches: a warp composes many maps at once.
__device__ __forceinline__ void ff_sum(float xh, float xl, float yh, float yl, float& rh, float& rl)
{
    float s, e;
    two_sum(xh, yh, s, e);
    e = __fadd_rn(e, __fadd_rn(xl, yl));
    e = fabsf(s) < INFINITY ? e : 0.0f;
    rh = __fadd_rn(s, e);
    rl = fabsf(s) < INFINITY ? __fsub_rn(e, __fsub_rn(rh, s)) : 0.0f;
}

__device__ __forceinline__ bool ff_less(float xh, float xl, float yh, float yl)
{
    return xh < yh || (xh == yh && xl < yl);
}

// x * y for finite float-float values: the exact product of the high parts by FMA (two-product), plus the
// cross terms, renormalised.
__device__ __forceinline__ void ff_mul(float xh, float xl, float yh, float yl, float& rh, float& rl)
{
    const float p = __fmul_rn(xh, yh);
    float e = __fmaf_rn(xh, yh, -p);
    e = __fmaf_rn(xh, yl, e);
    e = __fmaf_rn(xl, yh, e);
    rh = __fadd_rn(p, e);
    rl = __fsub_rn(e, __fsub_rn(rh, p));
}

// m1 first, then m2.  No branches: the constant map of a path's top is one on which the same formulas give
// a constant (a = -inf, +inf, 0 and +inf for the four float32 kinds), so only its flags are chosen.
template <int K>
__device__ __forceinline__ PMap<K> compose(const PMap<K>& m1, const PMap<K>& m2)
{
    PMap<K> r;
    r.flags = m2.flags & 1 ? m2.flags : m1.flags | m2.flags;
    if constexpr (K == kSum) {
        r.b = m2.flags & 1 ? m2.b : m1.b + m2.b;
    } else if constexpr (K == kAffine) {  // a2 * (a1 * x + b1) + b2
        ff_mul(m1.ah, m1.al, m2.ah, m2.al, r.ah, r.al);
        float th, tl;
        ff_mul(m2.ah, m2.al, m1.bh, m1.bl, th, tl);
        ff_sum(th, tl, m2.bh, m2.bl, r.bh, r.bl);
    } else if constexpr (K == kTrigger) {
        float th, tl, uh, ul;
        ff_sum(m1.bh, m1.bl, m2.bh, m2.bl, r.bh, r.bl);
        ff_sum(m2.ah, m2.al, -m1.bh, -m1.bl, th, tl);
        ff_sum(m1.ch, m1.cl, m2.bh, m2.bl, uh, ul);
        const bool holds = ff_less(m1.ch, m1.cl, m2.ah, m2.al);
        const bool later = holds && ff_less(m1.ah, m1.al, th, tl);
        r.ah = later ? th : m1.ah;
        r.al = later ? tl : m1.al;
        r.ch = holds ? m2.ch : uh;
        r.cl = holds ? m2.cl : ul;
    } else {
        ff_sum(m1.ah, m1.al, m2.ah, m2.al, r.ah, r.al);
        float th, tl;
        ff_sum(m1.bh, m1.bl, m2.ah, m2.al, th, tl);
        const bool take = K == kMinPlus ? ff_less(th, tl, m2.bh, m2.bl) : ff_less(m2.bh, m2.bl, th, tl);
        r.bh = take ? th : m2.bh;
        r.bl = take ? tl : m2.bl;
    }
    return r;
}

// The two kinds of numbers: float32 operations carry float-float values, float64 operations plain doubles.  A
// cell's sum s is its material plus its light inflow; total() adds what comes along its path.
struct F32 {
    using T = float;
    using V = FF;
    using Slot = float2;  // hi (NaN: no-data), lo
    static __device__ __forceinline__ void light(FF& s, bool& nan, float2 v)
    {
        nan |= isnan(v.x);
        float h, e;
        two_sum(s.hi, v.x, h, e);
        s.hi = h;
        s.lo = __fadd_rn(__fadd_rn(s.lo, e), v.y);
    }
    static __device__ __forceinline__ FF from(float x) { return FF{x, 0.0f}; }
    static __device__ __forceinline__ FF cell(FF s, float x) { return total(s, FF{x, 0.0f}); }
    static __device__ __forceinline__ FF total(FF x, FF s)
    {
        float h, e;
        two_sum(x.hi, s.hi, h, e);
        e = __fadd_rn(e, __fadd_rn(x.lo, s.lo));
        const float r = __fadd_rn(h, e);
        return FF{r, __fsub_rn(e, __fsub_rn(r, h))};
    }
    static __device__ __forceinline__ FF zero() { return FF{0.0f, 0.0f}; }
    static __device__ __forceinline__ float hi(FF v) { return v.hi; }
    static __device__ __forceinline__ Slot slot(FF v, bool nan)
    {
        return nan ? make_float2(__int_as_float(0x7fc00000), 0.0f) : make_float2(v.hi, v.lo);
    }
};
// Before, on the stage engine, float64 accu was bound by its chain of rounds: 3001 x 2777 with no-data 3375 us a call, as
// prefix sums along paths 279 us.
struct F64 {
    using T = double;
    using V = double;
    using Slot = double;
    static __device__ __forceinline__ void light(double& s, bool& nan, double v)
    {
        nan |= isnan(v);
        s += v;
    }
    static __device__ __forceinline__ double from(double x) { return x; }
    static __device__ __forceinline__ double cell(double s, double x) { return s + x; }
    static __device__ __forceinline__ double total(double x, double s) { return x + s; }
    static __device__ __forceinline__ double zero() { return 0.0; }
    static __device__ __forceinline__ double hi(double v) { return v; }
    static __device__ __forceinline__ double slot(double v, bool nan) { return nan ? qnan<double>() : v; }
};

// The rules of rule_f32 / rule_f64 on a finite total t (float-float: normalised), inputs in the domain.
template <Rule R>
__device__ __forceinline__ void rule_total(FF t, float b, FF& out, float& rem)
{
    if constexpr (R == Rule::fraction) {
        const float ph = __fmul_rn(b, t.hi);
        float pl = __fmaf_rn(b, t.hi, -ph);
        pl = __fmaf_rn(b, t.lo, pl);
        out.hi = __fadd_rn(ph, pl);
        out.lo = __fsub_rn(pl, __fsub_rn(out.hi, ph));
        const float h = __fsub_rn(t.hi, out.hi);  // |t| >= |out|: the rounding error of h is exact
        const float e = __fsub_rn(__fsub_rn(t.hi, h), out.hi);
        rem = __fadd_rn(h, __fadd_rn(e, __fsub_rn(t.lo, out.lo)));
    } else if constexpr (R == Rule::trigger) {
        const bool stays = t.hi < b || (t.hi == b && t.lo < 0.0f);
        rem = stays ? t.hi : 0.0f;
        out.hi = stays ? 0.0f : t.hi;
        out.lo = stays ? 0.0f : t.lo;
    } else {  // threshold, capacity: what is above b
        const bool above = t.hi > b || (t.hi == b && t.lo > 0.0f);
        const float h = __fsub_rn(t.hi, b);  // t.hi >= b >= 0 where it is used: exact error
        const float e = __fadd_rn(__fsub_rn(__fsub_rn(t.hi, h), b), t.lo);
        const float dh = __fadd_rn(h, e), dl = __fsub_rn(e, __fsub_rn(dh, h));
        if constexpr (R == Rule::threshold) {
            rem = above ? b : t.hi;
            out.hi = above ? dh : 0.0f;
            out.lo = above ? dl : 0.0f;
        } else {
            rem = above ? dh : 0.0f;
            out.hi = above ? b : t.hi;
            out.lo = above ? 0.0f : t.lo;
        }
    }
}
template <Rule R>
__device__ __forceinline__ void rule_total(double t, double b, double& out, double& rem)
{
    static_assert(R == Rule::accu, "float64 paths carry sums only");
    out = t;
}

// The map of one cell: s = its material plus the outflow of its light upstream neighbours, b its
// threshold, fraction, capacity or trigger (both 0 in a no-data cell).  By selects, as compose().
template <Rule R, int K, class V, class T>
__device__ __forceinline__ PMap<K> cell_map(bool top, V s, T b, bool nan)
{
    PMap<K> m;
    m.flags = (top ? 1 : 0) | (nan ? 2 : 0);
    if constexpr (K == kSum) {
        m.b = s;
    } else if constexpr (K == kAffine) {  // fraction * x + fraction * s; top: fraction * s
        m.ah = top ? 0.0f : b;
        m.al = 0.0f;
        ff_mul(b, 0.0f, s.hi, s.lo, m.bh, m.bl);
    } else if constexpr (K == kTrigger) {  // x + s where that reaches the trigger, else 0
        ff_sum(b, 0.0f, -s.hi, -s.lo, m.ah, m.al);
        const bool passes = m.ah <= 0.0f;
        m.ah = top ? INFINITY : m.ah;
        m.al = top ? 0.0f : m.al;
        m.bh = s.hi;
        m.bl = s.lo;
        m.ch = passes ? s.hi : 0.0f;
        m.cl = passes ? s.lo : 0.0f;
    } else if constexpr (K == kMaxPlus) {  // max(x + (s - threshold), 0); top: max(s - threshold, 0)
        float dh, dl;
        ff_sum(s.hi, s.lo, -b, 0.0f, dh, dl);
        const bool over = top && dh > 0.0f;
        m.ah = top ? -INFINITY : dh;
        m.al = top ? 0.0f : dl;
        m.bh = over ? dh : 0.0f;
        m.bl = over ? dl : 0.0f;
    } else {  // capacity: min(x + s, capacity); top: min(s, capacity)
        const bool under = top && ff_less(s.hi, s.lo, b, 0.0f);
        m.ah = top ? INFINITY : s.hi;
        m.al = top ? 0.0f : s.lo;
        m.bh = under ? s.hi : b;
        m.bl = under ? s.lo : 0.0f;
    }
    return m;
}

// Every word of a map, moved by f (shuffles and loads).
template <int K, class F>
__device__ __forceinline__ PMap<K> pm_each(const PMap<K>& m, F f)
{
    PMap<K> r;
    if constexpr (K == kSum) {
        r.b = f(m.b);
    } else {
        r.ah = f(m.ah);
        r.al = f(m.al);
        r.bh = f(m.bh);
        r.bl = f(m.bl);
    }
    r.flags = f(m.flags);
    if constexpr (K == kTrigger) {
        r.ch = f(m.ch);
        r.cl = f(m.cl);
    }
    return r;
}
template <int K>
__device__ __forceinline__ PMap<K> shfl_up(const PMap<K>& m, int d)
{
    return pm_each(m, [d](auto v) { return __shfl_up_sync(0xffffffffu, v, d); });
}
template <int K>
__device__ __forceinline__ PMap<K> shfl_down(const PMap<K>& m, int d)
{
    return pm_each(m, [d](auto v) { return __shfl_down_sync(0xffffffffu, v, d); });
}

// Exclusive scan of the threads' maps in thread order; `total` is the composition of all of them.
template <int K, int NT>
__device__ __forceinline__ PMap<K> block_excl_scan(const PMap<K>& v, PMap<K>* s_warp, PMap<K>& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    PMap<K> x = v;
    for (int d = 1; d < 32; d <<= 1) {
        if (__all_sync(0xffffffffu, lane < d || (x.flags & 1))) break;  // every map is a constant by now
        const PMap<K> y = shfl_up(x, d);
        if (lane >= d) x = compose<K>(y, x);
    }
    PMap<K> ex = shfl_up(x, 1);
    if (lane == 0) ex = pm_identity<K>();
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        PMap<K> w = lane < NT / 32 ? s_warp[lane] : pm_identity<K>();
        for (int d = 1; d < 32; d <<= 1) {
            const PMap<K> y = shfl_up(w, d);
            if (lane >= d) w = compose<K>(y, w);
        }
        if (lane < NT / 32) s_warp[lane] = w;
    }
    __syncthreads();
    total = s_warp[NT / 32 - 1];
    const PMap<K> r = warp ? compose<K>(s_warp[warp - 1], ex) : ex;
    __syncthreads();
    return r;
}

template <class N>
struct PathCall {
    const int32_t* __restrict__ order;
    const int32_t* __restrict__ path_slot;   // by position, at the bottoms of paths
    const int32_t* __restrict__ slot_first;  // by position (the engine's array minus its base)
    const typename N::T* __restrict__ a;     // material
    typename N::T as;
    const typename N::T* __restrict__ b;     // threshold / fraction / capacity / trigger
    typename N::T bs;
    typename N::T* out;
    typename N::T* rem;
    typename N::Slot* slots;                 // what leaves each path; written by a level, read by higher ones
    float2* dense;                           // both results by position, or nullptr: straight to out and rem
    unsigned long long* flag;
};

// The inputs of a cell are in the domain and not NaN.
template <Rule R, class T>
__device__ __forceinline__ bool in_domain(T e, T b)
{
    if constexpr (R == Rule::accu) return e >= T(0);
    else if constexpr (R == Rule::fraction) return e >= T(0) && b >= T(0) && b <= T(1);
    else return e >= T(0) && b >= T(0);
}

// The order entries of PER consecutive positions from `first` (a multiple of PER), read with vector
// loads; the position arrays are padded by one 8-position chunk, so a chunk that starts before the end
// of the array stays inside it.
template <int PER, class P>
__device__ __forceinline__ void load_order(const P& p, int64_t first, int32_t (&w)[PER])
{
    if (PER == 4) {
        const int4 x = __ldg(reinterpret_cast<const int4*>(p.order + first));
        w[0] = x.x; w[1 % PER] = x.y; w[2 % PER] = x.z; w[3 % PER] = x.w;
    } else if (PER == 2) {
        const int2 x = __ldg(reinterpret_cast<const int2*>(p.order + first));
        w[0] = x.x; w[1 % PER] = x.y;
    } else {
#pragma unroll
        for (int j = 0; j < PER; ++j) w[j] = __ldg(p.order + first + j);
    }
}

// Look-back of one level's launch: CTAs take tiles in ticket order.  Each tile publishes the composition of its own maps: a
// constant when a path's top is among its positions, so that nothing before the tile matters.  Tiles whose number is a
// multiple of 32 (fences) also publish the composition of the 32 tiles up to and including themselves (their group), or,
// at multiples of 1024, that of everything up to and including themselves (a prefix).  Status words carry the launch's
// epoch, so the arrays need no clearing between launches.
//
// A tile composes the tiles before it back to the nearest constant one, or to the fence before it, and from there the groups
// back to the nearest constant one or to a prefix.  Which ones these are depends on the layout alone, not on which CTA is how
// far: the same call gives the same bits every time, in plain doubles too.  The only chain of waits is that of the
// prefixes, one every 1024 tiles along a river.  accu (float64) over a basin of 3001 x 2777 takes 203 us, accu_trigger at
// 1500^2 124, accu over one path through 4000^2 cells 479; composing whatever tiles have published so far (every tile
// its prefix, so twice as many publications) 216, 136 and 538; prefixes every 32 tiles without groups 1171 on the last.
enum PathState { kOwn = 1, kGroup = 2, kConstant = 3, kConstantGroup = 4, kPrefix = 5 };
template <int K>
struct PathScan {
    int* status;  // [tiles] epoch << 3 | state
    PMap<K>* aggm;   // [tiles] the tile's own composition
    PMap<K>* inclm;  // [tiles] a fence's group or prefix
    int* ticket;  // zeroed before the launch
    int epoch;
    int polls;    // poll limit of one wait
};

constexpr int kPathPolls = 1 << 20;

template <int K>
__device__ __forceinline__ int path_state(const PathScan<K>& q, int tile)
{
    const int v = ld_acquire(q.status + tile);
    return (v >> 3) == q.epoch ? v & 7 : 0;
}
template <int K>
__device__ __forceinline__ void path_publish(const PathScan<K>& q, int tile, PMap<K>* to, const PMap<K>& m, int state)
{
    to[tile] = m;
    __threadfence();
    st_release(q.status + tile, (q.epoch << 3) | state);
}

// The lanes' maps composed, those of higher lanes (farther tiles) first, in every lane.
template <int K>
__device__ __forceinline__ PMap<K> compose_lanes(PMap<K> m)
{
    const int lane = threadIdx.x & 31;
    for (int d = 1; d < 32; d <<= 1) {
        const PMap<K> o = shfl_down(m, d);
        if (lane + d < 32) m = compose<K>(o, m);
    }
    return pm_each(m, [](auto v) { return __shfl_sync(0xffffffffu, v, 0); });
}

// Whether the lanes up to the first one of `ends` (all lanes without one) are ready; uniform.
__device__ __forceinline__ bool lanes_ready(unsigned ends, unsigned missing) { return !(missing & (ends ^ (ends - 1u))); }

// Warp 0: the composition of all tiles before `tile` (in every lane); publishes the group or prefix of a fence.  Waits are
// bounded: one that gives up (or finds that another one did) sets flag[1], after which the call is redone.
template <int K>
__device__ PMap<K> look_back(const PathScan<K>& q, int tile, const PMap<K>& total, unsigned long long* flag)
{
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, fence = (tile - 1) & ~31;
    const int near = tile - 1 - lane, far = fence - 32 * lane;  // a lane's tile behind the fence, and its fence
    const bool is_fence = (tile & 31) == 0 && !(total.flags & 1);
    int own = near > fence ? 0 : -1, group = far >= 0 ? 0 : -1;
    auto gave_up = [&] { return __any_sync(kAll, *reinterpret_cast<volatile unsigned long long*>(flag + 1) != 0) != 0; };
    // the tiles after the fence
    unsigned ends = 0;
    bool ready = false;
    for (int k = 0; k < q.polls && !ready; ++k) {
        if (own == 0) own = path_state(q, near);
        if (group >= 0 && group < kGroup) group = path_state(q, far);
        ends = __ballot_sync(kAll, own == kConstant);
        ready = lanes_ready(ends, __ballot_sync(kAll, own == 0));
        if (!ready) {
            if (gave_up()) break;
            __nanosleep(32);
        }
    }
    PMap<K> before = pm_identity<K>();
    if (ready) {
        const int stop = ends ? __ffs(ends) - 1 : 31;
        PMap<K> m = pm_identity<K>();
        if (own > 0 && lane <= stop) m = pm_each(q.aggm[near], [](const auto& v) { return __ldcg(&v); });
        before = compose_lanes<K>(m);
        if (is_fence && (ends || (tile & 1023)) && lane == 0)
            path_publish(q, tile, q.inclm, compose<K>(before, total), ends ? kConstantGroup : kGroup);
        if (ends) return before;
        // the groups up to the fence
        ready = false;
        for (int k = 0; k < q.polls && !ready; ++k) {
            if (group >= 0 && group < kGroup) group = path_state(q, far);
            ends = __ballot_sync(kAll, group >= kConstant);
            ready = ends && lanes_ready(ends, __ballot_sync(kAll, group >= 0 && group < kGroup));
            if (!ready) {
                if (gave_up()) break;
                __nanosleep(32);
            }
        }
    }
    if (!ready) {
        if (lane == 0) flag[1] = 1;
        return pm_identity<K>();
    }
    PMap<K> m = pm_identity<K>();
    if (lane <= __ffs(ends) - 1)
        m = pm_each(*(group == kConstant ? q.aggm + far : q.inclm + far), [](const auto& v) { return __ldcg(&v); });
    before = compose<K>(compose_lanes<K>(m), before);
    if (is_fence && !(tile & 1023) && lane == 0) path_publish(q, tile, q.inclm, compose<K>(before, total), kPrefix);
    return before;
}

// The positions of one thread in one chunk of a scan: PER consecutive positions from `first`, those in
// [lo, hi) active.  order() and gather() issue the loads, light() adds the light inflow, maps() composes the
// cells' maps, and store() applies, from the composition E of everything before the first position, each cell's
// rule.
template <class N, Rule R, int K, int PER, bool LIGHT>
struct Chunk {
    using T = typename N::T;
    int32_t w[PER];          // order entries: cell, top bit
    unsigned on;             // bit j: position j is active
    unsigned nan;            // bit j: no-data from the cell itself or its light inflow
    T e[PER], b[PER];
    typename N::V sum[PER];
    int32_t f[LIGHT ? PER + 1 : 1];  // the positions' first slots

    __device__ __forceinline__ int32_t first_slot(const PathCall<N>& p, int32_t first, int j) const
    {
        const bool used = ((on >> (j < PER ? j : PER - 1)) & 1u) || (j > 0 && ((on >> (j - 1)) & 1u));
        return used ? __ldg(p.slot_first + first + j) : 0;
    }

    // VEC: `first` is a multiple of PER and the order array is read with vector loads.
    template <bool VEC>
    __device__ __forceinline__ void order(const PathCall<N>& p, int32_t first, int32_t lo, int32_t hi)
    {
        on = 0;
#pragma unroll
        for (int j = 0; j < PER; ++j) on |= first + j >= lo && first + j < hi ? 1u << j : 0u;
        if (VEC) {
            if (on) load_order<PER>(p, first, w);
        } else {
#pragma unroll
            for (int j = 0; j < PER; ++j) w[j] = (on >> j) & 1u ? __ldg(p.order + first + j) : 0;
        }
    }

    __device__ __forceinline__ void gather(const PathCall<N>& p, int32_t first)
    {
        if constexpr (LIGHT) {
#pragma unroll
            for (int j = 0; j <= PER; ++j) f[j] = first_slot(p, first, j);
        }
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int32_t c = w[j] & 0x7fffffff;
            e[j] = p.as;
            b[j] = p.bs;
            if ((on >> j) & 1u) {
                if (p.a) e[j] = __ldg(p.a + c);
                if (R != Rule::accu && p.b) b[j] = __ldg(p.b + c);
            }
        }
    }

    // The cells' sums and the composition of their maps; inactive positions are the identity.
    __device__ __forceinline__ PMap<K> maps(const PathCall<N>& p, int32_t first)
    {
        nan = 0;
        if (LIGHT) {
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                sum[j] = N::zero();
                if (!((on >> j) & 1u)) continue;
                bool bad = false;
                for (int32_t k = f[j]; k < f[j + 1]; ++k) N::light(sum[j], bad, p.slots[k]);
                nan |= bad ? 1u << j : 0u;
            }
        }
        PMap<K> acc = pm_identity<K>();
        bool odd = false;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const bool act = (on >> j) & 1u;
            bool bad = LIGHT && ((nan >> j) & 1u);
            bad = bad || !in_domain<R>(e[j], b[j]);
            if constexpr (LIGHT) sum[j] = N::cell(sum[j], e[j]);
            else sum[j] = N::from(e[j]);
            // a trigger that nothing reaches is an ordinary map: its a is infinite, which compose() only compares
            odd |= act && !bad && !(N::hi(sum[j]) < T(INFINITY) && (R == Rule::trigger || b[j] < T(INFINITY)));
            if (bad) {
                sum[j] = N::zero();
                b[j] = T(0);
                nan |= 1u << j;
            }
            const PMap<K> m = cell_map<R, K>(w[j] < 0, sum[j], b[j], bad);
            if (act) acc = j == 0 ? m : compose<K>(acc, m);
        }
        if (odd) p.flag[1] = 1;  // +inf: the call is redone
        return acc;
    }

    // hi: the end of the CTA's positions, where a path ends.
    __device__ __forceinline__ void store(const PathCall<N>& p, int32_t first, int32_t hi, const PMap<K>& E)
    {
        // the position after this thread's last one: is it the top of a path (then the last one is a bottom)?
        const int32_t after = first + PER < hi ? __ldg(p.order + first + PER) : -1;
        // everything before the first position composes to a constant: a path's top is among it
        typename N::V x = E.value();
        bool xnan = (E.flags & 2) != 0, odd = false;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            if (!((on >> j) & 1u)) continue;
            const int32_t c = w[j] & 0x7fffffff;
            const bool top = w[j] < 0;
            xnan = ((nan >> j) & 1u) || (!top && xnan);
            const typename N::V t = top ? sum[j] : N::total(x, sum[j]);
            T rem = T(0);
            rule_total<R>(t, b[j], x, rem);
            odd |= !xnan && !(N::hi(t) < T(INFINITY));
            const T o = xnan ? qnan<T>() : N::hi(x), left = xnan ? qnan<T>() : rem;
            if (R != Rule::accu && p.dense) {
                p.dense[first + j] = make_float2((float)o, (float)left);
            } else {
                p.out[c] = o;
                if (R != Rule::accu) p.rem[c] = left;
            }
            const int32_t next = j + 1 < PER && first + j + 1 < hi ? w[(j + 1) % PER] : after;
            if (next < 0) {  // a path bottom
                const int32_t slot = __ldg(p.path_slot + first + j);
                if (slot >= 0) p.slots[slot] = N::slot(x, xnan);
            }
        }
        if (odd) p.flag[1] = 1;
    }
};

// The scan of one level with very long paths: tiles in ticket order, the composition of the tiles before each
// one by look-back.
template <class N, Rule R, int K, int PER, bool LIGHT>
__global__ void __launch_bounds__(kPathThreads, 4) k_path_level(PathCall<N> p, PathLevel v, PathScan<K> q)
{
    __shared__ PMap<K> s_warp[kPathThreads / 32];
    __shared__ PMap<K> s_prefix;
    __shared__ int s_tile;
    next_may_start();
    if (threadIdx.x == 0) s_tile = atomicAdd(q.ticket, 1);
    __syncthreads();
    const int tile = s_tile;
    const int32_t first = (v.p0 & ~(PER - 1)) + tile * (kPathThreads * PER) + (int32_t)threadIdx.x * PER;
    Chunk<N, R, K, PER, LIGHT> ch;
    ch.template order<true>(p, first, v.p0, v.p1);
    ch.gather(p, first);
    wait_for_previous();
    const PMap<K> acc = ch.maps(p, first);
    PMap<K> total;
    const PMap<K> E = block_excl_scan<K, kPathThreads>(acc, s_warp, total);
    if (threadIdx.x < 32) {
        // a level begins with a top
        if (threadIdx.x == 0) path_publish(q, tile, q.aggm, total, tile == 0 || (total.flags & 1) ? kConstant : kOwn);
        const PMap<K> before = tile ? look_back<K>(q, tile, total, p.flag) : pm_identity<K>();
        if (threadIdx.x == 0) s_prefix = before;
    }
    __syncthreads();
    ch.store(p, first, v.p1, compose<K>(s_prefix, E));
}

// The scan of one level with shorter paths: each CTA's range of positions begins and ends at path tops (`cut`, laid
// out once), so no path crosses from one CTA to another and CTAs do not wait for one another; a range is processed
// in chunks of kPathThreads * PER positions with the composition carried from chunk to chunk.  The next
// chunk's order is read before this chunk's scan, and its inputs before this chunk's rules, so that the two
// dependent loads overlap the arithmetic.
//
// Bound by instruction issue (54 % of the slots) and the waits for its loads: 230 thread instructions per position on level 0
// at 8192^2, 0.56 ms with its results by position (0.71 ms straight to the raster, bound by the requests of the scattered
// stores as well); with branches in the compositions, a second composition per cell in store() and 64-bit positions it was
// 486 and 1.0 ms.  accu_threshold at 16384^2: 8.4 -> 6.6 ms with these steps, 4.9 with the ones since.  Tried and slower: one thread per short path (up to 16, 64 or 256 cells) with the cell rule itself, sorted by
// length within a tile: 50 instructions per cell, but every lane of a store is a request of its own (8.3-10 ms at
// 16384^2, with the results of a tile collected in shared memory as well); CTAs of 128 threads (6.9 ms).
template <class N, Rule R, int K, int PER, bool LIGHT>
__global__ void __launch_bounds__(kPathThreads, 4)
    k_path_free(PathCall<N> p, PathLevel v, const int32_t* __restrict__ cut)
{
    __shared__ PMap<K> s_warp[kPathThreads / 32];
    __shared__ PMap<K> s_carry;
    constexpr int32_t T = kPathThreads * PER;
    next_may_start();
    const int32_t lo = __ldg(cut + v.cut0 + blockIdx.x), hi = __ldg(cut + v.cut0 + blockIdx.x + 1);
    if (threadIdx.x == 0) s_carry = pm_identity<K>();
    const int32_t at = (int32_t)threadIdx.x * PER;
    Chunk<N, R, K, PER, LIGHT> ch, nx;
    ch.template order<false>(p, lo + at, lo, hi);
    ch.gather(p, lo + at);
    wait_for_previous();
    for (int32_t c0 = lo; c0 < hi; c0 += T) {  // uniform
        const int32_t first = c0 + at;
        const bool more = c0 + T < hi;
        if (more) nx.template order<false>(p, first + T, lo, hi);
        const PMap<K> acc = ch.maps(p, first);
        PMap<K> total;
        // the scan's barriers come after thread 0's update of s_carry for the previous chunk
        const PMap<K> ex = block_excl_scan<K, kPathThreads>(acc, s_warp, total);
        const PMap<K> E = compose<K>(s_carry, ex);
        __syncthreads();  // every thread has read s_carry
        if (threadIdx.x == 0) s_carry = compose<K>(s_carry, total);
        if (more) nx.gather(p, first + T);
        ch.store(p, first, hi, E);
        ch = nx;
    }
}

// The results from their positions to the raster, a CTA per 64 x 64 tile; no-data cells (without a position) get NaN.
//
// Stored cell by cell while a level runs, each result is a partial write of a sector of its own, most of them after
// the rest of the sector has left L2: 2.4 of accu_threshold's 6.4 ms at 16384^2 (level 1: 1.21 ms, and 0.44 by position).
// By position they are dense, and a tile's positions are close together, so this kernel's reads hit L1 and its
// writes are whole rows: bound by memory, 0.88 ms at 16384^2 (20 bytes a cell, 6.1 TB/s).
__global__ void __launch_bounds__(256)
    k_path_spread(const int32_t* __restrict__ at, const float2* __restrict__ dense, int64_t rows, int64_t cols, int64_t tcols,
                  float* __restrict__ out, float* __restrict__ rem)
{
    constexpr int kCells = 8, kStep = 256 / kPathTile;
    const int64_t tr = blockIdx.x / tcols, tc = blockIdx.x - tr * tcols;
    const int64_t row0 = tr * kPathTile + threadIdx.x / kPathTile, col = tc * kPathTile + threadIdx.x % kPathTile;
    if (col >= cols) return;
#pragma unroll
    for (int h = 0; h < kPathTile / (kCells * kStep); ++h) {
        int32_t i[kCells];
        float2 v[kCells];
#pragma unroll
        for (int k = 0; k < kCells; ++k) {
            const int64_t r = row0 + (h * kCells + k) * kStep;
            i[k] = r < rows ? __ldcs(at + r * cols + col) : -1;
        }
#pragma unroll
        for (int k = 0; k < kCells; ++k) v[k] = i[k] >= 0 ? __ldg(dense + i[k]) : make_float2(qnan<float>(), qnan<float>());
#pragma unroll
        for (int k = 0; k < kCells; ++k) {
            const int64_t r = row0 + (h * kCells + k) * kStep;
            if (r >= rows) continue;
            __stcs(out + r * cols + col, v[k].x);
            __stcs(rem + r * cols + col, v[k].y);
        }
    }
}

__device__ __forceinline__ double from_lane(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
__device__ __forceinline__ float2 from_lane(float2 v, int lane)
{
    return make_float2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}
__device__ __forceinline__ FF from_lane(FF v, int lane)
{
    return FF{__shfl_sync(0xffffffffu, v.hi, lane), __shfl_sync(0xffffffffu, v.lo, lane)};
}

// What a step takes besides the flow along the path, from the lane that holds it.  bits: number of values added after that
// flow (the first in `then`), kFlow when there is one, kAlone when nothing is added before it, kNone for no-data.
constexpr unsigned kFlow = 16, kAlone = 32, kNone = 64;
template <class Visitor>
struct RedoStep {
    decltype(Visitor::Total::t) t;
    typename Visitor::Up then;
    unsigned bits;
    typename Visitor::T x, y;
    template <class Total, class Up, class T>
    static __device__ __forceinline__ RedoStep from(const Total& s, Up then, unsigned bits, T x, T y, int lane)
    {
        return RedoStep{from_lane(s.t, lane), from_lane(then, lane), __shfl_sync(0xffffffffu, bits, lane),
                        __shfl_sync(0xffffffffu, x, lane), __shfl_sync(0xffffffffu, y, lane)};
    }
};

// A slot without its value yet: a NaN that no rule gives.  A value is one word, so it needs no fence.
constexpr unsigned long long kEmptySlot = ~0ull;
template <class Up>
__device__ __forceinline__ bool read_slot(const unsigned long long* p, Up& u)
{
    static_assert(sizeof(Up) == sizeof(unsigned long long), "a slot is one word");
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    memcpy(&u, &w, sizeof u);
    return w != kEmptySlot;
}
template <class Up>
__device__ __forceinline__ void write_slot(unsigned long long* p, Up u)
{
    unsigned long long w;
    memcpy(&w, &u, sizeof w);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}

// A call redone cell by cell (flag[1] of the engine: infinite values, or a look-back wait that gave up), with the cell rule of
// the walk engine, so the results are that engine's bit for bit.  Persistent warps empty the slots, then take chunks
// of positions in ticket order, each the paths whose tops lie in it.  A warp's lanes load what 32 positions need besides
// the flow along their path, and the next 32 positions' inputs while the warp takes these steps one after the other,
// every lane all of them, or path by path where these are short.  It waits for the slots that its positions take: their
// paths are of lower levels, so lie at lower positions, in chunks of earlier tickets, held by warps that run.  Waits are
// bounded, by far more than the paths before can take; when one gives up, the last warp readies the counters of the walk over
// cells and sets walk[1].
//
// Bound by the chain of steps along the longest paths (55 to 120 ns a step), on large rasters also by issue (0.06 to 0.08
// ns a cell).  With one infinite cell, 1500^2 / 3000^2 / 8192^2: accu (float64) 0.89 / 2.1 / 8.9 ms a call, accu_trigger 0.79 /
// 1.9 / 7.7 ms; by the walk over cells (a dependent counter and its fences per step) 5.5 / 19 / 130 and 6.3 / 26 / 124 ms.
// Path by path up to 12 cells: 1 x 2000000 of short paths 247 -> 111 us (accu float64), 500000 x 8 685 -> 520.
constexpr int kRedoThreads = 256, kRedoChunk = 256, kRedoFill = 8192, kRedoShort = 12;
struct PathRedo {
    const int32_t* order;
    const int32_t* path_slot;
    const int32_t* slot_first;          // by position (the engine's array minus its base)
    unsigned long long* slots;
    int64_t npos, slot_base, nslots;
    const unsigned long long* flag;
    unsigned long long* walk;           // [2]
    unsigned* ctl;                      // ticket, filled chunks of slots, finished warps, a wait gave up
    long long polls;                    // poll limit of one wait
    const uint32_t* count;              // what the walk's counters start from
    uint32_t* work;
    int64_t nwords;
};

// One position of a window: its order entry and inputs, loaded ahead.
template <class Visitor>
struct RedoCell {
    typename Visitor::T x, y;
    unsigned mask;       // upstream neighbours
    int32_t slot;        // first of its slots
    __device__ __forceinline__ void load(const PathRedo& q, const Visitor& v, int64_t i, int32_t w)
    {
        const int32_t c = w & 0x7fffffff;
        const bool in = i < q.npos;
        x = in ? v.first(c) : 0;
        y = in ? v.second(c) : 0;
        mask = in ? __ldg(v.upmask + c) : 0u;
        slot = in && i >= q.slot_base ? __ldg(q.slot_first + i) : 0;
    }
};

// The paths whose tops lie in [at, stop); false: a wait gave up.
template <class Visitor>
__device__ __forceinline__ bool redo_chunk(const PathRedo& q, Visitor& v, int64_t at, int64_t stop)
{
    using Up = typename Visitor::Up;
    using T = typename Visitor::T;
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t p1 = q.npos, first = next_top(q.order, at, stop);
    if (first >= stop) return true;
    // order entries of the window and of the next one
    int32_t w = first + lane < p1 ? __ldg(q.order + first + lane) : -1;
    int32_t w1 = first + 32 + lane < p1 ? __ldg(q.order + first + 32 + lane) : -1;
    RedoCell<Visitor> cell;
    cell.load(q, v, first + lane, w);
    int32_t before_c = -1;  // the cell before the window's first
    Up flow{};
    for (int64_t i0 = first; i0 < p1; i0 += 32) {
        const int32_t c = w & 0x7fffffff;
        // the last window ends where the first path that another chunk takes begins
        const int64_t i = i0 + lane;
        const unsigned ends = __ballot_sync(kAll, i >= p1 || (i >= stop && w < 0));
        const int steps = ends ? __ffs(ends) - 1 : 32;
        const bool on = lane < steps;
        // the flow along the path (none into its top) comes in the place of its neighbour: values before it and after
        const int32_t up = __shfl_up_sync(kAll, c, 1), from = lane ? up : before_c;
        int before = 0;
        bool along = false;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (!((cell.mask >> k) & 1u) || along) continue;
            if (c + nb_dr(k) * v.cols + nb_dc(k) == from) along = true;
            else ++before;
        }
        const int n = on ? __popc(cell.mask) - (along ? 1 : 0) : 0;
        Up u[8];
        bool missing = n > 0;
        for (long long k = 0; __any_sync(kAll, missing); ++k) {
            if (k >= q.polls || __any_sync(kAll, *reinterpret_cast<volatile unsigned*>(q.ctl + 3) != 0)) return false;
            if (missing) {
                missing = false;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j < n) missing |= !read_slot(q.slots + cell.slot + j, u[j]);
            }
            if (k) __nanosleep(128);
        }
        // the next window's inputs
        RedoCell<Visitor> ahead;
        ahead.load(q, v, i + 32, w1);
        const int32_t w2 = i + 64 < p1 ? __ldg(q.order + i + 64) : -1;
        // (branches for the whole warp where a sum is rare: float64 additions that no lane needs take their time too)
        typename Visitor::Total s;
        Up then{};
        const int most = __reduce_max_sync(kAll, n);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j >= most) break;
            if (__any_sync(kAll, j < n && j < before))
                if (j < n && j < before) Visitor::add(s, u[j]);
            if (j < n && j == before) then = u[j];
        }
        const unsigned after = (unsigned)max(0, n - before);
        const unsigned bits = after | (along ? kFlow : 0u) | (along && before == 0 ? kAlone : 0u) | (s.nan ? kNone : 0u);
        Up mine{};
        T rest = T(0);
        const unsigned tops = __ballot_sync(kAll, w < 0);
        // how far a lane is from the first one of its path in the window
        const int offset = lane - (31 - __clz((tops | 1u) & (0xffffffffu >> (31 - lane))));
        const int longest = __reduce_max_sync(kAll, on ? offset : 0) + 1;
        if (longest <= kRedoShort) {  // short paths side by side
            for (int j = 0; j < longest; ++j) {
                Up in = from_lane(mine, lane ? lane - 1 : 0);
                if (lane == 0) in = flow;
                const bool turn = on && offset == j;
                typename Visitor::Total t = s;
                if (along && before == 0) t = Visitor::total(in);
                if (__any_sync(kAll, turn && along && before > 0))
                    if (along && before > 0) Visitor::add(t, in);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (k >= most) break;
                    if (__any_sync(kAll, turn && k >= before && k < n))
                        if (k >= before && k < n) Visitor::add(t, u[k]);
                }
                T r;
                const Up o = Visitor::apply(t, cell.x, cell.y, r);
                mine = turn ? o : mine;
                rest = turn ? r : rest;
            }
            flow = from_lane(mine, max(steps - 1, 0));
        } else if (__all_sync(kAll, n == 0)) {  // nothing but the flow along paths
            T x = __shfl_sync(kAll, cell.x, 0), y = __shfl_sync(kAll, cell.y, 0);
            for (int j = 0; j < steps; ++j) {
                const T x1 = __shfl_sync(kAll, cell.x, (j + 1) & 31), y1 = __shfl_sync(kAll, cell.y, (j + 1) & 31);
                // 0 + flow is the flow, bit for bit
                const typename Visitor::Total t = (tops >> j) & 1u ? typename Visitor::Total{} : Visitor::total(flow);
                T r;
                flow = Visitor::apply(t, x, y, r);
                mine = lane == j ? flow : mine;
                rest = lane == j ? r : rest;
                x = x1;
                y = y1;
            }
        } else {
            RedoStep<Visitor> now = RedoStep<Visitor>::from(s, then, bits, cell.x, cell.y, 0);
            for (int j = 0; j < steps; ++j) {
                const RedoStep<Visitor> next = RedoStep<Visitor>::from(s, then, bits, cell.x, cell.y, (j + 1) & 31);
                typename Visitor::Total t{now.t, (now.bits & kNone) != 0};
                if (now.bits & kAlone) t = Visitor::total(flow);
                else if (now.bits & kFlow) Visitor::add(t, flow);
                const unsigned more = now.bits & 15u;
                if (more) Visitor::add(t, now.then);
                if (more > 1u) {
                    const int b = __shfl_sync(kAll, before, j);
#pragma unroll
                    for (int k = 1; k < 8; ++k) {
                        const Up o = from_lane(u[k], j);
                        if (k > b && k < b + (int)more) Visitor::add(t, o);
                    }
                }
                T r;
                flow = Visitor::apply(t, now.x, now.y, r);
                mine = lane == j ? flow : mine;
                rest = lane == j ? r : rest;
                now = next;
            }
        }
        // results, and at the bottoms of paths what flows on
        int32_t below = __shfl_down_sync(kAll, w, 1);
        const int32_t next_w = __shfl_sync(kAll, w1, 0);
        if (lane == 31) below = next_w;
        if (on) {
            v.store(c, mine, rest);
            if (below < 0) {
                const int32_t slot = __ldg(q.path_slot + i);
                if (slot >= 0) write_slot(q.slots + slot, mine);
            }
        }
        if (steps < 32) break;
        before_c = __shfl_sync(kAll, c, 31);
        w = w1;
        w1 = w2;
        cell = ahead;
    }
    return true;
}

template <class Visitor>
__global__ void __launch_bounds__(kRedoThreads) k_path_redo(PathRedo q, Visitor v)
{
    constexpr unsigned kAll = 0xffffffffu;
    next_may_start();
    wait_for_previous();
    if (q.flag[1] == 0) return;
    const int lane = threadIdx.x & 31;
    unsigned *ticket = q.ctl, *filled = q.ctl + 1, *finished = q.ctl + 2, *gave_up = q.ctl + 3;
    const int64_t fills = (q.nslots + kRedoFill - 1) / kRedoFill;
    bool all_filled = false, ok = true;
    while (ok) {
        unsigned taken = 0;
        if (lane == 0) taken = atomicAdd(ticket, 1u);
        const int64_t k = __shfl_sync(kAll, taken, 0);
        if (k < fills) {
            for (int64_t i = k * kRedoFill + lane; i < min(q.nslots, (k + 1) * kRedoFill); i += 32) q.slots[i] = kEmptySlot;
            __syncwarp();
            if (lane == 0) {
                __threadfence();
                atomicAdd(filled, 1u);
            }
            continue;
        }
        for (long long j = 0; !all_filled; ++j) {
            all_filled = __all_sync(kAll, ld_acquire(filled) >= fills);
            if (j >= q.polls) break;
        }
        const int64_t at = (k - fills) * kRedoChunk;
        if (at >= q.npos) break;
        ok = all_filled && redo_chunk(q, v, at, min(at + kRedoChunk, q.npos));
        if (!ok && lane == 0) atomicExch(gave_up, 1u);
    }
    unsigned ends = 0;
    if (lane == 0) {
        __threadfence();
        ends = atomicAdd(finished, 1u);
    }
    ends = __shfl_sync(kAll, ends, 0);
    if (ends + 1u == gridDim.x * (kRedoThreads / 32) && *reinterpret_cast<volatile unsigned*>(gave_up)) {
        if (lane == 0) q.walk[1] = 1;
        for (int64_t j = lane; j < q.nwords; j += 32) q.work[j] = q.count[j];
    }
}

template <class T>
__global__ void k_path_no_data(const uint8_t* fd, int64_t n, T* out, T* rem)
{
    for (int64_t i = grid_stride_begin(); i < n; i += grid_stride())
        if (__ldg(fd + i) == kNoData) {
            out[i] = qnan<T>();
            if (rem) rem[i] = qnan<T>();
        }
}

static bool path_engine_off()
{
    const char* e = getenv("LUE_GB300_ENGINE");
    return e && (e[0] == 'w' || e[0] == 's');
}

// The path layout of t, built on first use; nullptr when the engine does not apply.  at: for rules with two results, the
// positions by cell, or nullptr where the levels write straight to the raster.
static int path_core_get(lue_gpu_topology* t, cudaStream_t stream, const PathCore** out, const int32_t** at)
{
    *out = nullptr;
    TopologyCore* core = t->core;
    if (core->stats.cycle_cells > 0) return LUE_GPU_OK;
    std::lock_guard<std::mutex> lock(core->stage_mutex);
    if (!core->paths && !core->paths_unavailable) {
        PathCore* pc = nullptr;
        const int rc = path_core_build(core, t->work_count, stream, &pc);
        if (rc == LUE_GPU_ERANGE) {
            core->paths_unavailable = true;
            return LUE_GPU_OK;
        }
        if (rc) return rc;
        core->paths = pc;
        core->bytes += pc->bytes;
    }
    if (at && core->paths) {
        // not while the call is captured: the allocation would be refused
        if (!core->paths->at_decided && !capturing(stream)) {
            if (int rc = path_at_build(core, core->paths, stream)) return rc;
            if (core->paths->at) core->bytes += core->n * 4;
        }
        *at = core->paths->at;
    }
    *out = core->paths;
    return LUE_GPU_OK;
}

void path_buffers_free(lue_gpu_topology* t)
{
    void* const buffers[2] = {t->path_maps, t->path_dense};
    pool_release(buffers, 2);
    t->path_dense = nullptr;
    t->path_maps = nullptr;
    t->path_ctl = nullptr;
    t->path_slots = nullptr;
}

// path_ctl: the redo flag and the walk's (two words of 8 bytes each), one ticket per level and the control words of
// k_path_redo, zeroed before each call, then the status words of the scan tiles.
constexpr int kPathRedoCtl = 4;
constexpr size_t kPathCtlZeroed =
    4 * sizeof(unsigned long long) + (kPathMaxLevels + 2 + kPathRedoCtl) * sizeof(int);

static int path_buffers(lue_gpu_topology* t, const PathCore* pc, cudaStream_t stream)
{
    if (t->path_maps) return LUE_GPU_OK;
    const char* what = "path engine buffers";
    if (const char* e = getenv("LUE_GB300_PATH_NO_MEMORY"))
        if (e[0] == 'b') return fail(LUE_GPU_ENOMEM, "path engine buffers: no memory (test hook)");
    if (capturing(stream))  // the buffers would belong to the graph
        return fail(LUE_GPU_ECUDA, std::string(what) + ": the first call of a handle cannot be captured (call "
                                                       "lue_gpu_topology_prepare on it first)");
    const int64_t nt = std::max<int64_t>(pc->tiles, 1), ns = std::max<int64_t>(pc->nslots, 1);
    const size_t ctl = kPathCtlZeroed + nt * sizeof(int);
    Arena plan;  // the offsets of the three in one allocation
    const size_t maps_at = plan.add(2 * nt * sizeof(PMap<kTrigger>)), ctl_at = plan.add(ctl),
                 slots_at = plan.add(ns * sizeof(double));
    void* base = nullptr;
    if (int rc = pool_allocate(&base, plan.bytes(), stream, what)) return rc;
    char* const b = static_cast<char*>(base);
    t->path_maps = b + maps_at;
    t->path_ctl = b + ctl_at;
    t->path_slots = b + slots_at;
    if (int rc = cuda_status(cudaMemsetAsync(t->path_ctl, 0, ctl, stream), what)) {
        path_buffers_free(t);
        return rc;
    }
    t->path_epoch = 0;
    t->scratch_bytes += (int64_t)plan.bytes();
    return LUE_GPU_OK;
}

// The two results of a call by position, for a handle's first call that spreads them; nullptr without the memory, or when
// that call is captured: the levels write straight to the raster.
static float2* path_dense(lue_gpu_topology* t, const PathCore* pc, cudaStream_t stream)
{
    if (!t->path_dense && !t->path_dense_tried && !capturing(stream)) {
        t->path_dense_tried = true;
        if (pc->npos > 0 && !pool_allocate(&t->path_dense, pc->npos * 8, stream, "path results"))
            t->scratch_bytes += pc->npos * 8;
    }
    return static_cast<float2*>(t->path_dense);
}

int path_prepare(lue_gpu_topology* t, cudaStream_t stream)
{
    const PathCore* pc = nullptr;
    const int32_t* at = nullptr;
    if (int rc = path_core_get(t, stream, &pc, &at)) return rc;
    return pc ? path_buffers(t, pc, stream) : LUE_GPU_OK;
}

// A level reads its order, its inputs and its first slots while the level before still runs.  Level 0 follows whatever
// wrote the inputs, so it starts after it.
template <class N, Rule R, int K, int PER, bool LIGHT>
static void launch_level(bool free, unsigned blocks, cudaStream_t stream, const PathCall<N>& p, const PathLevel& v,
                         const PathScan<K>& q, const int32_t* cut)
{
    if (!LIGHT) {
        if (free) k_path_free<N, R, K, PER, LIGHT><<<blocks, kPathThreads, 0, stream>>>(p, v, cut);
        else k_path_level<N, R, K, PER, LIGHT><<<blocks, kPathThreads, 0, stream>>>(p, v, q);
    } else {
        if (free) launch_after(k_path_free<N, R, K, PER, LIGHT>, blocks, kPathThreads, 0, stream, p, v, cut);
        else launch_after(k_path_level<N, R, K, PER, LIGHT>, blocks, kPathThreads, 0, stream, p, v, q);
    }
}

template <class N, Rule R, int K, class Visitor>
static int path_run(lue_gpu_topology* t, const PathCore* pc, const int32_t* at, const typename N::T* a, typename N::T as,
                    const typename N::T* b, typename N::T bs, typename N::T* out, typename N::T* rem,
                    const Visitor& redo, cudaStream_t stream, const char* what)
{
    const TopologyCore* core = t->core;
    const int64_t n = core->n;
    const int64_t nt_max = std::max<int64_t>(pc->tiles, 1);
    unsigned long long* flag = static_cast<unsigned long long*>(t->path_ctl);
    int* tickets = reinterpret_cast<int*>(flag + 4);
    int* redo_ctl = tickets + kPathMaxLevels + 2;
    int* status = redo_ctl + kPathRedoCtl;
    if (int rc = cuda_status(cudaMemsetAsync(flag, 0, kPathCtlZeroed, stream), what)) return rc;
    int launches = 0;
    float2* dense = at ? path_dense(t, pc, stream) : nullptr;
    if (pc->npos < n && !dense) {
        k_path_no_data<<<grid_for(n, 256), 256, 0, stream>>>(core->fd, n, out, rem);
        ++launches;
    }
    const PathCall<N> p{pc->order, pc->path_slot, pc->slot_first - pc->slot_base, a, as, b, bs, out, rem,
                        static_cast<typename N::Slot*>(t->path_slots), dense, flag};
    // test hooks: LUE_GB300_PATH_FREE_LONGEST (levels with longer paths use the look-back scan; 0: every
    // level) and LUE_GB300_PATH_POLLS (poll limit of a look-back wait; 0: every wait gives up at once,
    // and the walk engine redoes the call)
    int free_longest = -1, polls = kPathPolls;
    if (const char* e = getenv("LUE_GB300_PATH_FREE_LONGEST")) free_longest = std::max(0, atoi(e));
    if (const char* e = getenv("LUE_GB300_PATH_POLLS")) polls = std::max(0, atoi(e));
    PMap<K>* aggm = static_cast<PMap<K>*>(t->path_maps);
    for (size_t l = 0; l < pc->levels.size(); ++l) {
        const PathLevel& v = pc->levels[l];
        if (++t->path_epoch >= (1 << 28)) {  // status words of old launches could match again: clear them
            t->path_epoch = 1;
            if (int rc = cuda_status(cudaMemsetAsync(status, 0, nt_max * sizeof(int), stream), what)) return rc;
        }
        const int T = kPathThreads * v.per;
        const bool free = v.longest <= (free_longest >= 0 ? free_longest : path_free_longest(v.per));
        const unsigned blocks =
            free ? (unsigned)v.ncut : (unsigned)((v.p1 - (v.p0 & ~(v.per - 1)) + T - 1) / T);
        if (blocks == 0) continue;
        const PathScan<K> q{status, aggm, aggm + nt_max, tickets + l, t->path_epoch, polls};
        if (l == 0) {
            if (v.per == 1) launch_level<N, R, K, 1, false>(free, blocks, stream, p, v, q, pc->cut);
            else launch_level<N, R, K, 4, false>(free, blocks, stream, p, v, q, pc->cut);
        } else {
            if (v.per == 1) launch_level<N, R, K, 1, true>(free, blocks, stream, p, v, q, pc->cut);
            else launch_level<N, R, K, 2, true>(free, blocks, stream, p, v, q, pc->cut);
        }
        ++launches;
    }
    if constexpr (R != Rule::accu) {
        if (dense) {
            const int64_t tcols = (core->cols + kPathTile - 1) / kPathTile, trows = (core->rows + kPathTile - 1) / kPathTile;
            k_path_spread<<<(unsigned)(trows * tcols), 256, 0, stream>>>(at, dense, core->rows, core->cols, tcols, out, rem);
            ++launches;
        }
    }
    // the redo behind it; test hook: LUE_GB300_PATH_REDO_POLLS (poll limit of its waits; 0: each gives up at once, and
    // the walk engine does the call).  A step along a path takes about a microsecond, and so does a poll.
    int64_t chain = 0;
    for (const PathLevel& v : pc->levels) chain += v.longest;
    long long redo_polls = (1ll << 20) + 4 * chain + pc->npos / 64;
    if (const char* e = getenv("LUE_GB300_PATH_REDO_POLLS")) redo_polls = std::max(0, atoi(e));
    const PathRedo r{pc->order, pc->path_slot, p.slot_first, static_cast<unsigned long long*>(t->path_slots), pc->npos,
                     pc->slot_base, pc->nslots, flag, flag + 2, reinterpret_cast<unsigned*>(redo_ctl), redo_polls,
                     reinterpret_cast<const uint32_t*>(core->count), t->work_count, words_for(n)};
    launch_after(k_path_redo<Visitor>, grid_for(pc->npos, kRedoChunk * (kRedoThreads / 32), 152 * 4), kRedoThreads, 0, stream,
                 r, redo);
    WalkGrid g{core->fd, core->count, t->work_count, core->rows, core->cols, n};
    launch_after(k_walk_if<Visitor>, grid_for(n, 256), 256, 0, stream, g, redo, (const unsigned long long*)(flag + 2));
    count_launches(launches + 2);
    return cuda_status(cudaGetLastError(), what);
}

template <Rule R, int K>
static int path_run_f32(lue_gpu_topology* t, const PathCore* pc, const int32_t* at, const float* a, float as,
                        const float* b, float bs, float* out, float* rem, cudaStream_t stream, const char* what)
{
    const RouteF32<R> redo{t->core->upmask, a, as, b, bs, out, rem, t->lo, t->core->cols};
    return path_run<F32, R, K>(t, pc, at, a, as, b, bs, out, rem, redo, stream, what);
}

// Layout and buffers for a call; *pc is nullptr when there are none, also for want of memory: the stage engine, which
// then takes the call, builds other structures, which may fit (the layout takes 20 bytes a cell while it is built).
static int path_ready(lue_gpu_topology* t, cudaStream_t stream, const PathCore** pc, const int32_t** at)
{
    int rc = path_core_get(t, stream, pc, at);
    if (!rc && *pc) rc = path_buffers(t, *pc, stream);
    if (rc != LUE_GPU_ENOMEM) return rc;
    *pc = nullptr;
    return LUE_GPU_OK;
}

// A call in place: its inputs are overwritten before a redo would read them.
static bool overlap(const lue_gpu_topology* t, const void* in, const void* out, size_t size)
{
    const char *a = static_cast<const char*>(in), *b = static_cast<const char*>(out);
    const size_t bytes = (size_t)t->core->n * size;
    return a && b && a < b + bytes && b < a + bytes;
}

int path_route_f32(lue_gpu_topology* t, int rule, const float* a, float as, const float* b, float bs, float* out,
                   float* rem, cudaStream_t stream, bool* done)
{
    *done = false;
    if (path_engine_off()) return LUE_GPU_OK;
    if (rule < (int)Rule::threshold || rule > (int)Rule::trigger) return LUE_GPU_OK;
    if (rule == (int)Rule::trigger &&
        (overlap(t, a, out, 4) || overlap(t, a, rem, 4) || overlap(t, b, out, 4) || overlap(t, b, rem, 4)))
        return LUE_GPU_OK;
    const PathCore* pc = nullptr;
    const int32_t* at = nullptr;
    if (int rc = path_ready(t, stream, &pc, &at)) return rc;
    if (!pc) return LUE_GPU_OK;
    *done = true;
    if (rule == (int)Rule::threshold)
        return path_run_f32<Rule::threshold, kMaxPlus>(t, pc, at, a, as, b, bs, out, rem, stream,
                                                       "accu_threshold_f32 (paths)");
    if (rule == (int)Rule::fraction)
        return path_run_f32<Rule::fraction, kAffine>(t, pc, at, a, as, b, bs, out, rem, stream,
                                                     "accu_fraction_f32 (paths)");
    if (rule == (int)Rule::trigger)
        return path_run_f32<Rule::trigger, kTrigger>(t, pc, at, a, as, b, bs, out, rem, stream,
                                                     "accu_trigger_f32 (paths)");
    return path_run_f32<Rule::capacity, kMinPlus>(t, pc, at, a, as, b, bs, out, rem, stream, "accu_capacity_f32 (paths)");
}

int path_accu_f64(lue_gpu_topology* t, const double* a, double as, double* out, cudaStream_t stream, bool* done)
{
    *done = false;
    if (path_engine_off() || overlap(t, a, out, 8)) return LUE_GPU_OK;
    const PathCore* pc = nullptr;
    if (int rc = path_ready(t, stream, &pc, nullptr)) return rc;
    if (!pc) return LUE_GPU_OK;
    *done = true;
    const RouteF64<Rule::accu> redo{t->core->upmask, a, as, nullptr, 0.0, out, nullptr, t->core->cols};
    return path_run<F64, Rule::accu, kSum>(t, pc, nullptr, a, as, nullptr, 0.0, out, nullptr, redo, stream,
                                           "accu_f64 (paths)");
}

}  // namespace lue_gb300
