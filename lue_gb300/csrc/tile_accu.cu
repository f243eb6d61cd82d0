// tile_accu.cu — tiled accu engine (see tile_accu.cuh): topology build and per-call kernels.
#include <algorithm>
#include <cstring>

#include "tile_accu.cuh"
#include "topology.cuh"

namespace lue_gb300 {

typedef unsigned __int128 u128;

__device__ __forceinline__ u128 to_u128(uint4 v)
{
    return ((u128)v.w << 96) | ((u128)v.z << 64) | ((u128)v.y << 32) | (u128)v.x;
}
__device__ __forceinline__ uint4 from_u128(u128 v)
{
    return make_uint4((unsigned)v, (unsigned)(v >> 32), (unsigned)(v >> 64), (unsigned)(v >> 96));
}
__device__ __forceinline__ u128 shfl_up_u128(u128 v, int d)
{
    uint4 a = from_u128(v);
    a.x = __shfl_up_sync(0xffffffffu, a.x, d);
    a.y = __shfl_up_sync(0xffffffffu, a.y, d);
    a.z = __shfl_up_sync(0xffffffffu, a.z, d);
    a.w = __shfl_up_sync(0xffffffffu, a.w, d);
    return to_u128(a);
}
__device__ __forceinline__ u128 shfl_down_u128(u128 v, int d)
{
    uint4 a = from_u128(v);
    a.x = __shfl_down_sync(0xffffffffu, a.x, d);
    a.y = __shfl_down_sync(0xffffffffu, a.y, d);
    a.z = __shfl_down_sync(0xffffffffu, a.z, d);
    a.w = __shfl_down_sync(0xffffffffu, a.w, d);
    return to_u128(a);
}

constexpr u128 kPoison = (u128)1 << 96;                 // one no-data exit
constexpr u128 kValueMask = ((u128)1 << 96) - 1;

// Fixed-point scale: values are stored as round(v * 2^F).  F is chosen per call from an upper bound on
// the material total (in 2^-16 units) so that every prefix sum stays below 2^95.
__device__ __forceinline__ int fixed_point_bits(unsigned long long total_units)
{
    int bl = total_units ? 64 - __clzll((long long)total_units) : 0;
    int f = 111 - bl;
    return f > 100 ? 100 : (f < -100 ? -100 : f);
}

// |x| * 2^F rounded to nearest (ties up; 0 below 2^-40, 0 from 2^128 up), as a 128-bit two's-complement
// integer with the sign of x.  Built from 32-bit words: the 24-bit mantissa shifted by s & 31 spans two
// words, placed at word s >> 5, so no 128-bit variable shift is needed.
__device__ __forceinline__ u128 float_to_fixed(float x, int F)
{
    const unsigned bits = __float_as_uint(x);
    const unsigned e8 = (bits >> 23) & 0xFFu;
    const unsigned mant = (bits & 0x7FFFFFu) | (e8 ? 0x800000u : 0u);
    const int s = (int)(e8 ? e8 : 1u) - 150 + F;  // value = mant * 2^(e - 150) * 2^F
    unsigned long long lo = 0, hi = 0;
    if (s >= 0) {
        if (s < 104) {
            const int k = s >> 5;
            const unsigned b = (unsigned)s & 31u;
            const unsigned w0 = mant << b, w1 = __funnelshift_l(mant, 0u, b);
            const unsigned long long pair = ((unsigned long long)w1 << 32) | w0;
            const unsigned long long up = (unsigned long long)w0 << 32;
            lo = k == 0 ? pair : (k == 1 ? up : 0ull);
            hi = k == 1 ? (unsigned long long)w1 : (k == 2 ? pair : (k == 3 ? up : 0ull));
        }
    } else if (s > -40) {
        lo = ((unsigned long long)mant + (1ull << (-s - 1))) >> (-s);
    }
    if (bits >> 31) {  // two's complement
        hi = ~hi + (lo == 0 ? 1ull : 0ull);
        lo = 0ull - lo;
    }
    return ((u128)hi << 64) | lo;
}

__device__ __forceinline__ u128 exit_value_fixed(float2 v, int F)
{
    if (isnan(v.x) || isnan(v.y)) return kPoison;
    return float_to_fixed(v.x, F) + float_to_fixed(v.y, F);
}

// ---------------------------------------------------------------------------------------------------
// Build
// ---------------------------------------------------------------------------------------------------

struct TileGeom {
    int64_t rows, cols, trows, tcols;
};

__device__ __forceinline__ int64_t tile_of(const TileGeom& g, int64_t r, int64_t c)
{
    return (r / kTile) * g.tcols + c / kTile;
}

// Whether the flow of in-tile cell (rin, cin) leaves the tile but not the array.
__device__ __forceinline__ bool leaves_tile(const uint8_t* __restrict__ fd, const TileGeom& g, int64_t tr, int64_t tc,
                                            int rin, int cin)
{
    const int64_t r = tr * kTile + rin, c = tc * kTile + cin;
    int dr, dc;
    if (r >= g.rows || c >= g.cols) return false;
    const uint8_t code = __ldg(fd + r * g.cols + c);
    if (code == kNoData || !d8_offset(code, dr, dc)) return false;
    const int64_t rd = r + dr, cd = c + dc;
    if (rd < 0 || rd >= g.rows || cd < 0 || cd >= g.cols) return false;
    return rin + dr < 0 || rin + dr >= kTile || cin + dc < 0 || cin + dc >= kTile;
}

// Exits of a tile, one warp each: a 64-bit word per tile row (bit c: that cell is an exit; only border cells can
// be), the exits in the rows before each row, and their number.
__global__ void __launch_bounds__(256) k_exit_bitmap(const uint8_t* __restrict__ fd, TileGeom g, uint64_t* bitmap,
                                                     uint16_t* rowpref, int32_t* count)
{
    __shared__ uint64_t s_rows[8][kTile];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t tile = (int64_t)blockIdx.x * 8 + warp;
    if (tile >= g.trows * g.tcols) return;
    const int64_t tr = tile / g.tcols, tc = tile - tr * g.tcols;
    uint64_t* rows = s_rows[warp];
    for (int k = 0; k < 2; ++k) {  // the whole first and last row
        const int rin = k * (kTile - 1);
        const unsigned lo = __ballot_sync(0xffffffffu, leaves_tile(fd, g, tr, tc, rin, lane));
        const unsigned hi = __ballot_sync(0xffffffffu, leaves_tile(fd, g, tr, tc, rin, lane + 32));
        if (lane == 0) rows[rin] = ((uint64_t)hi << 32) | lo;
    }
    for (int rin = 1 + lane; rin < kTile - 1; rin += 32)
        rows[rin] = (leaves_tile(fd, g, tr, tc, rin, 0) ? 1ull : 0ull) |
                    (leaves_tile(fd, g, tr, tc, rin, kTile - 1) ? 1ull << (kTile - 1) : 0ull);
    __syncwarp();
    int before = 0;
    for (int k = 0; k < 2; ++k) {
        const int rin = 32 * k + lane;
        const uint64_t m = rows[rin];
        const int n = __popcll(m);
        int x = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        bitmap[tile * kTile + rin] = m;
        rowpref[tile * kTile + rin] = (uint16_t)(before + x - n);
        before += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) count[tile] = before;
}

// The number of exits of the raster, one warp per tile.
__global__ void __launch_bounds__(256) k_exit_count(const uint8_t* __restrict__ fd, TileGeom g, unsigned long long* total)
{
    const int lane = threadIdx.x & 31;
    const int64_t tile = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (tile >= g.trows * g.tcols) return;
    const int64_t tr = tile / g.tcols, tc = tile - tr * g.tcols;
    int n = 0;
#pragma unroll
    for (int k = 0; k < kTile; k += 32) {
        const int i = k + lane;
        n += leaves_tile(fd, g, tr, tc, 0, i) + leaves_tile(fd, g, tr, tc, kTile - 1, i);
        if (i > 0 && i < kTile - 1) n += leaves_tile(fd, g, tr, tc, i, 0) + leaves_tile(fd, g, tr, tc, i, kTile - 1);
    }
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0 && n) atomicAdd(total, (unsigned long long)n);
}

// Exclusive sums of up to two arrays of n counts (one CTA), with their totals at [n].
__global__ void __launch_bounds__(1024) k_tile_scan(const int32_t* a, int32_t* a_base, const int32_t* b, int32_t* b_base,
                                                    int64_t n)
{
    __shared__ int s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < (b ? 2 : 1); ++k) {
        const int32_t* x = k ? b : a;
        int32_t* base = k ? b_base : a_base;
        const int64_t per = (n + 1023) / 1024;
        const int64_t i0 = min(n, (int64_t)threadIdx.x * per), i1 = min(n, i0 + per);
        int sum = 0;
        for (int64_t i = i0; i < i1; ++i) sum += x[i];
        int v = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        if (lane == 31) s_warp[warp] = v;
        __syncthreads();
        int before = v - sum;
        for (int w = 0; w < warp; ++w) before += s_warp[w];
        for (int64_t i = i0; i < i1; ++i) {
            base[i] = before;
            before += x[i];
        }
        if (threadIdx.x == 1023) base[n] = before;
        __syncthreads();
    }
}

__device__ __forceinline__ int32_t exit_id_of(const TileGeom& g, const int32_t* exit_base, const uint64_t* bitmap,
                                               const uint16_t* rowpref, int64_t r, int64_t c)
{
    int64_t tile = tile_of(g, r, c);
    int rin = (int)(r % kTile), cin = (int)(c % kTile);
    uint64_t word = bitmap[tile * kTile + rin];
    return exit_base[tile] + rowpref[tile * kTile + rin] + __popcll(word & ((1ull << cin) - 1ull));
}

constexpr int kExitCounters = 5;  // children, children to come, positions handed out, depth, position seen

__global__ void k_exit_list(TileGeom g, const uint64_t* bitmap, const uint16_t* rowpref, const int32_t* exit_base,
                            uint16_t* exit_local, uint32_t* exit_cell, uint32_t* size, int32_t* zero, int64_t stride)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.trows * g.tcols * kTile) return;
    int64_t tile = i / kTile;
    int rin = (int)(i % kTile);
    int64_t tr = tile / g.tcols, tc = tile % g.tcols;
    uint64_t m = bitmap[i];
    int32_t id = exit_base[tile] + rowpref[i];
    while (m) {
        int cin = __ffsll((long long)m) - 1;
        m &= m - 1;
        exit_local[id] = (uint16_t)(rin * kTile + cin);
        exit_cell[id] = (uint32_t)((tr * kTile + rin) * g.cols + tc * kTile + cin);
        size[id] = 1;
        for (int k = 0; k < kExitCounters; ++k) zero[k * stride + id] = 0;
        ++id;
    }
}

// Border cell b (0..251: N row, S row, W column, E column without corners) of a tile.
__device__ __forceinline__ void border_cell(int b, int& rin, int& cin)
{
    if (b < kTile) { rin = 0; cin = b; }
    else if (b < 2 * kTile) { rin = kTile - 1; cin = b - kTile; }
    else if (b < 3 * kTile - 2) { rin = b - 2 * kTile + 1; cin = 0; }
    else { rin = b - (3 * kTile - 2) + 1; cin = kTile - 1; }
}

// The border cell at (rin, cin).
__device__ __forceinline__ int border_index(int rin, int cin)
{
    if (rin == 0) return cin;
    if (rin == kTile - 1) return kTile + cin;
    return (cin == 0 ? 2 * kTile : 3 * kTile - 2) + rin - 1;
}

// Parent of every exit: the root of its downstream cell in that cell's tile, if an exit.  plus: the cells from the exit
// to its parent.
// The roots come from k_tile_forest, which walks to them in shared memory: walking here, a round trip to memory per
// cell, took 33 us at 2048^2 instead of 6.
__global__ void k_exit_parent(const uint8_t* __restrict__ fd, TileGeom g, const int32_t* nexit, const uint32_t* exit_cell,
                              const int32_t* exit_base, const uint64_t* bitmap, const uint16_t* rowpref,
                              const uint32_t* __restrict__ border_root, int32_t* parent, int32_t* nchild, int32_t* pending,
                              int32_t* plus)
{
    int64_t y = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (y >= *nexit) return;
    const int64_t cell = exit_cell[y];
    int64_t r = cell / g.cols, c = cell % g.cols;
    int dr, dc;
    d8_offset(fd[cell], dr, dc);
    r += dr;
    c += dc;
    int32_t p = -1;
    if (fd[r * g.cols + c] != kNoData) {
        const int64_t tile = tile_of(g, r, c);
        const uint32_t root = border_root[tile * kBorderCells + border_index((int)(r % kTile), (int)(c % kTile))];
        const int rin = (int)((root & kIndexMask) >> 6), cin = (int)(root & 63u);
        const uint64_t m = bitmap[tile * kTile + rin];
        if ((m >> cin) & 1ull)
            p = exit_base[tile] + rowpref[tile * kTile + rin] + __popcll(m & ((1ull << cin) - 1ull));
        plus[y] = (int32_t)(root >> 12) + 1;
    }
    parent[y] = p;
    if (p >= 0) {
        atomicAdd(nchild + p, 1);
        atomicAdd(pending + p, 1);
    }
}

// Subtree sizes, downstream levels and depth of the exit forest, with the counter walk of walk.cuh on the coarse
// forest.  level: on entry each exit's level within its tile.  A subtree below a cycle never finishes.
__global__ void k_exit_sizes(const int32_t* nexit, const int32_t* parent, const int32_t* nchild, const int32_t* plus,
                             int32_t* pending, uint32_t* size, int32_t* level, int32_t* depth, int* max_depth)
{
    int64_t y = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (y >= *nexit || nchild[y] != 0) return;
    uint32_t s = 1;
    int32_t d = 1, lv = level[y];
    for (;;) {
        int32_t p = parent[y];
        if (p < 0) {
            if (d > *(volatile int*)max_depth) atomicMax(max_depth, d);
            return;
        }
        atomicAdd(size + p, s);
        atomicMax(depth + p, d + 1);
        atomicMax(level + p, lv + plus[y]);
        __threadfence();
        if (atomicSub(pending + p, 1) != 1) return;
        __threadfence();
        s = atomicAdd(size + p, 0u);
        d = atomicAdd(depth + p, 0);
        lv = atomicAdd(level + p, 0);
        y = p;
    }
}

// The exit forest in post-order: link[y] = (offset of y's position from its parent's, the parent); the subtrees of a
// parent's children follow one another in any order.
__global__ void k_exit_offsets(const int32_t* nexit, const int32_t* parent, const int32_t* pending, const uint32_t* size,
                               uint32_t* acc, unsigned* root_acc, int2* link, int* cyclic)
{
    const int64_t y = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool in = y < *nexit;
    const int32_t p = in ? parent[y] : 0;
    const unsigned own = in ? size[y] : 0u;
    if (in && pending[y] != 0) atomicExch(cyclic, 1);
    // roots: one atomic per warp
    unsigned x = in && p < 0 ? own : 0u;
    const unsigned mine = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned z = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += z;
    }
    unsigned base = 0;
    if (lane == 31 && x) base = atomicAdd(root_acc, x);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (!in) return;
    const unsigned off = p >= 0 ? atomicAdd(acc + p, own) - size[p] : base + x - mine - 1u;
    link[y] = make_int2((int)(off + own), p);
}

// Pointer jumping, in place: position(y) = offset + position(parent) holds for every link at any time, and a link is
// read and written as one 8-byte word.
__global__ void k_jump(int64_t nexit, int2* link)
{
    const int64_t y = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (y >= nexit) return;
    unsigned long long* words = reinterpret_cast<unsigned long long*>(link);
    const unsigned long long w = __ldcg(words + y);
    const int j = (int)(w >> 32);
    if (j < 0) return;
    const unsigned long long wj = __ldcg(words + j);
    __stcg(words + y, (wj & 0xFFFFFFFF00000000ull) | (unsigned)((unsigned)w + (unsigned)wj));
}

// Positions from the links, checked: every post-order position must be a distinct index in [0, nexit) with start <= pos
// (the per-call kernels scatter and gather with them, so the build refuses a forest that fails this check).
__global__ void k_exit_positions(int64_t nexit, const int2* link, const uint32_t* size, uint32_t* pos, uint32_t* start,
                                 int32_t* seen, int* error)
{
    int64_t y = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (y >= nexit) return;
    const int2 l = link[y];
    const uint32_t p = (uint32_t)l.x, s = p - size[y] + 1u;
    if (l.y >= 0 || p >= (uint64_t)nexit || s > p) {
        pos[y] = start[y] = 0;
        atomicExch(error, 1);
        return;
    }
    pos[y] = p;
    start[y] = s;
    if (atomicAdd(seen + p, 1) != 0) atomicExch(error, 1);
}

// ---------------------------------------------------------------------------------------------------
// Build: per-tile flow forests in post-order
// ---------------------------------------------------------------------------------------------------

constexpr uint16_t kNoCell = 0xFFFFu;

// 49 KB: four CTAs of k_tile_forest on an SM.
struct __align__(16) TileSmem {
    uint32_t cell[kTileCells];     // high half: in-tile inflows to come, then the cell's round (its downstream level within
                                   // the tile), then its subtree's first position; low half: the size of its subtree
    uint16_t dsl[kTileCells];      // downstream cell inside the tile, or kNoCell
    uint16_t queue[kTileCells];    // cells in the order they become ready (each cell once)
    uint16_t rstart[kTileCells + 1];  // round starts in the queue
    __align__(16) uint8_t up[kTileCells];  // in-tile upstream mask
    uint8_t fd[kHalo][kHalo + 2];  // flow direction with a one-cell halo (255 outside the array)
    int warp_tot[kTileThreads / 32];
    int edges;                     // flow edges into the tile
    int rounds;
    int round_count[3];            // cells queued for the next rounds (a ring of three counters)
};

// Downstream cell of in-tile cell (rin, cin) with flow direction `code`, if the flow goes to another cell of the tile;
// q: the neighbour (nb_dr order) that the cell is to it.
__device__ __forceinline__ bool tile_downstream(unsigned code, int rin, int cin, int& d, int& q)
{
    const unsigned pad = code - 1u;  // numeric pad: 0 .. 8 from the lower left, 4 in the middle
    if (pad > 8u || pad == 4u) return false;
    const int up = (int)(pad * 11u >> 5), right = (int)pad - 3 * up;  // 0, 1, 2
    const int r = rin + 1 - up, c = cin + right - 1;
    d = r * kTile + c;
    const int seen = up * 3 + 2 - right;
    q = seen - (seen > 4);
    return (unsigned)r < (unsigned)kTile && (unsigned)c < (unsigned)kTile;
}

// Load the flow direction with halo; fill in-tile upstream masks, cell words and downstream indices, and
// queue the cells without in-tile inflow (the first round).  Returns the number of queued cells.
__device__ __forceinline__ int tile_prepare(TileSmem& sm, const uint8_t* __restrict__ fd, const TileGeom& g,
                                            int64_t tr, int64_t tc)
{
    const int t = threadIdx.x, lane = t & 31;
    for (int hr = t >> 5; hr < kHalo; hr += kTileThreads / 32) {
        const int64_t r = tr * kTile + hr - 1;
        const bool row_in = r >= 0 && r < g.rows;
        for (int hc = lane; hc < kHalo; hc += 32) {
            const int64_t c = tc * kTile + hc - 1;
            sm.fd[hr][hc] = row_in && c >= 0 && c < g.cols ? __ldg(fd + r * g.cols + c) : kNoData;
        }
    }
    uint32_t* up = reinterpret_cast<uint32_t*>(sm.up);
    for (int i = t; i < kTileCells; i += kTileThreads) sm.cell[i] = 1u;
    for (int i = t; i < kTileCells / 4; i += kTileThreads) up[i] = 0u;
    if (t < 3) sm.round_count[t] = 0;
    if (t == 3) sm.edges = 0;
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < kTileCells / kTileThreads; ++k) {
        const int i = t + k * kTileThreads, rin = i >> 6, cin = i & 63;
        int d = kNoCell, e, q;
        if (tile_downstream(sm.fd[rin + 1][cin + 1], rin, cin, e, q) &&
            sm.fd[(e >> 6) + 1][(e & 63) + 1] != kNoData) {
            d = e;
            atomicAdd(sm.cell + d, 0x10000u);
            atomicOr(up + (d >> 2), 1u << (8 * (d & 3) + q));
        }
        sm.dsl[i] = (uint16_t)d;
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < kTileCells / kTileThreads; ++k) {
        // first round: valid cells without in-tile inflow (warp-aggregated queue appends)
        const int i = t + k * kTileThreads;
        const bool start = sm.cell[i] == 1u && sm.fd[(i >> 6) + 1][(i & 63) + 1] != kNoData;
        const unsigned ballot = __ballot_sync(0xffffffffu, start);
        int base = 0;
        if (lane == 0 && ballot) base = atomicAdd(&sm.round_count[0], __popc(ballot));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (start) sm.queue[base + __popc(ballot & ((1u << lane) - 1u))] = (uint16_t)i;
    }
    __syncthreads();
    return sm.round_count[0];
}

// In-tile linear offset of neighbour q (NW N NE W E SW S SE).
__device__ __forceinline__ int tile_nb_offset(int q)
{
    static_assert(kTile == 64, "neighbour offsets are packed for 64-cell rows");
    // -65 -64 -63 -1 +1 +63 +64 +65 as signed bytes
    return (int)(signed char)(unsigned)(0x41403F01FFC1C0BFull >> (8 * q));
}

// Neighbour index (0..7, NW N NE W E SW S SE) of in-tile cell c as seen from its downstream cell d.
__device__ __forceinline__ int nb_index_from(int d, int c)
{
    const int idx = ((c >> 6) - (d >> 6) + 1) * 3 + ((c & 63) - (d & 63) + 1);
    return idx < 4 ? idx : idx - 1;
}

// Exclusive prefix of one int per thread over the block; `total` gets the block sum.
__device__ __forceinline__ int block_exclusive_int(int v, int* warp_tot, int& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    int before = 0;
    total = 0;
    for (int w = 0; w < kTileThreads / 32; ++w) {
        const int s = warp_tot[w];
        before += w < warp ? s : 0;
        total += s;
    }
    __syncthreads();  // warp_tot may be reused
    return before + x - v;
}

// Build: the flow forest of one tile (CTA per tile), in post-order.  A cell's in-tile upstream cells
// (its subtree) get the positions start .. pos - 1 and the cell itself pos, so that the accu of any cell
// is the difference of two prefix sums over the material laid out in post-order.  Cells with a no-data
// flow direction (or outside the array) take the positions after the valid cells, flagged kNoValue.
// Also: each exit's scan slots (its own, and the one before its subtree), the cells' and exits' levels within the
// tile, and, per border cell, which outside neighbours drain into it.
// Bound by issue and by the chain of rounds (2048^2 fractal terrain: 126 us, 2.1 instructions per cycle; with separate
// sweeps for counts and sizes, block barriers in every round and the tables stored cell by cell 264 us).
__global__ void __launch_bounds__(kTileThreads)
    k_tile_forest(const uint8_t* __restrict__ fd, TileGeom g, const int32_t* __restrict__ exit_base,
                  const uint16_t* __restrict__ exit_local, uint16_t* cell_at, uint16_t* prev_at,
                  uint32_t* exit_span, uint8_t* border_in, int32_t* nslot, int32_t* nedge, int32_t* exit_level,
                  int32_t* __restrict__ level, uint32_t* __restrict__ border_root, int* error, int* cyclic)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileSmem& sm = *reinterpret_cast<TileSmem*>(smem_raw);
    const int64_t tr = blockIdx.y, tc = blockIdx.x;  // grid = (tile columns, tile rows)
    const int64_t tile = tr * g.tcols + tc;
    const int t = threadIdx.x, lane = t & 31;
    uint16_t* rstart = sm.rstart;
    const uint16_t* sz = reinterpret_cast<const uint16_t*>(sm.cell);  // [2 i] subtree size of cell i
    uint16_t* st = reinterpret_cast<uint16_t*>(sm.cell) + 1;          // [2 i] its round, then its first position
    int head = 0, count = tile_prepare(sm, fd, g, tr, tc), r = 0;
    // rounds: a round holds the cells whose in-tile upstream cells are all in earlier rounds; each hands its subtree's
    // size down.  No round has more cells than the one before it: from the first with at most 32 on, one warp goes
    // on without block barriers.
    while (count > 32) {
        int* next = &sm.round_count[(r + 1) % 3];
        const int next_base = head + count;
        if (t == 0) {
            rstart[r] = (uint16_t)head;
            sm.round_count[(r + 2) % 3] = 0;  // read by everyone two rounds ago
        }
        for (int k0 = 0; k0 < count; k0 += kTileThreads) {
            const int k = k0 + t;
            int d = kNoCell;
            bool ready = false;
            if (k < count) {
                const int i = sm.queue[head + k];
                const unsigned size = sm.cell[i] & 0xFFFFu;
                sm.cell[i] = ((unsigned)r << 16) | size;
                d = sm.dsl[i];
                if (d != kNoCell) ready = atomicAdd(sm.cell + d, size - 0x10000u) >> 16 == 1u;
            }
            unsigned ballot = __ballot_sync(0xffffffffu, ready);
            int base = 0;
            if (lane == 0 && ballot) base = atomicAdd(next, __popc(ballot));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (ready) sm.queue[next_base + base + __popc(ballot & ((1u << lane) - 1u))] = (uint16_t)d;
        }
        __syncthreads();
        head = next_base;
        count = *next;
        ++r;
    }
    const int wide = r;  // rounds of more than 32 cells
    if (t < 32) {
        int i = t < count ? sm.queue[head + t] : kNoCell, d = i != kNoCell ? sm.dsl[i] : kNoCell;
        unsigned size = i != kNoCell ? sm.cell[i] & 0xFFFFu : 0u;
        while (count > 0) {
            if (t == 0) rstart[r] = (uint16_t)head;
            if (i != kNoCell) sm.cell[i] = ((unsigned)r << 16) | size;
            bool ready = false;
            int after = kNoCell;
            if (d != kNoCell) {
                after = sm.dsl[d];
                const unsigned old = atomicAdd(sm.cell + d, size - 0x10000u);
                ready = old >> 16 == 1u;
                size = (old + size) & 0xFFFFu;
            }
            const unsigned ballot = __ballot_sync(0xffffffffu, ready);
            head += count;
            count = __popc(ballot);
            if (ready) sm.queue[head + __popc(ballot & ((1u << lane) - 1u))] = (uint16_t)d;
            i = ready ? d : kNoCell;
            d = ready ? after : kNoCell;
            ++r;
        }
        if (t == 0) {
            rstart[r] = (uint16_t)head;
            sm.rounds = r;
        }
    }
    // per border cell, the neighbours outside the tile that drain into it
    unsigned outside = 0;
    if (t < kBorderCells) {
        int rin, cin;
        border_cell(t, rin, cin);
        if (sm.fd[rin + 1][cin + 1] != kNoData) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int hr = rin + nb_dr(q), hc = cin + nb_dc(q);
                if (hr >= 0 && hr < kTile && hc >= 0 && hc < kTile) continue;
                if (sm.fd[hr + 1][hc + 1] == nb_inflow_code(q)) outside |= 1u << q;
            }
        }
        border_in[tile * kBorderCells + t] = (uint8_t)outside;
        if (outside) {  // where that flow leaves the tile or ends
            int i = rin * kTile + cin, steps = 0;
            for (int d; (d = sm.dsl[i]) != kNoCell && steps < kTileCells; ++steps) i = d;
            border_root[tile * kBorderCells + t] = (uint32_t)i | ((uint32_t)steps << 12);
        }
    }
    const int slots = __syncthreads_count(outside != 0);
    int edges = __popc(outside);
    edges = __reduce_add_sync(0xffffffffu, edges);
    if (lane == 0) atomicAdd(&sm.edges, edges);
    __syncthreads();
    if (t == 0) {
        nslot[tile] = slots;
        nedge[tile] = sm.edges;
    }
    const int rounds = sm.rounds, nvalid = rstart[rounds];
    // roots (valid cells without an in-tile downstream cell) and invalid cells, in cell order: warp w owns the cells
    // 512 w .. 512 w + 511
    const int own = (t >> 5) * (kTileCells / (kTileThreads / 32)) + lane;
    int root_sum = 0, invalid = 0;
    for (int i = own; i < own + 512; i += 32) {
        if (sm.fd[(i >> 6) + 1][(i & 63) + 1] == kNoData) ++invalid;
        else if (sm.dsl[i] == kNoCell) root_sum += sz[2 * i];
    }
    root_sum = __reduce_add_sync(0xffffffffu, root_sum);
    invalid = __reduce_add_sync(0xffffffffu, invalid);
    int root_total, invalid_total;
    int root_base = block_exclusive_int(lane == 31 ? root_sum : 0, sm.warp_tot, root_total);
    int invalid_base = root_total + block_exclusive_int(lane == 31 ? invalid : 0, sm.warp_tot, invalid_total);
    root_base = __shfl_sync(0xffffffffu, root_base, 31);
    invalid_base = __shfl_sync(0xffffffffu, invalid_base, 31);
    const int32_t e0 = exit_base[tile], ne = exit_base[tile + 1] - e0;
    if (nvalid + invalid_total != kTileCells) {  // uniform: cells on a cycle never become ready
        // only the levels: -1 on the cycle (no cell drains out of one, so all others are in the queue)
        uint32_t* ready = reinterpret_cast<uint32_t*>(sm.up);
        for (int w = t; w < kTileCells / 32; w += kTileThreads) ready[w] = 0;
        __syncthreads();
        for (int k = t; k < nvalid; k += kTileThreads) atomicOr(ready + (sm.queue[k] >> 5), 1u << (sm.queue[k] & 31));
        __syncthreads();
        for (int i = t; i < kTileCells; i += kTileThreads) {
            const int64_t row = tr * kTile + (i >> 6), col = tc * kTile + (i & 63);
            if (row < g.rows && col < g.cols)
                level[row * g.cols + col] = (ready[i >> 5] >> (i & 31)) & 1u ? (int32_t)st[2 * i] : -1;
        }
        for (int e = t; e < ne; e += kTileThreads) exit_level[e0 + e] = st[2 * exit_local[e0 + e]];
        if (t == 0) atomicExch(cyclic, 1);
        return;
    }
    // levels within the tile
    for (int i = t; i < kTileCells; i += kTileThreads) {
        const int64_t row = tr * kTile + (i >> 6), col = tc * kTile + (i & 63);
        if (row < g.rows && col < g.cols)
            level[row * g.cols + col] = sm.fd[(i >> 6) + 1][(i & 63) + 1] == kNoData ? -1 : (int32_t)st[2 * i];
    }
    for (int e = t; e < ne; e += kTileThreads) exit_level[e0 + e] = st[2 * exit_local[e0 + e]];
    __syncthreads();
    // first positions of roots and invalid cells; the others' offset from their downstream cell's: after the siblings
    // that come before them
    for (int i = own; i < own + 512; i += 32) {
        const bool bad = sm.fd[(i >> 6) + 1][(i & 63) + 1] == kNoData;
        const int d = sm.dsl[i];
        const int size = !bad && d == kNoCell ? sz[2 * i] : 0;
        const unsigned bads = __ballot_sync(0xffffffffu, bad);
        if (bad) st[2 * i] = (uint16_t)(invalid_base + __popc(bads & ((1u << lane) - 1u)));
        invalid_base += __popc(bads);
        if (__any_sync(0xffffffffu, size != 0)) {
            int x = size;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (size) st[2 * i] = (uint16_t)(root_base + x - size);
            root_base += __shfl_sync(0xffffffffu, x, 31);
        }
        if (d != kNoCell) {
            int o = 0;
            for (unsigned m = sm.up[d] & ((1u << nb_index_from(d, i)) - 1u); m; m &= m - 1)
                o += sz[2 * (d + tile_nb_offset(__ffs(m) - 1))];
            st[2 * i] = (uint16_t)o;
        }
    }
    __syncthreads();
    // positions, downstream first; the narrow rounds read the next round's cells ahead
    if (t < 32) {
        int q = rounds - 1, k = q >= wide ? rstart[q] + t : 0;
        int i = q >= wide && k < rstart[q + 1] ? sm.queue[k] : kNoCell, d = i != kNoCell ? sm.dsl[i] : kNoCell;
        for (; q >= wide; --q) {
            int i1 = kNoCell, d1 = kNoCell;
            if (q > wide && rstart[q - 1] + t < rstart[q]) {
                i1 = sm.queue[rstart[q - 1] + t];
                d1 = sm.dsl[i1];
            }
            if (d != kNoCell) st[2 * i] += st[2 * d];
            __syncwarp();
            i = i1;
            d = d1;
        }
    }
    __syncthreads();
    for (int q = wide - 1; q >= 0; --q) {
        for (int k = rstart[q] + t; k < rstart[q + 1]; k += kTileThreads) {
            const int i = sm.queue[k], d = sm.dsl[i];
            if (d != kNoCell) st[2 * i] += st[2 * d];
        }
        __syncthreads();
    }
    // positions, checked distinct (every position 0 .. 4095 once), the first positions of the roots'
    // subtrees (segment heads), then the tables by position
    const int64_t T = tile * kRunPositions;
    // the tables are put together here: written cell by cell, each value would be a memory request of its own
    uint16_t *s_cell = sm.queue, *s_prev = sm.rstart;
    uint32_t* seen = reinterpret_cast<uint32_t*>(sm.up);
    uint32_t* heads = seen + kRunPositions / 32;
    for (int w = t; w < kRunPositions / 32; w += kTileThreads) {
        seen[w] = 0;
        heads[w] = 0;
    }
    __syncthreads();
    for (int i = t; i < kTileCells; i += kTileThreads) {
        const bool valid = sm.fd[(i >> 6) + 1][(i & 63) + 1] != kNoData;
        const int s0 = st[2 * i], p = s0 + sz[2 * i] - 1;
        bool bad = p >= kRunPositions || s0 > p;
        if (!bad) bad = (atomicOr(&seen[p >> 5], 1u << (p & 31)) >> (p & 31)) & 1u;
        if (bad) {
            *error = 1;
            continue;
        }
        if (!valid || sm.dsl[i] == kNoCell) atomicOr(&heads[s0 >> 5], 1u << (s0 & 31));
    }
    __syncthreads();
    for (int i = t; i < kTileCells; i += kTileThreads) {
        const bool valid = sm.fd[(i >> 6) + 1][(i & 63) + 1] != kNoData;
        const int s0 = st[2 * i], p = s0 + sz[2 * i] - 1;
        if (p >= kRunPositions || s0 > p) continue;  // reported above
        const bool head = (heads[p >> 5] >> (p & 31)) & 1u;
        s_cell[run_table_index(p)] =
            (uint16_t)(i | (valid ? 0u : kNoValue) | (head ? kSegHead : 0u) | (s0 == p ? kLoneCell : 0u));
        s_prev[run_table_index(p)] = (uint16_t)(8 * (s0 > 0 ? scan_slot(s0 - 1) : kZeroSlot));
    }
    __syncthreads();
    static_assert(kRunPositions == kTileCells, "the tables are staged in arrays of one value per cell");
    for (int i = t; i < kRunPositions / 8; i += kTileThreads) {
        reinterpret_cast<uint4*>(cell_at + T)[i] = reinterpret_cast<const uint4*>(s_cell)[i];
        reinterpret_cast<uint4*>(prev_at + T)[i] = reinterpret_cast<const uint4*>(s_prev)[i];
    }
    if (t < kRunPositions / 32 && seen[t] != 0xFFFFFFFFu) *error = 1;
    for (int e = t; e < ne; e += kTileThreads) {
        const int loc = exit_local[e0 + e];
        const int s0 = st[2 * loc], p = s0 + sz[2 * loc] - 1;
        exit_span[e0 + e] = (uint32_t)scan_slot(p) | ((uint32_t)(s0 > 0 ? scan_slot(s0 - 1) : kZeroSlot) << 16);
    }
}

// ---------------------------------------------------------------------------------------------------
// Per call
// ---------------------------------------------------------------------------------------------------
//
// A tile CTA works in two orders.  Material and results move between HBM and shared memory in cell
// order (row-major float4 rows, coalesced).  Thread t owns the post-order positions 16 t .. 16 t + 15:
// it gathers their material from shared memory through cell_at (one 4-byte read per cell), converts it
// to fixed point and takes the prefix sum of its run in registers; a warp scan and the warp totals give
// the run's offset, and each inclusive prefix is written to shared memory once.  The accu of a cell is
// then its own prefix minus the prefix just before its subtree (prev_at).
//
// Inside a tile the material is summed in 64-bit fixed point, round(x * 2^F), with F chosen per tile
// from a bound on the tile's total (4096 times its largest term, plus what enters through its border)
// so that the total stays below 2^62: prefix sums over the post-order are then exact, and so is every
// subtree sum taken as their difference (modulo 2^64, exact because the true sum is < 2^64).  A term
// x > 0 is represented to within 2^-(F+1) absolute; a tile whose smallest positive term would carry
// fewer than 19 bits (x * 2^F < 2^19) or that holds +inf asks for the walk engine instead.

constexpr float kMinQuantum = 524288.0f;  // 2^19

__device__ __forceinline__ float pow2f(int e) { return __int_as_float((127 + e) << 23); }  // -126 <= e <= 127

// Largest F <= 126 with bound * 2^F < 2^62 (0 for bound 0).
__device__ __forceinline__ int tile_scale(float bound)
{
    if (!(bound > 0.0f)) return 0;
    const int e = (int)((__float_as_uint(bound) >> 23) & 0xFFu) - 126;  // bound < 2^e
    return min(62 - e, 126);
}

// Bound on a tile's total from the bits of its largest term (4096 terms below 2^(e - 126)) and of the
// largest sum entering through its border (at most 252 of them); +inf when beyond float range.
__device__ __forceinline__ float tile_bound(unsigned max_bits, unsigned src_bits)
{
    const int e = (int)(max_bits >> 23);
    const float local = e > 240 ? INFINITY : pow2f(e - 114);
    return (local + 256.0f * __uint_as_float(src_bits)) * 1.0009765625f;
}

// Conversions between float and 64-bit fixed point in integer arithmetic.  GB300 executes the 64-bit
// float <-> integer conversion instructions on its float64 pipe, which runs at a small fraction of the
// integer rate; these run on the integer pipes.

// round(x * 2^F) for finite x >= 0 with x * 2^F < 2^63 (ties away from zero).
__device__ __forceinline__ unsigned long long float_to_fixed64(float x, int F)
{
    const unsigned b = __float_as_uint(x);
    const unsigned e = b >> 23;
    const unsigned m = (b & 0x7FFFFFu) | (e ? 0x800000u : 0u);
    const int s = (int)(e ? e : 1u) - 150 + F;  // x * 2^F = m * 2^s
    const unsigned rs = s < 0 ? (unsigned)min(-s, 31) : 0u;
    const unsigned r = rs ? (m + (1u << (rs - 1))) >> rs : m;
    return (unsigned long long)r << (s > 0 ? s : 0);
}

// x * 2^F exactly, for x == 0 or a normal x >= 0 with x * 2^F >= 2^23 (no bit is shifted out).
__device__ __forceinline__ unsigned long long float_to_fixed64_exact(float x, float scale_hi)
{
    // scale_hi = 2^(F - 32).  The high and low 32-bit halves by float arithmetic, every step exact: a
    // power-of-two scaling, the truncation of a value below 2^30 with at most 24 significant bits, its
    // fraction (the bits under the binary point), and that fraction times 2^32 (an integer: no bit of
    // x * 2^F lies below 2^0).  Three conversions and three float operations instead of a 64-bit shift.
    const float y = __fmul_rn(x, scale_hi);
    const unsigned hi = __float2uint_rz(y);
    const float frac = __fsub_rn(y, __uint2float_rz(hi));
    const unsigned lo = __float2uint_rz(__fmul_rn(frac, 4294967296.0f));
    return ((unsigned long long)hi << 32) | lo;
}

// A 96-bit fixed-point value v * 2^-F, rounded to float (the bits below the top 64 are dropped).
__device__ __forceinline__ float fixed128_to_float(u128 v, int F)
{
    const unsigned long long hi = (unsigned long long)(v >> 64);
    if (hi == 0) return ldexpf(__ull2float_rn((unsigned long long)v), -F);
    const int shift = 64 - __clzll((long long)hi);
    return ldexpf(__ull2float_rn((unsigned long long)(v >> shift)), shift - F);
}

// Cells of a tile by thread in cell order: thread t holds the 4 x 4 cells (row (t + 256 j) / 16,
// columns 4 ((t + 256 j) % 16) .. + 3), j = 0..3, so that a row of the tile is 16 float4.
__device__ __forceinline__ int quad_cell(int j)
{
    const int k = threadIdx.x + kTileThreads * j;
    return (k >> 4) * kTile + (k & 15) * 4;
}

__device__ __forceinline__ float4 load_quad(const float* __restrict__ p, const TileGeom& g, int64_t r, int64_t c,
                                            bool vec, float fill)
{
    if (vec) {
        if (r < g.rows && c < g.cols) return __ldg(reinterpret_cast<const float4*>(p + r * g.cols + c));
        return make_float4(fill, fill, fill, fill);
    }
    float v[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) v[x] = (r < g.rows && c + x < g.cols) ? __ldg(p + r * g.cols + c + x) : fill;
    return make_float4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ void store_quad(float* __restrict__ p, const TileGeom& g, int64_t r, int64_t c, bool vec,
                                           float4 v)
{
    if (r >= g.rows) return;
    if (vec) {
        if (c < g.cols) *reinterpret_cast<float4*>(p + r * g.cols + c) = v;
        return;
    }
    const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int x = 0; x < 4; ++x)
        if (c + x < g.cols) p[r * g.cols + c + x] = w[x];
}

struct TileForest {
    const uint16_t* cell_at;
    const uint16_t* prev_at;
    const float* inflow;
};

// Shared memory of a tile CTA of pass 1 or pass 3 (dynamic: 53 KB, four CTAs per SM).
struct __align__(16) TileCallSmem {
    unsigned long long S[kScanSlotCount];  // inclusive prefix sums by scan slot; S[kZeroSlot] = 0
    float M[kTileCells];                   // material plus what enters, in cell order; then the results
    alignas(16) unsigned long long warp_tot[kTileThreads / 32];
    alignas(16) unsigned red[2][kTileThreads / 32];
    alignas(16) unsigned warp_mn[kTileThreads / 32];
    alignas(16) float warp_sum[kTileThreads / 32];
    float seg_hi[kTileThreads / 32], seg_lo[kTileThreads / 32];  // pass 1: warp totals of the segmented scan
    int seg_head[kTileThreads / 32];
    float carry_hi[kTileThreads], carry_lo[kTileThreads];        // pass 1: what each run's first segment carries in
    uint8_t run_first[kTileThreads];                             // pass 1: first segment head of each run (16: none)
    int quit;                                                    // the CTA leaves; the CTA is the last one
};

// The thread's run of a per-position table (cell_at or prev_at): eight coalesced 4-byte loads.
__device__ __forceinline__ void load_run(const uint16_t* __restrict__ table, uint32_t (&w)[kRunWords])
{
    const uint32_t* p = reinterpret_cast<const uint32_t*>(table) + threadIdx.x;
#pragma unroll
    for (int i = 0; i < kRunWords; ++i) w[i] = __ldg(p + i * kTileThreads);
}
__device__ __forceinline__ unsigned run_at(const uint32_t (&w)[kRunWords], int j)
{
    return (w[j >> 1] >> (16 * (j & 1))) & 0xFFFFu;
}

// Material of the tile in cell order (0 outside the array), by quads of 4 cells (quad_cell).
__device__ __forceinline__ void load_material(float4 (&x)[4], const float* __restrict__ ext, float ext_s,
                                              const TileGeom& g, int64_t tr, int64_t tc, bool vec)
{
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int cell = quad_cell(j);
        x[j] = ext ? load_quad(ext, g, tr * kTile + (cell >> 6), tc * kTile + (cell & 63), vec, 0.0f)
                   : make_float4(ext_s, ext_s, ext_s, ext_s);
    }
}

// The material total in 2^-16 units at or beyond this makes the tile engine hand the call to the walk
// engine (the 128-bit fixed point of the exit forest keeps 96 value bits).
constexpr unsigned long long kTotalLimit = 1000000000000000000ull;

// total[0], summed by pass 1 with 64-bit atomics (exact, so the order does not matter), and total[1]: the
// tile engine's result stands when neither says otherwise.
__device__ __forceinline__ bool tile_fallback(const unsigned long long* total)
{
    return *reinterpret_cast<const volatile unsigned long long*>(total + 1) != 0 || total[0] >= kTotalLimit;
}

// Exits per thread of a scan block: 8 (63 registers, four CTAs per SM) where the scan fills the GPU, 2 on small
// rasters, where fewer exits in a row per thread end the launch sooner.
constexpr int kScanItems = 8, kScanItemsSmall = 2;
constexpr int kScanPolls = 1 << 20;  // poll limit of one look-back wait (a second at most)

__device__ __forceinline__ u128 block_exclusive_u128(u128 v, u128* warp_tot, u128& block_total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u128 x = v;
    for (int d = 1; d < 32; d <<= 1) {
        u128 y = shfl_up_u128(x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    if (warp == 0) {
        u128 w = lane < kTileThreads / 32 ? warp_tot[lane] : (u128)0;
        for (int d = 1; d < 32; d <<= 1) {
            u128 y = shfl_up_u128(w, d);
            if (lane >= d) w += y;
        }
        if (lane < kTileThreads / 32) warp_tot[lane] = w;
    }
    __syncthreads();
    u128 before = warp ? warp_tot[warp - 1] : (u128)0;
    block_total = warp_tot[kTileThreads / 32 - 1];
    __syncthreads();
    return before + x - v;
}

// The exit forest's 128-bit inclusive scan, one chunk of consecutive scan blocks (256 x ITEMS exits each)
// per CTA, with as many CTAs as fit on the GPU at once.  CTAs take chunks in ticket order; each sums its
// chunk, publishes the sum (flag 1), then warp 0 adds up the sums of the chunks before it, 32 at a time,
// until it meets a chunk that has published the sum up to and including itself (flag 2); the CTA
// publishes its own (flag 2) and scans its chunk again, block by block, from that prefix.  A CTA waits
// only for chunks with smaller tickets, held by CTAs that started earlier, and those publish their own
// sums before they wait for anything: no chain of waits forms.  Every wait is bounded: a wait that gives
// up (or sees that one did) sets total[1] = 2, after which the walk engine redoes the call.
// ctl = the ticket, then the chunk flags, zeroed before the call.
template <int ITEMS>
__global__ void __launch_bounds__(kTileThreads)
    k_scan_exits(const float2* __restrict__ P, int64_t n, int64_t chunk_blocks, unsigned long long* total,
                 unsigned* ctl, uint4* look_aggr, uint4* look_incl, uint4* __restrict__ S, int polls)
{
    constexpr int64_t kBlock = kTileThreads * ITEMS;
    __shared__ u128 warp_tot[kTileThreads / 32];
    __shared__ u128 prefix_sh;
    __shared__ unsigned ticket_sh;
    __shared__ int abort_sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    next_may_start();
    wait_for_previous();
    // one thread decides, so that the whole CTA leaves or stays
    if (threadIdx.x == 0) ticket_sh = tile_fallback(total) ? ~0u : atomicAdd(ctl, 1u);
    __syncthreads();
    if (ticket_sh == ~0u) return;
    const int64_t g = ticket_sh;
    unsigned* flag = ctl + 1;
    const int F = fixed_point_bits(total[0]);
    const int64_t first = g * chunk_blocks * kBlock;
    const int64_t last = min(n, first + chunk_blocks * kBlock);
    // the chunk's sum
    u128 s = 0;
    for (int64_t b0 = first; b0 < last; b0 += kBlock) {
        const int64_t base = b0 + (int64_t)threadIdx.x * ITEMS;
#pragma unroll
        for (int k = 0; k < ITEMS; ++k)
            if (base + k < last) s += exit_value_fixed(__ldcg(P + base + k), F);
    }
    u128 bt;
    block_exclusive_u128(s, warp_tot, bt);
    if (warp == 0) {
        if (g == 0) {
            if (lane == 0) {
                look_incl[0] = from_u128(bt);
                st_release(flag, 2u);
                prefix_sh = 0;
                abort_sh = 0;
            }
        } else {
            if (lane == 0) {
                look_aggr[g] = from_u128(bt);
                st_release(flag + g, 1u);
            }
            u128 prefix = 0;
            bool failed = false;
            for (int64_t top = g - 1;; top -= 32) {
                const int64_t j = top - lane;
                unsigned f = 2u;  // before chunk 0: nothing (never reached: chunk 0 publishes flag 2)
                u128 x = 0;
                if (j >= 0) {
                    int k = 0;
                    for (; k < polls; ++k) {
                        f = ld_acquire(flag + j);
                        if (f != 0u) break;
                        if (*reinterpret_cast<volatile unsigned long long*>(total + 1)) k = polls - 1;
                        __nanosleep(64);
                    }
                    if (k >= polls) f = 0u;
                }
                if (__ballot_sync(0xffffffffu, f == 0u)) {
                    failed = true;
                    break;
                }
                const unsigned incl = __ballot_sync(0xffffffffu, f == 2u);
                const int stop = incl ? __ffs(incl) - 1 : 31;  // lanes 0..stop count
                if (j >= 0 && lane <= stop) x = to_u128(__ldcg(f == 2u ? look_incl + j : look_aggr + j));
                for (int d = 16; d > 0; d >>= 1) x += shfl_down_u128(x, d);
                prefix += x;  // lane 0 holds the window's sum
                if (incl) break;
            }
            if (lane == 0) {
                if (failed) {
                    total[1] = 2ull;
                } else {
                    look_incl[g] = from_u128(prefix + bt);
                    st_release(flag + g, 2u);
                }
                prefix_sh = prefix;
                abort_sh = failed ? 1 : 0;
            }
        }
    }
    __syncthreads();
    if (abort_sh) return;
    u128 carry = prefix_sh;
    for (int64_t b0 = first; b0 < last; b0 += kBlock) {
        const int64_t base = b0 + (int64_t)threadIdx.x * ITEMS;
        u128 v[ITEMS];
        u128 t = 0;
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            v[k] = base + k < last ? exit_value_fixed(__ldcg(P + base + k), F) : (u128)0;
            t += v[k];
        }
        u128 blk;
        u128 run = carry + block_exclusive_u128(t, warp_tot, blk);
        carry += blk;
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            run += v[k];
            if (base + k < last) S[base + k] = from_u128(run);
        }
    }
}

// What enters an inflow slot (a border cell receiving flow from other tiles): the exact sum of the subtree
// sums of the exits draining into it (each a difference of two inclusive prefix sums of the exit
// forest), rounded to float once; NaN when one of them holds a no-data exit.
struct TileSlots {
    const int32_t* base;   // [ntiles + 1] first slot of each tile
    const int32_t* at;     // tile * kSlotStride + border index
    const int32_t* first;  // first edge
    const int2* edge;
    const uint4* S;        // written by the kernel before: no read-only loads
};
__device__ __forceinline__ float slot_inflow(const TileSlots& q, int64_t i, int F)
{
    u128 src = 0;
    for (int32_t k = __ldg(q.first + i), k1 = __ldg(q.first + i + 1); k < k1; ++k) {
        const int2 e = __ldg(q.edge + k);
        src += to_u128(__ldcg(q.S + e.x)) - (e.y >= 0 ? to_u128(__ldcg(q.S + e.y)) : (u128)0);
    }
    return (src >> 96) ? __int_as_float(0x7fc00000) : fixed128_to_float(src & kValueMask, F);
}
__global__ void k_slot_inflow(int64_t nslot, TileSlots q, float* __restrict__ inflow, const unsigned long long* total)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nslot || tile_fallback(total)) return;
    inflow[__ldg(q.at + i)] = slot_inflow(q, i, fixed_point_bits(total[0]));
}

// Build, a CTA per tile: its inflow slots and their upstream exits, in border order (one thread per tile took 316 us
// at 2048^2, this 6.5 us).
__global__ void __launch_bounds__(kTileThreads)
    k_slot_fill(TileGeom g, const uint8_t* __restrict__ border_in, const int32_t* __restrict__ exit_base,
                const uint64_t* bitmap, const uint16_t* rowpref, const int32_t* __restrict__ slot_base,
                const int32_t* __restrict__ edge_base, const uint32_t* __restrict__ exit_pos,
                const uint32_t* __restrict__ exit_start, int32_t* slot_at, int32_t* slot_first, int2* slot_edge,
                int64_t nexit, int* error)
{
    __shared__ int warp_tot[kTileThreads / 32];
    const int64_t tr = blockIdx.y, tc = blockIdx.x, tile = tr * g.tcols + tc;
    const int t = threadIdx.x;
    const unsigned m0 = t < kBorderCells ? border_in[tile * kBorderCells + t] : 0u;
    int total;
    const int32_t s = slot_base[tile] + block_exclusive_int(m0 != 0, warp_tot, total);
    int32_t e = edge_base[tile] + block_exclusive_int(__popc(m0), warp_tot, total);
    if (tile == g.trows * g.tcols - 1 && t == 0) slot_first[slot_base[tile + 1]] = edge_base[tile + 1];
    if (!m0) return;
    int rin, cin;
    border_cell(t, rin, cin);
    slot_at[s] = (int32_t)(tile * kSlotStride + t);
    slot_first[s] = e;
    for (unsigned m = m0; m; m &= m - 1) {
        const int q = __ffs(m) - 1;
        // a neighbour draining in is an exit of its tile
        const int64_t y = exit_id_of(g, exit_base, bitmap, rowpref, tr * kTile + rin + nb_dr(q), tc * kTile + cin + nb_dc(q));
        if (y >= nexit) {
            atomicExch(error, 1);
            return;
        }
        const uint32_t st = exit_start[y];
        slot_edge[e++] = make_int2((int)exit_pos[y], st ? (int)(st - 1u) : -1);
    }
}

// Build, a CTA per tile: the downstream level of every cell, from its level within the tile (k_tile_forest) and the
// levels of the exits that drain into the tile (k_exit_sizes): each inflow raises the cells below it, up to the first
// that is at least as high already.  Cells on a cycle keep -1: those that have it from k_tile_forest, and those below an
// exit that k_exit_sizes did not finish (pending; nullptr without cycles).  And the raster's statistics [valid, ridge,
// outlet, sink, cycle, largest level].
// A walk over the cells of the whole raster (k_walk) is bound by the longest flow path, a memory round trip per cell:
// 0.99 ms at 2048^2, where k_exit_sizes, which takes those steps from tile to tile, and this kernel take 19 and 33 us.
constexpr int kOnCycle = 0x7fffffff;
__global__ void __launch_bounds__(kTileThreads)
    k_tile_levels(const uint8_t* __restrict__ fd, TileGeom g, const int32_t* __restrict__ exit_base,
                  const uint64_t* bitmap, const uint16_t* rowpref, const uint8_t* __restrict__ border_in,
                  const int32_t* __restrict__ exit_level, const int32_t* __restrict__ pending, int64_t nexit,
                  int32_t* __restrict__ level, unsigned long long* stats)
{
    __shared__ int lv[kTileCells];
    __shared__ uint8_t code[kTileCells];
    __shared__ int tally[6];
    const int64_t tr = blockIdx.y, tc = blockIdx.x, tile = tr * g.tcols + tc;
    const int t = threadIdx.x, lane = t & 31;
    // thread t: column t & 63 of every fourth row
    constexpr int kCells = kTileCells / kTileThreads, kStep = kTileThreads / kTile;
    const int64_t row0 = tr * kTile + (t >> 6), col = tc * kTile + (t & 63), cell0 = row0 * g.cols + col, step = kStep * g.cols;
    const int rows = col < g.cols ? (int)min((int64_t)kTile, max((int64_t)0, g.rows - row0)) : 0;  // this thread's, by kStep
    if (t < 6) tally[t] = 0;
    unsigned c[kCells];
    int l[kCells];
#pragma unroll
    for (int k = 0; k < kCells; ++k) {  // all loads before the first use
        const bool in = k * kStep < rows;
        c[k] = in ? fd[cell0 + k * step] : kNoData;
        l[k] = in ? level[cell0 + k * step] : -1;
    }
#pragma unroll
    for (int k = 0; k < kCells; ++k) {
        code[t + k * kTileThreads] = (uint8_t)c[k];
        lv[t + k * kTileThreads] = c[k] != kNoData && l[k] < 0 ? kOnCycle : l[k];
    }
    __syncthreads();
    const unsigned from = t < kBorderCells ? border_in[tile * kBorderCells + t] : 0u;
    if (from) {
        int r, c, in = 0;
        border_cell(t, r, c);
        for (unsigned m = from; m; m &= m - 1) {
            const int q = __ffs(m) - 1;
            const int64_t y = exit_id_of(g, exit_base, bitmap, rowpref, tr * kTile + r + nb_dr(q), tc * kTile + c + nb_dc(q));
            if (y < nexit) in = max(in, pending && pending[y] != 0 ? kOnCycle : exit_level[y] + 1);
        }
        // At most one step per cell: a cycle inside the tile stops the walk, as its cells have the highest value.  The walk
        // waits for its loads only, not for the maximum: whoever raised a cell first goes on below it.
        for (int i = r * kTile + c; *(volatile int*)(lv + i) < in; in += in != kOnCycle) {
            atomicMax(lv + i, in);
            int d, q;
            if (!tile_downstream(code[i], i >> 6, i & 63, d, q) || code[d] == kNoData) break;
            i = d;
        }
    }
    __syncthreads();
    int valid = 0, ridge = 0, outlet = 0, sink = 0, cycle = 0, most = 0;
#pragma unroll
    for (int k = 0; k < kCells; ++k) {
        const unsigned c = code[t + k * kTileThreads];
        if (c == kNoData) continue;
        ++valid;
        const int l = lv[t + k * kTileThreads];
        level[cell0 + k * step] = l == kOnCycle ? -1 : l;
        if (l == kOnCycle) {
            ++cycle;
            continue;
        }
        ridge += l == 0;  // a cell has level 0 when nothing drains into it
        const unsigned pad = c - 1u;  // numeric pad: 0 .. 8 from the lower left, 4 in the middle
        if (pad > 8u || pad == 4u) {
            ++sink;
        } else {
            const int up = (int)(pad * 11u >> 5), right = (int)pad - 3 * up;
            const int64_t row = row0 + k * kStep + 1 - up, to = col + right - 1;
            outlet += row < 0 || row >= g.rows || to < 0 || to >= g.cols;
        }
        most = max(most, l);
    }
    valid = __reduce_add_sync(0xffffffffu, valid);
    ridge = __reduce_add_sync(0xffffffffu, ridge);
    outlet = __reduce_add_sync(0xffffffffu, outlet);
    sink = __reduce_add_sync(0xffffffffu, sink);
    cycle = __reduce_add_sync(0xffffffffu, cycle);
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) {
        atomicAdd(tally + 0, valid);
        atomicAdd(tally + 1, ridge);
        atomicAdd(tally + 2, outlet);
        atomicAdd(tally + 3, sink);
        atomicAdd(tally + 4, cycle);
        atomicMax(tally + 5, most);
    }
    __syncthreads();
    if (t < 5 && tally[t]) atomicAdd(stats + t, (unsigned long long)tally[t]);
    if (t == 5 && (unsigned long long)tally[5] > *(volatile unsigned long long*)(stats + 5))
        atomicMax(stats + 5, (unsigned long long)tally[5]);
}

// Inclusive prefix sums (modulo 2^64) of the thread runs a[0..15] over the whole tile, written to S by
// scan slot.  Ends with a block barrier.
__device__ __forceinline__ void tile_prefix(TileCallSmem& sm, unsigned long long (&a)[kRun])
{
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
    for (int j = 1; j < kRun; ++j) a[j] += a[j - 1];
    unsigned long long x = a[kRun - 1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sm.warp_tot[warp] = x;
    __syncthreads();
    unsigned long long off = x - a[kRun - 1];
    const ulonglong2* wt = reinterpret_cast<const ulonglong2*>(sm.warp_tot);  // 16-byte loads
#pragma unroll
    for (int w = 0; w < kTileThreads / 64; ++w) {
        const ulonglong2 v = wt[w];
        off += (2 * w < warp ? v.x : 0ull) + (2 * w + 1 < warp ? v.y : 0ull);
    }
    unsigned long long* run = sm.S + kRunSlots * t;  // 136-byte runs
#pragma unroll
    for (int j = 0; j < kRun; ++j) {
        a[j] += off;  // the thread keeps its own prefixes
        run[j] = a[j];
    }
    if (t == 0) sm.S[kZeroSlot] = 0ull;
    __syncthreads();
}

// Poison counts (slow path): inclusive prefix counts over the post-order of the flagged terms, written as
// 32-bit counts by scan slot over S (free until the value scan).  Ends with a block barrier.
__device__ __forceinline__ void poison_counts(TileCallSmem& sm, unsigned bad)
{
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    unsigned run = __popc(bad);
    unsigned x = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sm.warp_tot[warp] = x;
    __syncthreads();
    unsigned off = x - run;
    for (int w = 0; w < warp; ++w) off += (unsigned)sm.warp_tot[w];
    unsigned* C = reinterpret_cast<unsigned*>(sm.S);
    unsigned c = off;
#pragma unroll
    for (int j = 0; j < kRun; ++j) {
        c += (bad >> j) & 1u;
        C[kRunSlots * t + j] = c;
    }
    if (t == 0) C[kZeroSlot] = 0u;
    __syncthreads();
}

// The thread's run in post-order: the material of each position (0 for no-data cells and cells outside
// the array), after a block barrier that follows the stores to M.
__device__ __forceinline__ void gather_run(const TileCallSmem& sm, const uint32_t (&ca)[kRunWords], float (&x)[kRun])
{
#pragma unroll
    for (int j = 0; j < kRun; ++j) {
        const unsigned w = run_at(ca, j);
        const float v = sm.M[w & kIndexMask];
        x[j] = (w & kNoValue) ? 0.0f : v;
    }
}

// NaN or negative terms of a run (slow path): flagged in the returned mask, then 0 (-0 counts as 0).
__device__ __forceinline__ unsigned clean_run(float (&x)[kRun])
{
    unsigned bad = 0;
#pragma unroll
    for (int j = 0; j < kRun; ++j) {
        if (!(x[j] >= 0.0f)) bad |= 1u << j;
        x[j] = x[j] >= 0.0f ? fabsf(x[j]) : 0.0f;
    }
    return bad;
}

// Float-float pieces of pass 1: x + y with the rounding error of the high parts kept in lo (no
// renormalisation), and the segmented-scan combination of (sum since the last segment head, has a head).
struct SegSum {
    float hi, lo;
    bool head;
};
__device__ __forceinline__ void ff_acc(float& hi, float& lo, float x)
{
    const float s = __fadd_rn(hi, x);
    const float bp = __fsub_rn(s, hi);
    const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(x, bp));
    hi = s;
    lo = __fadd_rn(lo, e);
}
// a, then b
__device__ __forceinline__ SegSum seg_combine(const SegSum& a, const SegSum& b)
{
    if (b.head) return b;
    SegSum r{a.hi, __fadd_rn(a.lo, b.lo), a.head};
    ff_acc(r.hi, r.lo, b.hi);
    return r;
}
__device__ __forceinline__ SegSum seg_shfl_up(const SegSum& v, int d)
{
    return SegSum{__shfl_up_sync(0xffffffffu, v.hi, d), __shfl_up_sync(0xffffffffu, v.lo, d),
                  __shfl_up_sync(0xffffffffu, (int)v.head, d) != 0};
}

// Pass 1: the local value of every exit (the accu of its in-tile subtree) to P, in the exit forest's
// post-order; an upper bound of the tile's material total in 2^-16 units added to total[0] (64-bit
// atomics: exact, whatever the order; total[1] is set instead, asking for the walk engine, on +inf, a
// total beyond float range, a dynamic range the 64-bit fixed point of pass 3 cannot hold, or a sum that
// wraps), and the statistics pass 3 takes its fixed-point scale from (so that it needs no reduction of its
// own).  Exits are roots of the tile's forest; the subtrees of the roots are consecutive runs of
// positions (segments, each starting at a flagged head), so an exit's value is the sum of its segment: a
// segmented prefix sum in float-float (relative error about 2^-35 of the segment's total in the worst
// case, no cancellation), computed on the float pipes.  A NaN or negative term makes its segment NaN,
// and with it the exit: no-data flows on from there through the exit forest.
//
// tile_exits: the tile's part of pass 1, from the material (xm) and the cell table (ca) in registers.  On return M
// holds the material in cell order.  False: the walk engine must redo the call.  units: thread 0's share of
// total[0] (kTotalLimit or more: out of range).
__device__ __forceinline__ bool tile_exits(TileCallSmem& sm, const float4 (&xm)[4], const uint32_t (&ca)[kRunWords],
                                           int ne, uint32_t span, uint32_t epos, float2* __restrict__ P,
                                           TileStat& st, unsigned long long& units)
{
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
    for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(sm.M + quad_cell(j)) = xm[j];
    __syncthreads();
    // over the valid positions: the largest raw bits (a sign bit or NaN: pass 3's slow path), the largest
    // and smallest positive bits of the terms that are >= 0, and their float sum; and the segmented sums of
    // the run, with the run's summary for the scan across threads
    unsigned raw = 0, mx = 0, mn = 0xFFFFFFFFu;
    float sum = 0.0f;
    SegSum run{0.0f, 0.0f, false};
    int first_head = kRun;
    float2* L = reinterpret_cast<float2*>(sm.S);
#pragma unroll
    for (int j = 0; j < kRun; ++j) {
        const unsigned w = run_at(ca, j);
        const float m = sm.M[w & kIndexMask];
        const float x = (w & kNoValue) ? 0.0f : m;
        const unsigned b = __float_as_uint(x);
        raw = max(raw, b);
        const bool ok = x >= 0.0f;
        const unsigned a = ok ? (b & 0x7FFFFFFFu) : 0u;
        mx = max(mx, a);
        mn = min(mn, a - 1u);
        sum += ok ? x : 0.0f;
        const float v = ok || isnan(x) ? x : __int_as_float(0x7fc00000);  // negative: NaN
        if (w & kSegHead) {
            if (!run.head) first_head = j;
            run = SegSum{v, 0.0f, true};
        } else {
            ff_acc(run.hi, run.lo, v);
        }
        L[kRunSlots * t + j] = make_float2(run.hi, run.lo);
    }
    raw = __reduce_max_sync(0xffffffffu, raw);
    mx = __reduce_max_sync(0xffffffffu, mx);
    mn = __reduce_min_sync(0xffffffffu, mn);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    // exclusive segmented scan of the run summaries across the tile: what a segment that starts before
    // this run carries into it
    SegSum inc = run;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const SegSum y = seg_shfl_up(inc, d);
        if (lane >= d) inc = seg_combine(y, inc);
    }
    SegSum exc = seg_shfl_up(inc, 1);
    if (lane == 0) exc = SegSum{0.0f, 0.0f, false};
    if (lane == 0) {
        sm.red[0][warp] = raw;
        sm.red[1][warp] = mx;
        sm.warp_mn[warp] = mn;
        sm.warp_sum[warp] = sum;
    }
    if (lane == 31) {
        sm.seg_hi[warp] = inc.hi;
        sm.seg_lo[warp] = inc.lo;
        sm.seg_head[warp] = inc.head;
    }
    __syncthreads();
    // the warps' summaries: lane i of every warp takes warp (i & 7)'s; the block's largest and smallest bits
    // by warp reductions, the sum (thread 0's is used) and a segmented scan over each group of eight lanes
    // by three shuffle steps; the carry into this warp is lane warp - 1's inclusive scan
    static_assert(kTileThreads == 256, "eight warps per tile CTA");
    const int w8 = lane & 7;
    raw = __reduce_max_sync(0xffffffffu, sm.red[0][w8]);
    mx = __reduce_max_sync(0xffffffffu, sm.red[1][w8]);
    mn = __reduce_min_sync(0xffffffffu, sm.warp_mn[w8]);
    sum = sm.warp_sum[w8];
    SegSum ws{sm.seg_hi[w8], sm.seg_lo[w8], sm.seg_head[w8] != 0};
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const SegSum y = seg_shfl_up(ws, o);
        if (w8 >= o) ws = seg_combine(y, ws);
    }
    const int src = warp > 0 ? warp - 1 : 0;
    SegSum before{__shfl_sync(0xffffffffu, ws.hi, src), __shfl_sync(0xffffffffu, ws.lo, src),
                  __shfl_sync(0xffffffffu, (int)ws.head, src) != 0};
    if (warp == 0) before = SegSum{0.0f, 0.0f, false};
    const SegSum carry = seg_combine(before, exc);
    sm.run_first[t] = (uint8_t)first_head;
    sm.carry_hi[t] = carry.hi;
    sm.carry_lo[t] = carry.lo;
    const float bound = tile_bound(mx, 0u);
    const int F = tile_scale(bound);
    if (mx >= 0x7F800000u || !(bound < 1.0e38f) ||
        (mn != 0xFFFFFFFFu && __uint_as_float(mn + 1u) * pow2f(F) < kMinQuantum))
        return false;  // uniform: every thread has the same reductions
    __syncthreads();
    if (t < ne) {
        // the exit's position is the end of its segment; a segment that starts in an earlier run also
        // holds what that run's carry brings
        const int slot = (int)(span & 0xFFFFu), r = slot / kRunSlots, j = slot - kRunSlots * r;
        float hi = L[slot].x, lo = L[slot].y;
        if (j < sm.run_first[r]) {
            lo = __fadd_rn(lo, sm.carry_lo[r]);
            ff_acc(hi, lo, sm.carry_hi[r]);
        }
        const float h = __fadd_rn(hi, lo);
        P[epos] = isnan(h) ? make_float2(__int_as_float(0x7fc00000), 0.0f) : make_float2(h, __fsub_rn(lo, __fsub_rn(h, hi)));
    }
    if (t == 0) {
        const double u = ldexp((double)sum * (1.0 + 1.0 / 1024.0) + ldexp(1.0, -100), 16) + 64.0;
        units = u < (double)kTotalLimit ? (unsigned long long)u : kTotalLimit;
    }
    st = TileStat{bound, mn, raw > 0x7F800000u ? 1u : 0u, 0u};
    return true;
}

// Small rasters (kSmallTiles): a call is bound by its launches, so work that would be a launch of its own, after
// all CTAs of a pass, is done by the CTA that finishes it last (an atomic counter; no CTA waits for another).
struct TileTail {
    int64_t ntiles, nexit;
    unsigned* done;               // [2] finished CTAs of pass 1 and of pass 3
    uint4* S;                     // pass 1: the exit forest's prefix sums, or null (k_scan_exits computes them)
    unsigned long long* redo;     // pass 3: redo[1] = the walk engine must redo the call
    const uint32_t* count;        // pass 3: inflow counts to reset the walk's counters with when it must
    uint32_t* work;
    int64_t nwords;
    unsigned* ctl;                // pass 3: all of the call's control words, left at 0 for the next call
    int64_t nctl;
};

// Whether the CTA is the last of the launch to get here; everything the others wrote before is then visible.  Ends
// with a block barrier.
__device__ __forceinline__ bool last_cta(int& flag, unsigned* done, int64_t n)
{
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) flag = atomicAdd(done, 1u) == (unsigned)(n - 1);
    __syncthreads();
    const bool last = flag;
    if (last) __threadfence();
    __syncthreads();
    return last;
}

// Most exits whose scan one CTA does within pass 1's launch: 16 per thread, about 3 us (a launch of its own takes 5
// us and more).
constexpr int64_t kTailExits = 4096;

__device__ __forceinline__ void tail_scan(const float2* P, int64_t n, const unsigned long long* total, uint4* S)
{
    constexpr int64_t kBlock = kTileThreads * kScanItems;
    __shared__ u128 warp_tot[kTileThreads / 32];
    const int F = fixed_point_bits(*reinterpret_cast<const volatile unsigned long long*>(total));
    u128 carry = 0;
    for (int64_t b0 = 0; b0 < n; b0 += kBlock) {
        const int64_t base = b0 + (int64_t)threadIdx.x * kScanItems;
        u128 v[kScanItems], t = 0;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            v[k] = base + k < n ? exit_value_fixed(__ldcg(P + base + k), F) : (u128)0;
            t += v[k];
        }
        u128 blk;
        u128 run = carry + block_exclusive_u128(t, warp_tot, blk);
        carry += blk;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            run += v[k];
            if (base + k < n) S[base + k] = from_u128(run);
        }
    }
}

// vec: material rows can be read as float4 (16-byte aligned, columns a multiple of 4).
template <bool SMALL>
__global__ void __launch_bounds__(kTileThreads, 4)
    k_tile_exits(TileGeom g, const float* __restrict__ ext, float ext_s, bool vec, TileForest f,
                 const int32_t* __restrict__ exit_base, const uint32_t* __restrict__ exit_span,
                 const uint32_t* __restrict__ exit_pos, float2* P, unsigned long long* total,
                 TileStat* __restrict__ stat, TileTail q)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileCallSmem& sm = *reinterpret_cast<TileCallSmem*>(smem_raw);
    const int64_t tr = blockIdx.y, tc = blockIdx.x;  // grid = (tile columns, tile rows)
    const int64_t tile = tr * g.tcols + tc;
    const int t = threadIdx.x;
    if (SMALL) next_may_start();
    float4 xm[4];
    load_material(xm, ext, ext_s, g, tr, tc, vec);
    uint32_t ca[kRunWords];
    load_run(f.cell_at + tile * kRunPositions, ca);
    const int32_t e0 = __ldg(exit_base + tile), ne = __ldg(exit_base + tile + 1) - e0;
    uint32_t span = 0, epos = 0;
    if (t < ne) {  // a tile has at most 252 exits (its border cells)
        span = __ldg(exit_span + e0 + t);
        epos = __ldg(exit_pos + e0 + t);
    }
    TileStat st{};
    unsigned long long units = 0;
    if (!tile_exits(sm, xm, ca, ne, span, epos, P, st, units)) {
        if (t == 0) atomicOr(total + 1, 1ull);
    } else if (t == 0) {
        // the sum may wrap
        if (units >= kTotalLimit || atomicAdd(total, units) + units < units) atomicOr(total + 1, 1ull);
        stat[tile] = st;
    }
    if (SMALL && q.S && last_cta(sm.quit, q.done, q.ntiles)) {
        if (t == 0)  // total[0] has changed during this launch
            sm.quit = tile_fallback(total) ||
                      *reinterpret_cast<const volatile unsigned long long*>(total) >= kTotalLimit;
        __syncthreads();
        if (!sm.quit) tail_scan(P, q.nexit, total, q.S);
    }
}

// Pass 3: the result of every cell: the accu of its in-tile subtree, where each border cell's material
// carries what enters it from other tiles (the exact subtree sums of the exits draining into it, rounded
// to float once, added to the cell's material in float), in one fixed-point scan per tile.
//
// The scale F comes from pass 1's bound on the tile's material plus the float sum of what enters, so no
// block reduction of the terms is needed; a tile whose smallest positive term would get fewer than 19
// bits sets the fallback flag total[1], and the walk engine redoes the call.  Fast path (no NaN or
// negative term and nothing NaN entering): gather, convert, scan, and for every cell with in-tile upstream
// cells its prefix minus the prefix before its subtree; a cell without in-tile upstream cells keeps its
// material (plus what enters) in M, which is its result.  Slow path: NaN / negative terms count as 0 and
// are counted along the post-order; a cell whose subtree holds one is NaN.
//
// tile_enter: the warps' statistics of what enters (before a block barrier); tile_result: the rest, from M (the
// material in cell order) and the tables in registers.  False: the walk engine must redo the call.
__device__ __forceinline__ void tile_enter(TileCallSmem& sm, float entering)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // over what enters: NaN anywhere, the float sum, and the smallest positive bits minus one
    const bool enan = isnan(entering);
    const float eclean = enan ? 0.0f : entering;
    float esum = eclean;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) esum += __shfl_xor_sync(0xffffffffu, esum, o);
    const unsigned emn = __reduce_min_sync(0xffffffffu, __float_as_uint(eclean) - 1u);
    const unsigned enan_any = __any_sync(0xffffffffu, enan);
    if (lane == 0) {
        sm.warp_sum[warp] = esum;
        sm.red[0][warp] = emn;
        sm.red[1][warp] = enan_any;
    }
}

__device__ __forceinline__ TileStat tile_stat(const TileStat* stat, int64_t tile)
{
    const uint4 w = __ldcg(reinterpret_cast<const uint4*>(stat) + tile);  // written by the launch before
    return TileStat{__uint_as_float(w.x), w.y, w.z, w.w};
}

// One thread decides whether the CTA leaves (other CTAs may set the flag meanwhile); read after a block barrier.
__device__ __forceinline__ void tile_decide(TileCallSmem& sm, unsigned long long* total)
{
    const bool fb = tile_fallback(total);
    if (fb && *reinterpret_cast<volatile unsigned long long*>(total + 1) == 0) total[1] = 1ull;
    sm.quit = fb;
}

__device__ __forceinline__ bool tile_result(TileCallSmem& sm, const TileGeom& g, int64_t tr, int64_t tc, bool vec,
                                            float* __restrict__ out, const uint32_t (&ca)[kRunWords],
                                            const uint32_t (&pv)[kRunWords], const TileStat& st, float entering,
                                            int ecell)
{
    const int t = threadIdx.x;
    if (ecell >= 0) {  // material out of the domain stays visible as NaN (the cell and all below are NaN)
        const float mat = sm.M[ecell];
        sm.M[ecell] = mat >= 0.0f ? mat + entering : __int_as_float(0x7fc00000);
    }
    // over the eight warps, by 16-byte loads; the sum in the same order in every thread
    static_assert(kTileThreads == 256, "eight warps per tile CTA");
    const float4 s0 = *reinterpret_cast<const float4*>(sm.warp_sum);
    const float4 s1 = *reinterpret_cast<const float4*>(sm.warp_sum + 4);
    const uint4 m0 = *reinterpret_cast<const uint4*>(sm.red[0]), m1 = *reinterpret_cast<const uint4*>(sm.red[0] + 4);
    const uint4 n0 = *reinterpret_cast<const uint4*>(sm.red[1]), n1 = *reinterpret_cast<const uint4*>(sm.red[1] + 4);
    const float in_total = 0.0f + s0.x + s0.y + s0.z + s0.w + s1.x + s1.y + s1.z + s1.w;
    const unsigned mn = min(min(min(min(st.min_bits, m0.x), min(m0.y, m0.z)), min(m0.w, m1.x)),
                            min(min(m1.y, m1.z), m1.w));
    const unsigned nan_in = n0.x | n0.y | n0.z | n0.w | n1.x | n1.y | n1.z | n1.w;
    const float bound = (st.bound + in_total) * 1.0009765625f;
    const int F = tile_scale(bound);
    if (!(bound < 1.0e38f) || (mn != 0xFFFFFFFFu && __uint_as_float(mn + 1u) * pow2f(F) < kMinQuantum))
        return false;  // uniform
    const bool exact = mn == 0xFFFFFFFFu || __uint_as_float(mn + 1u) * pow2f(F) >= 8388608.0f;
    const bool clean = !st.bad && !nan_in;  // uniform
    __syncthreads();  // M holds what enters
    float x[kRun];
    gather_run(sm, ca, x);
    unsigned poisoned = 0;  // bit j: the subtree of run entry j holds a NaN or negative term
    if (!clean) {
        poison_counts(sm, clean_run(x));
        const unsigned* C = reinterpret_cast<const unsigned*>(sm.S);
#pragma unroll
        for (int j = 0; j < kRun; ++j)
            if (C[kRunSlots * t + j] != C[run_at(pv, j) >> 3]) poisoned |= 1u << j;
        __syncthreads();  // S and warp_tot are free for the value scan
    }
    unsigned long long a[kRun];
    if (exact) {
#pragma unroll
        for (int j = 0; j < kRun; ++j) a[j] = float_to_fixed64_exact(x[j], pow2f(F - 32));
    } else {
#pragma unroll
        for (int j = 0; j < kRun; ++j) a[j] = float_to_fixed64(x[j], F);
    }
    tile_prefix(sm, a);
    // results by position, put in cell order into M; a cell without in-tile upstream cells keeps its
    // material (plus what enters) there on the fast path, which is its result
    const float nan = __int_as_float(0x7fc00000);
    const float unscale = pow2f(-F);
    const unsigned char* Sb = reinterpret_cast<const unsigned char*>(sm.S);  // prev_at: byte offsets
    // the subtree's sum (its prefix, a[j], minus the prefix before it, < 2^62) to float: two 32-bit
    // conversions, each rounded to nearest, and one fused rounding of their sum: within about one unit
    // in the last place, and exact when it has at most 24 significant bits
    auto result = [&](unsigned long long s_own, unsigned p) {
        const unsigned long long v = s_own - *reinterpret_cast<const unsigned long long*>(Sb + p);
        return __fmaf_rn(__uint2float_rn((unsigned)(v >> 32)), 4294967296.0f, __uint2float_rn((unsigned)v)) *
               unscale;
    };
    if (clean && exact) {  // uniform
        // a valid lone cell already holds its result (its material plus what enters) in M: its lanes skip
        // the read of the prefix before it and the store (predicated, so no shared-memory traffic)
#pragma unroll
        for (int j = 0; j < kRun; ++j) {
            const unsigned w = run_at(ca, j);
            const bool keep = (w & (kLoneCell | kNoValue)) == kLoneCell;
            unsigned long long before = 0ull;
            if (!keep) before = *reinterpret_cast<const unsigned long long*>(Sb + run_at(pv, j));
            const unsigned long long v = a[j] - before;
            const float r = __fmaf_rn(__uint2float_rn((unsigned)(v >> 32)), 4294967296.0f,
                                      __uint2float_rn((unsigned)v)) * unscale;
            if (!keep) sm.M[w & kIndexMask] = (w & kNoValue) ? nan : r;
        }
    } else if (clean) {
#pragma unroll
        for (int j = 0; j < kRun; ++j) {
            const unsigned w = run_at(ca, j);
            const bool none = w & kNoValue;
            if (!none && (w & kLoneCell)) continue;  // keeps its material (plus what enters) in M
            const float r = result(a[j], run_at(pv, j));
            sm.M[w & kIndexMask] = none ? nan : r;
        }
    } else {
#pragma unroll
        for (int j = 0; j < kRun; ++j) {
            const unsigned w = run_at(ca, j);
            const bool none = (w & kNoValue) || ((poisoned >> j) & 1u);
            const float r = result(a[j], run_at(pv, j));
            sm.M[w & kIndexMask] = none ? nan : r;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int cell = quad_cell(j);
        store_quad(out, g, tr * kTile + (cell >> 6), tc * kTile + (cell & 63), vec,
                   *reinterpret_cast<const float4*>(sm.M + cell));
    }
    return true;
}

// SMALL: what enters comes from the tile's slots, computed here, instead of from the array that k_slot_inflow fills (one
// launch less; on a large raster that array is faster: accu at 16384^2 1.65 ms, 1.75 ms without it), and the kernel's
// loads begin before the kernel before it has ended.  Three CTAs per SM, since the registers for that would spill.
template <bool SMALL>
__global__ void __launch_bounds__(kTileThreads, SMALL ? 3 : 4)
    k_tile_accu(TileGeom g, const float* __restrict__ ext, float ext_s, bool vec, float* __restrict__ out,
                TileForest f, const TileStat* __restrict__ stat, unsigned long long* total, TileSlots slots, TileTail q)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileCallSmem& sm = *reinterpret_cast<TileCallSmem*>(smem_raw);
    const int64_t tr = blockIdx.y, tc = blockIdx.x;  // grid = (tile columns, tile rows)
    const int64_t tile = tr * g.tcols + tc;
    const int t = threadIdx.x;
    if (SMALL) next_may_start();
    if (!SMALL && t == 0) tile_decide(sm, total);
    float4 xm[4];
    load_material(xm, ext, ext_s, g, tr, tc, vec);
    uint32_t ca[kRunWords], pv[kRunWords];
    load_run(f.cell_at + tile * kRunPositions, ca);
    load_run(f.prev_at + tile * kRunPositions, pv);
    if (SMALL) {
        wait_for_previous();
        if (t == 0) tile_decide(sm, total);
    }
    const TileStat st = SMALL ? tile_stat(stat, tile) : stat[tile];
    // what enters through border cell t (0 where nothing does; NaN when no-data enters)
    float entering = 0.0f;
    int ecell = -1;
    if (t < kBorderCells) {
        int rin, cin;
        border_cell(t, rin, cin);
        ecell = rin * kTile + cin;
    }
    if (SMALL) {
        float* enter = sm.carry_hi;  // pass 1's
        enter[t] = 0.0f;
        const int32_t s0 = __ldg(slots.base + tile), ns = __ldg(slots.base + tile + 1) - s0;
        __syncthreads();
        if (t < ns && !sm.quit)
            enter[__ldg(slots.at + s0 + t) - (int)(tile * kSlotStride)] =
                slot_inflow(slots, s0 + t, fixed_point_bits(total[0]));
        __syncthreads();
        if (t < kBorderCells) entering = enter[t];
    } else if (t < kBorderCells) {
        entering = __ldg(f.inflow + tile * kSlotStride + t);
    }
    tile_enter(sm, entering);
#pragma unroll
    for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(sm.M + quad_cell(j)) = xm[j];
    __syncthreads();
    if (!sm.quit) {  // uniform
        if (!tile_result(sm, g, tr, tc, vec, out, ca, pv, st, entering, ecell) && t == 0) total[1] = 1ull;
    }
    if (SMALL && last_cta(sm.quit, q.done + 1, q.ntiles)) {
        if (t == 0) {
            sm.quit = tile_fallback(total);
            q.redo[1] = sm.quit;
        }
        __syncthreads();
        if (sm.quit)
            for (int64_t i = t; i < q.nwords; i += kTileThreads) q.work[i] = q.count[i];
        for (int64_t i = t; i < q.nctl; i += kTileThreads) q.ctl[i] = 0u;
    }
}

// ---------------------------------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------------------------------

static inline unsigned blocks_for(int64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

// Most exits that a raster of this shape can have: a cell whose flow leaves its tile lies beside another tile.
static int64_t most_exits(int64_t rows, int64_t cols)
{
    const int64_t trows = (rows + kTile - 1) / kTile, tcols = (cols + kTile - 1) / kTile;
    return 2 * ((trows - 1) * cols + (tcols - 1) * rows);
}

namespace {

// Arrays of the build only.
struct TileTemp {
    size_t ctl, bitmap, rowpref, count, nslot, nedge, edge_base, border_in, border_root, local, cell, size, counters, parent, plus, level,
        link, start;
};

struct TileControl {
    int cyclic, error, depth;
    unsigned roots;
    unsigned long long stats[6];
};

TileTemp plan_temp(int64_t nt, int64_t E, Arena& a)
{
    TileTemp p{};
    p.ctl = a.add(sizeof(TileControl));
    p.bitmap = a.add(nt * kTile * 8);
    p.rowpref = a.add(nt * kTile * 2);
    p.count = a.add(nt * 4);
    p.nslot = a.add(nt * 4);
    p.nedge = a.add(nt * 4);
    p.edge_base = a.add((nt + 1) * 4);
    p.border_in = a.add(nt * kBorderCells);
    p.border_root = a.add(nt * kBorderCells * 4);
    p.local = a.add(E * 2);
    p.cell = a.add(E * 4);
    p.size = a.add(E * 4);
    p.counters = a.add(E * 4 * kExitCounters);
    p.parent = a.add(E * 4);
    p.plus = a.add(E * 4);
    p.level = a.add(E * 4);
    p.link = a.add(E * 8);
    p.start = a.add(E * 4);
    return p;
}

}  // namespace

// From this many cells on, the exits are counted before the arrays are planned: a raster has about half of the most that
// its shape can have (16384^2: 8.2 of 16.7 million, 0.4 GB less in the topology and its scratch).  Below, the
// allocation, launch and synchronisation for it would cost more than the memory is worth (14 of 290 MB at 4000^2).
constexpr int64_t kCountExitsCells = int64_t(1) << 24;

int tile_exit_bound(const uint8_t* fd, int64_t rows, int64_t cols, cudaStream_t stream, int64_t* exits)
{
    *exits = most_exits(rows, cols);
    if (rows * cols < kCountExitsCells) return LUE_GPU_OK;
    const TileGeom g{rows, cols, (rows + kTile - 1) / kTile, (cols + kTile - 1) / kTile};
    Arena a;
    const size_t at = a.add(sizeof(unsigned long long));
    unsigned long long h = 0;
    if (int rc = cuda_status(a.allocate(), "exit count")) return rc;
    if (int rc = cuda_status(cudaMemsetAsync(a.at<char>(at), 0, sizeof h, stream), "exit count")) return rc;
    k_exit_count<<<blocks_for(g.trows * g.tcols, 8), 256, 0, stream>>>(fd, g, a.at<unsigned long long>(at));
    if (int rc = cuda_status(cudaGetLastError(), "exit count")) return rc;
    if (int rc = cuda_status(cudaMemcpyAsync(&h, a.at<char>(at), sizeof h, cudaMemcpyDeviceToHost, stream), "exit count"))
        return rc;
    if (int rc = cuda_status(cudaStreamSynchronize(stream), "exit count")) return rc;
    *exits = (int64_t)h;
    return LUE_GPU_OK;
}

int tile_core_plan(int64_t rows, int64_t cols, int64_t exits, Arena& core, TileCorePlan* p, Arena& scratch,
                   TileScratchPlan* sp)
{
    const int64_t nt = ((rows + kTile - 1) / kTile) * ((cols + kTile - 1) / kTile), E = exits;
    p->exits = E;
    if (E >= INT32_MAX) return fail(LUE_GPU_ERANGE, "tile topology: too many exits");
    const size_t before = core.bytes();
    p->exit_base = core.add((nt + 1) * 4);
    p->slot_base = core.add((nt + 1) * 4);
    p->cell_at = core.add(nt * kRunPositions * 2);
    p->prev_at = core.add(nt * kRunPositions * 2);
    // an inflow slot and its edges belong to exits of other tiles: at most E of each
    p->exit_span = core.add(E * 4);
    p->exit_pos = core.add(E * 4);
    p->slot_at = core.add(E * 4);
    p->slot_first = core.add((E + 1) * 4);
    p->slot_edge = core.add(E * 8);
    p->bytes = core.bytes() - before;
    tile_scratch_plan(nt, E, scratch, sp);
    Arena temp;
    plan_temp(nt, E, temp);
    scratch.reserve(temp.bytes());
    return LUE_GPU_OK;
}

// Builds the tile structures, the downstream levels and the raster's statistics (hstats: valid, ridge, outlet, sink,
// cycle, largest level) in the planned arenas, and readies the scratch.  core->tiles stays empty, and the levels and
// statistics are all there is, when the network has a flow cycle.  The build's own arrays lie in the handle's scratch.
int tile_core_build(TopologyCore* core, const Arena& arena, const TileCorePlan& plan, const Arena& scratch,
                    const TileScratchPlan& scratch_plan, cudaStream_t stream, unsigned long long* hstats)
{
    auto* tc = new (std::nothrow) TileCore();
    if (!tc) return fail(LUE_GPU_ENOMEM, "tile topology: host allocation");
    TileGeom g{core->rows, core->cols, (core->rows + kTile - 1) / kTile, (core->cols + kTile - 1) / kTile};
    tc->trows = g.trows;
    tc->tcols = g.tcols;
    tc->ntiles = g.trows * g.tcols;
    const int64_t nt = tc->ntiles, most = plan.exits;
    const dim3 grid((unsigned)g.tcols, (unsigned)g.trows);
    const unsigned exit_ctas = blocks_for(std::max<int64_t>(most, 1), 256);
    tc->bytes = (int64_t)plan.bytes;
    tc->exit_base = arena.at<int32_t>(plan.exit_base);
    tc->slot_base = arena.at<int32_t>(plan.slot_base);
    tc->cell_at = arena.at<uint16_t>(plan.cell_at);
    tc->prev_at = arena.at<uint16_t>(plan.prev_at);
    tc->exit_span = arena.at<uint32_t>(plan.exit_span);
    tc->exit_pos = arena.at<uint32_t>(plan.exit_pos);
    tc->slot_at = arena.at<int32_t>(plan.slot_at);
    tc->slot_first = arena.at<int32_t>(plan.slot_first);
    tc->slot_edge = arena.at<int2>(plan.slot_edge);
    Arena sizes;
    const TileTemp tmp = plan_temp(nt, most, sizes);
    TileControl* ctl = scratch.at<TileControl>(tmp.ctl);
    uint64_t* bitmap = scratch.at<uint64_t>(tmp.bitmap);
    uint16_t* rowpref = scratch.at<uint16_t>(tmp.rowpref);
    int32_t *count = scratch.at<int32_t>(tmp.count), *nslot = scratch.at<int32_t>(tmp.nslot),
            *nedge = scratch.at<int32_t>(tmp.nedge), *edge_base = scratch.at<int32_t>(tmp.edge_base);
    uint8_t* border_in = scratch.at<uint8_t>(tmp.border_in);
    uint16_t* exit_local = scratch.at<uint16_t>(tmp.local);
    uint32_t *exit_cell = scratch.at<uint32_t>(tmp.cell), *size = scratch.at<uint32_t>(tmp.size),
             *exit_start = scratch.at<uint32_t>(tmp.start), *border_root = scratch.at<uint32_t>(tmp.border_root);
    int32_t* nchild = scratch.at<int32_t>(tmp.counters);
    int32_t *pending = nchild + most, *depth = nchild + 2 * most, *seen = nchild + 3 * most;
    uint32_t* acc = reinterpret_cast<uint32_t*>(nchild + 4 * most);
    int32_t *parent = scratch.at<int32_t>(tmp.parent), *plus = scratch.at<int32_t>(tmp.plus),
            *exit_level = scratch.at<int32_t>(tmp.level);
    int2* link = scratch.at<int2>(tmp.link);
    int32_t *base = tc->exit_base, *nexit = base + nt, hexit = 0, hslot = 0;
    TileControl h{};
    int rc = 0;
#define TRY(call, what) \
    if ((rc = cuda_status((call), what))) goto error
    TRY(cudaFuncSetAttribute(k_tile_forest, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileSmem)),
        "tile topology: shared memory");
    TRY(cudaMemsetAsync(ctl, 0, sizeof(TileControl), stream), "tile topology");
    k_exit_bitmap<<<blocks_for(nt, 8), 256, 0, stream>>>(core->fd, g, bitmap, rowpref, count);
    k_tile_scan<<<1, 1024, 0, stream>>>(count, base, nullptr, nullptr, nt);
    k_exit_list<<<blocks_for(nt * kTile, 256), 256, 0, stream>>>(g, bitmap, rowpref, base, exit_local, exit_cell, size,
                                                                 nchild, most);
    k_tile_forest<<<grid, kTileThreads, sizeof(TileSmem), stream>>>(core->fd, g, base, exit_local, tc->cell_at, tc->prev_at,
                                                                    tc->exit_span, border_in, nslot, nedge, exit_level,
                                                                    core->level, border_root, &ctl->error, &ctl->cyclic);
    k_tile_scan<<<1, 1024, 0, stream>>>(nslot, tc->slot_base, nedge, edge_base, nt);
    k_exit_parent<<<exit_ctas, 256, 0, stream>>>(core->fd, g, nexit, exit_cell, base, bitmap, rowpref, border_root, parent,
                                                 nchild, pending, plus);
    k_exit_sizes<<<exit_ctas, 256, 0, stream>>>(nexit, parent, nchild, plus, pending, size, exit_level, depth, &ctl->depth);
    k_exit_offsets<<<exit_ctas, 256, 0, stream>>>(nexit, parent, pending, size, acc, &ctl->roots, link, &ctl->cyclic);
    TRY(cudaGetLastError(), "tile build");
    TRY(cudaMemcpyAsync(&hexit, nexit, sizeof hexit, cudaMemcpyDeviceToHost, stream), "tile exits");
    TRY(cudaMemcpyAsync(&h, ctl, sizeof h, cudaMemcpyDeviceToHost, stream), "tile build");
    TRY(cudaStreamSynchronize(stream), "tile build");
    if (h.cyclic) {
        k_tile_levels<<<grid, kTileThreads, 0, stream>>>(core->fd, g, base, bitmap, rowpref, border_in, exit_level, pending,
                                                         hexit, core->level, ctl->stats);
        TRY(cudaGetLastError(), "tile build");
        TRY(cudaMemcpyAsync(hstats, ctl->stats, sizeof h.stats, cudaMemcpyDeviceToHost, stream), "tile build");
        TRY(cudaStreamSynchronize(stream), "tile build");
        goto error;  // rc == LUE_GPU_OK
    }
    tc->nexit = hexit;
    tc->max_depth = std::max(h.depth, hexit > 0 ? 1 : 0);
    if (hexit > 0) {
        const unsigned ctas = blocks_for(hexit, 256);
        for (int64_t reach = 1; reach < tc->max_depth; reach *= 2) k_jump<<<ctas, 256, 0, stream>>>(hexit, link);
        k_exit_positions<<<ctas, 256, 0, stream>>>(hexit, link, size, tc->exit_pos, exit_start, seen, &ctl->error);
    }
    k_slot_fill<<<grid, kTileThreads, 0, stream>>>(g, border_in, base, bitmap, rowpref, tc->slot_base, edge_base, tc->exit_pos,
                                                   exit_start, tc->slot_at, tc->slot_first, tc->slot_edge, hexit,
                                                   &ctl->error);
    k_tile_levels<<<grid, kTileThreads, 0, stream>>>(core->fd, g, base, bitmap, rowpref, border_in, exit_level, nullptr,
                                                     hexit, core->level, ctl->stats);
    TRY(cudaGetLastError(), "tile build");
    TRY(cudaMemcpyAsync(&h, ctl, sizeof h, cudaMemcpyDeviceToHost, stream), "tile build");
    TRY(cudaMemcpyAsync(&hslot, tc->slot_base + nt, sizeof hslot, cudaMemcpyDeviceToHost, stream), "tile build");
    if ((rc = tile_scratch_clear(scratch, scratch_plan, stream))) goto error;
    TRY(cudaStreamSynchronize(stream), "tile build");
    if (h.error) {
        rc = fail(LUE_GPU_EINVAL, "tile topology: inconsistent tile or exit forest");
        goto error;
    }
    tc->nslot = hslot;
    std::memcpy(hstats, h.stats, sizeof h.stats);
    core->tiles = tc;
    return LUE_GPU_OK;
error:
    delete tc;
    return rc;
#undef TRY
}

// A handle's tile scratch, planned in its arena for up to nexit exits.
void tile_scratch_plan(int64_t ntiles, int64_t nexit, Arena& a, TileScratchPlan* p)
{
    const int64_t E = std::max<int64_t>(nexit, 1);
    const int64_t nb = (E + kTileThreads * kScanItemsSmall - 1) / (kTileThreads * kScanItemsSmall);
    p->P = a.add(E * sizeof(float2));
    p->S = a.add(E * sizeof(uint4));
    p->look_aggr = a.add(nb * sizeof(uint4));
    p->look_incl = a.add(nb * sizeof(uint4));
    // zeroed once: slots without inflow are never written, and
    // total[2], the finished CTAs of the passes, the scan's ticket, its block flags
    p->inflow = a.add(ntiles * kSlotStride * sizeof(float));
    p->ctl_bytes = 2 * sizeof(unsigned long long) + (3 + nb) * sizeof(unsigned);
    p->total = a.add(p->ctl_bytes);
    p->redo = a.add(2 * sizeof(unsigned long long));
    p->stat = a.add(ntiles * sizeof(TileStat));
}

void tile_scratch_take(const Arena& a, const TileScratchPlan& p, TileScratch* s)
{
    s->P = a.at<float2>(p.P);
    s->S = a.at<uint4>(p.S);
    s->inflow = a.at<float>(p.inflow);
    s->look_aggr = a.at<uint4>(p.look_aggr);
    s->look_incl = a.at<uint4>(p.look_incl);
    s->total = a.at<unsigned long long>(p.total);
    s->ctl_bytes = (int64_t)p.ctl_bytes;
    s->redo = a.at<unsigned long long>(p.redo);
    s->stat = a.at<TileStat>(p.stat);
}

int tile_scratch_clear(const Arena& a, const TileScratchPlan& p, cudaStream_t stream)
{
    return cuda_status(cudaMemsetAsync(a.at<char>(p.inflow), 0, p.total + p.ctl_bytes - p.inflow, stream), "tile scratch");
}

// CTAs of k_scan_exits that fit on the device at once (chunks of the exit-forest scan).  The result does
// not depend on it: the chunks' sums are exact.
static int64_t scan_ctas()
{
    static const int64_t n = [] {
        int dev = 0, sms = 0, per_sm = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_scan_exits<kScanItems>, kTileThreads, 0) != cudaSuccess ||
            sms <= 0 || per_sm <= 0) {
            cudaGetLastError();
            return (int64_t)152;
        }
        return (int64_t)sms * per_sm;
    }();
    return n;
}

// Rasters of up to this many tiles (2048 x 2048 cells) are bound by their launches and the latency of each: three or
// four launches that overlap take 22, 32 and 56 us a call at 256^2, 1024^2 and 2048^2, seven in turn 37, 46 and 63 us;
// at 2800^2 they take 101 us against 92 us.
constexpr int64_t kSmallTiles = 1024;

template <bool SMALL>
static bool tile_smem_ok()
{
    static const bool ok = cudaFuncSetAttribute(k_tile_exits<SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)sizeof(TileCallSmem)) == cudaSuccess &&
                           cudaFuncSetAttribute(k_tile_accu<SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)sizeof(TileCallSmem)) == cudaSuccess;
    return ok;
}

// accu (float32) on the tile engine.  Returns LUE_GPU_OK with (*redo)[1] set on the device when the material holds
// +inf or its total is beyond the fixed-point range; the caller then runs the walk engine, guarded by that flag,
// with its counters in `work` (reset here when *reset is true on return, else the caller resets them).
int tile_accu_f32(const TopologyCore* core, TileScratch* s, const float* ext, float ext_s, float* out, uint32_t* work,
                  cudaStream_t stream, const unsigned long long** redo, bool* reset)
{
    const TileCore* tc = core->tiles;
    TileGeom g{core->rows, core->cols, tc->trows, tc->tcols};
    const TileForest f{tc->cell_at, tc->prev_at, s->inflow};
    // rows move as float4 when the columns are a multiple of 4 and the arrays 16-byte aligned
    const bool cols4 = (core->cols & 3) == 0;
    const bool vec_in = cols4 && (!ext || (reinterpret_cast<uintptr_t>(ext) & 15) == 0);
    const bool vec_out = cols4 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    const bool small = tc->ntiles <= kSmallTiles;
    if (!(small ? tile_smem_ok<true>() : tile_smem_ok<false>()))
        return fail(LUE_GPU_ECUDA, "accu_f32 (tiles): shared memory attribute");
    const dim3 tile_grid((unsigned)tc->tcols, (unsigned)tc->trows);
    const int64_t E = tc->nexit;
    unsigned* done = reinterpret_cast<unsigned*>(s->total + 2);
    const bool tail = small && E <= kTailExits;
    const TileTail q{tc->ntiles, E, done, tail && E > 0 ? s->S : nullptr, s->redo,
                     reinterpret_cast<const uint32_t*>(core->count), work, words_for(core->n),
                     reinterpret_cast<unsigned*>(s->total), s->ctl_bytes / 4};
    const TileSlots slots{tc->slot_base, tc->slot_at, tc->slot_first, tc->slot_edge, s->S};
    *redo = small ? s->redo : s->total;
    *reset = small;
    // a small call leaves its control words at 0, unless one of its launches was refused
    if (!small || s->dirty)
        if (int rc = cuda_status(cudaMemsetAsync(s->total, 0, s->ctl_bytes, stream), "accu_f32 (tiles)")) return rc;
    s->dirty = small;
    constexpr size_t smem = sizeof(TileCallSmem);
    // test hook: LUE_GB300_TILE_REFUSE asks for more shared memory than there is, so that pass 3's launch is refused
    const size_t refused = getenv("LUE_GB300_TILE_REFUSE") ? size_t(1) << 20 : 0;
    if (small)
        k_tile_exits<true><<<tile_grid, kTileThreads, smem, stream>>>(g, ext, ext_s, vec_in, f, tc->exit_base,
                                                                      tc->exit_span, tc->exit_pos, s->P, s->total,
                                                                      s->stat, q);
    else
        k_tile_exits<false><<<tile_grid, kTileThreads, smem, stream>>>(g, ext, ext_s, vec_in, f, tc->exit_base,
                                                                       tc->exit_span, tc->exit_pos, s->P, s->total,
                                                                       s->stat, q);
    count_launches(1);
    if (E > 0 && !tail) {
        const int64_t block = kTileThreads * (small ? kScanItemsSmall : kScanItems);
        const int64_t nb = (E + block - 1) / block;
        const int64_t chunk_blocks = (nb + scan_ctas() - 1) / scan_ctas();
        const int64_t nchunk = (nb + chunk_blocks - 1) / chunk_blocks;
        // test hook: LUE_GB300_TILE_POLLS (poll limit of a look-back wait; 0: every wait gives up at once,
        // and the walk engine redoes the call)
        int polls = kScanPolls;
        if (const char* e = getenv("LUE_GB300_TILE_POLLS")) polls = std::max(0, atoi(e));
        if (small)
            launch_after(k_scan_exits<kScanItemsSmall>, (unsigned)nchunk, kTileThreads, 0, stream, s->P, E, chunk_blocks,
                         s->total, done + 2, s->look_aggr, s->look_incl, s->S, polls);
        else
            k_scan_exits<kScanItems><<<(unsigned)nchunk, kTileThreads, 0, stream>>>(
                s->P, E, chunk_blocks, s->total, done + 2, s->look_aggr, s->look_incl, s->S, polls);
        count_launches(1);
        if (!small && tc->nslot > 0) {
            k_slot_inflow<<<blocks_for(tc->nslot, 256), 256, 0, stream>>>(tc->nslot, slots, s->inflow, s->total);
            count_launches(1);
        }
    }
    if (small)
        launch_after(k_tile_accu<true>, tile_grid, kTileThreads, smem + refused, stream, g, ext, ext_s, vec_in && vec_out, out, f,
                     s->stat, s->total, slots, q);
    else
        k_tile_accu<false><<<tile_grid, kTileThreads, smem, stream>>>(g, ext, ext_s, vec_in && vec_out, out, f, s->stat,
                                                                      s->total, slots, q);
    count_launches(1);
    const int rc = cuda_status(cudaGetLastError(), "accu_f32 (tiles)");
    if (!rc) s->dirty = false;
    return rc;
}

}  // namespace lue_gb300
