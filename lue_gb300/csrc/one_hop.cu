// one_hop.cu — upstream, downstream and downstream_distance: one-hop and local operations on a D8
// raster (focal operations of radius 1 in the reference; no routing, no topology).
//
//   upstream ............ ALG/definition/upstream.hpp:9-160     sum of the material of the neighbours that
//                                                                drain into the cell (NW N NE W E SW S SE)
//   downstream .......... ALG/definition/downstream.hpp:9-158   material of the downstream cell
//   downstream_distance . ALG/definition/downstream_distance.hpp:9-75
//                                                                length of the step to the downstream cell
// (ALG/ = source/framework/algorithm/include/lue/framework/algorithm/)
//
// Value policies (ALG/flow_accumulation.hpp DefaultValuePolicies, ALG/policy/flow_direction_halo.hpp):
// no-data is 255 for flow directions and NaN for material; outside the array the flow directions point
// away from the array and the material is 0.
//
// upstream and downstream take their 3 x 3 windows from registers (window.cuh).
#include "window.cuh"

namespace lue_gb300 {

// Rows are taken from north to south, and each cell's material is added to the sum of the cell it drains
// into: first to a sum of the row below (whose sum begins there), then to one of its own row, then to one
// of the row above, so a sum takes its terms in the order NW N NE W E SW S SE.
template <bool EDGE>
__device__ __forceinline__ void upstream_window(const uint8_t* __restrict__ fd, int64_t rows, int64_t cols,
                                                const float* __restrict__ m, float* __restrict__ out)
{
    using T = float;
    const WindowAt<EDGE> w(rows, cols);
    if (w.idle()) return;
    unsigned f[kWindowRows + 2];
    T v[kWindowRows + 2];
    w.load(f, fd, (unsigned)kNoData);
    w.load(v, m, T(0));
    T sum[kWindowRows + 2];
#pragma unroll
    for (int j = 0; j < kWindowRows + 2; ++j) {
        const unsigned west = __shfl_up_sync(0xffffffffu, f[j], 1), east = __shfl_down_sync(0xffffffffu, f[j], 1);
        const T vw = __shfl_up_sync(0xffffffffu, v[j], 1), ve = __shfl_down_sync(0xffffffffu, v[j], 1);
        if (j + 1 <= kWindowRows) {
            T s = T(0);
            if (west == 3u) s += vw;
            if (f[j] == 2u) s += v[j];
            if (east == 1u) s += ve;
            sum[j + 1] = s;
        }
        if (j >= 1 && j <= kWindowRows) {
            if (west == 6u) sum[j] += vw;
            if (east == 4u) sum[j] += ve;
        }
        if (j >= 2) {
            T s = sum[j - 1];
            if (west == 9u) s += vw;
            if (f[j] == 8u) s += v[j];
            if (east == 7u) s += ve;
            if (f[j - 1] == kNoData || isnan(v[j - 1])) s = T(NAN);
            w.store(out, j - 2, s);
        }
    }
}

// float64: a warp's addition takes the float64 pipe 16 cycles whatever the number of lanes that need it, so each cell takes
// its upstream values one after the other, found by integer operations: as many additions per row of a warp as its
// busiest cell has inflows, less one, instead of eight and a comparison: 8192 x 8191 1290 -> 580 us, 500000 x 8 296 -> 137.
template <bool EDGE>
__device__ __forceinline__ void upstream_window(const uint8_t* __restrict__ fd, int64_t rows, int64_t cols,
                                                const double* __restrict__ m, double* __restrict__ out)
{
    const WindowAt<EDGE> w(rows, cols);
    if (w.idle()) return;
    unsigned f[kWindowRows + 2], mask[kWindowRows + 2];
    double v[kWindowRows + 2];
    w.load(f, fd, (unsigned)kNoData);
    w.load(v, m, 0.0);
    const int west_lane = (int)(threadIdx.x & 31) - 1;
#pragma unroll
    for (int j = 0; j < kWindowRows + 2; ++j) {
        if (j >= 2 && w.below(j - 2)) break;
        const unsigned west = __shfl_up_sync(0xffffffffu, f[j], 1), east = __shfl_down_sync(0xffffffffu, f[j], 1);
        if (j + 1 <= kWindowRows) mask[j + 1] = (west == 3u ? 1u : 0u) | (f[j] == 2u ? 2u : 0u) | (east == 1u ? 4u : 0u);
        if (j >= 1 && j <= kWindowRows) mask[j] |= (west == 6u ? 8u : 0u) | (east == 4u ? 16u : 0u);
        if (j < 2) continue;
        unsigned from = mask[j - 1] | (west == 9u ? 32u : 0u) | (f[j] == 8u ? 64u : 0u) | (east == 7u ? 128u : 0u);
        bool nan = f[j - 1] == kNoData || is_nan_bits(v[j - 1]);
        if (!w.result || nan) from = 0;
        double s = 0.0;
        bool first = true;
        while (__any_sync(0xffffffffu, from != 0)) {
            const int k = from ? __ffs(from) - 1 : 0, place = k + (k > 3);  // of the 3 x 3 cells, row by row
            const int row = (place * 11) >> 5, lane = west_lane + place - 3 * row;
            const double above = __shfl_sync(0xffffffffu, v[j - 2], lane), level = __shfl_sync(0xffffffffu, v[j - 1], lane),
                         below = __shfl_sync(0xffffffffu, v[j], lane);
            const double x = row == 0 ? above : (row == 1 ? level : below);
            const bool some = from != 0;
            from &= from - 1u;
            if (__any_sync(0xffffffffu, some && !first)) {
                const double sum = s + x;
                if (some && !first) s = sum;
            }
            // 0 + x: x, but 0 for -0
            if (some && first) s = __double_as_longlong(x) == (long long)0x8000000000000000ull ? 0.0 : x;
            nan |= some && is_nan_bits(x);
            if (some) first = false;
        }
        if (nan) s = NAN;
        w.store(out, j - 2, s);
    }
}

// Bound by instruction issue and DRAM about equally (9 B per float cell).  Before, one thread per cell with the
// codes staged byte by byte in shared memory: 599 us at 8192 x 8191; now 131 us (4.6 TB/s).
template <class T>
__global__ void __launch_bounds__(kWindowThreads)
    k_upstream(const uint8_t* __restrict__ fd, int64_t rows, int64_t cols, const T* __restrict__ m, T* __restrict__ out)
{
    if (window_inside(rows, cols)) upstream_window<false>(fd, rows, cols, m, out);
    else upstream_window<true>(fd, rows, cols, m, out);
}

// Code k of the keypad (1..9) points to column (k - 1) % 3 - 1 and row 1 - (k - 1) / 3, and 5 to the cell itself;
// outside the array the window holds 0, which is what a cell whose flow leaves the array gets.
template <class T, bool EDGE>
__device__ __forceinline__ void downstream_window(const uint8_t* __restrict__ fd, int64_t rows, int64_t cols,
                                                  const T* __restrict__ m, T* __restrict__ out)
{
    const WindowAt<EDGE> w(rows, cols);
    if (w.idle()) return;
    unsigned f[kWindowRows + 2];
    T v[kWindowRows + 2];
    w.load(f, fd, (unsigned)kNoData);  // the first and the last row are not used: no loads of them
    w.load(v, m, T(0));
    const int west = (int)(threadIdx.x & 31) - 1;
#pragma unroll
    for (int j = 1; j <= kWindowRows; ++j) {
        if (w.below(j - 1)) break;
        unsigned k = f[j] - 1u;
        if (k > 8u) k = 4u;  // no-data, or a code that is not a direction: a sink
        const unsigned north = (k * 11u) >> 5;  // k / 3: 0 the row below, 1 the cell's, 2 the row above
        const int from = west + (int)(k - 3u * north);  // 0 .. 31 in the lanes that give results
        const T below = __shfl_sync(0xffffffffu, v[j + 1], from);
        const T level = __shfl_sync(0xffffffffu, v[j], from);
        const T above = __shfl_sync(0xffffffffu, v[j - 1], from);
        T to = north == 0u ? below : (north == 1u ? level : above);
        if (f[j] == kNoData || isnan(v[j])) to = T(NAN);
        w.store(out, j - 1, to);
    }
}

// Bound as k_upstream.  Before, one thread per cell and a gather per cell: 324 us at 8192 x 8191; now 111 us (5.4 TB/s).
template <class T>
__global__ void __launch_bounds__(kWindowThreads)
    k_downstream(const uint8_t* __restrict__ fd, int64_t rows, int64_t cols, const T* __restrict__ m,
                 T* __restrict__ out)
{
    if (window_inside(rows, cols)) downstream_window<T, false>(fd, rows, cols, m, out);
    else downstream_window<T, true>(fd, rows, cols, m, out);
}

template <class T>
__global__ void k_downstream_distance(const uint8_t* __restrict__ fd, int64_t n, T cell, T diagonal,
                                      T* __restrict__ out)
{
    for (int64_t i = grid_stride_begin(); i < n; i += grid_stride()) {
        const uint8_t code = __ldg(fd + i);
        T d = T(0);
        if (code == kNoData) d = T(NAN);
        else if (code == 7 || code == 9 || code == 1 || code == 3) d = diagonal;
        else if (code == 8 || code == 4 || code == 6 || code == 2) d = cell;
        out[i] = d;
    }
}

template <class T>
static int one_hop(bool up, const uint8_t* fd, int64_t rows, int64_t cols, const T* m, T* out, void* stream,
                   const char* what)
{
    if (!fd || !m || !out) return fail(LUE_GPU_EINVAL, std::string(what) + ": NULL argument");
    if (rows <= 0 || cols <= 0) return fail(LUE_GPU_EINVAL, std::string(what) + ": non-positive extent");
    dim3 grid;
    unsigned threads = 0;
    if (!window_grid(rows, cols, grid, threads)) return fail(LUE_GPU_ERANGE, std::string(what) + ": more than 524280 rows");
    if (up)
        k_upstream<T><<<grid, threads, 0, (cudaStream_t)stream>>>(fd, rows, cols, m, out);
    else
        k_downstream<T><<<grid, threads, 0, (cudaStream_t)stream>>>(fd, rows, cols, m, out);
    count_launches(1);
    return cuda_status(cudaGetLastError(), what);
}

template <class T>
static int distance(const uint8_t* fd, int64_t rows, int64_t cols, T cell_size, T* out, void* stream)
{
    if (!fd || !out) return fail(LUE_GPU_EINVAL, "downstream_distance: NULL argument");
    if (rows <= 0 || cols <= 0) return fail(LUE_GPU_EINVAL, "downstream_distance: non-positive extent");
    const int64_t n = rows * cols;
    const T diagonal = (T)(sqrt(2.0) * (double)cell_size);
    k_downstream_distance<T><<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(fd, n, cell_size, diagonal, out);
    count_launches(1);
    return cuda_status(cudaGetLastError(), "downstream_distance");
}

}  // namespace lue_gb300

using namespace lue_gb300;

extern "C" int lue_gpu_upstream_f32(const uint8_t* fd, int64_t rows, int64_t cols, const float* material, float* out,
                                    void* stream)
{
    return one_hop<float>(true, fd, rows, cols, material, out, stream, "upstream_f32");
}
extern "C" int lue_gpu_upstream_f64(const uint8_t* fd, int64_t rows, int64_t cols, const double* material,
                                    double* out, void* stream)
{
    return one_hop<double>(true, fd, rows, cols, material, out, stream, "upstream_f64");
}
extern "C" int lue_gpu_downstream_f32(const uint8_t* fd, int64_t rows, int64_t cols, const float* material,
                                      float* out, void* stream)
{
    return one_hop<float>(false, fd, rows, cols, material, out, stream, "downstream_f32");
}
extern "C" int lue_gpu_downstream_f64(const uint8_t* fd, int64_t rows, int64_t cols, const double* material,
                                      double* out, void* stream)
{
    return one_hop<double>(false, fd, rows, cols, material, out, stream, "downstream_f64");
}
extern "C" int lue_gpu_downstream_distance_f32(const uint8_t* fd, int64_t rows, int64_t cols, float cell_size,
                                               float* out, void* stream)
{
    return distance<float>(fd, rows, cols, cell_size, out, stream);
}
extern "C" int lue_gpu_downstream_distance_f64(const uint8_t* fd, int64_t rows, int64_t cols, double cell_size,
                                               double* out, void* stream)
{
    return distance<double>(fd, rows, cols, cell_size, out, stream);
}
