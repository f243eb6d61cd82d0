// d8_flow_direction.cu — D8 flow direction from an elevation raster (the step before the routing path).
//
// Restates the reference's rule (ALG/definition/d8_flow_direction.hpp:45-147 and
// ALG/value_policies/d8_flow_direction.hpp:20-45, ALG/ = source/framework/algorithm/include/lue/framework/
// algorithm/): for each cell, the steepest unweighted drop among the neighbours in the order N, W, E, S,
// NW, NE, SW, SE, with a strict '>' (so the first of equal drops wins); no drop > 0 gives a sink (5).
// A NaN elevation gives the no-data direction 255; a NaN neighbour is skipped.  Outside the array the
// halo holds std::numeric_limits<E>::min() (the smallest positive normal value), so cells above it on
// the edge drain off the array.
//
// The 3 x 3 windows come from registers (window.cuh), so each elevation is read from HBM about once.
#include <cfloat>

#include "window.cuh"

namespace lue_gb300 {

template <class T>
__device__ __forceinline__ T halo_min();
template <>
__device__ __forceinline__ float halo_min<float>() { return FLT_MIN; }
template <>
__device__ __forceinline__ double halo_min<double>() { return DBL_MIN; }

template <bool EDGE>
__device__ __forceinline__ void d8_window(const float* __restrict__ z, int64_t rows, int64_t cols, uint8_t* __restrict__ fd)
{
    const WindowAt<EDGE> w(rows, cols);
    if (w.idle()) return;
    using T = float;
    T v[kWindowRows + 2], west[kWindowRows + 2], east[kWindowRows + 2];
    w.load(v, z, halo_min<T>());
#pragma unroll
    for (int j = 0; j < kWindowRows + 2; ++j) {
        if (j >= 2 && w.below(j - 2)) break;
        west[j] = __shfl_up_sync(0xffffffffu, v[j], 1);
        east[j] = __shfl_down_sync(0xffffffffu, v[j], 1);
        if (j < 2) continue;
        const T zc = v[j - 1];
        // candidates N, W, E, S, NW, NE, SW, SE (d8_flow_direction.hpp:57-145)
        const T zn[8] = {v[j - 2], west[j - 1], east[j - 1], v[j], west[j - 2], east[j - 2], west[j], east[j]};
        constexpr unsigned code[8] = {8, 4, 6, 2, 7, 9, 1, 3};
        unsigned dir = 5;
        T drop = T(0);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const T other = zc - zn[k];
            if (other > drop) {  // false for a NaN neighbour
                drop = other;
                dir = code[k];
            }
        }
        if (isnan(zc)) dir = kNoData;
        w.store(fd, j - 2, (uint8_t)dir);
    }
}

// float64: a warp's subtraction or comparison takes the float64 pipe 16 cycles.  The drop from a cell to a neighbour is that
// from the neighbour to the cell with its sign turned, so four subtractions a row give all eight, and drops, which only
// count when they are positive, are compared as integers.  A drop that is not a number counts as 0.  8192 x 8191: 2490 -> 709
// us, 500000 x 8: 566 -> 161.
template <bool EDGE>
__device__ __forceinline__ void d8_window(const double* __restrict__ z, int64_t rows, int64_t cols, uint8_t* __restrict__ fd)
{
    const WindowAt<EDGE> w(rows, cols);
    if (w.idle()) return;
    double v[kWindowRows + 2];
    w.load(v, z, halo_min<double>());
    constexpr long long kSign = (long long)0x8000000000000000ull;
    auto drop_of = [](double a, double b) {
        const double d = a - b;
        return is_nan_bits(d) ? 0ll : __double_as_longlong(d);
    };
    long long south = 0, south_east = 0, south_west = 0;  // of the row before, from its cells
    double east = 0.0;
#pragma unroll
    for (int j = 0; j <= kWindowRows; ++j) {
        if (j >= 1 && w.below(j - 1)) break;
        const double here = v[j], next_west = __shfl_up_sync(0xffffffffu, v[j + 1], 1),
                     next_east = __shfl_down_sync(0xffffffffu, v[j + 1], 1);
        const long long to_south = drop_of(here, v[j + 1]), to_south_east = drop_of(here, next_east),
                        to_south_west = drop_of(here, next_west);
        if (j >= 1) {
            const long long to_east = drop_of(here, east), from_west = __shfl_up_sync(0xffffffffu, to_east, 1);
            // candidates N, W, E, S, NW, NE, SW, SE (d8_flow_direction.hpp:57-145)
            const long long drops[8] = {south ^ kSign,
                                        from_west ^ kSign,
                                        to_east,
                                        to_south,
                                        __shfl_up_sync(0xffffffffu, south_east, 1) ^ kSign,
                                        __shfl_down_sync(0xffffffffu, south_west, 1) ^ kSign,
                                        to_south_west,
                                        to_south_east};
            constexpr unsigned code[8] = {8, 4, 6, 2, 7, 9, 1, 3};
            unsigned dir = 5;
            long long drop = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (drops[k] > drop) {  // false for a negative drop
                    drop = drops[k];
                    dir = code[k];
                }
            }
            if (is_nan_bits(here)) dir = kNoData;
            w.store(fd, j - 1, (uint8_t)dir);
        }
        south = to_south;
        south_east = to_south_east;
        south_west = to_south_west;
        east = next_east;
    }
}

// Bound by instruction issue.  Before, one thread per cell with a 32 x 8 tile in shared memory: 422 us at 8192 x 8191;
// now 172 us, with 32 registers (44: 194 us).
template <class T>
__global__ void __launch_bounds__(kWindowThreads, sizeof(T) == 4 ? 8 : 1)
    k_d8(const T* __restrict__ z, int64_t rows, int64_t cols, uint8_t* __restrict__ fd)
{
    if (window_inside(rows, cols)) d8_window<false>(z, rows, cols, fd);
    else d8_window<true>(z, rows, cols, fd);
}

template <class T>
static int d8(const T* z, int64_t rows, int64_t cols, uint8_t* fd, void* stream, const char* what)
{
    if (!z || !fd) return fail(LUE_GPU_EINVAL, std::string(what) + ": NULL argument");
    if (rows <= 0 || cols <= 0) return fail(LUE_GPU_EINVAL, std::string(what) + ": array shape must not be empty");
    dim3 grid;
    unsigned threads = 0;
    if (!window_grid(rows, cols, grid, threads)) return fail(LUE_GPU_ERANGE, std::string(what) + ": too many rows");
    k_d8<T><<<grid, threads, 0, (cudaStream_t)stream>>>(z, rows, cols, fd);
    count_launches(1);
    return cuda_status(cudaGetLastError(), what);
}

}  // namespace lue_gb300

extern "C" int lue_gpu_d8_flow_direction_f32(const float* elevation, int64_t rows, int64_t cols, uint8_t* flow_direction,
                                             void* stream)
{
    return lue_gb300::d8(elevation, rows, cols, flow_direction, stream, "d8_flow_direction_f32");
}

extern "C" int lue_gpu_d8_flow_direction_f64(const double* elevation, int64_t rows, int64_t cols,
                                             uint8_t* flow_direction, void* stream)
{
    return lue_gb300::d8(elevation, rows, cols, flow_direction, stream, "d8_flow_direction_f64");
}
