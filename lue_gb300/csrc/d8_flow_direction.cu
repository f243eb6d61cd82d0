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

template <class T, bool EDGE>
__device__ __forceinline__ void d8_window(const T* __restrict__ z, int64_t rows, int64_t cols, uint8_t* __restrict__ fd)
{
    const WindowAt<EDGE> w(rows, cols);
    if (w.idle()) return;
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

// Bound by instruction issue.  Before, one thread per cell with a 32 x 8 tile in shared memory: 422 us at 8192 x 8191;
// now 172 us, with 32 registers (44: 194 us).
template <class T>
__global__ void __launch_bounds__(kWindowThreads, sizeof(T) == 4 ? 8 : 1)
    k_d8(const T* __restrict__ z, int64_t rows, int64_t cols, uint8_t* __restrict__ fd)
{
    if (window_inside(rows, cols)) d8_window<T, false>(z, rows, cols, fd);
    else d8_window<T, true>(z, rows, cols, fd);
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
