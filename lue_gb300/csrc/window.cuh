// window.cuh — the 3 x 3 window of focal operations, in registers.
//
// A warp takes 32 adjacent columns and kWindowRows + 2 rows: lane l holds column l of every row, and its
// neighbours' values come by shuffles.  The outer lanes and rows are halo, so a warp gives the results of
// 30 x kWindowRows cells.  All loads of a warp are issued at once, before the first use, and each is one
// coalesced access per row whatever the raster's width: no shared memory, no barrier, no index division
// per halo element, and rows need not be aligned.  8 rows keep 20 loads of a thread in flight and cost 2
// halo rows, which the CTA above or below has brought into L2.
#pragma once

#include "common.cuh"

namespace lue_gb300 {

constexpr int kWindowRows = 8;
constexpr int kWindowCols = 30;                     // results per warp and row
constexpr int kWindowThreads = 256;                 // 8 warps side by side; fewer where one CTA is wide enough
constexpr int kWindowCtaCols = kWindowCols * (kWindowThreads / 32);

// EDGE: part of the CTA's windows lies outside the array (or the raster is too wide for 32-bit offsets), so every
// access is checked.  Inside, a row is one 32-bit offset from a base that the whole CTA shares: the checks and
// 64-bit addresses were about half of the instructions of these kernels, which issue bounds.
template <bool EDGE>
struct WindowAt {
    int64_t rows, cols, r0, c;  // r0: first row of the results; c: this lane's column
    unsigned off;               // this lane's offset (elements) from the window's first row, inside
    bool in, result;            // the column is in the array; the lane gives results

    __device__ __forceinline__ WindowAt(int64_t rows_, int64_t cols_) : rows(rows_), cols(cols_)
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int x = warp * kWindowCols + lane;
        r0 = (int64_t)blockIdx.y * kWindowRows;
        c = (int64_t)blockIdx.x * kWindowCtaCols + x - 1;
        off = (unsigned)x;
        in = !EDGE || (c >= 0 && c < cols);
        result = in && lane >= 1 && lane <= kWindowCols;
    }

    // Whether no column of the warp is in the array (uniform).
    __device__ __forceinline__ bool idle() const { return EDGE && c - (int)(threadIdx.x & 31) + 1 >= cols; }
    // Whether result row j lies below the array (uniform).
    __device__ __forceinline__ bool below(int j) const { return EDGE && r0 + j >= rows; }

    // Rows r0 - 1 .. r0 + kWindowRows of a raster at the lane's column; `outside` where there is no cell.
    template <class T, class R>
    __device__ __forceinline__ void load(R (&x)[kWindowRows + 2], const T* __restrict__ p, R outside) const
    {
        if (EDGE) {
#pragma unroll
            for (int j = 0; j < kWindowRows + 2; ++j) {
                const int64_t r = r0 + j - 1;
                x[j] = in && r >= 0 && r < rows ? (R)__ldg(p + r * cols + c) : outside;
            }
        } else {
            const T* q = p + (r0 - 1) * cols + (int64_t)blockIdx.x * kWindowCtaCols - 1;
#pragma unroll
            for (int j = 0; j < kWindowRows + 2; ++j) x[j] = (R)__ldg(q + (off + (unsigned)j * (unsigned)cols));
        }
    }

    // The result of row r0 + j.
    template <class T>
    __device__ __forceinline__ void store(T* __restrict__ p, int j, T v) const
    {
        if (EDGE) {
            const int64_t r = r0 + j;
            if (result && r < rows) p[r * cols + c] = v;
        } else {
            T* q = p + r0 * cols + (int64_t)blockIdx.x * kWindowCtaCols - 1;
            if (result) q[off + (unsigned)j * (unsigned)cols] = v;
        }
    }
};

// Whether every cell of the CTA's windows is in the array, at 32-bit offsets (uniform over the CTA).
__device__ __forceinline__ bool window_inside(int64_t rows, int64_t cols)
{
    return blockIdx.y > 0 && ((int64_t)blockIdx.y + 1) * kWindowRows < rows && blockIdx.x > 0 &&
           ((int64_t)blockIdx.x + 1) * kWindowCtaCols < cols && cols < (1 << 24);
}

// The grid and the threads of a windowed kernel; false when the raster has more rows than a grid holds.  On a narrow raster
// eight warps, of which one has results, fill the SMs with idle ones: float32 upstream, downstream and d8 of 500000 x 8
// 264, 234 and 286 us; with the warps that it takes 56, 51 and 54 us.
inline bool window_grid(int64_t rows, int64_t cols, dim3& grid, unsigned& threads)
{
    const int64_t y = (rows + kWindowRows - 1) / kWindowRows, warps = (cols + kWindowCols - 1) / kWindowCols;
    threads = (unsigned)(warps < kWindowThreads / 32 ? 32 * warps : kWindowThreads);
    grid = dim3((unsigned)((cols + kWindowCtaCols - 1) / kWindowCtaCols), (unsigned)y);
    return y <= 65535;
}

}  // namespace lue_gb300
