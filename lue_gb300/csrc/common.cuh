// common.cuh — shared device helpers: D8 decoding, neighbour tables, compensated arithmetic, status.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <utility>

#include "lue_gb300.h"

namespace lue_gb300 {

constexpr uint8_t kNoData = 255;

// Neighbour k of a cell, k = 0..7: NW, N, NE, W, E, SW, S, SE (row offset, column offset).
__host__ __device__ constexpr int nb_dr(int k) { return k < 3 ? -1 : (k < 5 ? 0 : 1); }
__host__ __device__ constexpr int nb_dc(int k)
{
    return (k == 0 || k == 3 || k == 5) ? -1 : ((k == 1 || k == 6) ? 0 : 1);
}

// Code neighbour k must carry to drain into the centre cell: the keypad code pointing back.
// NW neighbour drains SE (3), N -> S (2), NE -> SW (1), W -> E (6), E -> W (4), SW -> NE (9),
// S -> N (8), SE -> NW (7).
__host__ __device__ constexpr uint8_t nb_inflow_code(int k)
{
    return k == 0 ? 3 : k == 1 ? 2 : k == 2 ? 1 : k == 3 ? 6 : k == 4 ? 4 : k == 5 ? 9 : k == 6 ? 8 : 7;
}

// Keypad D8 code to offsets (flow_direction.hpp:7-35); anything else is a sink (0, 0).
__host__ __device__ inline bool d8_offset(uint8_t code, int& dr, int& dc)
{
    switch (code) {
        case 7: dr = -1; dc = -1; return true;
        case 8: dr = -1; dc = 0; return true;
        case 9: dr = -1; dc = 1; return true;
        case 4: dr = 0; dc = -1; return true;
        case 6: dr = 0; dc = 1; return true;
        case 1: dr = 1; dc = -1; return true;
        case 2: dr = 1; dc = 0; return true;
        case 3: dr = 1; dc = 1; return true;
        default: dr = 0; dc = 0; return false;
    }
}

// Downstream cell index of cell (r, c) with code `code`; false for sinks and for flow off the array.
__device__ inline bool downstream(uint8_t code, int64_t r, int64_t c, int64_t rows, int64_t cols, int64_t& d)
{
    int dr, dc;
    if (!d8_offset(code, dr, dc)) return false;
    int64_t rd = r + dr, cd = c + dc;
    if (rd < 0 || rd >= rows || cd < 0 || cd >= cols) return false;
    d = rd * cols + cd;
    return true;
}

// Error-free transformations (Knuth two-sum, FMA two-product) for float-float accumulation.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e)
{
    s = __fadd_rn(a, b);
    float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// Float-float accumulator: value = hi + lo with |lo| <= ulp(hi) / 2 after normalise().  A sum that is
// not finite keeps IEEE semantics (inf stays inf, NaN stays NaN) with lo = 0; the error terms of
// two_sum would otherwise turn inf into NaN.
struct FF {
    float hi, lo;
    __device__ __forceinline__ void add(float x)
    {
        float s, e;
        two_sum(hi, x, s, e);
        if (!isfinite(s)) {
            hi = s;
            lo = 0.0f;
            return;
        }
        hi = s;
        lo = __fadd_rn(lo, e);
    }
    __device__ __forceinline__ void add(float xh, float xl)
    {
        add(xh);
        if (isfinite(hi)) lo = __fadd_rn(lo, xl);
    }
    __device__ __forceinline__ void normalise()
    {
        float s = __fadd_rn(hi, lo);
        if (!isfinite(s)) {
            hi = s;
            lo = 0.0f;
            return;
        }
        lo = __fsub_rn(lo, __fsub_rn(s, hi));
        hi = s;
    }
};

// Loads that bypass L1: values written by other threads during the same kernel.
template <class T>
__device__ __forceinline__ T load_cg(const T* p)
{
    return __ldcg(p);
}

// On the integer pipes: a warp's float64 operation, comparisons included, takes the float64 pipe of a GB300 SM 16 cycles.
__device__ __forceinline__ bool is_nan_bits(double x)
{
    const unsigned lo = (unsigned)__double2loint(x);
    return (((unsigned)__double2hiint(x) & 0x7fffffffu) | ((lo | (0u - lo)) >> 31)) > 0x7ff00000u;
}

// Words by which CTAs wait for one another.
__device__ __forceinline__ int ld_acquire(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p)
{
    return (unsigned)ld_acquire(reinterpret_cast<const int*>(p));
}
__device__ __forceinline__ void st_release(int* p, int v)
{
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) { st_release(reinterpret_cast<int*>(p), (int)v); }

__device__ __forceinline__ int64_t grid_stride_begin() { return (int64_t)blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int64_t grid_stride() { return (int64_t)gridDim.x * blockDim.x; }

// Kernels of one call that follow each other on a stream (launch_after below): the next one starts while this one
// still runs, once every CTA of this one has said so (or ended), and reads what no earlier kernel of the call
// writes; it waits for the whole of this one before anything else.  Neither does anything in a kernel launched the
// ordinary way.
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Host side -----------------------------------------------------------------------------------------

void set_error(const std::string& msg);
// Kernel launches made by this library in this process (reported by lue_gpu_kernel_launches).
void count_launches(int n);
int fail(int status, const std::string& msg);
int cuda_status(cudaError_t err, const char* what);

// Launches a kernel that may start before the kernel before it on the stream has ended: it must call
// wait_for_previous() before it reads what that one (or an earlier one of the call) writes and before its own first
// write.  Errors are left to cudaGetLastError(), as with <<<>>>.
template <class... P, class... A>
inline void launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    c.attrs = &attr;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// Several device arrays in one allocation: plan them with add(), then allocate().  Frees it unless released.
class Arena {
    size_t bytes_ = 0;
    char* base_ = nullptr;
    bool owned_ = false;

public:
    Arena() = default;
    Arena(const Arena&) = delete;
    Arena& operator=(const Arena&) = delete;
    ~Arena()
    {
        if (owned_) cudaFree(base_);
    }
    size_t add(int64_t n)
    {
        const size_t at = bytes_;
        bytes_ += ((size_t)n + 255) & ~size_t(255);
        return at;
    }
    size_t bytes() const { return bytes_; }
    void reserve(size_t n) { bytes_ = bytes_ < n ? n : bytes_; }
    cudaError_t allocate()
    {
        const cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&base_), bytes_ ? bytes_ : 256);
        owned_ = e == cudaSuccess;
        return e;
    }
    void* release()
    {
        owned_ = false;
        return base_;
    }
    void swap(Arena& o)
    {
        std::swap(bytes_, o.bytes_);
        std::swap(base_, o.base_);
        std::swap(owned_, o.owned_);
    }
    template <class T>
    T* at(size_t offset) const
    {
        return reinterpret_cast<T*>(base_ + offset);
    }
};

// One thread per element, no grid-stride reuse (walk kernels: a thread that walks a long path must not
// also own later cells, or the walks chain up behind each other).
inline unsigned grid_all(int64_t n, int threads)
{
    int64_t b = (n + threads - 1) / threads;
    return (unsigned)(b < 1 ? 1 : b);
}

inline int grid_for(int64_t n, int threads, int max_blocks = 152 * 16)
{
    int64_t b = (n + threads - 1) / threads;
    if (b > max_blocks) b = max_blocks;
    if (b < 1) b = 1;
    return (int)b;
}

}  // namespace lue_gb300
