// CSR operands, CSR SpMV and CG / PCG / block-PCG for sm_100a.
//
// Replaces the reference's cuSPARSE SpMV (src/sparse/sparse_ops.cu:687-740) and its
// cuBLAS-driven adaptive solver loop (src/sparse/iterative_solver.cu:30-349), which
// synchronises with the host after every iteration.  Here:
//   * the int64 CSR structure is validated once and kept as int32 (4 B per index on the
//     HBM stream instead of 8 B);
//   * SpMV takes rows of up to eight nonzeros on average 32 at a time through shared memory, a
//     lane per row, and longer ones with 16 or 32 lanes per row and shuffle reductions;
//   * a CG / PCG solve is one cooperative kernel where that is the faster form (pcg_row_kernel,
//     pcg_loop_kernel): SpMV with the p.q dot, vector update with preconditioner apply and the
//     r.z / r.r dots, direction, with grid barriers between.  Elsewhere the same three steps are
//     kernels, repeated by a CUDA graph 'while' node; every dot is accumulated in FP64 per block
//     and finished by the last block to arrive, in a fixed order.  Either way the device decides
//     when the solve is done and the host reads the state once, after it.
#include "pm_common.cuh"
#include "pm_grid.cuh"
#include "pm_piece.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <limits>
#include <mutex>
#include <sstream>
#include <vector>

struct pm_csr
{
    int value_size = 0;
    int64_t rows = 0, cols = 0, nnz = 0;
    int* row_ptr = nullptr; // int32 copy of the validated row offsets
    int* col_idx = nullptr; // int32 copy of the validated column indices
    const void* values = nullptr;
    int threads_per_row = 1; // lanes per row of the heuristic
    int longest_row = 0;     // its nonzeros
    uint64_t serial = 0;     // no other operand of the process has it, also none that is created later
    int kernel = -1;         // -1: heuristic; 0: row-group stream; 1..32: lanes per row (autotuned or set)
    // streams on which products or fixed-iteration solves were queued (pm_csr_wait)
    mutable std::mutex used_lock;
    mutable std::vector<cudaStream_t> used;
    void queued_on(cudaStream_t stream) const
    {
        const std::lock_guard<std::mutex> lock(used_lock);
        if (std::find(used.begin(), used.end(), stream) == used.end())
            used.push_back(stream);
    }
};

namespace pm
{

// the SpMV shape of an operand: the row-group stream kernel, or TPR lanes per row
inline bool use_stream(const pm_csr* A) { return A->kernel == 0; }
inline int lanes_per_row(const pm_csr* A) { return A->kernel > 0 ? A->kernel : A->threads_per_row; }

template <typename T>
struct Eps;
template <>
struct Eps<float>
{
    static constexpr double value = 1.1920928955078125e-7;
};
template <>
struct Eps<double>
{
    static constexpr double value = 2.2204460492503131e-16;
};

namespace
{

constexpr long long kNone = 0x7fffffffffffffffLL;
constexpr int kReduceBlock = 256;
constexpr int kMaxReduceBlocks = 1024;

struct CsrCheck
{
    long long bad_offsets_row;
    long long bad_column;
    long long bad_value;
    int endpoints_bad;
    int longest; // nonzeros of a row
};

template <typename T>
__global__ void validate_csr_kernel(int64_t rows, int64_t cols, int64_t nnz, const int64_t* __restrict__ row_offsets,
                                    const int64_t* __restrict__ col_indices, const T* __restrict__ values,
                                    int* __restrict__ row_ptr32, int* __restrict__ col32, CsrCheck* check)
{
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t == 0 && (row_offsets[0] != 0 || row_offsets[rows] != nnz))
        check->endpoints_bad = 1;
    int longest = 0;
    for (int64_t r = t; r < rows; r += stride)
    {
        const int64_t b = row_offsets[r], e = row_offsets[r + 1];
        if (b < 0 || e < b || e > nnz)
            atomicMin(&check->bad_offsets_row, static_cast<long long>(r));
        row_ptr32[r] = static_cast<int>(b);
        longest = static_cast<int>(min(static_cast<int64_t>(INT32_MAX), max(e - b, static_cast<int64_t>(longest))));
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    if (longest > 0 && (threadIdx.x & 31) == 0)
        atomicMax(&check->longest, longest);
    if (t == 0)
        row_ptr32[rows] = static_cast<int>(nnz);
    for (int64_t p = t; p < nnz; p += stride)
    {
        const int64_t c = col_indices[p];
        if (c < 0 || c >= cols)
            atomicMin(&check->bad_column, static_cast<long long>(p));
        if (!isfinite(static_cast<double>(values[p])))
            atomicMin(&check->bad_value, static_cast<long long>(p));
        col32[p] = static_cast<int>(c);
    }
}

// row of A x with a TPR-wide sub-warp per row; x_at(c) is entry c of x; G > 0 of a lane's nonzeros are
// loaded at a time: columns and values, then the gathers, all in flight together; 0: one after the other,
// as the compiler unrolls them (see long_rows).  The order of a lane's sum is the same.
template <typename T, int TPR, int G, typename Gather>
__device__ __forceinline__ T csr_row_dot(const int* __restrict__ rp, const int* __restrict__ ci,
                                         const T* __restrict__ v, Gather&& x_at, int64_t row, bool valid, int lane)
{
    T sum = T(0);
    if (valid)
    {
        const int b = rp[row], e = rp[row + 1];
        if constexpr (G == 0)
        {
            for (int p = b + lane; p < e; p += TPR)
                sum += v[p] * x_at(ci[p]);
        }
        else
        {
            for (int p = b + lane; p < e; p += G * TPR)
            {
                int col[G];
                T val[G], xv[G];
#pragma unroll
                for (int k = 0; k < G; ++k)
                    if (p + k * TPR < e)
                    {
                        // a thread per row: streamed, no reuse
                        col[k] = TPR == 1 ? __ldcs(ci + p + k * TPR) : ci[p + k * TPR];
                        val[k] = TPR == 1 ? __ldcs(v + p + k * TPR) : v[p + k * TPR];
                    }
#pragma unroll
                for (int k = 0; k < G; ++k)
                    if (p + k * TPR < e)
                        xv[k] = x_at(col[k]);
#pragma unroll
                for (int k = 0; k < G; ++k)
                    if (p + k * TPR < e)
                        sum += val[k] * xv[k];
            }
        }
    }
#pragma unroll
    for (int o = TPR / 2; o > 0; o >>= 1)
        sum += __shfl_xor_sync(0xffffffffu, sum, o, TPR);
    return sum;
}

// ------------------------------------------------------------------ staged row tiles
// One lane per row with the matrix staged in shared memory.  A warp takes tiles of 32 consecutive
// rows; the tile's nonzeros are one contiguous range of columns and values, brought in by 16-byte
// asynchronous copies (coalesced, marked evict-first in L2 so that the vectors stay), and lane i
// then sums row i in storage order from shared memory.  Reading the
// same rows directly costs a lane-strided access per nonzero: 180 load wavefronts per 32 rows of
// seven FP64 nonzeros against about 100 here, and at 180 the load pipe (45 us for the 128^3
// Laplacian) is slower than HBM.
constexpr int kTileCap = 256; // most staged nonzeros per tile; longer tiles are taken in pieces
template <typename T, int CAP>
struct alignas(16) RowTile
{
    static_assert(CAP % 4 == 0, "whole 16-byte pieces");
    T val[CAP];
    int col[CAP];
};

__device__ __forceinline__ uint64_t evict_first_policy()
{
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(policy));
    return policy;
}

// 16 bytes global -> shared, of which the first `bytes` are read and the rest zero-filled
__device__ __forceinline__ void cp_async16_stream(void* dst, const void* src, int bytes, uint64_t policy)
{
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;\n" ::"r"(smem_addr(dst)), "l"(src),
                 "r"(bytes), "l"(policy)
                 : "memory");
}

// nonzeros [first, first + count) into the tile (first a multiple of four, count <= its capacity);
// nothing at or past `nnz` is read
template <typename T, int CAP>
__device__ __forceinline__ void tile_load(RowTile<T, CAP>& tile, const int* __restrict__ ci, const T* __restrict__ v,
                                          int first, int count, int nnz, uint64_t policy, int lane)
{
    constexpr int kPer = 16 / static_cast<int>(sizeof(T));
#pragma unroll
    for (int u = 0; u < (CAP + 127) / 128; ++u)
    {
        const int k = (u * 32 + lane) * 4;
        if (k < count)
            cp_async16_stream(tile.col + k, ci + first + k, piece_bytes(nnz - first - k, sizeof(int)), policy);
    }
#pragma unroll
    for (int u = 0; u < (CAP + 32 * kPer - 1) / (32 * kPer); ++u)
    {
        const int k = (u * 32 + lane) * kPer;
        if (k < count)
            cp_async16_stream(tile.val + k, v + first + k, piece_bytes(nnz - first - k, sizeof(T)), policy);
    }
}

// sum + the products of the staged positions [lo, hi), in order; gathers in groups of G
template <int G, typename T, int CAP, typename Gather>
__device__ __forceinline__ T tile_sum(const RowTile<T, CAP>& tile, int lo, int hi, T sum, Gather&& x_at)
{
    for (int base = lo; base < hi; base += G)
    {
        T xv[G];
#pragma unroll
        for (int k = 0; k < G; ++k)
            if (base + k < hi)
                xv[k] = x_at(tile.col[base + k]);
#pragma unroll
        for (int k = 0; k < G; ++k)
            if (base + k < hi)
                sum += tile.val[base + k] * xv[k];
    }
    return sum;
}

// the row [b, e) of a tile whose nonzeros are [first, end), its first piece staged; tiles longer
// than the capacity load their other pieces here
template <int G, typename T, int CAP, typename Gather>
__device__ __forceinline__ T tile_row(RowTile<T, CAP>& tile, const int* __restrict__ ci, const T* __restrict__ v,
                                      int b, int e, int first, int end, int nnz, uint64_t policy, int lane,
                                      Gather&& x_at)
{
    T sum = tile_sum<G>(tile, b - first, min(e - first, CAP), T(0), x_at);
    // unsigned: the step past the last piece need not fit in an int
    for (unsigned next = static_cast<unsigned>(first) + CAP; next < static_cast<unsigned>(end); next += CAP)
    {
        const int at = static_cast<int>(next);
        __syncwarp();
        tile_load(tile, ci, v, at, min(end - at, CAP), nnz, policy, lane);
        cp_async_commit();
        cp_async_wait<0>();
        __syncwarp();
        sum = tile_sum<G>(tile, max(b - at, 0), min(e - at, CAP), sum, x_at);
    }
    return sum;
}

// Every tile warp0, warp0 + warps, ...: done(row, sum) for each of its rows, by the row's lane.
// Values and columns 16-byte aligned; `stage`: the warp's tiles, two (the next one is on its way while
// one is summed) or one.
template <int BUFFERS, typename T, int CAP, typename Gather, typename Done>
__device__ __forceinline__ void csr_tiles(RowTile<T, CAP>* stage, int64_t rows, int nnz, const int* __restrict__ rp,
                                          const int* __restrict__ ci, const T* __restrict__ v, int64_t warp0,
                                          int64_t warps, Gather&& x_at, Done&& done)
{
    const int lane = threadIdx.x & 31;
    const uint64_t policy = evict_first_policy();
    const int64_t tiles = (rows + 31) / 32;
    auto bounds = [&](int64_t tile, int& b, int& e) {
        const int64_t row = tile * 32 + lane;
        b = e = nnz;
        if (row < rows)
        {
            b = rp[row];
            e = rp[row + 1];
        }
    };
    auto issue = [&](RowTile<T, CAP>& tile, int b, int e) {
        const int first = __shfl_sync(0xffffffffu, b, 0) & ~3;
        const int count = __shfl_sync(0xffffffffu, e, 31) - first;
        tile_load(tile, ci, v, first, min(count, CAP), nnz, policy, lane);
        cp_async_commit();
    };
    int b, e, nb, ne, buffer = 0;
    bounds(warp0, b, e);
    bounds(warp0 + warps, nb, ne);
    if (BUFFERS == 2)
        issue(stage[0], b, e);
    for (int64_t t = warp0; t < tiles; t += warps)
    {
        if (BUFFERS == 2)
            issue(stage[buffer ^ 1], nb, ne);
        else
            issue(stage[0], b, e);
        int fb, fe;
        bounds(t + 2 * warps, fb, fe);
        cp_async_wait<BUFFERS - 1>();
        __syncwarp();
        const int first = __shfl_sync(0xffffffffu, b, 0) & ~3;
        const int end = __shfl_sync(0xffffffffu, e, 31);
        constexpr int G = BUFFERS == 1 && sizeof(T) == 4 ? 4 : 8;
        const T sum = tile_row<G>(stage[buffer], ci, v, b, e, first, end, nnz, policy, lane, x_at);
        if (t * 32 + lane < rows)
            done(t * 32 + lane, sum);
        __syncwarp();
        b = nb;
        e = ne;
        nb = fb;
        ne = fe;
        if (BUFFERS == 2)
            buffer ^= 1;
    }
    cp_async_wait<0>();
}

// SpMV.  What bounds it is the gathers of x, and the matrix from HBM when it is cold.  One tile of ten
// nonzeros per row for each warp: a second buffer would take the L1 from the gathers (FP64 197 KB of shared
// memory an SM against 123) and a capacity of eight per row sends half the tiles of a mean of 7.9 through a
// second load.  us, directly read / two buffers of 256 / this, L2 warm: 600,000 rows of 7.9 in a random
// band FP64 24.7 / 33.0 / 22.7, FP32 18.2 / 19.4 / 16.5; 1.5M rows of 7.3 FP64 55.2 / 57.9 / 47.2, FP32
// 37.0 / 37.1 / 32.7; 128^3 grid FP64 37.0 / 35.0 / 35.0, FP32 26.5 / 28.4 / 26.8, cold FP64 45.1 / 41.0 /
// 39.0.  Five CTAs per SM and gathers in groups of four in FP32 (48 registers); FP64 spills there.
constexpr int kSpmvCap = 320;
constexpr int spmv_ctas(size_t value_size) { return value_size == 8 ? 4 : 5; } // of 256 threads per SM
template <typename T>
__global__ void __launch_bounds__(256, spmv_ctas(sizeof(T))) csr_tile_kernel(int64_t rows, int nnz,
                                                                             const int* __restrict__ rp,
                                                                             const int* __restrict__ ci,
                                                                             const T* __restrict__ v,
                                                                             const T* __restrict__ x,
                                                                             T* __restrict__ y)
{
    extern __shared__ __align__(16) unsigned char tile_smem[];
    csr_tiles<1>(reinterpret_cast<RowTile<T, kSpmvCap>*>(tile_smem) + (threadIdx.x >> 5), rows, nnz, rp, ci, v,
                 (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5, int64_t(gridDim.x) * (blockDim.x >> 5),
                 [&](int c) { return __ldg(x + c); }, [&](int64_t row, T sum) { y[row] = sum; });
}

// Row-group stream (chosen by pm_csr_set_kernel or the autotuner): a warp owns 32 consecutive rows.  Their nonzeros form one
// contiguous range, loaded coalesced in pieces of kStreamCap (values, columns, then the x
// gathers, all in flight together); products are staged in shared memory and lane i sums
// row i's products in column order.  The sum order is the row's storage order.
constexpr int kStreamCap = 256; // staged products per warp
constexpr int kStreamUnroll = kStreamCap / 32;

template <typename T, typename Gather>
__device__ __forceinline__ T csr_stream_rows(int64_t r0, int64_t rows, const int* __restrict__ rp,
                                             const int* __restrict__ ci, const T* __restrict__ v, Gather&& x_at,
                                             T* __restrict__ stage)
{
    const int lane = threadIdx.x & 31;
    const int64_t row = r0 + lane;
    const bool valid = row < rows;
    const int my_begin = valid ? rp[row] : 0;
    const int my_end = valid ? rp[row + 1] : 0;
    const int last = static_cast<int>(rows - 1 - r0 < 31 ? rows - 1 - r0 : 31);
    const int cb = __shfl_sync(0xffffffffu, my_begin, 0);
    const int ce = __shfl_sync(0xffffffffu, my_end, last);
    T sum = T(0);
    for (int base = cb; base < ce; base += kStreamCap)
    {
        const int n = ce - base < kStreamCap ? ce - base : kStreamCap;
        int col[kStreamUnroll];
        T val[kStreamUnroll];
#pragma unroll
        for (int u = 0; u < kStreamUnroll; ++u)
        {
            const int k = u * 32 + lane;
            if (k < n)
            {
                col[u] = __ldcs(ci + base + k);
                val[u] = __ldcs(v + base + k);
            }
        }
#pragma unroll
        for (int u = 0; u < kStreamUnroll; ++u)
        {
            const int k = u * 32 + lane;
            if (k < n)
                stage[k] = val[u] * x_at(col[u]);
        }
        __syncwarp();
        const int lo = my_begin > base ? my_begin : base;
        const int hi = my_end < base + n ? my_end : base + n;
        for (int k = lo; k < hi; ++k)
            sum += stage[k - base];
        __syncwarp();
    }
    return sum;
}

template <typename T>
__global__ void __launch_bounds__(256) csr_stream_kernel(int64_t rows, const int* __restrict__ rp,
                                                         const int* __restrict__ ci, const T* __restrict__ v,
                                                         const T* __restrict__ x, T* __restrict__ y)
{
    __shared__ T stage[8][kStreamCap];
    const int warp = threadIdx.x >> 5;
    const int64_t warps = int64_t(gridDim.x) * 8;
    for (int64_t wrow = (int64_t(blockIdx.x) * 8 + warp) * 32; wrow < rows; wrow += warps * 32)
    {
        const T sum = csr_stream_rows<T>(wrow, rows, rp, ci, v, [&](int c) { return __ldg(x + c); }, stage[warp]);
        if (wrow + (threadIdx.x & 31) < rows)
            y[wrow + (threadIdx.x & 31)] = sum;
    }
}

template <typename T, int TPR, int G>
__global__ void __launch_bounds__(256) csr_spmv_kernel(int64_t rows, const int* __restrict__ rp,
                                                       const int* __restrict__ ci, const T* __restrict__ v,
                                                       const T* __restrict__ x, T* __restrict__ y)
{
    const int64_t gid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x / TPR;
    const int lane = threadIdx.x % TPR;
    const int64_t first = gid / TPR;
    const int64_t span = (rows + stride - 1) / stride; // uniform trip count keeps shuffles convergent
    for (int64_t k = 0; k < span; ++k)
    {
        const int64_t row = first + k * stride;
        const bool valid = row < rows;
        const T sum =
            csr_row_dot<T, TPR, G>(rp, ci, v, [&](int c) { return __ldg(x + c); }, row, valid, lane);
        if (valid && lane == 0)
            y[row] = sum;
    }
}

// heuristic lanes per row: a lane per row up to 8 nonzeros per row on average (128^3 Laplacian FP64, cold:
// 39 us from staged tiles, 45 read in groups where the values are not aligned, 56 as a row-group stream),
// then 16 or 32
int pick_tpr(int64_t rows, int64_t nnz)
{
    const double mean = rows > 0 ? double(nnz) / double(rows) : 1.0;
    if (mean <= 8.0)
        return 1;
    int tpr = 16;
    while (tpr < 32 && tpr < mean)
        tpr <<= 1;
    return tpr;
}

// Rows of fourteen or more nonzeros per lane, on 32 lanes, are read eight of a lane's at a time (two rounds of
// loads for a row of 474 instead of fifteen, at 48-64 registers instead of 32): 24,000 rows of 474, L2 warm,
// FP32 22.7 -> 16.5 us, FP64 50.6 -> 28.9; 12,000 of 1,000, FP32 25.0 -> 16.5, FP64 57.5 -> 28.8.  Below that
// most of a round is empty and half the warps are gone: 24,000 rows of 400, 30 FP32 iterations 833 us one
// after the other against 880; 240,000 rows of 32, FP64 57 us against 97; an 80^3 27-point grid 112 against 213.
// A lone long row is a chain of its own, 6 ns a nonzero less in rounds; the rest pays 0.007 ns a nonzero of the
// matrix: 60,000 rows of 18, FP64, one of 5,000, 45 us one after the other and 21 in rounds; 240,000 rows of
// 18, one of 5,000, 47 and 72, one of 20,000, 168 and 72.
inline bool long_rows(const pm_csr* A)
{
    if (lanes_per_row(A) != 32 || A->nnz > INT32_MAX - 8 * 32) // positions a round past the end fit in an int
        return false;
    return A->nnz >= 14 * 32 * A->rows || (A->longest_row >= 256 && A->nnz <= 512 * int64_t(A->longest_row));
}

// one lane per row from staged tiles: the values (the caller's array) on a 16-byte boundary
template <typename T>
bool use_tiles(const pm_csr* A)
{
    return !use_stream(A) && lanes_per_row(A) == 1 && reinterpret_cast<uintptr_t>(A->values) % 16 == 0;
}

template <typename T>
void launch_spmv(const pm_csr* A, const T* x, T* y, cudaStream_t stream)
{
    if (A->rows == 0)
        return;
    const T* v = static_cast<const T*>(A->values);
    const int block = 256;
    if (use_stream(A))
    {
        csr_stream_kernel<T><<<grid_for(A->rows, 256, 1 << 20), 256, 0, stream>>>(A->rows, A->row_ptr, A->col_idx,
                                                                                    v, x, y);
        PM_LAUNCH_CHECK();
        return;
    }
    if (use_tiles<T>(A))
    {
        const size_t smem = size_t(block / 32) * sizeof(RowTile<T, kSpmvCap>);
        allow_smem(reinterpret_cast<const void*>(csr_tile_kernel<T>), smem);
        csr_tile_kernel<T><<<grid_for(A->rows, block, spmv_ctas(sizeof(T)) * sm_count()), block, smem, stream>>>(
            A->rows, static_cast<int>(A->nnz), A->row_ptr, A->col_idx, v, x, y);
        PM_LAUNCH_CHECK();
        return;
    }
    const unsigned grid = grid_for(A->rows * lanes_per_row(A), block, 65535);
    switch (lanes_per_row(A))
    {
    case 1: csr_spmv_kernel<T, 1, 8><<<grid, block, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, x, y); break;
    case 2: csr_spmv_kernel<T, 2, 0><<<grid, block, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, x, y); break;
    case 4: csr_spmv_kernel<T, 4, 0><<<grid, block, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, x, y); break;
    case 8: csr_spmv_kernel<T, 8, 0><<<grid, block, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, x, y); break;
    case 16: csr_spmv_kernel<T, 16, 0><<<grid, block, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, x, y); break;
    default:
        if (long_rows(A))
            csr_spmv_kernel<T, 32, 8><<<grid, block, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, x, y);
        else
            csr_spmv_kernel<T, 32, 0><<<grid, block, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, x, y);
        break;
    }
    PM_LAUNCH_CHECK();
}

// ------------------------------------------------------------------ PCG state
struct PcgState
{
    double rho;      // r.z of the current direction
    double alpha;
    double beta;
    double tolerance;
    double initial_squared;
    double residual_squared;
    int iterations;
    int max_iterations;
    int done;
    int converged;
    int breakdown;     // 1: not SPD / non-finite step
    int nonfinite_init;
    int timed_out;     // a grid barrier gave up
    long long jacobi_bad_row;
    unsigned int ticket[3];
    int chunks; // bodies run by the iteration graph
};

// ------------------------------------------------------------------ PCG in one launch
// The whole solve is one cooperative kernel: the SpMV, the vector updates and the dots of every
// iteration, with grid barriers in the place of kernel boundaries.  A graph of three kernels per
// iteration costs 10-14 us an iteration however small the system is.  Every dot is accumulated in
// FP64 per CTA; after the barrier each CTA sums the partials in the same fixed order, so all CTAs
// take the same alpha, beta and decisions and no result depends on scheduling.
//   pcg_row_kernel   up to 2,048 rows per SM, one lane per row: all vectors in registers, the
//                    matrix in shared memory (24^3 grid FP32: 5.6 us an iteration against 12.7;
//                    67^3 FP64: 13.2 against 23.4)
//   pcg_loop_kernel  KEEP: larger, or with a row past kLoneRow, while the residual fits in shared
//                    memory beside the staged tiles (128^3 FP64: 67 us an iteration against 79: no z,
//                    r out of L2, x and p in one pass; DRAM traffic 212 MB an iteration against 308);
//                    otherwise systems of few lanes in any SpMV shape (360 rows of 360: 9.5 us
//                    against 14.5)
// Everything else runs the graph: with one CTA of at most 1,024 threads per SM the vector phases
// of larger systems, and the block preconditioner's, have too few loads in flight (150^3 FP64: 145
// us an iteration against 132; 24,000 rows of 474 in FP64: 55 against 44).
constexpr int kLoopThreads = kGridMaxThreads;      // most threads of a CTA (one CTA per SM)
constexpr int kRowThreads = 512;                   // most threads of a CTA with one row per thread
// Staged nonzeros per tile beside the kept residual: 32 rows of 7.25.  What a tile takes is lost to the residual:
// 23 entries a thread in FP64 (2.18M rows) with 232, 21 (1.99M) with 256.  Longer rows on average take a second
// load per tile and are still faster than as kernels (30 iterations, FP64: 600,000 rows of 7.3 1.36 -> 1.14 ms,
// of 7.9 1.42 -> 1.20; 1.5M of 7.9 2.84 -> 2.64).
constexpr int kKeepCap = 232;
constexpr int kTileThreads = 640;                  // of a CTA that stages tiles of the matrix

template <typename T>
struct PcgLoop
{
    int64_t n;
    int nnz;
    const int* rp;
    const int* ci;
    const T* v;
    const T* b;
    T* x;
    T* r[2];
    T* z;
    T* p[2];
    T* q;
    T* inv;
    int mode; // 0: CG, 1: Jacobi, 2: the caller's block inverses
    const T* blocks;
    int64_t bs;
    double relative, absolute;
    Packet* mail;             // [2][CTA][CTA][2]
    const unsigned long long* epoch; // barriers of earlier launches end below it
    PcgState* st;
};

// preconditioned component i of the residual vector `r` (scalar Jacobi, caller blocks, none)
template <typename T, typename R>
__device__ __forceinline__ double apply_precond(int mode, int64_t i, R&& residual_at, const T* inv_diag,
                                                const T* blocks, int64_t bs)
{
    if (mode == 1)
        return static_cast<double>(inv_diag[i]) * residual_at(i);
    if (mode == 2)
    {
        const int64_t blk = i / bs, local = i - blk * bs;
        const T* row = blocks + blk * bs * bs + local * bs;
        double z = 0.0;
        for (int64_t c = 0; c < bs; ++c)
            z += static_cast<double>(row[c]) * residual_at(blk * bs + c);
        return z;
    }
    return residual_at(i);
}

// Jacobi inverse of row r: iterative_solver_kernels.cuh:104-131 semantics (sum of diagonal
// duplicates, 16*eps*rowscale guard); invalid rows are reported (lowest row) instead of NaN markers.
template <typename T>
__device__ __forceinline__ void jacobi_row(int64_t r, const int* __restrict__ rp, const int* __restrict__ ci,
                                           const T* __restrict__ v, T* inv, PcgState* st)
{
    double diag = 0.0;
    T most = T(0);
    bool found = false;
    constexpr int G = 8; // loads in flight
    const int* c = ci + rp[r];
    const T* w = v + rp[r];
    for (int left = rp[r + 1] - rp[r]; left > 0; left -= G, c += G, w += G)
    {
        int col[G];
        T value[G];
#pragma unroll
        for (int k = 0; k < G; ++k)
            if (k < left)
            {
                col[k] = c[k];
                value[k] = w[k];
            }
#pragma unroll
        for (int k = 0; k < G; ++k)
            if (k < left)
            {
                most = fmax(most, fabs(value[k]));
                if (col[k] == r)
                {
                    diag += static_cast<double>(value[k]);
                    found = true;
                }
            }
    }
    const double threshold = Eps<T>::value * static_cast<double>(most) * 16.0;
    const double reciprocal = 1.0 / diag;
    if (!found || !isfinite(diag) || diag <= threshold || !isfinite(reciprocal))
    {
        atomicMin(&st->jacobi_bad_row, static_cast<long long>(r));
        inv[r] = T(0);
    }
    else
    {
        inv[r] = static_cast<T>(reciprocal);
    }
}

// alpha = rho / p.q (alphaKernel semantics, iterative_solver_kernels.cuh:169-202); the step must
// also be representable in the vector type (the reference forms alpha in Scalar precision and
// treats its overflow as breakdown); false on breakdown
template <typename T>
__device__ __forceinline__ bool pcg_alpha(double rho, double den, double& alpha)
{
    alpha = 0.0;
    if (rho == 0.0 && den == 0.0)
        return true;
    if (!(isfinite(rho) && isfinite(den) && rho > 0.0 && den > 0.0))
        return false;
    alpha = rho / den;
    return isfinite(alpha) && isfinite(static_cast<double>(static_cast<T>(alpha)));
}

// end of an iteration (total = {r.z, r.r}): true when the solve is over, otherwise beta and rho
// are the next direction's (betaKernel semantics, iterative_solver_kernels.cuh:204-238)
template <typename T>
__device__ __forceinline__ bool pcg_finish(const double (&total)[2], double tolerance, int iterations,
                                           int max_iterations, double& rho, double& beta, int& converged,
                                           int& breakdown)
{
    const double next = total[0], residual = total[1];
    if (!isfinite(residual) || residual < 0.0)
    {
        breakdown = 1;
        return true;
    }
    if (sqrt(residual) <= tolerance)
    {
        converged = 1;
        return true;
    }
    if (iterations >= max_iterations)
        return true;
    beta = 0.0;
    if (!(rho == 0.0 && next == 0.0))
    {
        if (!(isfinite(rho) && isfinite(next) && rho > 0.0 && next > 0.0))
        {
            breakdown = 1;
            return true;
        }
        beta = next / rho;
        if (!isfinite(beta) || !isfinite(static_cast<double>(static_cast<T>(beta))))
        {
            breakdown = 1;
            return true;
        }
    }
    rho = next;
    return false;
}

// every row of A x_at over the grid: done(row, sum) once per row
// SHAPE: 0 row-group stream, 1 staged tiles (values 16-byte aligned), -1 a thread per row read
// directly, otherwise lanes per row
template <typename T, int SHAPE, int CAP, typename Gather, typename Done>
__device__ __forceinline__ void for_rows(const PcgLoop<T>& a, unsigned char* smem, Gather&& x_at, Done&& done)
{
    const int64_t thread = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t threads = int64_t(gridDim.x) * blockDim.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if constexpr (SHAPE == 1)
    {
        csr_tiles<2>(reinterpret_cast<RowTile<T, CAP>*>(smem) + 2 * warp, a.n, a.nnz, a.rp, a.ci, a.v, thread >> 5,
                  threads >> 5, x_at, done);
    }
    else if constexpr (SHAPE == 0)
    {
        T* stage = reinterpret_cast<T*>(smem) + warp * kStreamCap;
        for (int64_t wrow = (thread >> 5) * 32; wrow < a.n; wrow += threads)
        {
            const T sum = csr_stream_rows<T>(wrow, a.n, a.rp, a.ci, a.v, x_at, stage);
            if (wrow + lane < a.n)
                done(wrow + lane, sum);
        }
    }
    else
    {
        constexpr int TPR = SHAPE < 0 ? 1 : SHAPE;
        const int64_t first = thread / TPR, stride = threads / TPR;
        const int64_t span = (a.n + stride - 1) / stride; // uniform trip count keeps shuffles convergent
        for (int64_t k = 0; k < span; ++k)
        {
            const int64_t row = first + k * stride;
            // 1,024 threads leave no registers for more loads: two gathers per nonzero of p (360
            // rows of 360, FP64: 430 us for 30 iterations, 753 with eight)
            constexpr int G = TPR == 1 ? 8 : 1;
            const T sum = csr_row_dot<T, TPR, G>(a.rp, a.ci, a.v, x_at, row, row < a.n, lane % TPR);
            if (row < a.n && lane % TPR == 0)
                done(row, sum);
        }
    }
}

// Most threads of a CTA.  With one lane per row 640: 102 registers a thread (64 spill in FP64, 20%
// slower) and 74-109 KB of tiles, which leave room for the kept residual.
template <typename T>
__host__ __device__ constexpr int loop_threads(int shape)
{
    return shape <= 1 ? kTileThreads : kLoopThreads;
}

// KEEP (one lane per row, modes 0 and 1): every CTA keeps its residual entries in shared memory and
// the direction p = z + beta p, with the step of x along the old p, is a phase of its own.
// Otherwise (FUSE) both happen inside the SpMV, every gathered entry of p formed from z and the old
// p, which saves a grid barrier per iteration.  The arithmetic of every element is the same.
template <typename T, int SHAPE, bool KEEP>
__global__ void __launch_bounds__(loop_threads<T>(SHAPE), 1) pcg_loop_kernel(const PcgLoop<T> a)
{
    extern __shared__ __align__(16) unsigned char loop_smem[];
    __shared__ GridShared shared;
    PcgState* const st = a.st;
    constexpr bool FUSE = !KEEP;
    GridSync sync{a.mail, &st->timed_out, &shared, *a.epoch};
    if (threadIdx.x == 0)
        shared.failed = 0; // read after the first barrier's __syncthreads
    // a row's lane owns its entries in the vector phases too (block rows read their neighbours' q)
    constexpr bool kOwnRows = SHAPE == 1 || SHAPE == -1 || SHAPE == 0;
    constexpr int CAP = KEEP ? kKeepCap : kTileCap;
    T* const kept = reinterpret_cast<T*>(loop_smem + (blockDim.x >> 5) * 2 * sizeof(RowTile<T, CAP>));
    const int64_t thread = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t threads = int64_t(gridDim.x) * blockDim.x;
    const bool writer = thread == 0;
    T* const x = a.x;
    // ---- r = b - A x, z = M^-1 r, rho = r.z, ||r||^2 (the first direction is z)
    if (a.mode == 1)
        for (int64_t i = thread; i < a.n; i += threads)
            jacobi_row<T>(i, a.rp, a.ci, a.v, a.inv, st);
    for_rows<T, SHAPE, CAP>(a, loop_smem, [&](int c) { return x[c]; }, [&](int64_t row, T sum) { a.q[row] = sum; });
    if (!grid_barrier(sync))
        return;
    double mine[2] = {0.0, 0.0}, total[2];
    {
        auto res = [&](int64_t k) {
            return static_cast<double>(
                static_cast<T>(static_cast<double>(a.b[k]) - static_cast<double>(a.q[k])));
        };
        for (int64_t i = thread; i < a.n; i += threads)
        {
            const double ri = res(i);
            const T zi = static_cast<T>(apply_precond<T>(a.mode, i, res, a.inv, a.blocks, a.bs));
            if (KEEP)
                kept[(i / threads) * blockDim.x + threadIdx.x] = static_cast<T>(ri);
            else
                a.r[0][i] = static_cast<T>(ri);
            a.z[i] = zi;
            a.p[0][i] = zi;
            mine[0] += ri * static_cast<double>(zi);
            mine[1] += ri * ri;
        }
    }
    if (!grid_sum<2>(sync, mine, total, true))
        return;
    double rho = total[0], residual = total[1], alpha = 0.0, beta = 0.0;
    const double initial = sqrt(residual);
    const double tolerance = fmax(a.absolute, a.relative * initial);
    const int max_iterations = st->max_iterations;
    int iterations = 0, converged = 0, breakdown = 0;
    bool done = max_iterations <= 0;
    if (writer)
        st->initial_squared = residual;
    if (!isfinite(residual) || residual < 0.0)
    {
        if (writer)
            st->nonfinite_init = 1;
        done = true;
    }
    else if (initial <= tolerance)
    {
        converged = 1;
        done = true;
    }
    if (__ldcg(&st->jacobi_bad_row) != kNone)
        done = true;
    // ---- iterations: p0 holds the direction (FUSE: the old one once z is newer), r_in the residual
    T *r_in = a.r[0], *r_out = a.r[1], *p0 = a.p[0], *p1 = a.p[1];
    while (!done)
    {
        // direction p = z + beta p, with the step x += alpha p of the iteration before
        if (!FUSE && iterations > 0)
        {
            // z is r or inv r: formed again instead of stored and read back
            const T* own = kept + threadIdx.x;
#pragma unroll 4
            for (int64_t i = thread; i < a.n; i += threads, own += blockDim.x)
            {
                const double pi = static_cast<double>(p0[i]);
                const double ri = static_cast<double>(*own);
                const double zi =
                    a.mode == 1 ? static_cast<double>(static_cast<T>(static_cast<double>(a.inv[i]) * ri)) : ri;
                x[i] = static_cast<T>(static_cast<double>(x[i]) + alpha * pi);
                p0[i] = static_cast<T>(zi + beta * pi);
            }
            if (!grid_barrier(sync))
                return;
        }
        // q = A p and p.q
        double pq[1] = {0.0}, pq_total[1];
        if (FUSE && iterations > 0)
        {
            const T* const z = a.z;
            for_rows<T, SHAPE, CAP>(
                a, loop_smem,
                [&](int c) { return static_cast<T>(static_cast<double>(z[c]) + beta * static_cast<double>(p0[c])); },
                [&](int64_t row, T sum) {
                    const double old = static_cast<double>(p0[row]);
                    const T pn = static_cast<T>(static_cast<double>(z[row]) + beta * old);
                    x[row] = static_cast<T>(static_cast<double>(x[row]) + alpha * old);
                    p1[row] = pn;
                    a.q[row] = sum;
                    pq[0] += static_cast<double>(pn) * static_cast<double>(sum);
                });
            T* const t = p0;
            p0 = p1;
            p1 = t;
        }
        else
        {
            for_rows<T, SHAPE, CAP>(a, loop_smem, [&](int c) { return p0[c]; }, [&](int64_t row, T sum) {
                a.q[row] = sum;
                pq[0] += static_cast<double>(p0[row]) * static_cast<double>(sum);
            });
        }
        if (!grid_sum<1>(sync, pq, pq_total, !kOwnRows || a.mode == 2))
            return;
        if (!pcg_alpha<T>(rho, pq_total[0], alpha))
        {
            breakdown = 1;
            break; // x keeps the last completed step
        }
        // r -= alpha q, z = M^-1 r, r.z, r.r (r is ping-ponged: block rows read the old values)
        mine[0] = mine[1] = 0.0;
        if (a.mode == 2)
        {
            auto res = [&](int64_t k) {
                return static_cast<double>(
                    static_cast<T>(static_cast<double>(r_in[k]) - alpha * static_cast<double>(a.q[k])));
            };
            for (int64_t i = thread; i < a.n; i += threads)
            {
                const double ri = res(i);
                const T zi = static_cast<T>(apply_precond<T>(a.mode, i, res, a.inv, a.blocks, a.bs));
                r_out[i] = static_cast<T>(ri);
                a.z[i] = zi;
                mine[0] += ri * static_cast<double>(zi);
                mine[1] += ri * ri;
            }
        }
        else
        {
            T* own = kept + threadIdx.x;
#pragma unroll 4
            for (int64_t i = thread; i < a.n; i += threads, own += blockDim.x)
            {
                const T rt = static_cast<T>(static_cast<double>(KEEP ? *own : r_in[i]) -
                                            alpha * static_cast<double>(a.q[i]));
                const double ri = static_cast<double>(rt);
                const T zi = a.mode == 1 ? static_cast<T>(static_cast<double>(a.inv[i]) * ri) : rt;
                if (KEEP)
                    *own = rt;
                else
                    r_out[i] = rt;
                if (FUSE)
                    a.z[i] = zi;
                mine[0] += ri * static_cast<double>(zi);
                mine[1] += ri * ri;
            }
        }
        if (!grid_sum<2>(sync, mine, total, true))
            return;
        T* const swap = r_in;
        r_in = r_out;
        r_out = swap;
        iterations += 1;
        residual = total[1];
        done = pcg_finish<T>(total, tolerance, iterations, max_iterations, rho, beta, converged, breakdown);
        if (done) // the step of the last iteration
            for (int64_t i = thread; i < a.n; i += threads)
                x[i] = static_cast<T>(static_cast<double>(x[i]) + alpha * static_cast<double>(p0[i]));
    }
    if (writer)
    {
        st->residual_squared = residual;
        st->iterations = iterations;
        st->converged = converged;
        st->breakdown = breakdown;
    }
}

// Small systems, R rows per thread, modes 0 and 1: the matrix stays in shared memory and every
// vector entry in its row's registers through all iterations; only z and p go through L2, for the
// gathers.  Two barriers per iteration, as with FUSE, and the same arithmetic.
template <typename T, int R>
__global__ void __launch_bounds__(kRowThreads, 1) pcg_row_kernel(const PcgLoop<T> a)
{
    extern __shared__ __align__(16) unsigned char loop_smem[];
    __shared__ GridShared shared;
    PcgState* const st = a.st;
    GridSync sync{a.mail, &st->timed_out, &shared, *a.epoch};
    if (threadIdx.x == 0)
        shared.failed = 0; // read after the first barrier's __syncthreads
    const int lane = threadIdx.x & 31;
    // the warp's 32 R consecutive rows, 32 apart in a lane
    const int64_t row0 = ((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * (32 * R) + lane;
    RowTile<T, kTileCap * R>& tile = reinterpret_cast<RowTile<T, kTileCap * R>*>(loop_smem)[threadIdx.x >> 5];
    int b[R], e[R];
    T x[R], inv[R], r[R], z[R], p[R], q[R];
#pragma unroll
    for (int j = 0; j < R; ++j)
    {
        const int64_t row = row0 + 32 * j;
        b[j] = row < a.n ? a.rp[row] : a.nnz;
        e[j] = row < a.n ? a.rp[row + 1] : a.nnz;
    }
    const int first = __shfl_sync(0xffffffffu, b[0], 0), end = __shfl_sync(0xffffffffu, e[R - 1], 31);
    const bool staged = end - first <= kTileCap * R; // otherwise the rows are read directly
    if (staged)
    {
        for (int k = lane; k < end - first; k += 32)
        {
            tile.col[k] = a.ci[first + k];
            tile.val[k] = a.v[first + k];
        }
#pragma unroll
        for (int j = 0; j < R; ++j)
        {
            b[j] -= first;
            e[j] -= first;
        }
    }
    __syncwarp();
    auto row_sums = [&](auto&& x_at) {
#pragma unroll
        for (int j = 0; j < R; ++j)
        {
            q[j] = T(0);
            if (staged)
                q[j] = tile_sum<8>(tile, b[j], e[j], T(0), x_at);
            else
                for (int k = b[j]; k < e[j]; ++k)
                    q[j] += a.v[k] * x_at(a.ci[k]);
        }
    };
    T* const z_all = a.z;
    T *p_old = a.p[0], *p_new = a.p[1];
    double mine[2] = {0.0, 0.0}, total[2];
    row_sums([&](int c) { return a.x[c]; });
#pragma unroll
    for (int j = 0; j < R; ++j)
    {
        const int64_t row = row0 + 32 * j;
        x[j] = r[j] = z[j] = p[j] = T(0);
        inv[j] = T(1);
        if (row < a.n)
        {
            if (a.mode == 1)
            {
                jacobi_row<T>(row, a.rp, a.ci, a.v, a.inv, st);
                inv[j] = a.inv[row];
            }
            x[j] = a.x[row];
            r[j] = static_cast<T>(static_cast<double>(a.b[row]) - static_cast<double>(q[j]));
            const double ri = static_cast<double>(r[j]);
            p[j] = z[j] = a.mode == 1 ? static_cast<T>(static_cast<double>(inv[j]) * ri) : r[j];
            p_old[row] = z[j];
            mine[0] += ri * static_cast<double>(z[j]);
            mine[1] += ri * ri;
        }
    }
    if (!grid_sum<2>(sync, mine, total, true))
        return;
    double rho = total[0], residual = total[1], beta = 0.0;
    const double initial = sqrt(residual);
    const double tolerance = fmax(a.absolute, a.relative * initial);
    const int max_iterations = st->max_iterations;
    int iterations = 0, converged = 0, breakdown = 0;
    bool done = max_iterations <= 0;
    const bool writer = blockIdx.x == 0 && threadIdx.x == 0;
    if (writer)
        st->initial_squared = residual;
    if (!isfinite(residual) || residual < 0.0)
    {
        if (writer)
            st->nonfinite_init = 1;
        done = true;
    }
    else if (initial <= tolerance)
    {
        converged = 1;
        done = true;
    }
    if (__ldcg(&st->jacobi_bad_row) != kNone)
        done = true;
    while (!done)
    {
        if (iterations == 0)
        {
            row_sums([&](int c) { return p_old[c]; });
        }
        else
        {
            row_sums([&](int c) {
                return static_cast<T>(static_cast<double>(z_all[c]) + beta * static_cast<double>(p_old[c]));
            });
#pragma unroll
            for (int j = 0; j < R; ++j)
            {
                p[j] = static_cast<T>(static_cast<double>(z[j]) + beta * static_cast<double>(p[j]));
                if (row0 + 32 * j < a.n)
                    p_new[row0 + 32 * j] = p[j];
            }
            T* const t = p_old;
            p_old = p_new;
            p_new = t;
        }
        double pq[1] = {0.0}, pq_total[1];
#pragma unroll
        for (int j = 0; j < R; ++j) // rows past the end hold zeros
            pq[0] += static_cast<double>(p[j]) * static_cast<double>(q[j]);
        if (!grid_sum<1>(sync, pq, pq_total, false))
            return;
        double alpha;
        if (!pcg_alpha<T>(rho, pq_total[0], alpha))
        {
            breakdown = 1;
            break;
        }
        mine[0] = mine[1] = 0.0;
#pragma unroll
        for (int j = 0; j < R; ++j)
        {
            r[j] = static_cast<T>(static_cast<double>(r[j]) - alpha * static_cast<double>(q[j]));
            const double ri = static_cast<double>(r[j]);
            z[j] = a.mode == 1 ? static_cast<T>(static_cast<double>(inv[j]) * ri) : r[j];
            x[j] = static_cast<T>(static_cast<double>(x[j]) + alpha * static_cast<double>(p[j]));
            if (row0 + 32 * j < a.n)
                z_all[row0 + 32 * j] = z[j];
            mine[0] += ri * static_cast<double>(z[j]);
            mine[1] += ri * ri;
        }
        if (!grid_sum<2>(sync, mine, total, true))
            return;
        iterations += 1;
        residual = total[1];
        done = pcg_finish<T>(total, tolerance, iterations, max_iterations, rho, beta, converged, breakdown);
    }
    if (iterations > 0)
    {
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (row0 + 32 * j < a.n)
                a.x[row0 + 32 * j] = x[j];
    }
    if (writer)
    {
        st->residual_squared = residual;
        st->iterations = iterations;
        st->converged = converged;
        st->breakdown = breakdown;
    }
}

// ------------------------------------------------------------------ PCG as a graph of kernels
// Last block to arrive sums the per-block partials (fixed order) and runs `finish`.
template <int K, typename Finish>
__device__ __forceinline__ void reduce_partials(double (&mine)[K], double* partials, unsigned int* ticket,
                                                Finish&& finish)
{
    __shared__ double smem[kReduceBlock / 32];
    __shared__ bool last;
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        const double s = block_sum<double, kReduceBlock>(mine[k], smem);
        if (threadIdx.x == 0)
            partials[k * kMaxReduceBlocks + blockIdx.x] = s;
    }
    __threadfence();
    if (threadIdx.x == 0)
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last)
        return;
    __threadfence();
    double totals[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        double s = 0.0;
        for (int b = threadIdx.x; b < gridDim.x; b += blockDim.x)
            s += __ldcg(partials + k * kMaxReduceBlocks + b);
        totals[k] = block_sum<double, kReduceBlock>(s, smem);
    }
    if (threadIdx.x == 0)
    {
        *ticket = 0;
        finish(totals);
    }
}

template <typename T>
__global__ void jacobi_kernel(int64_t rows, const int* __restrict__ rp, const int* __restrict__ ci,
                              const T* __restrict__ v, T* __restrict__ inv, PcgState* st)
{
    for (int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; r < rows; r += int64_t(gridDim.x) * blockDim.x)
        jacobi_row<T>(r, rp, ci, v, inv, st);
}

// r = b - Ax (Ax in q), z = M^-1 r, p = z; rho = r.z, initial ||r||^2
template <typename T>
__global__ void __launch_bounds__(kReduceBlock) pcg_init_kernel(int64_t n, const T* __restrict__ b,
                                                                const T* __restrict__ q, T* __restrict__ r,
                                                                T* __restrict__ z, T* __restrict__ p, int mode,
                                                                const T* __restrict__ inv, const T* __restrict__ blocks,
                                                                int64_t bs, double relative, double absolute,
                                                                double* partials, PcgState* st)
{
    double mine[2] = {0.0, 0.0};
    auto res = [&](int64_t k) { return static_cast<double>(static_cast<T>(static_cast<double>(b[k]) - static_cast<double>(q[k]))); };
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    {
        const double ri = res(i);
        const T zi = static_cast<T>(apply_precond<T>(mode, i, res, inv, blocks, bs));
        r[i] = static_cast<T>(ri);
        z[i] = zi;
        p[i] = zi;
        mine[0] += ri * static_cast<double>(zi);
        mine[1] += ri * ri;
    }
    reduce_partials<2>(mine, partials, &st->ticket[0], [&](double (&tot)[2]) {
        st->rho = tot[0];
        st->initial_squared = tot[1];
        st->residual_squared = tot[1];
        const double initial = sqrt(tot[1]);
        st->tolerance = fmax(absolute, relative * initial);
        st->iterations = 0;
        st->beta = 0.0;
        if (!isfinite(tot[1]) || tot[1] < 0.0)
        {
            st->nonfinite_init = 1;
            st->done = 1;
        }
        else if (initial <= st->tolerance)
        {
            st->converged = 1;
            st->done = 1;
        }
        if (st->jacobi_bad_row != kNone)
            st->done = 1;
    });
}

// alpha = rho / p.q on the last block
template <typename T>
__device__ __forceinline__ void pcg_step(PcgState* st, double den, T)
{
    double alpha;
    if (!pcg_alpha<T>(st->rho, den, alpha))
    {
        st->breakdown = 1;
        st->done = 1;
        alpha = 0.0;
    }
    st->alpha = alpha;
}

// q = A p, alpha = rho / p.q
template <typename T, int TPR, int G>
__global__ void __launch_bounds__(kReduceBlock) pcg_spmv_kernel(int64_t rows, const int* __restrict__ rp,
                                                                const int* __restrict__ ci, const T* __restrict__ v,
                                                                const T* __restrict__ p, T* __restrict__ q,
                                                                double* partials, PcgState* st)
{
    if (st->done)
        return;
    double mine[1] = {0.0};
    const int64_t stride = int64_t(gridDim.x) * blockDim.x / TPR;
    const int lane = threadIdx.x % TPR;
    const int64_t first = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) / TPR;
    const int64_t span = (rows + stride - 1) / stride;
    for (int64_t k = 0; k < span; ++k)
    {
        const int64_t row = first + k * stride;
        const bool valid = row < rows;
        const T sum = csr_row_dot<T, TPR, G>(rp, ci, v, [&](int c) { return __ldg(p + c); }, row, valid, lane);
        if (valid && lane == 0)
        {
            q[row] = sum;
            mine[0] += static_cast<double>(p[row]) * static_cast<double>(sum);
        }
    }
    reduce_partials<1>(mine, partials, &st->ticket[1], [&](double (&tot)[1]) { pcg_step(st, tot[0], T(0)); });
}

// q = A p with the short-row stream layout, alpha = rho / p.q
template <typename T>
__global__ void __launch_bounds__(kReduceBlock) pcg_stream_spmv_kernel(int64_t rows, const int* __restrict__ rp,
                                                                       const int* __restrict__ ci,
                                                                       const T* __restrict__ v,
                                                                       const T* __restrict__ p, T* __restrict__ q,
                                                                       double* partials, PcgState* st)
{
    if (st->done)
        return;
    __shared__ T stage[kReduceBlock / 32][kStreamCap];
    double mine[1] = {0.0};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t warps = int64_t(gridDim.x) * (kReduceBlock / 32);
    for (int64_t wrow = (int64_t(blockIdx.x) * (kReduceBlock / 32) + warp) * 32; wrow < rows; wrow += warps * 32)
    {
        const T sum = csr_stream_rows<T>(wrow, rows, rp, ci, v, [&](int c) { return __ldg(p + c); }, stage[warp]);
        const int64_t row = wrow + lane;
        if (row < rows)
        {
            q[row] = sum;
            mine[0] += static_cast<double>(p[row]) * static_cast<double>(sum);
        }
    }
    reduce_partials<1>(mine, partials, &st->ticket[1], [&](double (&tot)[1]) { pcg_step(st, tot[0], T(0)); });
}

// q = A p from staged tiles, alpha = rho / p.q
template <typename T>
__global__ void __launch_bounds__(kReduceBlock, 4) pcg_tile_spmv_kernel(int64_t rows, int nnz,
                                                                        const int* __restrict__ rp,
                                                                        const int* __restrict__ ci,
                                                                        const T* __restrict__ v,
                                                                        const T* __restrict__ p, T* __restrict__ q,
                                                                        double* partials, PcgState* st)
{
    if (st->done)
        return;
    extern __shared__ __align__(16) unsigned char tile_smem[];
    double mine[1] = {0.0};
    csr_tiles<1>(reinterpret_cast<RowTile<T, kSpmvCap>*>(tile_smem) + (threadIdx.x >> 5), rows, nnz, rp, ci, v,
              (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5, int64_t(gridDim.x) * (blockDim.x >> 5),
              [&](int c) { return __ldg(p + c); }, [&](int64_t row, T sum) {
                  q[row] = sum;
                  mine[0] += static_cast<double>(p[row]) * static_cast<double>(sum);
              });
    reduce_partials<1>(mine, partials, &st->ticket[1], [&](double (&tot)[1]) { pcg_step(st, tot[0], T(0)); });
}

// x += alpha p, r -= alpha q, z = M^-1 r; convergence on ||r||, beta = r.z / rho.
// r is ping-ponged (r_in -> r_out) so block preconditioners read only old values.
template <typename T>
__global__ void __launch_bounds__(kReduceBlock) pcg_update_kernel(int64_t n, T* __restrict__ x,
                                                                  const T* __restrict__ p, const T* __restrict__ q,
                                                                  const T* __restrict__ r_in, T* __restrict__ r_out,
                                                                  T* __restrict__ z, int mode,
                                                                  const T* __restrict__ inv,
                                                                  const T* __restrict__ blocks, int64_t bs,
                                                                  double* partials, PcgState* st)
{
    if (st->done)
        return;
    const double alpha = st->alpha;
    double mine[2] = {0.0, 0.0};
    auto res = [&](int64_t k) {
        return static_cast<double>(static_cast<T>(static_cast<double>(r_in[k]) - alpha * static_cast<double>(q[k])));
    };
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    {
        x[i] = static_cast<T>(static_cast<double>(x[i]) + alpha * static_cast<double>(p[i]));
        const double ri = res(i);
        const T zi = static_cast<T>(apply_precond<T>(mode, i, res, inv, blocks, bs));
        r_out[i] = static_cast<T>(ri);
        z[i] = zi;
        mine[0] += ri * static_cast<double>(zi);
        mine[1] += ri * ri;
    }
    reduce_partials<2>(mine, partials, &st->ticket[2], [&](double (&tot)[2]) {
        st->iterations += 1;
        st->residual_squared = tot[1];
        double rho = st->rho, beta = st->beta;
        int converged = 0, breakdown = 0;
        st->done = pcg_finish<T>(tot, st->tolerance, st->iterations, st->max_iterations, rho, beta, converged,
                                 breakdown);
        st->rho = rho;
        st->beta = beta;
        st->converged = converged;
        st->breakdown = breakdown;
    });
}

template <typename T>
__global__ void pcg_direction_kernel(int64_t n, const T* __restrict__ z, T* __restrict__ p, const PcgState* st)
{
    if (st->done || st->iterations == 0) // the first iteration's direction is z itself (set by the init)
        return;
    const double beta = st->beta;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        p[i] = static_cast<T>(static_cast<double>(z[i]) + beta * static_cast<double>(p[i]));
}

// Condition of the CG / PCG iteration graph: another chunk while the solve is not done, at most
// max_iterations / kCgChunk + 1 chunks (the update kernel also ends the solve at max_iterations).
constexpr int kCgChunk = 4; // iterations per graph body (even: the residual ping-pong returns to r0)
__global__ void cg_continue_kernel(cudaGraphConditionalHandle handle, PcgState* st)
{
    if (threadIdx.x == 0 && blockIdx.x == 0)
    {
        const int chunks = st->chunks + 1;
        st->chunks = chunks;
        cudaGraphSetConditional(handle, !st->done && chunks <= st->max_iterations / kCgChunk + 1 ? 1u : 0u);
    }
}

__global__ void pcg_reset_kernel(PcgState* st, int max_iterations, unsigned long long* epoch)
{
    grid_next_launch(epoch);
    PcgState s{};
    s.max_iterations = max_iterations;
    s.jacobi_bad_row = kNone;
    *st = s;
}

// initial and final recurrence residuals of a fixed-iteration solve; NaN marks a breakdown
__global__ void fixed_finish_kernel(const PcgState* st, double* out)
{
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    const bool bad = st->breakdown || st->nonfinite_init || st->timed_out || st->jacobi_bad_row != kNone;
    out[0] = st->nonfinite_init ? nan : st->initial_squared;
    out[1] = bad ? nan : st->residual_squared;
}

} // namespace
} // namespace pm

struct pm_fixed_state
{
    double* residuals = nullptr; // device: initial, final squared residual
    cudaEvent_t event = nullptr;
    cudaStream_t stream = nullptr;
    int submitted = 0;
    ~pm_fixed_state()
    {
        if (event)
            cudaEventDestroy(event);
        if (residuals)
            cudaFree(residuals);
    }
};

struct pm_solver_workspace
{
    pm::DeviceBuffer buffer;
    pm::GridMail mail;
    void* host_state = nullptr; // pinned
    cudaEvent_t event = nullptr;
    // CG / PCG iteration graphs ('while' node around a chunk of iterations), one per operand set
    struct IterationGraph
    {
        uint64_t operand = 0; // its serial: an address may be another operand's by now
        const void* key[4] = {};
        int64_t n = -1;
        int shape = 0, mode = -1, value_size = 0;
        int64_t block_size = 0;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
    };
    IterationGraph graphs[4];
    int graph_next = 0;
    cudaStream_t capture_stream = nullptr;
    void drop_graphs()
    {
        for (auto& g : graphs)
        {
            if (g.exec)
                cudaGraphExecDestroy(g.exec);
            if (g.graph)
                cudaGraphDestroy(g.graph);
            g = IterationGraph{};
        }
    }
    ~pm_solver_workspace()
    {
        drop_graphs();
        if (capture_stream)
            cudaStreamDestroy(capture_stream);
        buffer.release();
        mail.buffer.release();
        if (host_state)
            cudaFreeHost(host_state);
        if (event)
            cudaEventDestroy(event);
    }
};

namespace pm
{
namespace
{

std::atomic<uint64_t> operand_count{0};

template <typename T>
void csr_create(cudaStream_t stream, int64_t rows, int64_t cols, int64_t nnz, const int64_t* ro, const int64_t* ci,
                const T* v, pm_csr** out)
{
    if (!out)
        fail(PM_INVALID_ARGUMENT, "CSR output handle pointer is null");
    if (rows < 0 || cols < 0 || nnz < 0)
        fail(PM_INVALID_ARGUMENT, "CSRMatrix dimensions must be non-negative");
    if (nnz > INT32_MAX - 1 || rows > INT32_MAX - 1 || cols > INT32_MAX)
        fail(PM_OVERFLOW_ERROR, "CSR operand exceeds the int32 index range of the device kernels");
    if (!ro || (nnz > 0 && (!ci || !v)))
        fail(PM_INVALID_ARGUMENT, "CSR arrays must be non-null");
    auto* A = new pm_csr();
    try
    {
        A->value_size = sizeof(T);
        A->rows = rows;
        A->cols = cols;
        A->nnz = nnz;
        A->values = v;
        A->threads_per_row = pick_tpr(rows, nnz);
        A->serial = ++operand_count;
        PM_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&A->row_ptr), (rows + 1) * sizeof(int), stream));
        PM_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&A->col_idx), (nnz > 0 ? nnz : 1) * sizeof(int), stream));
        CsrCheck* check = nullptr;
        PM_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&check), sizeof(CsrCheck), stream));
        CsrCheck init{kNone, kNone, kNone, 0, 0};
        PM_CUDA(cudaMemcpyAsync(check, &init, sizeof(init), cudaMemcpyHostToDevice, stream));
        validate_csr_kernel<T><<<grid_for(std::max(rows, nnz), 256, 4096), 256, 0, stream>>>(
            rows, cols, nnz, ro, ci, v, A->row_ptr, A->col_idx, check);
        PM_LAUNCH_CHECK();
        CsrCheck result{};
        PM_CUDA(cudaMemcpyAsync(&result, check, sizeof(result), cudaMemcpyDeviceToHost, stream));
        PM_CUDA(cudaFreeAsync(check, stream));
        PM_CUDA(cudaStreamSynchronize(stream));
        if (result.endpoints_bad)
            fail(PM_INVALID_ARGUMENT, "CSRMatrix row offsets must start at zero and end at nnz");
        if (result.bad_offsets_row != kNone)
        {
            std::ostringstream m;
            m << "CSRMatrix invalid row offsets at row " << result.bad_offsets_row;
            fail(PM_INVALID_ARGUMENT, m.str());
        }
        if (result.bad_column != kNone)
        {
            std::ostringstream m;
            m << "CSRMatrix column index out of range at position " << result.bad_column;
            fail(PM_INVALID_ARGUMENT, m.str());
        }
        if (result.bad_value != kNone)
        {
            std::ostringstream m;
            m << "CSRMatrix value is not finite at position " << result.bad_value;
            fail(PM_INVALID_ARGUMENT, m.str());
        }
        A->longest_row = result.longest;
    }
    catch (...)
    {
        cudaStreamSynchronize(stream);
        cudaFree(A->row_ptr);
        cudaFree(A->col_idx);
        delete A;
        throw;
    }
    *out = A;
}

template <typename T>
void csr_spmv(const pm_csr* A, cudaStream_t stream, const T* x, T* y)
{
    if (!A)
        fail(PM_INVALID_ARGUMENT, "CSR handle is null");
    if (A->value_size != static_cast<int>(sizeof(T)))
        fail(PM_INVALID_ARGUMENT, "spmv scalar type differs from the CSR operand");
    if (A->rows > 0 && (!y || (A->cols > 0 && !x)))
        fail(PM_INVALID_ARGUMENT, "spmv vectors must be non-null");
    if (x && x == y)
        fail(PM_INVALID_ARGUMENT, "spmv input and output data must not alias");
    A->queued_on(stream);
    launch_spmv<T>(A, x, y, stream);
}

// ------------------------------------------------------------------ SpMV autotuning
// Times every SpMV shape (row-group stream; 1, 2, 4, 8, 16, 32 lanes per row) on the operand with
// the caller's vectors and stream (one warm-up, then `reps` launches each, CUDA events) and keeps
// the fastest in the handle; the CG / PCG solvers use the same shape.  Shapes differ in the order
// of a row's additions, so the choice is part of a result's rounding; pm_csr_set_kernel pins one.
template <typename T>
int csr_autotune(pm_csr* A, cudaStream_t stream, const T* x, T* y, int reps)
{
    if (!A)
        fail(PM_INVALID_ARGUMENT, "CSR handle is null");
    if (A->value_size != static_cast<int>(sizeof(T)))
        fail(PM_INVALID_ARGUMENT, "autotune scalar type differs from the CSR operand");
    if (A->rows > 0 && (!y || (A->cols > 0 && !x)))
        fail(PM_INVALID_ARGUMENT, "autotune vectors must be non-null");
    if (x && x == y)
        fail(PM_INVALID_ARGUMENT, "spmv input and output data must not alias");
    if (A->rows == 0 || A->nnz == 0)
        return A->kernel;
    const int candidates[] = {0, 1, 2, 4, 8, 16, 32};
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    PM_CUDA(cudaEventCreate(&e0));
    PM_CUDA(cudaEventCreate(&e1));
    int best = A->kernel;
    float best_ms = 0.f;
    try
    {
        for (const int c : candidates)
        {
            A->kernel = c;
            launch_spmv<T>(A, x, y, stream);
            PM_CUDA(cudaEventRecord(e0, stream));
            for (int r = 0; r < reps; ++r)
                launch_spmv<T>(A, x, y, stream);
            PM_CUDA(cudaEventRecord(e1, stream));
            PM_CUDA(cudaEventSynchronize(e1));
            float ms = 0.f;
            PM_CUDA(cudaEventElapsedTime(&ms, e0, e1));
            if (c == candidates[0] || ms < best_ms)
            {
                best = c;
                best_ms = ms;
            }
        }
    }
    catch (...)
    {
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        throw;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    A->kernel = best;
    return best;
}

// ------------------------------------------------------------------ SpMM
// output (rows x k) = A input (cols x k), dense matrices column-major (leading dimension = rows).
// A warp owns 32 consecutive rows; their nonzero range is staged in shared memory in pieces of
// kStreamCap (columns, values, coalesced) and lane i forms row i of up to kSpmmCols output
// columns at a time, each sum from zero in storage order with one rounded multiply and one
// rounded add per term (the reference CPU spmm, sparse_ops_cpu.cpp:244-270).
constexpr int kSpmmCols = 8;

template <typename T>
__device__ __forceinline__ T mul_round(T a, T b)
{
    if constexpr (sizeof(T) == 8)
        return __dmul_rn(a, b);
    else
        return __fmul_rn(a, b);
}
template <typename T>
__device__ __forceinline__ T add_round(T a, T b)
{
    if constexpr (sizeof(T) == 8)
        return __dadd_rn(a, b);
    else
        return __fadd_rn(a, b);
}

template <typename T>
__global__ void __launch_bounds__(256) csr_spmm_kernel(int64_t rows, int64_t cols, int64_t k,
                                                       const int* __restrict__ rp, const int* __restrict__ ci,
                                                       const T* __restrict__ v, const T* __restrict__ in,
                                                       T* __restrict__ out)
{
    __shared__ int scol[8][kStreamCap];
    __shared__ T sval[8][kStreamCap];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t warps = int64_t(gridDim.x) * 8;
    for (int64_t wrow = (int64_t(blockIdx.x) * 8 + warp) * 32; wrow < rows; wrow += warps * 32)
    {
        const int64_t row = wrow + lane;
        const bool valid = row < rows;
        const int my_begin = valid ? rp[row] : 0;
        const int my_end = valid ? rp[row + 1] : 0;
        const int last = static_cast<int>(rows - 1 - wrow < 31 ? rows - 1 - wrow : 31);
        const int cb = __shfl_sync(0xffffffffu, my_begin, 0);
        const int ce = __shfl_sync(0xffffffffu, my_end, last);
        for (int64_t j0 = 0; j0 < k; j0 += kSpmmCols)
        {
            const int nj = k - j0 < kSpmmCols ? static_cast<int>(k - j0) : kSpmmCols;
            T sum[kSpmmCols];
#pragma unroll
            for (int j = 0; j < kSpmmCols; ++j)
                sum[j] = T(0);
            for (int base = cb; base < ce; base += kStreamCap)
            {
                const int n = ce - base < kStreamCap ? ce - base : kStreamCap;
                for (int e = lane; e < n; e += 32)
                {
                    scol[warp][e] = __ldg(ci + base + e);
                    sval[warp][e] = __ldg(v + base + e);
                }
                __syncwarp();
                const int lo = my_begin > base ? my_begin : base;
                const int hi = my_end < base + n ? my_end : base + n;
                for (int e = lo; e < hi; ++e)
                {
                    const T a = sval[warp][e - base];
                    const T* b = in + scol[warp][e - base];
#pragma unroll
                    for (int j = 0; j < kSpmmCols; ++j)
                        if (j < nj)
                            sum[j] = add_round(sum[j], mul_round(a, __ldg(b + (j0 + j) * cols)));
                }
                __syncwarp();
            }
            if (valid)
            {
#pragma unroll
                for (int j = 0; j < kSpmmCols; ++j)
                    if (j < nj)
                        out[(j0 + j) * rows + row] = sum[j];
            }
        }
    }
}

template <typename T>
void csr_spmm(const pm_csr* A, cudaStream_t stream, int64_t in_rows, int64_t in_cols, const T* in, int64_t out_rows,
              int64_t out_cols, T* out)
{
    if (!A)
        fail(PM_INVALID_ARGUMENT, "CSR handle is null");
    if (A->value_size != static_cast<int>(sizeof(T)))
        fail(PM_INVALID_ARGUMENT, "spmm scalar type differs from the CSR operand");
    if (in_rows < 0 || in_cols < 0 || out_rows < 0 || out_cols < 0)
        fail(PM_INVALID_ARGUMENT, "spmm dimensions must be non-negative");
    if (in_rows != A->cols)
    {
        std::ostringstream m;
        m << "spmm GPU dimension mismatch: CSR is " << A->rows << "x" << A->cols << ", input is " << in_rows << "x"
          << in_cols;
        fail(PM_RUNTIME_ERROR, m.str());
    }
    if (out_rows != A->rows || out_cols != in_cols)
    {
        std::ostringstream m;
        m << "spmm GPU output dimension mismatch: output is " << out_rows << "x" << out_cols << ", expected "
          << A->rows << "x" << in_cols;
        fail(PM_RUNTIME_ERROR, m.str());
    }
    if (in && in == out)
        fail(PM_INVALID_ARGUMENT, "spmm GPU input and output data must not alias");
    if (out_rows * out_cols == 0)
        return;
    if (!out || (A->nnz > 0 && !in))
        fail(PM_INVALID_ARGUMENT, "spmm matrices must be non-null");
    if (A->nnz == 0)
    {
        PM_CUDA(cudaMemsetAsync(out, 0, size_t(out_rows * out_cols) * sizeof(T), stream));
        return;
    }
    A->queued_on(stream);
    csr_spmm_kernel<T><<<grid_for(A->rows, 256, 1 << 20), 256, 0, stream>>>(A->rows, A->cols, in_cols, A->row_ptr,
                                                                             A->col_idx, static_cast<const T*>(A->values),
                                                                             in, out);
    PM_LAUNCH_CHECK();
}

// the workspace's arrays for a system of n rows
template <typename T>
struct PcgVectors
{
    PcgState* st;
    double* partials;
    T *r[2], *z, *p[2], *q, *inv;
    size_t bytes;
    PcgVectors(const pm_solver_workspace* ws, int64_t n)
    {
        Carver c;
        c.base = static_cast<char*>(ws->buffer.ptr);
        st = c.take<PcgState>(1);
        partials = c.take<double>(3 * kMaxReduceBlocks);
        for (T** v : {&r[0], &r[1], &z, &p[0], &q, &inv})
            *v = c.take<T>(n);
        // only the launches that form p inside the SpMV keep the old one beside it: one row per thread or group
        // of lanes, or four with rows in registers
        p[1] = n <= int64_t(4) * kRowThreads * kGridMaxCtas ? c.take<T>(n) : nullptr;
        bytes = c.offset;
    }
};

template <typename T>
void launch_pcg_spmv(const pm_csr* A, const T* p, T* q, double* partials, PcgState* st, unsigned grid,
                     cudaStream_t stream)
{
    const T* v = static_cast<const T*>(A->values);
    if (use_stream(A))
    {
        pcg_stream_spmv_kernel<T><<<grid, kReduceBlock, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, p, q,
                                                                     partials, st);
        PM_LAUNCH_CHECK();
        return;
    }
    // FP32 only: in FP64 a grid's rows are read faster directly (150^3, 30 iterations: 3.87 ms from tiles
    // against 3.74; FP32 2.60 against 2.93; 600,000 rows of 7.9, blocks of six: FP32 1.19 against 1.30)
    if (sizeof(T) == 4 && use_tiles<T>(A))
    {
        const size_t smem = size_t(kReduceBlock / 32) * sizeof(RowTile<T, kSpmvCap>);
        allow_smem(reinterpret_cast<const void*>(pcg_tile_spmv_kernel<T>), smem);
        pcg_tile_spmv_kernel<T><<<std::min<unsigned>(grid, 4 * sm_count()), kReduceBlock, smem, stream>>>(
            A->rows, static_cast<int>(A->nnz), A->row_ptr, A->col_idx, v, p, q, partials, st);
        PM_LAUNCH_CHECK();
        return;
    }
    switch (lanes_per_row(A))
    {
    case 1: pcg_spmv_kernel<T, 1, 8><<<grid, kReduceBlock, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, p, q, partials, st); break;
    case 2: pcg_spmv_kernel<T, 2, 0><<<grid, kReduceBlock, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, p, q, partials, st); break;
    case 4: pcg_spmv_kernel<T, 4, 0><<<grid, kReduceBlock, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, p, q, partials, st); break;
    case 8: pcg_spmv_kernel<T, 8, 0><<<grid, kReduceBlock, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, p, q, partials, st); break;
    case 16: pcg_spmv_kernel<T, 16, 0><<<grid, kReduceBlock, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, p, q, partials, st); break;
    default:
        if (long_rows(A))
            pcg_spmv_kernel<T, 32, 8><<<grid, kReduceBlock, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, p, q,
                                                                          partials, st);
        else
            pcg_spmv_kernel<T, 32, 0><<<grid, kReduceBlock, 0, stream>>>(A->rows, A->row_ptr, A->col_idx, v, p, q,
                                                                          partials, st);
        break;
    }
    PM_LAUNCH_CHECK();
}

// The iteration graph of one operand set (matrix and its SpMV shape, solution, preconditioner and
// the workspace's buffer), built on first use and kept in the workspace: a CUDA graph 'while' node
// whose body is kCgChunk iterations (direction, SpMV with p.q, update with the dots) and
// cg_continue_kernel, so the device decides when the solve is done.
template <typename T>
cudaGraphExec_t cg_iteration_graph(pm_solver_workspace* ws, const pm_csr* A, T* x, const T* blocks, int64_t bs,
                                   int mode)
{
    const int64_t n = A->rows;
    const int shape = use_stream(A) ? 0 : lanes_per_row(A);
    const void* key[4] = {A->values, x, blocks, ws->buffer.ptr};
    for (auto& g : ws->graphs)
        if (g.exec && g.operand == A->serial && g.n == n && g.shape == shape && g.mode == mode &&
            g.block_size == bs && g.value_size == int(sizeof(T)) && std::equal(key, key + 4, g.key))
            return g.exec;
    if (!ws->capture_stream)
        PM_CUDA(cudaStreamCreateWithFlags(&ws->capture_stream, cudaStreamNonBlocking));
    auto& slot = ws->graphs[ws->graph_next];
    ws->graph_next = (ws->graph_next + 1) % 4;
    if (slot.exec)
        cudaGraphExecDestroy(slot.exec);
    if (slot.graph)
        cudaGraphDestroy(slot.graph);
    slot = pm_solver_workspace::IterationGraph{};
    const PcgVectors<T> u(ws, n);
    PcgState* const st = u.st;
    double* const partials = u.partials;
    T *const r0 = u.r[0], *const r1 = u.r[1], *const z = u.z, *const p = u.p[0], *const q = u.q, *const inv = u.inv;
    const unsigned vgrid = grid_for(n, kReduceBlock, kMaxReduceBlocks);
    const unsigned sgrid = use_stream(A) ? grid_for(n, kReduceBlock, kMaxReduceBlocks)
                                         : grid_for(n * lanes_per_row(A), kReduceBlock, kMaxReduceBlocks);
    cudaGraph_t graph = nullptr;
    PM_CUDA(cudaGraphCreate(&graph, 0));
    cudaGraphConditionalHandle handle = 0;
    cudaGraph_t body = nullptr;
    {
        const cudaError_t made = cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault);
        cudaGraphNodeParams cp{};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = handle;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        cudaGraphNode_t node = nullptr;
        const cudaError_t added = made == cudaSuccess ? cudaGraphAddNode(&node, graph, nullptr, 0, &cp) : made;
        if (added != cudaSuccess)
        {
            cudaGraphDestroy(graph);
            fail(PM_CUDA_ERROR, std::string("CUDA iterative solver: conditional graph node: ") +
                                    cudaGetErrorString(added));
        }
        body = cp.conditional.phGraph_out[0];
    }
    const cudaStream_t cs = ws->capture_stream;
    PM_CUDA(cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    for (int k = 0; k < kCgChunk; ++k)
    {
        T* r_in = (k & 1) ? r1 : r0;
        T* r_out = (k & 1) ? r0 : r1;
        pcg_direction_kernel<T><<<vgrid, kReduceBlock, 0, cs>>>(n, z, p, st);
        launch_pcg_spmv<T>(A, p, q, partials, st, sgrid, cs);
        pcg_update_kernel<T><<<vgrid, kReduceBlock, 0, cs>>>(n, x, p, q, r_in, r_out, z, mode, inv, blocks, bs,
                                                              partials, st);
    }
    cg_continue_kernel<<<1, 32, 0, cs>>>(handle, st);
    cudaGraph_t captured = nullptr;
    const cudaError_t cap = cudaStreamEndCapture(cs, &captured);
    cudaGraphExec_t exec = nullptr;
    const cudaError_t inst = cap == cudaSuccess ? cudaGraphInstantiate(&exec, graph, 0) : cap;
    if (inst != cudaSuccess)
    {
        cudaGraphDestroy(graph);
        fail(PM_CUDA_ERROR, std::string("CUDA iterative solver: iteration graph: ") + cudaGetErrorString(inst));
    }
    slot.operand = A->serial;
    std::copy(key, key + 4, slot.key);
    slot.n = n;
    slot.shape = shape;
    slot.mode = mode;
    slot.block_size = bs;
    slot.value_size = int(sizeof(T));
    slot.graph = graph;
    slot.exec = exec;
    return exec;
}

// smem: this launch's shared memory, most_smem: that of the kernel's largest launch
template <typename T, typename Kernel>
bool launch_cooperative(Kernel kernel, PcgLoop<T>& a, unsigned ctas, unsigned threads, size_t smem, size_t most_smem,
                        cudaStream_t stream)
{
    allow_smem(reinterpret_cast<const void*>(kernel), most_smem);
    void* args[] = {&a};
    return launch_resident(reinterpret_cast<const void*>(kernel), ctas, threads, args, smem, stream);
}

// One cooperative launch of the whole solve where it is the faster form (see pcg_loop_kernel);
// false where it is not.  One CTA per SM at most: they wait for one another, so all must be resident.
// A lane that sums a longer row alone holds up the whole launch.  Every gathered entry of p formed from two
// vectors, it takes 103 ns a nonzero in FP64 and 67 in FP32 (36 and 30 from staged tiles, 67 and 65 as kernels
// that read directly).  Jacobi PCG, 30 iterations, us, as kernels / rows in registers / staged tiles with the
// kept residual: 60,000 rows of 5 and one of 128, FP64 748 / 600 / 508, FP32 701 / 443 / 452; one of 1,000,
// 2,555 / 2,753 / 1,214 and 2,104 / 1,711 / 986.  Blocks of six, FP32, one of 1,000: one launch 2,166,
// kernels 1,437; FP64 1,935 and 2,469, but one of 12,000 25.2 ms and 24.0.
constexpr int kLoneRow = 128;
constexpr int kLoneBlockRow = 8192;

template <typename T, int SHAPE>
bool launch_pcg_loop_shape(PcgLoop<T>& a, size_t warp_smem, int lanes, int longest_row, cudaStream_t stream)
{
    const int most = std::min(sm_count(), kGridMaxCtas);
    if constexpr (SHAPE == 1)
    {
        constexpr size_t kSmem = 226 * 1024; // of the 227 KB a CTA may have; the rest is static
        if (a.mode != 2 && a.n <= int64_t(4) * kRowThreads * most && longest_row <= kLoneRow)
        {
            const auto launch_rows = [&](auto kernel, int per_thread) {
                unsigned block = 256;
                if (a.n > int64_t(block) * per_thread * most)
                    block = kRowThreads;
                const size_t warp = size_t(kTileCap) * per_thread * (sizeof(T) + sizeof(int));
                return launch_cooperative(kernel, a, grid_for(a.n, static_cast<int>(block) * per_thread, most), block,
                                          warp * (block / 32), warp * (kRowThreads / 32), stream);
            };
            if (a.n <= int64_t(kRowThreads) * most)
                return launch_rows(pcg_row_kernel<T, 1>, 1);
            if (a.n <= int64_t(2) * kRowThreads * most)
                return launch_rows(pcg_row_kernel<T, 2>, 2);
            return launch_rows(pcg_row_kernel<T, 4>, 4);
        }
        const unsigned ctas = grid_for(a.n, kTileThreads, most);
        const int64_t per_thread = (a.n + int64_t(ctas) * kTileThreads - 1) / (int64_t(ctas) * kTileThreads);
        const size_t kept = size_t(per_thread) * kTileThreads * sizeof(T);
        const size_t staged = kTileThreads / 32 * 2 * sizeof(RowTile<T, kKeepCap>);
        if (a.mode != 2 && kept <= kSmem - staged)
            return launch_cooperative(pcg_loop_kernel<T, 1, true>, a, ctas, kTileThreads, staged + kept, kSmem, stream);
        warp_smem = 2 * sizeof(RowTile<T, kTileCap>);
    }
    if ((SHAPE == -1 || SHAPE == 1) && longest_row > (SHAPE == 1 && sizeof(T) == 8 ? kLoneBlockRow : kLoneRow))
        return false;
    // few lanes: one row per thread (or group of lanes)
    constexpr unsigned kMost = loop_threads<T>(SHAPE);
    const int64_t wanted = a.n * lanes;
    if (wanted > int64_t(kMost) * most)
        return false;
    unsigned threads = 256;
    while (threads < kMost && wanted > int64_t(threads) * most)
        threads = std::min(2 * threads, kMost);
    return launch_cooperative(pcg_loop_kernel<T, SHAPE, false>, a, grid_for(wanted, static_cast<int>(threads), most),
                              threads, warp_smem * (threads / 32), warp_smem * (kMost / 32), stream);
}

template <typename T>
bool launch_pcg_loop(const pm_csr* A, PcgLoop<T>& a, cudaStream_t stream)
{
    if (use_stream(A))
        return launch_pcg_loop_shape<T, 0>(a, kStreamCap * sizeof(T), 1, A->longest_row, stream);
    if (use_tiles<T>(A))
        return launch_pcg_loop_shape<T, 1>(a, 0, 1, A->longest_row, stream);
    switch (lanes_per_row(A))
    {
    case 1: return launch_pcg_loop_shape<T, -1>(a, 0, 1, A->longest_row, stream);
    case 2: return launch_pcg_loop_shape<T, 2>(a, 0, 2, A->longest_row, stream);
    case 4: return launch_pcg_loop_shape<T, 4>(a, 0, 4, A->longest_row, stream);
    case 8: return launch_pcg_loop_shape<T, 8>(a, 0, 8, A->longest_row, stream);
    case 16: return launch_pcg_loop_shape<T, 16>(a, 0, 16, A->longest_row, stream);
    default: return launch_pcg_loop_shape<T, 32>(a, 0, 32, A->longest_row, stream);
    }
}

// Queues a solve: one cooperative launch, or the initial residual and then the iterations as kernels
// (from the operand set's graph, or one by one when `graph` is false).  Returns the device state.
template <typename T>
PcgState* queue_pcg(pm_solver_workspace* ws, const pm_csr* A, const T* b, T* x, const T* blocks, int64_t bs, int mode,
                    double relative, double absolute, int max_iterations, bool graph, cudaStream_t stream)
{
    const int64_t n = A->rows;
    ws->buffer.ensure(PcgVectors<T>(ws, n).bytes + 256, stream, "IterativeSolverWorkspace");
    const PcgVectors<T> u(ws, n);
    ws->mail.open(stream, "IterativeSolverWorkspace");
    const T* v = static_cast<const T*>(A->values);
    pcg_reset_kernel<<<1, 1, 0, stream>>>(u.st, max_iterations, ws->mail.epoch());
    PM_LAUNCH_CHECK();
    PcgLoop<T> a{n, static_cast<int>(A->nnz), A->row_ptr, A->col_idx, v, b, x, {u.r[0], u.r[1]}, u.z, {u.p[0], u.p[1]},
                 u.q, u.inv, mode, blocks, bs, relative, absolute, ws->mail.packets(), ws->mail.epoch(), u.st};
    if (launch_pcg_loop<T>(A, a, stream))
        return u.st;
    if (mode == 1)
    {
        jacobi_kernel<T><<<grid_for(n, 256, 4096), 256, 0, stream>>>(n, A->row_ptr, A->col_idx, v, u.inv, u.st);
        PM_LAUNCH_CHECK();
    }
    const unsigned vgrid = grid_for(n, kReduceBlock, kMaxReduceBlocks);
    launch_spmv<T>(A, x, u.q, stream);
    pcg_init_kernel<T><<<vgrid, kReduceBlock, 0, stream>>>(n, b, u.q, u.r[0], u.z, u.p[0], mode, u.inv, blocks, bs,
                                                            relative, absolute, u.partials, u.st);
    PM_LAUNCH_CHECK();
    if (graph && max_iterations > 0)
    {
        const cudaGraphExec_t exec = cg_iteration_graph<T>(ws, A, x, blocks, bs, mode);
        PM_CUDA(cudaMemsetAsync(&u.st->chunks, 0, sizeof(int), stream));
        PM_CUDA(cudaGraphLaunch(exec, stream));
    }
    else
    {
        const unsigned sgrid = use_stream(A) ? vgrid : grid_for(n * lanes_per_row(A), kReduceBlock, kMaxReduceBlocks);
        for (int k = 0; k < max_iterations; ++k)
        {
            if (k > 0)
            {
                pcg_direction_kernel<T><<<vgrid, kReduceBlock, 0, stream>>>(n, u.z, u.p[0], u.st);
                PM_LAUNCH_CHECK();
            }
            launch_pcg_spmv<T>(A, u.p[0], u.q, u.partials, u.st, sgrid, stream);
            pcg_update_kernel<T><<<vgrid, kReduceBlock, 0, stream>>>(n, x, u.p[0], u.q, u.r[k & 1], u.r[(k & 1) ^ 1],
                                                                      u.z, mode, u.inv, blocks, bs, u.partials, u.st);
            PM_LAUNCH_CHECK();
        }
    }
    return u.st;
}

// mode: 0 = CG, 1 = Jacobi PCG, 2 = caller block inverses
template <typename T>
void solve(pm_solver_workspace* ws, cudaStream_t stream, const pm_csr* A, const T* b, T* x, const T* blocks,
           int64_t bs, const pm_solver_options* o, pm_solver_report* report, int mode)
{
    if (!ws || !A || !o || !report)
        fail(PM_INVALID_ARGUMENT, "solver arguments must be non-null");
    *report = pm_solver_report{0, 0, 0.0, 0.0};
    if (o->max_iterations < 0 || !std::isfinite(o->relative_tolerance) || o->relative_tolerance < 0.0 ||
        o->relative_tolerance > 1.0 || !std::isfinite(o->absolute_tolerance) || o->absolute_tolerance < 0.0)
        fail(PM_INVALID_ARGUMENT, "invalid CUDA iterative solver options");
    if (A->value_size != static_cast<int>(sizeof(T)))
        fail(PM_INVALID_ARGUMENT, "solver scalar type differs from the CSR operand");
    if (A->rows != A->cols)
        fail(PM_INVALID_ARGUMENT, "CUDA iterative solver requires square A and Nx1 rhs/solution");
    const int64_t n = A->rows;
    if (n > 0 && (!b || !x))
        fail(PM_INVALID_ARGUMENT, "solver vectors must be non-null");
    if (b && b == x)
        fail(PM_INVALID_ARGUMENT, "CUDA iterative solver rhs and solution must not alias");
    if (mode == 2)
    {
        if (bs <= 0 || n % bs != 0 || !blocks)
            fail(PM_INVALID_ARGUMENT, "CUDA block PCG requires complete row-major inverse diagonal blocks");
        if (static_cast<const void*>(blocks) == static_cast<const void*>(b) ||
            static_cast<const void*>(blocks) == static_cast<const void*>(x))
            fail(PM_INVALID_ARGUMENT, "CUDA block PCG inverse blocks must not alias rhs or solution");
    }
    if (n == 0)
    {
        report->converged = 1;
        return;
    }
    if (!ws->host_state)
        PM_CUDA(cudaMallocHost(&ws->host_state, sizeof(PcgState)));
    if (!ws->event)
        PM_CUDA(cudaEventCreateWithFlags(&ws->event, cudaEventDisableTiming));
    const PcgState* st = queue_pcg<T>(ws, A, b, x, blocks, bs, mode, o->relative_tolerance, o->absolute_tolerance,
                                      o->max_iterations, true, stream);
    PM_CUDA(cudaMemcpyAsync(ws->host_state, st, sizeof(PcgState), cudaMemcpyDeviceToHost, stream));
    PM_CUDA(cudaEventRecord(ws->event, stream));
    PM_CUDA(cudaEventSynchronize(ws->event));
    const PcgState s = *static_cast<PcgState*>(ws->host_state);
    for (int k = 0; k < s.chunks * (3 * kCgChunk + 1); ++k) // the kernels a graph ran
        count_launch();
    if (s.timed_out)
        fail(PM_CUDA_ERROR, "CUDA iterative solver: a grid barrier did not complete");
    if (s.jacobi_bad_row != kNone)
    {
        std::ostringstream m;
        m << "pcg Jacobi diagonal is missing, non-positive, or near zero at row " << s.jacobi_bad_row;
        fail(PM_RUNTIME_ERROR, m.str());
    }
    if (s.nonfinite_init)
        fail(PM_RUNTIME_ERROR, "CUDA iterative solver initial residual is not finite");
    report->initial_residual = std::sqrt(s.initial_squared);
    report->iterations = s.iterations;
    report->final_residual = std::sqrt(std::max(0.0, s.residual_squared));
    report->converged = s.converged;
    if (s.breakdown)
        fail(PM_RUNTIME_ERROR, "CUDA iterative solver breakdown: matrix is not numerically SPD");
    if (!s.converged && o->require_convergence)
    {
        std::ostringstream m;
        m << "CUDA iterative solver did not converge in " << s.iterations
          << " iterations; final residual=" << report->final_residual;
        fail(PM_RUNTIME_ERROR, m.str());
    }
}

// Exactly `iterations` CG (mode 0) or Jacobi-PCG (mode 1) steps with no host check
// (fixedSolve, src/sparse/iterative_solver.cu:166-233): tolerance 0, so the device state only
// stops early on an exact zero residual or a breakdown.
template <typename T>
pm_fixed_state* fixed_solve(pm_solver_workspace* ws, cudaStream_t stream, const pm_csr* A, const T* b, T* x,
                            int iterations, int mode)
{
    if (!ws || !A)
        fail(PM_INVALID_ARGUMENT, "solver arguments must be non-null");
    if (iterations < 0)
        fail(PM_INVALID_ARGUMENT, "fixed CUDA iterative solver iterations must be non-negative");
    if (A->value_size != static_cast<int>(sizeof(T)))
        fail(PM_INVALID_ARGUMENT, "solver scalar type differs from the CSR operand");
    if (A->rows != A->cols)
        fail(PM_INVALID_ARGUMENT, "CUDA iterative solver requires square A and Nx1 rhs/solution");
    const int64_t n = A->rows;
    if (n > 0 && (!b || !x))
        fail(PM_INVALID_ARGUMENT, "solver vectors must be non-null");
    if (b && b == x)
        fail(PM_INVALID_ARGUMENT, "CUDA iterative solver rhs and solution must not alias");
    auto* state = new pm_fixed_state();
    try
    {
        state->stream = stream;
        state->submitted = iterations;
        PM_CUDA(cudaMalloc(reinterpret_cast<void**>(&state->residuals), 2 * sizeof(double)));
        PM_CUDA(cudaEventCreateWithFlags(&state->event, cudaEventDisableTiming));
        if (n == 0)
        {
            PM_CUDA(cudaMemsetAsync(state->residuals, 0, 2 * sizeof(double), stream));
            PM_CUDA(cudaEventRecord(state->event, stream));
            return state;
        }
        A->queued_on(stream);
        const PcgState* st = queue_pcg<T>(ws, A, b, x, static_cast<const T*>(nullptr), 0, mode, 0.0, 0.0, iterations,
                                          false, stream);
        fixed_finish_kernel<<<1, 1, 0, stream>>>(st, state->residuals);
        PM_LAUNCH_CHECK();
        PM_CUDA(cudaEventRecord(state->event, stream));
    }
    catch (...)
    {
        delete state;
        throw;
    }
    return state;
}

void fixed_finalize(const pm_fixed_state* state, const pm_solver_options* o, pm_solver_report* report)
{
    if (!o || !report)
        fail(PM_INVALID_ARGUMENT, "finalize arguments must be non-null");
    if (!std::isfinite(o->relative_tolerance) || o->relative_tolerance < 0.0 || o->relative_tolerance > 1.0 ||
        !std::isfinite(o->absolute_tolerance) || o->absolute_tolerance < 0.0)
        fail(PM_INVALID_ARGUMENT, "invalid CUDA iterative solver options");
    if (!state || !state->event)
        fail(PM_LOGIC_ERROR, "fixed CUDA iterative solver state is empty or closed");
    const cudaError_t status = cudaEventQuery(state->event);
    if (status == cudaErrorNotReady)
        fail(PM_LOGIC_ERROR, "finalizeIterativeSolverReport requires caller stream synchronization");
    PM_CUDA(status);
    double host[2] = {0.0, 0.0};
    PM_CUDA(cudaMemcpy(host, state->residuals, sizeof(host), cudaMemcpyDeviceToHost));
    if (!std::isfinite(host[0]) || !std::isfinite(host[1]) || host[0] < 0.0 || host[1] < 0.0)
        fail(PM_RUNTIME_ERROR, "fixed CUDA iterative solver breakdown: residual is not finite");
    *report = pm_solver_report{0, 0, 0.0, 0.0};
    report->iterations = state->submitted;
    report->initial_residual = std::sqrt(host[0]);
    report->final_residual = std::sqrt(host[1]);
    const double tolerance = std::max(o->absolute_tolerance, o->relative_tolerance * report->initial_residual);
    report->converged = report->final_residual <= tolerance;
    if (!report->converged && o->require_convergence)
    {
        std::ostringstream m;
        m << "fixed CUDA iterative solver did not converge in " << report->iterations
          << " iterations; final residual=" << report->final_residual;
        fail(PM_RUNTIME_ERROR, m.str());
    }
}

} // namespace
} // namespace pm

extern "C" {

int pm_csr_create_f32(pm_stream_t stream, int64_t rows, int64_t cols, int64_t nnz, const int64_t* ro,
                      const int64_t* ci, const float* v, pm_csr** out)
{
    return pm::guarded([&] { pm::csr_create<float>(stream, rows, cols, nnz, ro, ci, v, out); });
}
int pm_csr_create_f64(pm_stream_t stream, int64_t rows, int64_t cols, int64_t nnz, const int64_t* ro,
                      const int64_t* ci, const double* v, pm_csr** out)
{
    return pm::guarded([&] { pm::csr_create<double>(stream, rows, cols, nnz, ro, ci, v, out); });
}
#define PM_FIXED(KIND, MODE, SFX, T)                                                                              \
    int pm_##KIND##_fixed_iterations_async_##SFX(pm_solver_workspace* ws, pm_stream_t s, const pm_csr* A, const T* b, \
                                                  T* x, int iterations, pm_fixed_state** state)                    \
    {                                                                                                              \
        return pm::guarded([&] {                                                                                   \
            if (!state)                                                                                            \
                pm::fail(PM_INVALID_ARGUMENT, "fixed solver state pointer is null");                               \
            *state = pm::fixed_solve<T>(ws, s, A, b, x, iterations, MODE);                                         \
        });                                                                                                        \
    }
PM_FIXED(cg, 0, f32, float)
PM_FIXED(cg, 0, f64, double)
PM_FIXED(pcg, 1, f32, float)
PM_FIXED(pcg, 1, f64, double)
#undef PM_FIXED

int pm_fixed_state_finalize(const pm_fixed_state* state, const pm_solver_options* o, pm_solver_report* report)
{
    return pm::guarded([&] { pm::fixed_finalize(state, o, report); });
}

void pm_fixed_state_destroy(pm_fixed_state* state)
{
    if (state)
    {
        if (state->event)
            cudaEventSynchronize(state->event);
        delete state;
        cudaGetLastError(); // a captured event cannot be waited for: not the next call's error
    }
}

void pm_csr_destroy(pm_csr* A)
{
    if (A)
    {
        cudaFree(A->row_ptr); // stream-ordered memory: it does not wait for kernels that still read it
        cudaFree(A->col_idx);
        delete A;
    }
}
int pm_csr_wait(const pm_csr* A)
{
    return pm::guarded([&] {
        if (!A)
            pm::fail(PM_INVALID_ARGUMENT, "CSR handle is null");
        std::vector<cudaStream_t> streams;
        {
            const std::lock_guard<std::mutex> lock(A->used_lock);
            streams.swap(A->used);
        }
        for (const cudaStream_t stream : streams)
        {
            cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
            if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess)
                cudaGetLastError(); // the legacy stream beside a capture: it cannot be waited for either
            else if (capture == cudaStreamCaptureStatusNone)
                PM_CUDA(cudaStreamSynchronize(stream));
        }
    });
}
int pm_csr_set_values(pm_csr* A, const void* values)
{
    return pm::guarded([&] {
        if (!A || (A->nnz > 0 && !values))
            pm::fail(PM_INVALID_ARGUMENT, "CSR handle and values must be non-null");
        A->values = values;
    });
}
int pm_csr_spmv_f32(const pm_csr* A, pm_stream_t stream, const float* x, float* y)
{
    return pm::guarded([&] { pm::csr_spmv<float>(A, stream, x, y); });
}
int pm_csr_spmv_f64(const pm_csr* A, pm_stream_t stream, const double* x, double* y)
{
    return pm::guarded([&] { pm::csr_spmv<double>(A, stream, x, y); });
}

int pm_csr_spmm_f32(const pm_csr* A, pm_stream_t stream, int64_t input_rows, int64_t input_cols, const float* input,
                    int64_t output_rows, int64_t output_cols, float* output)
{
    return pm::guarded(
        [&] { pm::csr_spmm<float>(A, stream, input_rows, input_cols, input, output_rows, output_cols, output); });
}
int pm_csr_spmm_f64(const pm_csr* A, pm_stream_t stream, int64_t input_rows, int64_t input_cols, const double* input,
                    int64_t output_rows, int64_t output_cols, double* output)
{
    return pm::guarded(
        [&] { pm::csr_spmm<double>(A, stream, input_rows, input_cols, input, output_rows, output_cols, output); });
}

int pm_csr_autotune_f32(pm_csr* A, pm_stream_t stream, const float* x, float* y, int* kernel)
{
    return pm::guarded([&] {
        const int k = pm::csr_autotune<float>(A, stream, x, y, 5);
        if (kernel)
            *kernel = k;
    });
}
int pm_csr_autotune_f64(pm_csr* A, pm_stream_t stream, const double* x, double* y, int* kernel)
{
    return pm::guarded([&] {
        const int k = pm::csr_autotune<double>(A, stream, x, y, 5);
        if (kernel)
            *kernel = k;
    });
}
int pm_csr_set_kernel(pm_csr* A, int kernel)
{
    return pm::guarded([&] {
        if (!A)
            pm::fail(PM_INVALID_ARGUMENT, "CSR handle is null");
        if (!(kernel == -1 || kernel == 0 || kernel == 1 || kernel == 2 || kernel == 4 || kernel == 8 ||
              kernel == 16 || kernel == 32))
            pm::fail(PM_INVALID_ARGUMENT, "SpMV kernel must be -1 (heuristic), 0 (row-group stream) or 1, 2, 4, "
                                          "8, 16, 32 lanes per row");
        A->kernel = kernel;
    });
}
int pm_csr_kernel(const pm_csr* A, int* kernel, int* heuristic_lanes)
{
    return pm::guarded([&] {
        if (!A)
            pm::fail(PM_INVALID_ARGUMENT, "CSR handle is null");
        if (kernel)
            *kernel = A->kernel;
        if (heuristic_lanes)
            *heuristic_lanes = A->threads_per_row;
    });
}

int pm_solver_workspace_create(pm_solver_workspace** out)
{
    return pm::guarded([&] {
        if (!out)
            pm::fail(PM_INVALID_ARGUMENT, "workspace output pointer is null");
        *out = new pm_solver_workspace();
    });
}
void pm_solver_workspace_destroy(pm_solver_workspace* ws) { delete ws; }
int pm_solver_workspace_close(pm_solver_workspace* ws)
{
    return pm::guarded([&] {
        if (!ws)
            pm::fail(PM_INVALID_ARGUMENT, "workspace is null");
        ws->drop_graphs(); // they hold pointers into the buffer released here
        ws->buffer.release();
        ws->mail.buffer.release();
    });
}

#define PM_SOLVER_API(SFX, T)                                                                                      \
    int pm_cg_##SFX(pm_solver_workspace* ws, pm_stream_t s, const pm_csr* A, const T* b, T* x,                      \
                    const pm_solver_options* o, pm_solver_report* r)                                                \
    {                                                                                                               \
        return pm::guarded([&] { pm::solve<T>(ws, s, A, b, x, nullptr, 0, o, r, 0); });                            \
    }                                                                                                               \
    int pm_pcg_##SFX(pm_solver_workspace* ws, pm_stream_t s, const pm_csr* A, const T* b, T* x,                     \
                     const pm_solver_options* o, pm_solver_report* r)                                               \
    {                                                                                                               \
        return pm::guarded([&] { pm::solve<T>(ws, s, A, b, x, nullptr, 0, o, r, o && o->use_jacobi ? 1 : 0); });  \
    }                                                                                                               \
    int pm_block_pcg_##SFX(pm_solver_workspace* ws, pm_stream_t s, const pm_csr* A, const T* b, T* x,               \
                           const T* blocks, int64_t bs, const pm_solver_options* o, pm_solver_report* r)            \
    {                                                                                                               \
        return pm::guarded([&] { pm::solve<T>(ws, s, A, b, x, blocks, bs, o, r, 2); });                            \
    }

PM_SOLVER_API(f32, float)
PM_SOLVER_API(f64, double)

} // extern "C"
