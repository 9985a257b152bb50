// Deterministic COO -> CSR for sm_100a.
//
// Contract (src/sparse/sparse_ops_cpu.cpp:24-134): the output equals a stable sort of the
// triplets by (row, col) followed by an in-order combination of duplicates (first value
// taken as is, the rest added one by one in input order).
//
// Design: instead of a device-wide radix sort of packed (row, col) keys, the triplets are
// bucketed by row with integer atomics (positions inside a row bucket are arbitrary), and
// every row segment is then sorted by the unique 64-bit key (col << 32 | source offset).
// Because the key contains the source offset, any correct sort yields the one order that
// the stable sort defines -- the result does not depend on scheduling.  Segments are sorted
// where they fit: <= 16 entries in registers (one thread per row), <= 2048 in shared memory
// (one CTA per row), longer rows by CTA-local merge passes in global memory.  Runs are then
// combined serially in key order, which reproduces the reference's left-to-right sums bit for
// bit.  Errors are recorded in a device status (lowest offending offset, as the reference's
// CooStatus, src/sparse/coo_to_csr.cu:22-29) and read by pm_coo_status().
#include "pm_common.cuh"

#include <climits>
#include <cmath>
#include <sstream>

namespace pm
{
namespace
{

constexpr unsigned long long kNoOffset = 0x7fffffffffffffffULL;
constexpr uint64_t kPadKey = ~uint64_t(0);
constexpr int kShortMax = 16;       // register-sorted segment length
constexpr int kLongCap = 2048;      // shared-memory segment length
constexpr int kLongThreads = 256;
constexpr int kMergeItems = kLongCap / kLongThreads;

struct CooStatus
{
    unsigned long long invalid_source;
    unsigned long long invalid_value;
    unsigned long long mismatch_actual;
    unsigned long long mismatch_expected;
    long long actual_nnz;
    int long_count;
    int pad;
};

// (key, value) of one scattered triplet: a single 16-byte store into its row bucket
template <typename T>
struct alignas(16) CooRec
{
    uint64_t key;
    T value;
};

__device__ __forceinline__ uint32_t key_col(uint64_t key) { return static_cast<uint32_t>(key >> 32); }
__device__ __forceinline__ unsigned source_of(uint64_t key) { return static_cast<unsigned>(key & 0xffffffffu); }

template <typename T>
__device__ __forceinline__ bool finite_value(T v)
{
    return isfinite(static_cast<double>(v));
}

// a fresh status and empty buckets
__global__ void __launch_bounds__(256) init_kernel(CooStatus* status, int* __restrict__ bucket_sizes, int64_t rows)
{
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < rows; i += int64_t(gridDim.x) * blockDim.x)
        bucket_sizes[i] = 0;
    if (blockIdx.x > 0 || threadIdx.x > 0)
        return;
    status->invalid_source = kNoOffset;
    status->invalid_value = kNoOffset;
    status->mismatch_actual = kNoOffset;
    status->mismatch_expected = kNoOffset;
    status->actual_nnz = 0;
    status->long_count = 0;
    status->pad = 0;
}

// 1) validate the row and reserve a slot inside its bucket (columns and values are checked by the
// scatter, which reads them anyway)
__global__ void __launch_bounds__(256) count_kernel(const int64_t* __restrict__ rows, int64_t count, int64_t row_count,
                                                    int* __restrict__ bucket_sizes, int* __restrict__ slots,
                                                    CooStatus* status)
{
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= count)
        return;
    const int64_t row = __ldcs(rows + i);
    if (row < 0 || row >= row_count)
    {
        atomicMin(&status->invalid_source, static_cast<unsigned long long>(i));
        slots[i] = -1;
        return;
    }
    slots[i] = atomicAdd(&bucket_sizes[row], 1);
}

// 2) scatter (key, value) into the row buckets as one 16-byte record per triplet (the sorts
// below read the records and write the sorted keys and values).  Shuffled triplets land all over
// the records, and a partial sector that leaves L2 before its neighbour arrives costs a read and a
// write of memory.  Pass k of a larger input therefore writes only the records of the k-th window of
// kScatterWindow bytes, which stays in L2: pass 0 turns every slot into the record's position, the
// others read that and, for their own triplets, the column and value again.  16M triplets of FP64:
// 603 us in one pass, 456 in four (conversion 1,152 against 1,005 us; 128 MB windows 1,132, 48 MB 1,048).
// Triplets that come in some order gain nothing from it: a warp whose records lie within one window's length
// writes all of them in pass 0 and skips the others.  Conversions of 8-entry rows, us, in one pass /
// this / windows for every warp, FP64: 16M shuffled 1,261 / 1,187 / 1,179; in row order 732 / 763 / 838;
// rows within 10,000 of their place 879 / 893 / 1,010; FP32: 1,349 / 1,235 / 1,228, 765 / 802 / 862,
// 1,005 / 1,028 / 1,123.
constexpr size_t kScatterWindow = size_t(64) << 20;
// Longer inputs take one pass: from six on the passes over ordered triplets cost what they save elsewhere
// (25M of FP32: shuffled 2,135 in one pass, 1,943 in six; rows within 60,000 of their place 1,485 and 1,569).
constexpr int kScatterPasses = 5;
// a CTA's kPer * 256 triplets; ranges: every warp's least and greatest positions where pass 0 left some to the
// others
template <typename T, bool FIRST, int kPer>
__device__ __forceinline__ void scatter_group(const int64_t* __restrict__ rows,
                                              const int64_t* __restrict__ cols, const T* __restrict__ values,
                                              int64_t count, int64_t col_count, int* __restrict__ slots,
                                              const int* __restrict__ bucket_start, CooRec<T>* __restrict__ recs,
                                              int64_t lo, int64_t hi, int2* __restrict__ ranges, CooStatus* status)
{
    const int64_t i0 = int64_t(blockIdx.x) * (kPer * 256) + threadIdx.x;
    int pos[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k)
    {
        const int64_t i = i0 + k * 256;
        pos[k] = i < count ? __ldcs(slots + i) : -1;
    }
    if constexpr (FIRST)
    {
#pragma unroll
        for (int k = 0; k < kPer; ++k)
            if (pos[k] >= 0)
                pos[k] += bucket_start[__ldcs(rows + i0 + k * 256)];
        if (hi < count)
        {
            int least = INT_MAX, greatest = -1;
#pragma unroll
            for (int k = 0; k < kPer; ++k)
                if (pos[k] >= 0)
                {
                    least = min(least, pos[k]);
                    greatest = max(greatest, pos[k]);
                }
            least = __reduce_min_sync(0xffffffffu, least);
            greatest = __reduce_max_sync(0xffffffffu, greatest);
            const bool left = greatest - least >= hi; // hi: a window's records
            if (left)
            {
#pragma unroll
                for (int k = 0; k < kPer; ++k)
                    if (pos[k] >= 0)
                        __stcs(slots + i0 + k * 256, pos[k]);
            }
            else
                hi = count; // all of them here
            if ((threadIdx.x & 31) == 0)
                ranges[blockIdx.x * 8 + (threadIdx.x >> 5)] = left ? make_int2(least, greatest) : make_int2(INT_MAX, -1);
        }
    }
    int64_t col[kPer];
    T value[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k)
    {
        const int64_t i = i0 + k * 256;
        // the first pass checks every column and value, also those of triplets whose rows the count
        // rejected
        if (FIRST ? i < count : pos[k] >= lo && pos[k] < hi)
        {
            col[k] = __ldcs(cols + i);
            value[k] = values ? __ldcs(values + i) : T(0);
        }
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k)
    {
        const int64_t i = i0 + k * 256;
        if (FIRST && i < count)
        {
            if (col[k] < 0 || col[k] >= col_count)
                atomicMin(&status->invalid_source, static_cast<unsigned long long>(i));
            if (!finite_value(value[k]))
                atomicMin(&status->invalid_value, static_cast<unsigned long long>(i));
        }
        if (pos[k] >= lo && pos[k] < hi)
        {
            CooRec<T> r;
            r.key = (static_cast<uint64_t>(col[k]) << 32) | static_cast<uint64_t>(i);
            r.value = value[k];
            recs[pos[k]] = r;
        }
    }
}

template <typename T, int kPer>
__global__ void __launch_bounds__(256) scatter_kernel(const int64_t* __restrict__ rows, const int64_t* __restrict__ cols,
                                                      const T* __restrict__ values, int64_t count, int64_t col_count,
                                                      int* __restrict__ slots, const int* __restrict__ bucket_start,
                                                      CooRec<T>* __restrict__ recs, int64_t hi,
                                                      int2* __restrict__ ranges, CooStatus* status)
{
    scatter_group<T, true, kPer>(rows, cols, values, count, col_count, slots, bucket_start, recs, 0, hi,
                                 ranges, status);
}

template <typename T, int kPer>
__global__ void __launch_bounds__(256) scatter_window_kernel(const int64_t* __restrict__ cols,
                                                             const T* __restrict__ values, int64_t count,
                                                             int* __restrict__ slots, CooRec<T>* __restrict__ recs,
                                                             int64_t lo, int64_t hi, int2* __restrict__ ranges)
{
    const int2 range = ranges[blockIdx.x * 8 + (threadIdx.x >> 5)];
    if (range.y < lo || range.x >= hi)
        return;
    scatter_group<T, false, kPer>(nullptr, cols, values, count, 0, slots, nullptr, recs, lo, hi, nullptr, nullptr);
}

// odd-even merge network over N register-resident (key, value) pairs (63 comparators for 16; a
// bitonic network takes 80); indices are compile-time
template <int N, typename T>
__device__ __forceinline__ void register_sort(uint64_t (&k)[N], T (&v)[N])
{
#pragma unroll
    for (int p = 1; p < N; p <<= 1)
    {
#pragma unroll
        for (int d = p; d > 0; d >>= 1)
        {
#pragma unroll
            for (int i = 0; i < N; ++i)
            {
                // i is the lower end of a comparator (i, i + d) of this step
                const int j = i - d % p;
                if (j >= 0 && (j / d) % 2 == 0 && i + d < N && i / (2 * p) == (i + d) / (2 * p))
                {
                    const uint64_t a = k[i], b = k[i + d];
                    const bool swap = a > b;
                    const T va = v[i], vb = v[i + d];
                    k[i] = swap ? b : a;
                    k[i + d] = swap ? a : b;
                    v[i] = swap ? vb : va;
                    v[i + d] = swap ? va : vb;
                }
            }
        }
    }
}

// 3) short rows whose sorted keys are read later: one thread per row, sorted in registers; long rows
// are queued
template <typename T>
__global__ void __launch_bounds__(128) sort_short_kernel(const int* __restrict__ bucket_start, int64_t row_count,
                                                         const CooRec<T>* __restrict__ recs,
                                                         uint64_t* __restrict__ keys, T* __restrict__ values,
                                                         int* __restrict__ unique_count, int* __restrict__ long_rows,
                                                         CooStatus* status)
{
    const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r >= row_count)
        return;
    const int start = bucket_start[r];
    const int len = bucket_start[r + 1] - start;
    if (len > kShortMax)
    {
        long_rows[atomicAdd(&status->long_count, 1)] = static_cast<int>(r);
        return;
    }
    if (len <= 1)
    {
        if (len == 1)
        {
            const CooRec<T> one = recs[start];
            keys[start] = one.key;
            values[start] = one.value;
        }
        unique_count[r] = len;
        return;
    }
    uint64_t k[kShortMax];
    T v[kShortMax];
#pragma unroll
    for (int q = 0; q < kShortMax; ++q)
    {
        if (q < len)
        {
            const CooRec<T> one = recs[start + q];
            k[q] = one.key;
            v[q] = one.value;
        }
        else
        {
            k[q] = kPadKey;
            v[q] = T(0);
        }
    }
    register_sort<kShortMax, T>(k, v);
    int unique = 0;
    uint32_t previous = 0;
#pragma unroll
    for (int q = 0; q < kShortMax; ++q)
    {
        if (q < len)
        {
            keys[start + q] = k[q];
            values[start + q] = v[q];
            const uint32_t col = key_col(k[q]);
            unique += (q == 0 || col != previous) ? 1 : 0;
            previous = col;
        }
    }
    unique_count[r] = unique;
}

// 3') the count phase of a conversion needs only the unique count of a short row (the fill sorts
// it): its columns are compared with one another, no sort.  A warp takes 32 rows, whose columns are
// one contiguous run brought into shared memory by coalesced loads when it has at most kTileRecs
// records (a lane reading its own row takes a line per record: 224 load wavefronts per 32 rows of
// seven against about 70).  2,097,152 rows of 7.6 entries: 42 us, against 151 for sorting them.
constexpr int kTileWarps = 8;
constexpr int kTileRecs = 384; // twelve per row
template <typename T>
__global__ void __launch_bounds__(32 * kTileWarps) count_short_kernel(const int* __restrict__ bucket_start,
                                                                      int64_t row_count,
                                                                      const CooRec<T>* __restrict__ recs,
                                                                      int* __restrict__ unique_count,
                                                                      int* __restrict__ long_rows, CooStatus* status)
{
    __shared__ uint32_t tiles[kTileWarps][kTileRecs];
    const int lane = threadIdx.x & 31;
    uint32_t* const tile = tiles[threadIdx.x >> 5];
    const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t at = r < row_count ? r : row_count;
    const int start = bucket_start[at], end = bucket_start[r < row_count ? r + 1 : row_count];
    const int len = end - start;
    const int first = __shfl_sync(0xffffffffu, start, 0), total = __shfl_sync(0xffffffffu, end, 31) - first;
    const bool staged = total <= kTileRecs;
    if (staged)
    {
        // asynchronous copies: all in flight together
        for (int k = lane; k < total; k += 32)
            cp_async4(tile + k, reinterpret_cast<const uint32_t*>(&recs[first + k].key) + 1);
        cp_async_commit();
        cp_async_wait<0>();
    }
    __syncwarp();
    if (r >= row_count)
        return;
    if (len > kShortMax)
    {
        long_rows[atomicAdd(&status->long_count, 1)] = static_cast<int>(r);
        return;
    }
    // columns are below 2^32 - 1: the padding is one more distinct value
    uint32_t col[kShortMax];
#pragma unroll
    for (int q = 0; q < kShortMax; ++q)
        col[q] = q < len ? (staged ? tile[start - first + q] : key_col(recs[start + q].key)) : 0xffffffffu;
    int unique = 1;
#pragma unroll
    for (int q = 1; q < kShortMax; ++q)
    {
        bool seen = false;
#pragma unroll
        for (int e = 0; e < q; ++e)
            seen |= col[e] == col[q];
        unique += seen ? 0 : 1;
    }
    unique_count[r] = unique - (len < kShortMax ? 1 : 0);
}

// bitonic sort of m (power of two, <= kLongCap) staged pairs in shared memory
template <typename T>
__device__ void smem_bitonic(uint64_t* sk, T* sv, int m)
{
    for (int size = 2; size <= m; size <<= 1)
    {
        for (int stride = size >> 1; stride > 0; stride >>= 1)
        {
            for (int i = threadIdx.x; i < m; i += blockDim.x)
            {
                const int j = i ^ stride;
                if (j > i)
                {
                    const bool ascending = (i & size) == 0;
                    const uint64_t a = sk[i], b = sk[j];
                    if ((a > b) == ascending)
                    {
                        sk[i] = b;
                        sk[j] = a;
                        const T t = sv[i];
                        sv[i] = sv[j];
                        sv[j] = t;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// merge-path split of diagonal d between sorted runs a[0..na) and b[0..nb) (unique keys)
__device__ __forceinline__ int merge_split(const uint64_t* a, int na, const uint64_t* b, int nb, int d)
{
    int lo = d > nb ? d - nb : 0;
    int hi = d < na ? d : na;
    while (lo < hi)
    {
        const int mid = (lo + hi) >> 1;
        if (a[mid] < b[d - mid - 1])
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// 4) long rows: one CTA per row.  <= kLongCap entries are sorted in shared memory; longer
// rows are sorted chunk by chunk and merged pairwise in global memory (ping-pong with
// `spare`), all inside the CTA.  Also counts the distinct columns of the row.
template <typename T>
__global__ void __launch_bounds__(kLongThreads) sort_long_kernel(const int* __restrict__ bucket_start,
                                                                 const CooRec<T>* __restrict__ recs,
                                                                 uint64_t* __restrict__ keys, T* __restrict__ values,
                                                                 uint64_t* __restrict__ spare_keys,
                                                                 T* __restrict__ spare_values,
                                                                 int* __restrict__ unique_count,
                                                                 const int* __restrict__ long_rows,
                                                                 const CooStatus* __restrict__ status)
{
    __shared__ uint64_t sk[kLongCap];
    __shared__ T sv[kLongCap];
    __shared__ int reduce[kLongThreads / 32];
    const int long_count = status->long_count;
    for (int li = blockIdx.x; li < long_count; li += gridDim.x)
    {
        const int r = long_rows[li];
        const int start = bucket_start[r];
        const int len = bucket_start[r + 1] - start;
        uint64_t* rk = keys + start;
        T* rv = values + start;
        // chunk sorts
        for (int c0 = 0; c0 < len; c0 += kLongCap)
        {
            const int n = min(kLongCap, len - c0);
            int m = 1;
            while (m < n)
                m <<= 1;
            for (int i = threadIdx.x; i < m; i += blockDim.x)
            {
                if (i < n)
                {
                    const CooRec<T> one = recs[start + c0 + i];
                    sk[i] = one.key;
                    sv[i] = one.value;
                }
                else
                {
                    sk[i] = kPadKey;
                    sv[i] = T(0);
                }
            }
            __syncthreads();
            smem_bitonic<T>(sk, sv, m);
            for (int i = threadIdx.x; i < n; i += blockDim.x)
            {
                rk[c0 + i] = sk[i];
                rv[c0 + i] = sv[i];
            }
            __syncthreads();
        }
        // merge passes (only rows longer than one chunk)
        uint64_t* src_k = rk;
        T* src_v = rv;
        uint64_t* dst_k = spare_keys + start;
        T* dst_v = spare_values + start;
        for (int width = kLongCap; width < len; width <<= 1)
        {
            for (int tile = 0; tile < len; tile += kLongCap)
            {
                const int pair = tile / (2 * width) * (2 * width);
                const int na = min(width, len - pair);
                const int nb = max(0, min(width, len - pair - width));
                const uint64_t* a = src_k + pair;
                const uint64_t* b = a + na;
                const T* av = src_v + pair;
                const T* bv = av + na;
                int d = tile - pair + threadIdx.x * kMergeItems;
                if (d < na + nb)
                {
                    int i = merge_split(a, na, b, nb, d);
                    int j = d - i;
                    for (int q = 0; q < kMergeItems && d + q < na + nb; ++q)
                    {
                        const bool take_a = i < na && (j >= nb || a[i] < b[j]);
                        dst_k[pair + d + q] = take_a ? a[i] : b[j];
                        dst_v[pair + d + q] = take_a ? av[i] : bv[j];
                        i += take_a ? 1 : 0;
                        j += take_a ? 0 : 1;
                    }
                }
            }
            __syncthreads();
            uint64_t* tk = src_k;
            src_k = dst_k;
            dst_k = tk;
            T* tv = src_v;
            src_v = dst_v;
            dst_v = tv;
        }
        if (src_k != rk)
        {
            for (int i = threadIdx.x; i < len; i += blockDim.x)
            {
                rk[i] = src_k[i];
                rv[i] = src_v[i];
            }
            __syncthreads();
        }
        // distinct columns
        int local = 0;
        for (int i = threadIdx.x; i < len; i += blockDim.x)
            local += (i == 0 || key_col(rk[i]) != key_col(rk[i - 1])) ? 1 : 0;
        const int unique = block_sum<int, kLongThreads>(local, reduce);
        if (threadIdx.x == 0)
            unique_count[r] = unique;
        __syncthreads();
    }
}

// the status' count, and the row offsets into the caller's array (out, may be null)
__global__ void __launch_bounds__(256) finish_status_kernel(const int64_t* __restrict__ row_offsets, int64_t row_count,
                                                            int64_t expected, CooStatus* status,
                                                            int64_t* __restrict__ out)
{
    if (out)
        for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i <= row_count;
             i += int64_t(gridDim.x) * blockDim.x)
            out[i] = row_offsets[i];
    if (blockIdx.x > 0 || threadIdx.x > 0)
        return;
    const long long actual = row_offsets[row_count];
    status->actual_nnz = actual;
    if (expected >= 0 && actual != expected)
    {
        status->mismatch_actual = static_cast<unsigned long long>(actual);
        status->mismatch_expected = static_cast<unsigned long long>(expected);
    }
}

template <typename T>
__device__ __forceinline__ void emit(int64_t at, int64_t capacity, uint32_t col, T sum, int64_t* col_out, T* val_out)
{
    if (at < capacity)
    {
        col_out[at] = col;
        val_out[at] = sum;
    }
}

// 5) combine runs of short rows: one thread per row, serial left-to-right sums
template <typename T>
__global__ void __launch_bounds__(128) write_short_kernel(const int* __restrict__ bucket_start, int64_t row_count,
                                                          const uint64_t* __restrict__ keys,
                                                          const T* __restrict__ values,
                                                          const int64_t* __restrict__ row_offsets, int64_t capacity,
                                                          int64_t* __restrict__ col_out, T* __restrict__ val_out,
                                                          CooStatus* status)
{
    const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r >= row_count)
        return;
    const int start = bucket_start[r];
    const int len = bucket_start[r + 1] - start;
    if (len > kShortMax || len == 0)
        return;
    int64_t at = row_offsets[r];
    uint32_t col = key_col(keys[start]);
    T sum = values[start];
    for (int q = 1; q < len; ++q)
    {
        const uint64_t key = keys[start + q];
        const uint32_t c = key_col(key);
        if (c != col)
        {
            emit(at++, capacity, col, sum, col_out, val_out);
            col = c;
            sum = values[start + q];
        }
        else
        {
            sum += values[start + q];
            if (!finite_value(sum))
                atomicMin(&status->invalid_value, static_cast<unsigned long long>(source_of(key)));
        }
    }
    emit(at, capacity, col, sum, col_out, val_out);
}

// The len <= N records at `in`, in key order: every pair of keys is compared once and counts towards
// the rank of the larger one (four instructions a pair; a comparator of a sorting network moves two
// keys and two values in fourteen), ranks are packed four bits each, and the records are read again
// in that order.  Keys are unique.
template <int N, typename T>
__device__ __forceinline__ void ordered_row(const CooRec<T>* in, int len, CooRec<T> (&row)[kShortMax])
{
    uint64_t rank = 0, order = 0;
    {
        uint64_t k[N];
#pragma unroll
        for (int q = 0; q < N; ++q)
            k[q] = q < len ? in[q].key : kPadKey;
#pragma unroll
        for (int q = 1; q < N; ++q)
#pragma unroll
            for (int e = 0; e < q; ++e)
                rank += k[q] < k[e] ? uint64_t(1) << (4 * e) : uint64_t(1) << (4 * q);
    }
#pragma unroll
    for (int q = 0; q < N; ++q)
        order |= uint64_t(q) << (4 * ((rank >> (4 * q)) & 15));
#pragma unroll
    for (int q = 0; q < N; ++q)
        if (q < len)
            row[q] = in[(order >> (4 * q)) & 15];
}

// 5') the same from the scattered records: every short row is put in key order (the count phase kept
// only its unique count) and its runs combined serially in key order.  A warp's 32 rows are one
// contiguous run of records and one of output entries; both pass through shared memory, so that
// memory is read and written in whole lines (kTileRecs records and no long row among them; otherwise
// each lane reads and writes its own row).  2,097,152 rows of 7.6 entries: 148 us, against 205 with the
// network and a lane's own loads and stores; what is left waits on the loads of a warp's tile.
template <typename T>
__global__ void __launch_bounds__(32 * kTileWarps) write_short_resort_kernel(const int* __restrict__ bucket_start,
                                                                 int64_t row_count, const CooRec<T>* __restrict__ recs,
                                                                 const int64_t* __restrict__ row_offsets,
                                                                 int64_t capacity, int64_t* __restrict__ col_out,
                                                                 T* __restrict__ val_out, CooStatus* status)
{
    union Tile
    {
        CooRec<T> in[kTileRecs];
        struct
        {
            T val[kTileRecs];
            uint32_t col[kTileRecs];
        } out;
        __device__ Tile() {}
    };
    extern __shared__ __align__(16) unsigned char tile_smem[];
    const int lane = threadIdx.x & 31;
    Tile& tile = reinterpret_cast<Tile*>(tile_smem)[threadIdx.x >> 5];
    const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t r0 = r < row_count ? r : row_count, r1 = r < row_count ? r + 1 : row_count;
    const int start = bucket_start[r0], end = bucket_start[r1];
    const int len = end - start;
    const int first = __shfl_sync(0xffffffffu, start, 0), total = __shfl_sync(0xffffffffu, end, 31) - first;
    const int most = __reduce_max_sync(0xffffffffu, len);
    const bool staged = total <= kTileRecs && most <= kShortMax;
    int64_t at = row_offsets[r0];
    const int64_t out0 = __shfl_sync(0xffffffffu, at, 0);
    const int out_total = static_cast<int>(__shfl_sync(0xffffffffu, row_offsets[r1], 31) - out0);
    if (staged)
    {
        for (int k = lane; k < total; k += 32)
            cp_async16(tile.in + k, recs + first + k);
        cp_async_commit();
        cp_async_wait<0>();
    }
    __syncwarp();
    const bool own = len > 0 && len <= kShortMax;
    const CooRec<T>* const mine = staged ? tile.in + (start - first) : recs + start;
    const int n = own ? len : 0;
    CooRec<T> row[kShortMax]; // in key order
    if (most <= 8)
        ordered_row<8, T>(mine, n, row);
    else if (most <= 12)
        ordered_row<12, T>(mine, n, row);
    else
        ordered_row<16, T>(mine, n, row);
    __syncwarp(); // the tile's input is read before its output is written
    if (own)
    {
        auto put = [&](int64_t to, uint32_t c, T sum) {
            if (staged)
            {
                tile.out.col[to - out0] = c;
                tile.out.val[to - out0] = sum;
            }
            else
                emit(to, capacity, c, sum, col_out, val_out);
        };
        uint32_t col = key_col(row[0].key);
        T sum = row[0].value;
#pragma unroll
        for (int q = 1; q < kShortMax; ++q)
        {
            if (q < len)
            {
                const uint32_t c = key_col(row[q].key);
                if (c != col)
                {
                    put(at++, col, sum);
                    col = c;
                    sum = row[q].value;
                }
                else
                {
                    sum += row[q].value;
                    if (!finite_value(sum))
                        atomicMin(&status->invalid_value, static_cast<unsigned long long>(source_of(row[q].key)));
                }
            }
        }
        put(at, col, sum);
    }
    if (!staged)
        return;
    __syncwarp();
    for (int e = lane; e < out_total; e += 32)
        emit(out0 + e, capacity, tile.out.col[e], tile.out.val[e], col_out, val_out);
}

// 6) combine runs of long rows: one CTA per row; run heads found by a block scan, each
// head thread sums its run serially in key order
template <typename T>
__global__ void __launch_bounds__(kLongThreads) write_long_kernel(const int* __restrict__ bucket_start,
                                                                  const uint64_t* __restrict__ keys,
                                                                  const T* __restrict__ values,
                                                                  const int64_t* __restrict__ row_offsets,
                                                                  int64_t capacity, int64_t* __restrict__ col_out,
                                                                  T* __restrict__ val_out,
                                                                  const int* __restrict__ long_rows,
                                                                  CooStatus* status)
{
    __shared__ int scan[kLongThreads / 32 + 1];
    const int long_count = status->long_count;
    for (int li = blockIdx.x; li < long_count; li += gridDim.x)
    {
        const int r = long_rows[li];
        const int start = bucket_start[r];
        const int len = bucket_start[r + 1] - start;
        const uint64_t* rk = keys + start;
        const T* rv = values + start;
        int64_t carry = row_offsets[r];
        for (int c0 = 0; c0 < len; c0 += kLongThreads)
        {
            const int i = c0 + threadIdx.x;
            const bool head = i < len && (i == 0 || key_col(rk[i]) != key_col(rk[i - 1]));
            int chunk_heads = 0;
            const int ordinal = block_exclusive_scan<int, kLongThreads>(head ? 1 : 0, scan, chunk_heads);
            if (head)
            {
                const uint32_t col = key_col(rk[i]);
                T sum = rv[i];
                for (int q = i + 1; q < len && key_col(rk[q]) == col; ++q)
                {
                    sum += rv[q];
                    if (!finite_value(sum))
                        atomicMin(&status->invalid_value, static_cast<unsigned long long>(source_of(rk[q])));
                }
                emit(carry + ordinal, capacity, col, sum, col_out, val_out);
            }
            carry += chunk_heads;
        }
    }
}

} // namespace
} // namespace pm

// =========================================================================== workspace
struct pm_sparse_workspace
{
    pm::DeviceBuffer buffer;
    bool status_pending = false; // a conversion was enqueued and not yet checked
    bool prepared = false;       // count phase enqueued; fill may follow
    int value_size = 0;
    int64_t rows = 0, cols = 0, count = 0;
    // carved device arrays of the last prepared conversion
    pm::CooStatus* status = nullptr;
    int* bucket_sizes = nullptr;
    int* bucket_start = nullptr;
    int* slots = nullptr;
    uint64_t* keys = nullptr;
    void* values = nullptr;
    uint64_t* spare_keys = nullptr;
    void* spare_values = nullptr;
    int* unique_count = nullptr;
    int* long_rows = nullptr;
    int64_t* row_offsets = nullptr;
    void* scan_scratch = nullptr;
    void* recs = nullptr;             // the scattered (key, value) records of the last conversion
    bool short_rows_kept = true;      // short rows' sorted keys / values are stored (else re-sorted at fill)
};

namespace pm
{

void require_values(int64_t count, const void* values)
{
    if (count > 0 && !values)
        fail(PM_INVALID_ARGUMENT, "cooToCsr GPU triplet pointers must be non-null");
}

void check_metadata(int64_t rows, int64_t cols, int64_t count)
{
    if (rows < 0 || cols < 0 || count < 0)
        fail(PM_INVALID_ARGUMENT, "cooToCsr GPU dimensions must be non-negative");
    if (count > INT_MAX || rows >= INT_MAX || cols > int64_t(UINT32_MAX))
        fail(PM_OVERFLOW_ERROR, "cooToCsr GPU dimensions exceed the supported packed-key range");
}

template <typename T>
void coo_prepare(pm_sparse_workspace* ws, cudaStream_t stream, int64_t rows, int64_t cols, int64_t count,
                 const int64_t* row_indices, const int64_t* col_indices, const T* values, bool keep_sorted, bool filled)
{
    if (!ws)
        fail(PM_INVALID_ARGUMENT, "cooToCsr GPU workspace is null");
    check_metadata(rows, cols, count);
    if (ws->status_pending)
        fail(PM_LOGIC_ERROR, "SparseOpsWorkspace status must be checked before another COO conversion");
    if (count > 0 && (!row_indices || !col_indices))
        fail(PM_INVALID_ARGUMENT, "cooToCsr GPU triplet pointers must be non-null");
    const size_t scan_bytes = scan_scratch_bytes(rows + 1, sizeof(int64_t)) + scan_scratch_bytes(rows + 1, sizeof(int));
    const size_t n = static_cast<size_t>(count > 0 ? count : 1);
    const size_t R = static_cast<size_t>(rows + 1);
    Carver plan;
    plan.take<CooStatus>(1);
    plan.take<int>(R);
    plan.take<int>(R + 1);
    plan.take<int>(n);
    plan.take<uint64_t>(n);
    plan.take<T>(n);
    plan.take<uint64_t>(n);
    plan.take<T>(n);
    plan.take<int>(R);
    plan.take<int>(R);
    plan.take<int64_t>(R + 1);
    plan.take<char>(scan_bytes);
    plan.take<CooRec<T>>(n);
    ws->buffer.ensure(plan.offset + 256, stream, "SparseOpsWorkspace");
    Carver carve;
    carve.base = static_cast<char*>(ws->buffer.ptr);
    ws->status = carve.take<CooStatus>(1);
    ws->bucket_sizes = carve.take<int>(R);
    ws->bucket_start = carve.take<int>(R + 1);
    ws->slots = carve.take<int>(n);
    ws->keys = carve.take<uint64_t>(n);
    ws->values = carve.take<T>(n);
    ws->spare_keys = carve.take<uint64_t>(n);
    ws->spare_values = carve.take<T>(n);
    ws->unique_count = carve.take<int>(R);
    ws->long_rows = carve.take<int>(R);
    ws->row_offsets = carve.take<int64_t>(R + 1);
    ws->scan_scratch = carve.take<char>(scan_bytes);
    CooRec<T>* recs = carve.take<CooRec<T>>(n);
    ws->recs = recs;
    ws->short_rows_kept = keep_sorted;
    ws->rows = rows;
    ws->cols = cols;
    ws->count = count;
    ws->value_size = sizeof(T);

    init_kernel<<<grid_for(count > 0 ? rows : 1, 256, 4 * sm_count()), 256, 0, stream>>>(ws->status, ws->bucket_sizes,
                                                                                         count > 0 ? rows : 0);
    PM_LAUNCH_CHECK();
    ws->status_pending = true;
    ws->prepared = true;
    if (count == 0)
    {
        // empty input: every bucket is empty (callers read bucket_start / unique_count)
        PM_CUDA(cudaMemsetAsync(ws->bucket_start, 0, (rows + 1) * sizeof(int), stream));
        PM_CUDA(cudaMemsetAsync(ws->unique_count, 0, (rows > 0 ? rows : 1) * sizeof(int), stream));
        PM_CUDA(cudaMemsetAsync(ws->row_offsets, 0, (rows + 1) * sizeof(int64_t), stream));
        finish_status_kernel<<<1, 1, 0, stream>>>(ws->row_offsets, rows, -1, ws->status, nullptr);
        PM_LAUNCH_CHECK();
        return;
    }
    T* sorted_values = static_cast<T*>(ws->values);
    count_kernel<<<grid_for(count, 256), 256, 0, stream>>>(row_indices, count, rows, ws->bucket_sizes, ws->slots,
                                                           ws->status);
    PM_LAUNCH_CHECK();
    exclusive_scan<int, int>(ws->bucket_sizes, ws->bucket_start, rows, ws->scan_scratch, stream);
    {
        const int64_t window = kScatterWindow / sizeof(CooRec<T>);
        const bool windows = count > window && count <= kScatterPasses * window;
        // four triplets per thread once they fill the chip (2,048 threads per SM)
        const bool many = count > int64_t(sm_count()) * 2048 * 4;
        const unsigned groups = grid_for(count, 4 * 256);
        int2* const ranges = reinterpret_cast<int2*>(ws->keys); // written by the sorts, after the passes
        if (many)
            scatter_kernel<T, 4><<<groups, 256, 0, stream>>>(row_indices, col_indices, values, count, cols, ws->slots,
                                                             ws->bucket_start, recs, windows ? window : count, ranges,
                                                             ws->status);
        else
            scatter_kernel<T, 1><<<grid_for(count, 256), 256, 0, stream>>>(row_indices, col_indices, values, count,
                                                                           cols, ws->slots, ws->bucket_start, recs,
                                                                           count, ranges, ws->status);
        PM_LAUNCH_CHECK();
        for (int64_t lo = window; windows && lo < count; lo += window)
        {
            scatter_window_kernel<T, 4><<<groups, 256, 0, stream>>>(col_indices, values, count, ws->slots, recs, lo,
                                                                    lo + window, ranges);
            PM_LAUNCH_CHECK();
        }
    }
    if (rows > 0)
    {
        if (keep_sorted)
            sort_short_kernel<T><<<grid_for(rows, 128), 128, 0, stream>>>(ws->bucket_start, rows, recs, ws->keys,
                                                                          sorted_values, ws->unique_count,
                                                                          ws->long_rows, ws->status);
        else
            count_short_kernel<T><<<grid_for(rows, 32 * kTileWarps), 32 * kTileWarps, 0, stream>>>(
                ws->bucket_start, rows, recs, ws->unique_count, ws->long_rows, ws->status);
        PM_LAUNCH_CHECK();
        sort_long_kernel<T><<<2 * sm_count(), kLongThreads, 0, stream>>>(
            ws->bucket_start, recs, ws->keys, sorted_values, ws->spare_keys, static_cast<T*>(ws->spare_values),
            ws->unique_count, ws->long_rows, ws->status);
        PM_LAUNCH_CHECK();
    }
    exclusive_scan<int, int64_t>(ws->unique_count, ws->row_offsets, rows, ws->scan_scratch, stream);
    if (filled)
        return; // the fill that follows writes the status
    finish_status_kernel<<<1, 1, 0, stream>>>(ws->row_offsets, rows, -1, ws->status, nullptr);
    PM_LAUNCH_CHECK();
}

template void coo_prepare<float>(pm_sparse_workspace*, cudaStream_t, int64_t, int64_t, int64_t, const int64_t*,
                                  const int64_t*, const float*, bool, bool);
template void coo_prepare<double>(pm_sparse_workspace*, cudaStream_t, int64_t, int64_t, int64_t, const int64_t*,
                                   const int64_t*, const double*, bool, bool);

CooView coo_view(const pm_sparse_workspace* ws)
{
    return CooView{ws->rows, ws->count, ws->bucket_start, ws->keys, ws->unique_count, ws->row_offsets};
}

// Host read of the status of an internal (sort-only) use of the workspace.
int64_t coo_internal_status(pm_sparse_workspace* ws, cudaStream_t stream, const char* operation)
{
    CooStatus status{};
    PM_CUDA(cudaMemcpyAsync(&status, ws->status, sizeof(status), cudaMemcpyDeviceToHost, stream));
    PM_CUDA(cudaStreamSynchronize(stream));
    ws->status_pending = false;
    if (status.invalid_source != kNoOffset)
    {
        std::ostringstream m;
        m << operation << ": block index out of range at entry " << status.invalid_source;
        fail(PM_OUT_OF_RANGE, m.str());
    }
    return status.actual_nnz;
}

namespace
{

template <typename T>
void coo_fill(pm_sparse_workspace* ws, cudaStream_t stream, int64_t nnz, int64_t* row_offsets, int64_t* col_out,
              T* val_out, bool async_api)
{
    if (!ws || !ws->prepared)
        fail(PM_LOGIC_ERROR, "cooToCsr fill requires a preceding count on the same workspace");
    if (ws->value_size != static_cast<int>(sizeof(T)))
        fail(PM_INVALID_ARGUMENT, "cooToCsr fill scalar type differs from the counted triplets");
    ws->buffer.bind(stream, "SparseOpsWorkspace");
    if (nnz < 0)
        fail(PM_INVALID_ARGUMENT, "cooToCsr output nnz must be non-negative");
    if (ws->count == 0 && nnz != 0)
        fail(PM_RUNTIME_ERROR, "cooToCsrAsync empty input requires output nnz=0");
    if (!row_offsets || (nnz > 0 && (!col_out || !val_out)))
        fail(PM_INVALID_ARGUMENT, "cooToCsr output pointers must be non-null");
    finish_status_kernel<<<grid_for(ws->rows + 1, 256, 8 * sm_count()), 256, 0, stream>>>(ws->row_offsets, ws->rows, nnz,
                                                                                          ws->status, row_offsets);
    PM_LAUNCH_CHECK();
    if (ws->count == 0 || ws->rows == 0)
        return;
    const T* sorted_values = static_cast<const T*>(ws->values);
    if (ws->short_rows_kept)
        write_short_kernel<T><<<grid_for(ws->rows, 128), 128, 0, stream>>>(ws->bucket_start, ws->rows, ws->keys,
                                                                           sorted_values, ws->row_offsets, nnz,
                                                                           col_out, val_out, ws->status);
    else
    {
        constexpr size_t kSmem = kTileWarps * kTileRecs * sizeof(CooRec<T>);
        static_assert(kSmem <= 48 * 1024, "the default shared memory of a kernel");
        write_short_resort_kernel<T><<<grid_for(ws->rows, 32 * kTileWarps), 32 * kTileWarps, kSmem, stream>>>(
            ws->bucket_start, ws->rows, static_cast<const CooRec<T>*>(ws->recs), ws->row_offsets, nnz, col_out,
            val_out, ws->status);
    }
    PM_LAUNCH_CHECK();
    write_long_kernel<T><<<2 * sm_count(), kLongThreads, 0, stream>>>(ws->bucket_start, ws->keys, sorted_values,
                                                                      ws->row_offsets, nnz, col_out, val_out,
                                                                      ws->long_rows, ws->status);
    PM_LAUNCH_CHECK();
    (void)async_api;
}

template <typename T>
int coo_async(pm_sparse_workspace* ws, cudaStream_t stream, int64_t rows, int64_t cols, int64_t count,
              const int64_t* ri, const int64_t* ci, const T* v, int64_t nnz, int64_t* ro, int64_t* co, T* vo)
{
    return guarded([&] {
        if (v && vo && static_cast<const void*>(v) == static_cast<const void*>(vo))
            fail(PM_INVALID_ARGUMENT, "cooToCsrAsync values and output must not alias");
        if (count == 0 && nnz != 0)
        {
            check_metadata(rows, cols, count);
            fail(PM_RUNTIME_ERROR, "cooToCsrAsync empty input requires output nnz=0");
        }
        require_values(count, v);
        // an output that the fill refuses leaves the count behind it, with its status
        const bool fills = nnz >= 0 && ro && (nnz == 0 || (co && vo));
        coo_prepare<T>(ws, stream, rows, cols, count, ri, ci, v, false, fills);
        coo_fill<T>(ws, stream, nnz, ro, co, vo, true);
    });
}

} // namespace
} // namespace pm

extern "C" {

int pm_sparse_workspace_create(pm_sparse_workspace** out)
{
    return pm::guarded([&] {
        if (!out)
            pm::fail(PM_INVALID_ARGUMENT, "workspace output pointer is null");
        *out = new pm_sparse_workspace();
    });
}

void pm_sparse_workspace_destroy(pm_sparse_workspace* ws)
{
    if (ws)
    {
        ws->buffer.release();
        delete ws;
    }
}

int pm_sparse_workspace_close(pm_sparse_workspace* ws)
{
    return pm::guarded([&] {
        if (!ws)
            pm::fail(PM_INVALID_ARGUMENT, "workspace is null");
        ws->buffer.release();
        ws->status_pending = false;
        ws->prepared = false;
    });
}

size_t pm_sparse_workspace_capacity(const pm_sparse_workspace* ws) { return ws ? ws->buffer.bytes : 0; }

int pm_coo_to_csr_count_f32(pm_sparse_workspace* ws, pm_stream_t stream, int64_t rows, int64_t cols, int64_t count,
                            const int64_t* ri, const int64_t* ci, const float* v)
{
    return pm::guarded([&] {
        pm::require_values(count, v);
        pm::coo_prepare<float>(ws, stream, rows, cols, count, ri, ci, v, false);
    });
}
int pm_coo_to_csr_count_f64(pm_sparse_workspace* ws, pm_stream_t stream, int64_t rows, int64_t cols, int64_t count,
                            const int64_t* ri, const int64_t* ci, const double* v)
{
    return pm::guarded([&] {
        pm::require_values(count, v);
        pm::coo_prepare<double>(ws, stream, rows, cols, count, ri, ci, v, false);
    });
}
int pm_coo_to_csr_fill_f32(pm_sparse_workspace* ws, pm_stream_t stream, int64_t nnz, int64_t* ro, int64_t* co,
                           float* vo)
{
    return pm::guarded([&] {
        if (ws)
            ws->status_pending = true;
        pm::coo_fill<float>(ws, stream, nnz, ro, co, vo, false);
    });
}
int pm_coo_to_csr_fill_f64(pm_sparse_workspace* ws, pm_stream_t stream, int64_t nnz, int64_t* ro, int64_t* co,
                           double* vo)
{
    return pm::guarded([&] {
        if (ws)
            ws->status_pending = true;
        pm::coo_fill<double>(ws, stream, nnz, ro, co, vo, false);
    });
}
int pm_coo_to_csr_async_f32(pm_sparse_workspace* ws, pm_stream_t stream, int64_t rows, int64_t cols, int64_t count,
                            const int64_t* ri, const int64_t* ci, const float* v, int64_t nnz, int64_t* ro,
                            int64_t* co, float* vo)
{
    return pm::coo_async<float>(ws, stream, rows, cols, count, ri, ci, v, nnz, ro, co, vo);
}
int pm_coo_to_csr_async_f64(pm_sparse_workspace* ws, pm_stream_t stream, int64_t rows, int64_t cols, int64_t count,
                            const int64_t* ri, const int64_t* ci, const double* v, int64_t nnz, int64_t* ro,
                            int64_t* co, double* vo)
{
    return pm::coo_async<double>(ws, stream, rows, cols, count, ri, ci, v, nnz, ro, co, vo);
}

int pm_coo_status(pm_sparse_workspace* ws, const char* operation, int64_t* nnz_out)
{
    return pm::guarded([&] {
        if (!ws)
            pm::fail(PM_INVALID_ARGUMENT, "workspace is null");
        const char* name = operation ? operation : "cooToCsrAsync";
        if (nnz_out)
            *nnz_out = 0;
        if (!ws->buffer.bound || !ws->status)
            return;
        const cudaError_t query = cudaStreamQuery(ws->buffer.stream);
        if (query == cudaErrorNotReady)
            pm::fail(PM_LOGIC_ERROR, "SparseOpsWorkspace::checkStatus requires stream synchronization first");
        PM_CUDA(query);
        pm::CooStatus status{};
        PM_CUDA(cudaMemcpy(&status, ws->status, sizeof(status), cudaMemcpyDeviceToHost));
        ws->status_pending = false;
        if (nnz_out)
            *nnz_out = status.actual_nnz;
        if (status.invalid_source != pm::kNoOffset)
        {
            std::ostringstream m;
            m << name << ": coordinate out of range at source offset " << status.invalid_source;
            ws->prepared = false;
            pm::fail(PM_OUT_OF_RANGE, m.str());
        }
        if (status.invalid_value != pm::kNoOffset)
        {
            std::ostringstream m;
            m << name << ": non-finite value at source offset " << status.invalid_value;
            ws->prepared = false;
            pm::fail(PM_INVALID_ARGUMENT, m.str());
        }
        if (status.mismatch_actual != pm::kNoOffset)
        {
            std::ostringstream m;
            m << name << ": output nnz is " << status.mismatch_expected << ", but duplicate-combined nnz is "
              << status.mismatch_actual;
            pm::fail(PM_RUNTIME_ERROR, m.str());
        }
    });
}

} // extern "C"

// =========================================================================== allocation-free variant
// COO -> CSR for callers that must not allocate device memory at call time: for example a
// host application that hands the library a fixed device-memory budget at start-up and owns
// every allocation after that, or a latency-critical loop where a cudaMalloc could block or
// fail in the middle of a run.  The scratch of the conversion (row buckets, sort keys, scan
// partials, status) lives in one file-scope device array of kStaticScratchBytes, created when
// the library's device code is loaded on a GPU and held by every GPU that loads the library
// until the process exits.  Inputs are limited to kStaticMaxTriplets triplets and
// kStaticMaxRows rows so that the scratch always fits.  All calls share the array: calls
// that overlap on one GPU, from any stream or host thread, race on it, so serialise them;
// each device has its own copy.  Each call clears what must start at zero.
namespace pm
{
namespace
{
constexpr int64_t kStaticMaxTriplets = 65536;
constexpr int64_t kStaticMaxRows = 65536;
constexpr size_t kStaticScratchBytes = size_t(8) << 20;
} // namespace
} // namespace pm

static __device__ __align__(256) unsigned char g_static_coo_scratch[pm::kStaticScratchBytes];

namespace pm
{
namespace
{

// Device address of g_static_coo_scratch in the current device's context.  The host-side name
// of the array is only a stand-in, so the address is looked up with that device current.  It
// is looked up on every call (cudaGetSymbolAddress allocates nothing): a cached address would
// outlive a cudaDeviceReset, after which the module is loaded again and the array may move.
// The first call on a device loads the library's device code there; issue that first call
// before any stream capture.
void* static_scratch_address()
{
    void* address = nullptr;
    const cudaError_t rc = cudaGetSymbolAddress(&address, g_static_coo_scratch);
    if (rc != cudaSuccess || !address)
        fail(PM_CUDA_ERROR, std::string("cudaGetSymbolAddress(static COO scratch): ") + cudaGetErrorString(rc));
    return address;
}

// Bytes coo_prepare carves for (rows, count) triplets of type T (same layout, same order).
template <typename T>
size_t static_plan_bytes(int64_t rows, int64_t count)
{
    const size_t scan_bytes = scan_scratch_bytes(rows + 1, sizeof(int64_t)) + scan_scratch_bytes(rows + 1, sizeof(int));
    const size_t n = static_cast<size_t>(count > 0 ? count : 1);
    const size_t R = static_cast<size_t>(rows + 1);
    Carver plan;
    plan.take<CooStatus>(1);
    plan.take<int>(R);
    plan.take<int>(R + 1);
    plan.take<int>(n);
    plan.take<uint64_t>(n);
    plan.take<T>(n);
    plan.take<uint64_t>(n);
    plan.take<T>(n);
    plan.take<int>(R);
    plan.take<int>(R);
    plan.take<int64_t>(R + 1);
    plan.take<char>(scan_bytes);
    plan.take<CooRec<T>>(n);
    return plan.offset + 256;
}

template <typename T>
void coo_static(cudaStream_t stream, int64_t rows, int64_t cols, int64_t count, const int64_t* ri, const int64_t* ci,
                const T* v, int64_t capacity, int64_t* ro, int64_t* co, T* vo, int64_t* nnz_out)
{
    check_metadata(rows, cols, count);
    if (count > kStaticMaxTriplets || rows > kStaticMaxRows)
    {
        std::ostringstream m;
        m << "cooToCsr (static scratch): at most " << kStaticMaxTriplets << " triplets and " << kStaticMaxRows
          << " rows are supported, got " << count << " triplets and " << rows << " rows";
        fail(PM_INVALID_ARGUMENT, m.str());
    }
    require_values(count, v);
    if (capacity < 0 || !ro || (capacity > 0 && (!co || !vo)))
        fail(PM_INVALID_ARGUMENT, "cooToCsr (static scratch): output pointers must be non-null");
    if (v && vo && static_cast<const void*>(v) == static_cast<const void*>(vo))
        fail(PM_INVALID_ARGUMENT, "cooToCsrAsync values and output must not alias");
    const size_t need = static_plan_bytes<T>(rows, count);
    if (need > kStaticScratchBytes)
        fail(PM_INVALID_ARGUMENT, "cooToCsr (static scratch): scratch plan exceeds the static array");
    // a workspace whose storage is the static array: it never grows, so nothing is allocated
    void* const base = static_scratch_address();
    pm_sparse_workspace ws;
    ws.buffer.ptr = base;
    ws.buffer.bytes = kStaticScratchBytes;
    coo_prepare<T>(&ws, stream, rows, cols, count, ri, ci, v, false);
    PM_CUDA(cudaStreamSynchronize(stream));
    int64_t nnz = 0;
    int status = pm_coo_status(&ws, "cooToCsr", &nnz);
    if (status != PM_OK)
        throw Error(status, pm_last_error());
    if (nnz > capacity)
    {
        std::ostringstream m;
        m << "cooToCsr (static scratch): output capacity " << capacity << " is below the duplicate-combined nnz "
          << nnz;
        fail(PM_RUNTIME_ERROR, m.str());
    }
    ws.status_pending = true;
    coo_fill<T>(&ws, stream, nnz, ro, co, vo, false);
    PM_CUDA(cudaStreamSynchronize(stream));
    if (ws.buffer.ptr != base)
        fail(PM_RUNTIME_ERROR, "cooToCsr (static scratch): scratch storage changed unexpectedly");
    status = pm_coo_status(&ws, "cooToCsr", nullptr);
    if (status != PM_OK)
        throw Error(status, pm_last_error());
    if (nnz_out)
        *nnz_out = nnz;
}

} // namespace
} // namespace pm

extern "C" {

int pm_coo_to_csr_static_f32(pm_stream_t stream, int64_t rows, int64_t cols, int64_t count, const int64_t* ri,
                             const int64_t* ci, const float* v, int64_t capacity, int64_t* ro, int64_t* co, float* vo,
                             int64_t* nnz_out)
{
    return pm::guarded([&] { pm::coo_static<float>(stream, rows, cols, count, ri, ci, v, capacity, ro, co, vo, nnz_out); });
}

int pm_coo_to_csr_static_f64(pm_stream_t stream, int64_t rows, int64_t cols, int64_t count, const int64_t* ri,
                             const int64_t* ci, const double* v, int64_t capacity, int64_t* ro, int64_t* co, double* vo,
                             int64_t* nnz_out)
{
    return pm::guarded([&] { pm::coo_static<double>(stream, rows, cols, count, ri, ci, v, capacity, ro, co, vo, nnz_out); });
}

} // extern "C"
