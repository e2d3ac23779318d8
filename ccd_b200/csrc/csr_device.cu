// csr_device.cu -- the row-major copy of the matrix (computeXBeta's row sums,
// the MM cycle; ModelSpecifics.hpp:313-361 walks the columns per row) built on
// the device from the uploaded column-major arrays.
//
// Pass 1 counts each row's entries (one CTA per column, an atomic add per
// entry: within a column a row appears once), and a CTA per tile of rows turns
// the counts into row offsets (an exclusive scan) and finds the longest row.  Pass 2 places every entry at its row's cursor (an atomic
// fetch-add; the order inside a row is then the arrival order) and sorts each
// row by column with one thread per row.  A row holds each column at most
// once, so the sorted layout is unique: per row the columns in increasing
// order, the same bytes as the host build (csr_host.cpp) whatever the
// arrival order.  Insertion sort is near linear here because the CTAs of
// pass 2 start in column order.
#include "csr_device.h"

#include <cstdint>

#include "types.h"

namespace ccdb {
namespace {

constexpr int kCT = 256;         // threads of the per-column kernels
constexpr int kST = 1024;        // threads of the scan
constexpr int kSPer = 4;         // rows per scan thread
constexpr int kTile = kST * kSPer;

struct ColRange {
    int64_t cb, vb, n;
    bool has_rows, has_vals;
};

__device__ __forceinline__ ColRange col_range(const CsrDeviceArgs& a, int j) {
    ColRange c;
    const uint8_t f = a.fmt[j];
    c.has_rows = (f == F_SPARSE || f == F_INDICATOR);
    c.has_vals = (f == F_SPARSE || f == F_DENSE);
    c.cb = a.col_ptr[j];
    c.vb = a.val_ptr[j];
    c.n = c.has_rows ? a.col_ptr[j + 1] - c.cb : a.K;
    return c;
}

__global__ void __launch_bounds__(kCT) csr_count_kernel(CsrDeviceArgs a, int32_t* counts) {
    for (int j = blockIdx.x; j < a.J; j += gridDim.x) {
        const ColRange c = col_range(a, j);
        for (int64_t p = threadIdx.x; p < c.n; p += kCT) {
            const int64_t k = c.has_rows ? (int64_t)__ldg(a.rows + c.cb + p) : p;
            atomicAdd(counts + k, 1);
        }
    }
}

// Entries of each tile of kTile rows, and the longest row.
__global__ void __launch_bounds__(kST) csr_tile_kernel(const int32_t* counts, int64_t K, int64_t* tile_sum,
                                                        int32_t* max_row) {
    __shared__ int64_t s_sum[kST / 32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t r0 = (int64_t)blockIdx.x * kTile + (int64_t)tid * kSPer;
    int64_t sum = 0;
    int32_t longest = 0;
#pragma unroll
    for (int i = 0; i < kSPer; ++i) {
        const int32_t c = (r0 + i < K) ? counts[r0 + i] : 0;
        sum += c;
        longest = max(longest, c);
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) {
        s_sum[wid] = sum;
        atomicMax(max_row, longest);
    }
    __syncthreads();
    if (tid == 0) {
        int64_t t = 0;
        for (int w = 0; w < kST / 32; ++w) t += s_sum[w];
        tile_sum[blockIdx.x] = t;
    }
}

// The exclusive scan of one tile: each thread has a run of kSPer rows, the thread
// sums are scanned across the CTA (warp shuffles, then the warp totals), and the
// tiles before it are added up by the CTA itself, so the tiles need no order.
// 130,000 rows: 12 us for both kernels, where one CTA that walked the tiles took 170.
__global__ void __launch_bounds__(kST) csr_scan_kernel(const int32_t* counts, int64_t K, const int64_t* tile_sum,
                                                        int64_t* row_ptr, int64_t* cursor) {
    __shared__ int64_t s_warp[kST / 32], s_part[kST / 32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    int64_t before = 0;
    for (int t = tid; t < (int)blockIdx.x; t += kST) before += tile_sum[t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 0) s_part[wid] = before;
    const int64_t r0 = (int64_t)blockIdx.x * kTile + (int64_t)tid * kSPer;
    int32_t c[kSPer];
    int64_t mine = 0;
#pragma unroll
    for (int i = 0; i < kSPer; ++i) {
        c[i] = (r0 + i < K) ? counts[r0 + i] : 0;
        mine += c[i];
    }
    // inclusive scan of the thread sums within the warp
    int64_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    int64_t at = incl - mine;
    for (int w = 0; w < kST / 32; ++w) at += s_part[w] + (w < wid ? s_warp[w] : 0);
#pragma unroll
    for (int i = 0; i < kSPer; ++i)
        if (r0 + i < K) {
            row_ptr[r0 + i] = at;
            cursor[r0 + i] = at;
            at += c[i];
            if (r0 + i == K - 1) row_ptr[K] = at;
        }
}

__global__ void __launch_bounds__(kCT) csr_place_kernel(CsrDeviceArgs a, int64_t* cursor, int32_t* col,
                                                         double* val) {
    for (int j = blockIdx.x; j < a.J; j += gridDim.x) {
        const ColRange c = col_range(a, j);
        for (int64_t p = threadIdx.x; p < c.n; p += kCT) {
            const int64_t k = c.has_rows ? (int64_t)__ldg(a.rows + c.cb + p) : p;
            const double x = c.has_vals ? __ldg(a.vals + c.vb + p) : 1.0;
            const int64_t q = (int64_t)atomicAdd(reinterpret_cast<unsigned long long*>(cursor + k), 1ull);
            col[q] = j;
            val[q] = x;
        }
    }
}

// One thread per row: insertion sort of the row's (column, value) pairs by
// column (columns are distinct within a row).
// Without values every one is 1, and only the columns move (2.6 million entries: 54
// us, 112 with the values).
template <bool VALUES>
__global__ void __launch_bounds__(kCT) csr_sort_kernel(const int64_t* row_ptr, int64_t K, int32_t* col,
                                                        double* val) {
    for (int64_t k = (int64_t)blockIdx.x * kCT + threadIdx.x; k < K; k += (int64_t)gridDim.x * kCT) {
        const int64_t lo = row_ptr[k], hi = row_ptr[k + 1];
        for (int64_t i = lo + 1; i < hi; ++i) {
            const int32_t cj = col[i];
            const double vj = VALUES ? val[i] : 1.0;
            int64_t q = i - 1;
            while (q >= lo && col[q] > cj) {
                col[q + 1] = col[q];
                if (VALUES) val[q + 1] = val[q];
                --q;
            }
            col[q + 1] = cj;
            if (VALUES) val[q + 1] = vj;
        }
    }
}

unsigned col_grid(int32_t J) { return (unsigned)(J < 65535 ? (J > 0 ? J : 1) : 65535); }

}  // namespace

cudaError_t csr_device_count(const CsrDeviceArgs& a, int32_t* counts, int64_t* tile_sum, int64_t* row_ptr,
                             int64_t* cursor, int32_t* max_row, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(counts, 0, sizeof(int32_t) * (size_t)(a.K > 0 ? a.K : 1), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(max_row, 0, sizeof(int32_t), s);
    if (e != cudaSuccess) return e;
    csr_count_kernel<<<col_grid(a.J), kCT, 0, s>>>(a, counts);
    const unsigned tiles = (unsigned)((a.K + kTile - 1) / kTile);
    csr_tile_kernel<<<tiles, kST, 0, s>>>(counts, a.K, tile_sum, max_row);
    csr_scan_kernel<<<tiles, kST, 0, s>>>(counts, a.K, tile_sum, row_ptr, cursor);
    return cudaGetLastError();
}

int64_t csr_device_tiles(int64_t K) { return (K + kTile - 1) / kTile; }

cudaError_t csr_device_fill(const CsrDeviceArgs& a, const int64_t* row_ptr, int64_t* cursor, int32_t* col,
                            double* val, cudaStream_t s) {
    csr_place_kernel<<<col_grid(a.J), kCT, 0, s>>>(a, cursor, col, val);
    const int64_t blocks = (a.K + kCT - 1) / kCT;
    const unsigned grid = (unsigned)(blocks < 4096 ? (blocks > 0 ? blocks : 1) : 4096);
    if (a.has_values) csr_sort_kernel<true><<<grid, kCT, 0, s>>>(row_ptr, a.K, col, val);
    else csr_sort_kernel<false><<<grid, kCT, 0, s>>>(row_ptr, a.K, col, val);
    return cudaGetLastError();
}

}  // namespace ccdb
