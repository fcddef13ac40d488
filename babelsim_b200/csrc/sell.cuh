// Sliced-ELL ("SELL-32") storage of the off-diagonal part of a sparse matrix.
//
// Rows are grouped in slices of 32 (one warp).  Inside slice s every row is
// padded to the slice's widest row w_s and the slice is stored column-major:
// entry k of row 32 s + l sits at sptr[s] + 32 k + l.  A warp sweeping its
// slice therefore reads each column-index and value step as one contiguous
// 128-byte (int32) / 256-byte (FP64) or 128-byte (FP32) transaction, one thread
// per row, and issues its gathers four entries at a time.  Padding entries are
// (column = own row, value = 0), so they gather an already cached value and add
// nothing.  Rows past n in the last slice carry (column 0, value 0).
#pragma once

#include "bsg_internal.h"

#include <algorithm>
#include <vector>

namespace bsg {

constexpr int kSellC = 32;
// Entries each thread loads before it gathers (memory-level parallelism of a row sweep).
// 8 against 4: 39.5 against 40.5 ms per outer iteration on the 1M-cell cavity (6: 39.8).
#ifndef BSG_SELL_BATCH
#define BSG_SELL_BATCH 8
#endif
constexpr int kSellBatch = BSG_SELL_BATCH;

template <class T>
struct SellMat {
    int n = 0;
    int nslices = 0;
    const int* sptr = nullptr;  // nslices + 1 entry offsets
    const int* col = nullptr;
    const T* val = nullptr;
    const T* diag = nullptr;    // n
    bool stream = false;        // entries pass L1 by
};

// Entries of a large matrix pass L1 by: each is used once per sweep, and kept in L1 they push out the
// vectors that neighbouring rows gather.  A small one gains from what L1 still holds of it from the
// sweep before.  By bytes of entries, kept / passed by (ms of pressure and momentum solves per outer
// iteration): Voronoi 40 MB 9.1 / 10.4, 54 MB 10.0 / 10.6, 85 MB 15.9 / 15.1, 96 MB 16.7 / 15.6, 228 MB
// 33.1 / 32.6; 2D cavity 39 MB 7.5 / 7.8; momentum and k-omega on a 1M-cell channel, 74 MB, 11.7 / 10.2.
inline bool sellStreams(long long entries, int value_bytes) { return entries * (4 + value_bytes) > (64LL << 20); }

// Slice offsets (entries) of a CSR pattern.
inline std::vector<int> sellOffsets(int rows, const int* ptr) {
    const int nslices = (rows + kSellC - 1) / kSellC;
    std::vector<int> sptr(nslices + 1, 0);
    for (int s = 0; s < nslices; ++s) {
        int w = 0;
        for (int i = kSellC * s; i < std::min(rows, kSellC * (s + 1)); ++i) w = std::max(w, ptr[i + 1] - ptr[i]);
        sptr[s + 1] = sptr[s] + kSellC * w;
    }
    return sptr;
}

#ifdef __CUDACC__
// A matrix entry's load, past L1 if STREAM (see sellStreams).
__device__ __forceinline__ int streamLoad(const int* p) {
    int x;
    asm("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(x) : "l"(p));
    return x;
}
__device__ __forceinline__ float streamLoad(const float* p) {
    float x;
    asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(x) : "l"(p));
    return x;
}
__device__ __forceinline__ double streamLoad(const double* p) {
    double x;
    asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(x) : "l"(p));
    return x;
}
template <bool STREAM, class T>
__device__ __forceinline__ T entryLoad(const T* p) {
    return STREAM ? streamLoad(p) : __ldg(p);
}
// sum_k a_ik y(col_ik) over this lane's row of slice s (lane = row within the slice).
// Entries go in batches of kSellBatch: all index and value loads of a batch first, then
// all its gathers; the entries past the last full batch follow one at a time.  (A
// predicated last batch, which would shorten a row's chain of dependent load rounds,
// measured slower on the 1M-cell pressure solves: 36.8 against 31.0 ms per outer
// iteration.)
template <bool STREAM, class T, class Y>
__device__ __forceinline__ T sellRowAs(const SellMat<T>& A, int s, int lane, Y y) {
    const int beg = A.sptr[s];
    const int w = (A.sptr[s + 1] - beg) >> 5;
    const int* __restrict__ c = A.col + beg + lane;
    const T* __restrict__ v = A.val + beg + lane;
    T a0 = T(0), a1 = T(0);
    int k = 0;
    for (; k + kSellBatch <= w; k += kSellBatch) {
        int cc[kSellBatch];
        T vv[kSellBatch];
#pragma unroll
        for (int u = 0; u < kSellBatch; ++u) {
            cc[u] = entryLoad<STREAM>(c + 32 * (k + u));
            vv[u] = entryLoad<STREAM>(v + 32 * (k + u));
        }
        T yy[kSellBatch];
#pragma unroll
        for (int u = 0; u < kSellBatch; ++u) yy[u] = y(cc[u]);
#pragma unroll
        for (int u = 0; u < kSellBatch; u += 2) {
            a0 += vv[u] * yy[u];
            if (u + 1 < kSellBatch) a1 += vv[u + 1] * yy[u + 1];
        }
    }
    for (; k < w; ++k) a0 += entryLoad<STREAM>(v + 32 * k) * y(entryLoad<STREAM>(c + 32 * k));
    return a0 + a1;
}
template <class T, class Y>
__device__ __forceinline__ T sellRow(const SellMat<T>& A, int s, int lane, Y y) {
    return A.stream ? sellRowAs<true>(A, s, lane, y) : sellRowAs<false>(A, s, lane, y);
}

// The same row sum split over K consecutive lanes (K a power of two, 2..32): lane q
// of the group takes entries q, q + K, ... of row r of slice s, and the group's
// partial sums are combined in a fixed butterfly order, so every lane of the
// group returns the same, deterministic total.  For levels whose slices leave
// warps idle: the dependent index -> gather chain of a wide row gets K times
// shorter.  Every lane of the warp must call it (the butterfly uses the full mask).
template <class T, class Y>
__device__ __forceinline__ T sellRowSplit(const SellMat<T>& A, int s, int r, int q, int K, Y y) {
    const int beg = A.sptr[s];
    const int w = (A.sptr[s + 1] - beg) >> 5;
    const int* __restrict__ c = A.col + beg + r;
    const T* __restrict__ v = A.val + beg + r;
    T a0 = T(0), a1 = T(0);
    int k = q;
    for (; k + K < w; k += 2 * K) {
        const int c0 = __ldg(c + 32 * k), c1 = __ldg(c + 32 * (k + K));
        const T v0 = __ldg(v + 32 * k), v1 = __ldg(v + 32 * (k + K));
        const T y0 = y(c0), y1 = y(c1);
        a0 += v0 * y0;
        a1 += v1 * y1;
    }
    if (k < w) a0 += __ldg(v + 32 * k) * y(__ldg(c + 32 * k));
    T a = a0 + a1;
    for (int o = K >> 1; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

// Padded columns of a CSR pattern, one block per slice: padding entries hold their own row, rows
// past n column 0.
static __global__ void kSellColumns(int n, const int* __restrict__ ptr, const int* __restrict__ col,
                                    const int* __restrict__ sptr, int* __restrict__ scol) {
    const int s = blockIdx.x, beg = sptr[s], count = sptr[s + 1] - beg;
    for (int e = threadIdx.x; e < count; e += blockDim.x) {
        const int i = kSellC * s + (e & 31), k = e >> 5;
        int c = 0;
        if (i < n) c = k < ptr[i + 1] - ptr[i] ? col[ptr[i] + k] : i;
        scol[beg + e] = c;
    }
}
inline void sellColumns(int n, const int* ptr, const int* col, const int* sptr, int* scol, cudaStream_t stream) {
    if (n > 0) kSellColumns<<<(n + kSellC - 1) / kSellC, 128, 0, stream>>>(n, ptr, col, sptr, scol);
    BSG_CUDA(cudaGetLastError());
}

// Values of a CSR matrix (FP64) scattered into SELL positions, converted to T;
// diag and omega/diag converted alongside.  Padding entries are never written.
template <class T>
__global__ void kCsrToSell(int n, const int* __restrict__ ptr, const double* __restrict__ val,
                           const double* __restrict__ diag, const int* __restrict__ sptr, double omega,
                           T* __restrict__ sval, T* __restrict__ sdiag, T* __restrict__ rd) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int base = sptr[i >> 5] + (i & 31);
    const int k0 = ptr[i], len = ptr[i + 1] - k0;
    for (int j = 0; j < len; ++j) sval[base + 32 * j] = static_cast<T>(val[k0 + j]);
    if (sdiag) sdiag[i] = static_cast<T>(diag[i]);
    if (rd) rd[i] = static_cast<T>(omega / diag[i]);
}
#endif

}  // namespace bsg
