// CTA groups of the persistent solver kernels (device code, sm_100a).
//
// A persistent kernel runs one cooperative launch per solve and separates its
// phases by barriers instead of kernel launches.  GridGroup is the whole
// cooperative grid; SegmentGroup is a contiguous range of its CTAs that owns one
// system of a batch, so one launch can solve several independent systems side by
// side.  Both synchronise through groupBarrier, whose every wait is bounded, and
// gridSum is the deterministic reduction both use.
#pragma once

#include "bsg_internal.h"
#include "per_device.h"

#include <algorithm>

#ifdef __CUDACC__
#include <cooperative_groups.h>
#endif

namespace bsg {

// Thread-block clusters the small-system kernels run on: one system per cluster, at most
// this many CTAs (16 is the hardware's non-portable maximum).
constexpr int kMaxClusterCtas = 16;

// Systems of one batched launch: their arguments are one kernel argument (constant bank: read where they
// are used they take no registers; from global or shared memory they spilled the solvers' loops), which
// CUDA limits to kKernelArgumentBytes.
constexpr int kBatchArgs = 128;
constexpr std::size_t kKernelArgumentBytes = 32764;
#ifdef __CUDACC__
constexpr long long kBarrierCycles = 4000000000LL;  // about 2 s at the B200's clock

// Barrier of n CTAs on one word: every CTA adds 1 per barrier (red.release at gpu scope, after
// __syncthreads, so it covers the whole CTA's writes) and polls with acquiring loads until the
// count reaches its own barrier number times n (compared as a signed difference, so the count may
// wrap; it is zero before each launch).  Against an atomic whose result tells the phase, followed
// by relaxed polling and one fence, the reduction needs no round trip before the first poll and the
// loads no fence after the last: 1.98 against 2.20 us per barrier with one store before and one
// gather after it, 148 CTAs of 1024 threads (a release flag written by the last CTA: 2.48 us).
// All CTAs of a cooperative launch are resident, so the count is always reached unless a CTA
// skipped the barrier; the wait is bounded all the same: past kBarrierCycles the
// CTA records an abort (and, first of all, where it was and what it saw) and
// returns, and later barriers of the group stop waiting, so the launch ends and
// the host reports status 3 instead of hanging the GPU.
__device__ __forceinline__ void arriveRelease(unsigned* word) {
    asm volatile("red.add.release.gpu.global.u32 [%0], %1;" ::"l"(word), "r"(1u) : "memory");
}
__device__ __forceinline__ unsigned loadAcquire(const unsigned* word) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
    return v;
}

// Thread 0's barrier bookkeeping lives in shared memory, out of the registers of
// the kernels' hot loops: the number of this CTA's latest barrier and where the
// launch records it.
struct BarrierBook {
    unsigned seq;
    unsigned* progress;
};
__device__ __forceinline__ BarrierBook& barrierBook() {
    __shared__ BarrierBook book;
    return book;
}
__device__ __forceinline__ void openBarrierBook(const SegmentBarrier* bar) {
    if (threadIdx.x == 0) barrierBook() = BarrierBook{0u, bar->progress};
}

// Thread 0's part of a barrier: arrive, wait for the count (bounded), acquire.
// Returns 1 when it left on the group's abort (its own timeout or another CTA's).
__device__ __forceinline__ int arriveAndWait(SegmentBarrier* bar, int n) {
    if (n == 1) return 0;  // a group of one CTA: the block barriers around this call are enough
    arriveRelease(&bar->count);
    BarrierBook& book = barrierBook();
    const unsigned seq = ++book.seq, target = seq * static_cast<unsigned>(n);
    // recorded after the arrival, so the release above never waits on this store
    if (book.progress) book.progress[blockIdx.x] = seq;
    long long t0 = 0;
    for (unsigned spins = 1;; ++spins) {
        const unsigned cur = loadAcquire(&bar->count);
        if (static_cast<int>(cur - target) >= 0) return 0;
        if ((spins & 255u) != 0u) continue;
        if (*reinterpret_cast<volatile int*>(&bar->abort)) return 1;
        const long long now = clock64();
        if (spins == 256u) {
            t0 = now;
        } else if (now - t0 > kBarrierCycles) {
            if (atomicCAS(&bar->who, 0, static_cast<int>(blockIdx.x) + 1) == 0) {
                bar->where = seq;
                bar->seen = cur - (target - static_cast<unsigned>(n));  // arrivals at this barrier
            }
            __threadfence();
            atomicExch(&bar->abort, 1);
            return 1;
        }
    }
}

// Returns thread 0's result of arriveAndWait: the same value for every thread of
// the CTA, so a loop that stops on it stops in all of them.  Inlined: with one CTA per SM a call
// would save its caller's live registers to local memory around every barrier and read them back
// from L2 after it, since the acquire empties L1 (33k-cell PCG solves 3.37 against 2.77 ms, the
// 200k-cell O-grid's 49.8 against 41.9 ms).
__device__ __forceinline__ int groupBarrier(SegmentBarrier* bar, int n) {
    __shared__ int aborted;
    __syncthreads();
    if (threadIdx.x == 0) aborted = arriveAndWait(bar, n);
    __syncthreads();
    // the next write to `aborted` comes after the next barrier's first __syncthreads,
    // which every thread reaches only after this read
    return aborted;
}

// aborted(): this CTA has left a wait on the group's abort (sticky, uniform within
// the CTA; for stopping loops).  failed(): the group's flag in memory, read once
// at the end for the launch's status, since a CTA may pass every barrier it
// reaches after another CTA gave up.
struct GridGroup {
    SegmentBarrier* bar;
    int stop = 0;
    __device__ explicit GridGroup(SegmentBarrier* b) : bar(b) { openBarrierBook(b); }
    __device__ __forceinline__ int rank() const { return blockIdx.x; }
    __device__ __forceinline__ int size() const { return gridDim.x; }
    __device__ __forceinline__ bool aborted() const { return stop != 0; }
    __device__ __forceinline__ bool failed() const { return *reinterpret_cast<volatile int*>(&bar->abort) != 0; }
    __device__ __forceinline__ void sync() { stop |= groupBarrier(bar, gridDim.x); }
};

struct SegmentGroup {
    int cta0, ncta;
    SegmentBarrier* bar;
    int stop = 0;
    __device__ SegmentGroup(int c0, int n, SegmentBarrier* b) : cta0(c0), ncta(n), bar(b) { openBarrierBook(b); }
    __device__ __forceinline__ int rank() const { return blockIdx.x - cta0; }
    __device__ __forceinline__ int size() const { return ncta; }
    __device__ __forceinline__ bool aborted() const { return stop != 0; }
    __device__ __forceinline__ bool failed() const { return *reinterpret_cast<volatile int*>(&bar->abort) != 0; }
    __device__ __forceinline__ void sync() { stop |= groupBarrier(bar, ncta); }
};

// One thread-block cluster as a group: its barrier is the hardware's cluster barrier
// (release/acquire at cluster scope), 0.2-0.3 us for 16 CTAs against 1.3 us for the grid barrier
// above on 148 CTAs and 1.2 us for any barrier on a global word.  The CTAs of a cluster are
// scheduled together, so there is nothing to abort.
struct ClusterGroup {
    __device__ __forceinline__ int rank() const {
        unsigned r;
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
        return static_cast<int>(r);
    }
    __device__ __forceinline__ int size() const {
        unsigned r;
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
        return static_cast<int>(r);
    }
    __device__ __forceinline__ bool aborted() const { return false; }
    __device__ __forceinline__ bool failed() const { return false; }
    __device__ __forceinline__ void sync() {
        asm volatile(
            "barrier.cluster.arrive.release.aligned;\n\t"
            "barrier.cluster.wait.acquire.aligned;" ::
                : "memory");
    }
};

struct Lanes {
    int lane, gwarp, nwarps, gthread, nthreads;
};

template <int BS, class G>
__device__ __forceinline__ Lanes lanes(const G& g) {
    Lanes c;
    c.gthread = g.rank() * BS + threadIdx.x;
    c.nthreads = g.size() * BS;
    c.lane = threadIdx.x & 31;
    c.gwarp = c.gthread >> 5;
    c.nwarps = c.nthreads >> 5;
    return c;
}

// Lanes per row on a level: the largest power of two (at most 32) that still
// gives every (slice, lane-group) unit its own warp; 1 on the fine levels.
__device__ __forceinline__ int splitOf(int nslices, int nwarps) {
    int K = 1;
    while (K < 32 && static_cast<long long>(nslices) * K * 2 <= nwarps) K *= 2;
    return K;
}

// Unit u of a split sweep: slice s, the row r within it and this lane's part q.
struct SplitUnit {
    int s, r, q;
};
__device__ __forceinline__ SplitUnit splitUnit(int u, int K, int lane) {
    const int rows = 32 / K;
    return {u / K, (u % K) * rows + lane / K, lane % K};
}

// The device that attributes set now belong to.
inline int currentDevice() {
    int device = 0;
    BSG_CUDA(cudaGetDevice(&device));
    return device;
}

// Lets Kernel take up to `bytes` (the same in every call) of dynamic shared memory on this device.
template <auto Kernel>
void allowSharedMemory(int bytes) {
    static PerDevice done;
    done.get(currentDevice(), [&] {
        BSG_CUDA(cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        return 1;
    });
}

// CTAs per cluster for Kernel at `block` threads and up to `smem` bytes of dynamic shared
// memory: 16 where the device can place such a cluster, else the portable 8.
template <auto Kernel>
int clusterCtas(int block, int smem = 0) {
    static PerDevice ctas;
    return ctas.get(currentDevice(), [&] {
        int n = 0;
        if (cudaFuncSetAttribute(Kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(kMaxClusterCtas);
            cfg.blockDim = dim3(block);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute at{};
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = kMaxClusterCtas;
            at.val.clusterDim.y = at.val.clusterDim.z = 1;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, Kernel, &cfg) != cudaSuccess) n = 0;
        }
        cudaGetLastError();
        return n > 0 ? kMaxClusterCtas : 8;
    });
}

// `clusters` clusters of Kernel on the context's stream, with `smem` (at most `max_smem`) bytes
// of dynamic shared memory per CTA.
template <auto Kernel, class... A>
void launchCluster(Context& ctx, int clusters, int block, int smem, int max_smem, A... args) {
    const int ctas = clusterCtas<Kernel>(block, max_smem);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(clusters * ctas);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx.stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    BSG_CUDA(cudaLaunchKernelEx(&cfg, Kernel, args...));
    ctx.launched();
}

// Warp 0's part of a sum over the n CTAs of a group: the CTA's totals into `part`, the
// barrier, and every CTA's totals summed back in a fixed order into tot.
template <int NV, int BS>
__device__ __forceinline__ int sumThroughBarrier(SegmentBarrier* bar, int rank, int n, const double (*sh)[BS / 32],
                                                     double* part, double* tot) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        double x = lane < BS / 32 ? sh[j][lane] : 0.0;
#pragma unroll
        for (int o = BS / 64; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) part[rank * NV + j] = x;
    }
    int stop = 0;
    if (lane == 0) stop = arriveAndWait(bar, n);
    __syncwarp();
    double x[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) x[j] = 0.0;
    // read at L2 (ld.global.cg): every CTA must see exactly the totals the others see,
    // whatever its SM's L1 still holds of the previous sum on this half
    for (int b = lane; b < n; b += 32)
#pragma unroll
        for (int j = 0; j < NV; ++j) x[j] += __ldcg(part + b * NV + j);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x[j] += __shfl_xor_sync(0xffffffffu, x[j], o);
        if (lane == 0) tot[j] = x[j];
    }
    return stop;
}

// Deterministic sum of NV values (FP64) over a group; every CTA returns the same totals, in a
// fixed order (warps, CTAs).  It is a barrier of the group too, with two block barriers around
// warp 0's work.  `buf` alternates between two halves of `partial` (kSumValues doubles per CTA
// each, whatever NV is, so the halves of sums of different widths do not overlap) so a fast
// block's next write never overtakes a slow block's read of the previous sum.
constexpr int kSumValues = 10;
template <int NV, int BS, class G>
__device__ __forceinline__ void gridSum(G& g, double v[NV], double* partial, int& buf) {
    static_assert(NV <= kSumValues && BS / 32 <= 32, "one warp adds the block's warps");
    __shared__ double sh[NV][BS / 32];
    __shared__ double tot[NV];
    __shared__ int stopped;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        double x = v[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) sh[j][warp] = x;
    }
    __syncthreads();
    if (warp == 0) {
        const int stop = sumThroughBarrier<NV, BS>(g.bar, g.rank(), g.size(), sh,
                                                   partial + static_cast<long long>(buf) * g.size() * kSumValues, tot);
        if (lane == 0) stopped = stop;
    }
    __syncthreads();
    // sh, tot and stopped are next written behind the next sum's first block barrier, past every read here
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = tot[j];
    g.stop |= stopped;
    buf ^= 1;
}

// The same sum over a cluster: every CTA writes its totals into a slot of every CTA's shared
// memory, one cluster barrier orders them, and each CTA adds the slots in rank order.  The
// slots alternate with `buf`, so a CTA one sum ahead writes the other half.
template <int NV, int BS>
__device__ void gridSum(ClusterGroup& g, double v[NV], double*, int& buf) {
    static_assert(NV <= BS / 32 && BS / 32 <= 32, "one warp per value");
    __shared__ double sh[NV][BS / 32];
    __shared__ double slots[2][NV][kMaxClusterCtas];
    __shared__ double tot[NV];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rank = g.rank(), size = g.size();
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        double x = v[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) sh[j][warp] = x;
    }
    __syncthreads();
    if (warp < NV) {
        double x = lane < BS / 32 ? sh[warp][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane < size) *cooperative_groups::this_cluster().map_shared_rank(&slots[buf][warp][rank], lane) = x;
    }
    g.sync();
    if (warp < NV) {
        double x = lane < size ? slots[buf][warp][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) tot[warp] = x;
    }
    __syncthreads();
    // sh and tot are next written after the next barrier of the group, past every read here
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = tot[j];
    buf ^= 1;
}

#endif

#ifdef __CUDACC__
// The system whose CTA range [begin[s], begin[s + 1]) holds this block.
__device__ __forceinline__ int systemOfBlock(const int* begin, int count) {
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (begin[mid] <= static_cast<int>(blockIdx.x)) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
#endif

// CTA ranges of a batch's systems in one cooperative launch: begin[i]..begin[i+1], about
// `slices_per_cta` level-0 slices each and at least one CTA, scaled down in proportion (keeping one each) when
// the batch exceeds the resident grid.  Within the grid a system's share is its own size's alone,
// so its arithmetic does not depend on its neighbours.
std::vector<int> allotCtas(const std::vector<long long>& slices, int slices_per_cta, int capacity);

// The systems of a batch's launches, one after another: [c[i], c[i + 1]).  A launch takes up to kBatchArgs
// systems (and no more than CTAs), but past kBatchSideBySide of them only while each still gets the CTAs its size
// asks for: 64 cavities of 512 cells take 0.33 ms for a pressure solve in one launch and 0.65 in two,
// 64 of 4096 cells, which fill the GPU 37 at a time, 1.60 in one and 1.41 in two.
constexpr int kBatchSideBySide = 32;
std::vector<std::size_t> batchLaunches(const std::vector<long long>& slices, int slices_per_cta, int capacity);

}  // namespace bsg
