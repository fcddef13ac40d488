// Aggregation AMG: host structure setup once per mesh, device numeric setup per
// matrix version, device V-cycle.  See amg.h for the design.
#include "amg.h"
#include "amg_setup.h"
#include "bsg_device.cuh"
#include "pcg_sell.cuh"

#include <algorithm>
#include <cmath>
#include <numeric>

namespace bsg {

struct AmgPreconditioner::Level {
    int n = 0;
    long long nnz = 0;
    // matrix of this level (level 0 borrows the caller's arrays)
    DeviceArray<int> ptr, col;
    DeviceArray<double> diag, val;
    const int* dptr = nullptr;
    const int* dcol = nullptr;
    const double* ddiag = nullptr;
    const double* dval = nullptr;
    DeviceArray<double> rdiag;           // omega / diag for damped Jacobi
    // transfer to the next coarser level
    DeviceArray<int> agg;                // fine row -> coarse row
    DeviceArray<int> agg_ptr, agg_rows;  // coarse row -> fine rows
    DeviceArray<int> cslot_ptr, cslot_src, cintra_ptr, cintra_src;
    // work vectors
    DeviceArray<double> x, b, t;
    // coarsest level
    DeviceArray<double> dense;           // coarsest level: n x n inverse, row-major
    // SELL-32 copies for the persistent solver (pcg_sell.cuh)
    int nslices = 0;
    long long sell_entries = 0;
    DeviceArray<int> s_ptr, s_col;
    DeviceArray<double> s_val;           // FP64 values (FP64 V-cycle; on level 0 also the Krylov matrix)
    DeviceArray<double> w;               // first Jacobi sweep (FP64 V-cycle)
    DeviceArray<float> s_val32, diag32, rd32, x32, b32, w32, t32;
    // tree numbering (pcg_tree.cuh): maps, the columns' positions, and the level's vectors, all in the
    // preconditioner's tree_store_
    int npos = 0;
    int *t_row = nullptr, *t_rank = nullptr, *t_pos = nullptr, *t_pcol = nullptr, *at = nullptr;  // at: row -> position
    int4* t_memb = nullptr;
    double *tb = nullptr, *tw = nullptr, *te = nullptr;
    // SELL-32 pattern from the level's CSR: row pointers on the host, both arrays on the device.
    void buildSell(const int* hptr, const int* dptr_, const int* dcol_, cudaStream_t s) {
        const std::vector<int> sptr = sellOffsets(n, hptr);
        nslices = static_cast<int>(sptr.size()) - 1;
        sell_entries = sptr.back();
        s_ptr.upload(sptr, s);
        s_col.resize(std::max<long long>(sell_entries, 1));
        sellColumns(n, dptr_, dcol_, s_ptr.data(), s_col.data(), s);
    }
};

namespace {
constexpr int kBlock = 256;
// Largest level whose whole V-cycle is kept as a dense matrix (8 MB at 1024 rows, read from L2).
constexpr int kFoldRows = 1200;
// Smallest system whose coarse-correction scale is tried out (24 CG iterations cost it about 0.3 ms).
constexpr int kTuneRows = 2048;

__global__ void kGatherInts(int n, const int* __restrict__ index, const int* __restrict__ table, int* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = table[index[i]];
}

__global__ void kRdiag(int n, double omega, const double* __restrict__ d, double* __restrict__ rd) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) rd[i] = omega / d[i];
}

// Coarse Galerkin values: fixed-order gathers over precomputed fine contributions.
__global__ void kGalerkin(int nc, const int* __restrict__ agg_ptr, const int* __restrict__ agg_rows,
                          const int* __restrict__ cintra_ptr, const int* __restrict__ cintra_src,
                          const int* __restrict__ cptr, const int* __restrict__ cslot_ptr,
                          const int* __restrict__ cslot_src, const double* __restrict__ fdiag,
                          const double* __restrict__ fval, double* __restrict__ cdiag, double* __restrict__ cval) {
    const int I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= nc) return;
    double d = 0.0;
    for (int k = agg_ptr[I]; k < agg_ptr[I + 1]; ++k) d += fdiag[agg_rows[k]];
    for (int k = cintra_ptr[I]; k < cintra_ptr[I + 1]; ++k) d += fval[cintra_src[k]];
    cdiag[I] = d;
    for (int c = cptr[I]; c < cptr[I + 1]; ++c) {
        double v = 0.0;
        for (int k = cslot_ptr[c]; k < cslot_ptr[c + 1]; ++k) v += fval[cslot_src[k]];
        cval[c] = v;
    }
}

// In-place Gauss-Jordan inverse of the coarsest matrix (SPD, so no pivoting),
// one block; each step stages the pivot row and column in shared memory and
// every thread updates its share of the n x n entries.
__global__ void kDenseInverse(int n, const int* __restrict__ ptr, const int* __restrict__ col,
                              const double* __restrict__ diag, const double* __restrict__ val, double* __restrict__ M) {
    extern __shared__ double sh[];
    double* prow = sh;
    double* pcol = sh + n;
    const int nn = n * n;
    for (int e = threadIdx.x; e < nn; e += blockDim.x) M[e] = 0.0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        M[static_cast<long long>(i) * n + i] = diag[i];
        for (int k = ptr[i]; k < ptr[i + 1]; ++k) M[static_cast<long long>(i) * n + col[k]] += val[k];
    }
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        const double p = 1.0 / M[static_cast<long long>(k) * n + k];
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            prow[j] = M[static_cast<long long>(k) * n + j];
            pcol[j] = M[static_cast<long long>(j) * n + k];
        }
        __syncthreads();
        for (int e = threadIdx.x; e < nn; e += blockDim.x) {
            const int i = e / n, j = e - i * n;
            double v;
            if (i == k) v = j == k ? p : prow[j] * p;
            else if (j == k) v = -pcol[i] * p;
            else v = M[e] - pcol[i] * prow[j] * p;
            M[e] = v;
        }
        __syncthreads();
    }
}

// The same inverse in blocks of kInvBlock pivots on one thread-block cluster, the matrix in its CTAs'
// shared memory: CTA q owns rows [q*rows, (q+1)*rows), a multiple of the block.  Per block, with D its
// diagonal block and R its rows: the owner inverts D (one warp, Gauss-Jordan), forms D^-1 R, keeps it as
// its rows (D^-1 in the block's own columns) and leaves a copy in memory; after a cluster barrier every
// CTA reads that panel and takes it off its other rows, whose entries C in the block's columns
// become -C D^-1.  2 n^3 flops are little (0.2 GFLOP at 440 rows); what counts is the chain, which is
// two barriers and two block-wide passes per 16 pivots instead of one of each per pivot: see the
// figures at kAmgCoarsestRows.
constexpr int kInvBlock = 16;
constexpr int kInvThreads = 256;
// Largest coarsest level: 16 CTAs of 32 rows keep 440 rows (rows x n + the panel, 169 KB).  Time of one
// inverse, pivot by pivot on 8 CTAs against in blocks on 16:
//   256 rows 1.00 / 0.40 ms, 294 rows 1.10 / 0.40 ms, 400 rows 2.50 / 0.55 ms.
constexpr int kAmgCoarsestRows = 440;

__global__ void __launch_bounds__(kInvThreads, 1)
    kDenseInverseBlocked(int n, int rows, const int* __restrict__ ptr, const int* __restrict__ col,
                         const double* __restrict__ diag, const double* __restrict__ val, double* panel,
                         double* __restrict__ M) {
    extern __shared__ double sh[];
    double* Ml = sh;                                          // rows x n, this CTA's rows
    double* R = sh + static_cast<long long>(rows) * n;        // kInvBlock x n, the block's rows
    __shared__ double D[kInvBlock][kInvBlock + 1];
    ClusterGroup g;
    const int q = g.rank(), tid = threadIdx.x, lane = tid & 31;
    const int r0 = min(n, q * rows), nr = min(n, r0 + rows) - r0;
    for (int e = tid; e < nr * n; e += kInvThreads) Ml[e] = 0.0;
    __syncthreads();
    for (int li = tid; li < nr; li += kInvThreads) {
        const int i = r0 + li;
        Ml[static_cast<long long>(li) * n + i] = diag[i];
        for (int k = ptr[i]; k < ptr[i + 1]; ++k) Ml[static_cast<long long>(li) * n + col[k]] += val[k];
    }
    __syncthreads();
    for (int b0 = 0; b0 < n; b0 += kInvBlock) {
        const int nb = min(kInvBlock, n - b0);
        const bool owner = b0 >= r0 && b0 < r0 + nr;
        double* out = panel + static_cast<long long>((b0 / kInvBlock) & 1) * kInvBlock * n;
        if (owner) {
            double* rowsB = Ml + static_cast<long long>(b0 - r0) * n;
            if (tid < 32) {  // D^-1
                for (int e = lane; e < nb * nb; e += 32) D[e / nb][e % nb] = rowsB[static_cast<long long>(e / nb) * n + b0 + e % nb];
                __syncwarp();
                for (int k = 0; k < nb; ++k) {
                    const double p = 1.0 / D[k][k];
                    double next[kInvBlock * kInvBlock / 32];
#pragma unroll
                    for (int u = 0; u < kInvBlock * kInvBlock / 32; ++u) {
                        const int e = lane + 32 * u, i = e / kInvBlock, j = e % kInvBlock;
                        next[u] = 0.0;
                        if (i >= nb || j >= nb) continue;
                        if (i == k) next[u] = j == k ? p : D[k][j] * p;
                        else if (j == k) next[u] = -D[i][k] * p;
                        else next[u] = D[i][j] - D[i][k] * D[k][j] * p;
                    }
                    __syncwarp();
#pragma unroll
                    for (int u = 0; u < kInvBlock * kInvBlock / 32; ++u) {
                        const int e = lane + 32 * u, i = e / kInvBlock, j = e % kInvBlock;
                        if (i < nb && j < nb) D[i][j] = next[u];
                    }
                    __syncwarp();
                }
            }
            __syncthreads();
            for (int j = tid; j < n; j += kInvThreads) {  // one column of D^-1 R per thread
                const bool own = j >= b0 && j < b0 + nb;
                double in[kInvBlock];
#pragma unroll
                for (int k = 0; k < kInvBlock; ++k) in[k] = k < nb ? rowsB[static_cast<long long>(k) * n + j] : 0.0;
                for (int i = 0; i < nb; ++i) {
                    double v = 0.0;
                    if (own) v = D[i][j - b0];
                    else
#pragma unroll
                        for (int k = 0; k < kInvBlock; ++k) v += (k < nb ? D[i][k] : 0.0) * in[k];
                    rowsB[static_cast<long long>(i) * n + j] = v;
                    out[static_cast<long long>(i) * n + j] = v;
                }
            }
        }
        g.sync();  // the panel is in memory
#pragma unroll 8
        for (int e = tid; e < nb * n; e += kInvThreads) R[e] = out[e];
        __syncthreads();
        // four rows at a time, so an entry of R is read once for four updates
        const int warp = tid >> 5, warps = kInvThreads / 32;
        for (int l0 = 4 * warp; l0 < nr; l0 += 4 * warps) {
            if (owner && l0 >= b0 - r0 && l0 < b0 - r0 + nb) continue;  // blocks are multiples of four rows
            const int m = min(4, nr - l0);
            double c[4][kInvBlock];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int k = 0; k < kInvBlock; ++k)
                    c[i][k] = i < m && k < nb ? Ml[static_cast<long long>(l0 + i) * n + b0 + k] : 0.0;
            __syncwarp();  // every lane has C before any of it is overwritten
            for (int j = lane; j < n; j += 32) {
                const bool own = j >= b0 && j < b0 + nb;
                double v[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = own || i >= m ? 0.0 : Ml[static_cast<long long>(l0 + i) * n + j];
#pragma unroll
                for (int k = 0; k < kInvBlock; ++k) {
                    const double r = k < nb ? R[k * n + j] : 0.0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] -= c[i][k] * r;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i < m) Ml[static_cast<long long>(l0 + i) * n + j] = v[i];
            }
        }
        __syncthreads();  // rows, and R, before the next block (the panel alternates between two halves)
    }
    for (int e = tid; e < nr * n; e += kInvThreads) M[static_cast<long long>(r0) * n + e] = Ml[e];
}

// foldCoarse, first pass: column j of Y = M T, one block per j.  Column j of T has 1 - a_jj w_j at
// j's aggregate and -a_ij w_j at each neighbour's.
__global__ void kFoldColumns(int n, int nc, const int* __restrict__ ptr, const int* __restrict__ col,
                             const double* __restrict__ diag, const double* __restrict__ val,
                             const double* __restrict__ rd, const int* __restrict__ agg, const double* __restrict__ M,
                             double* __restrict__ Y) {
    const int j = blockIdx.x;
    const double wj = rd[j];
    const int k0 = ptr[j], k1 = ptr[j + 1];
    for (int c = threadIdx.x; c < nc; c += blockDim.x) {
        double y = (1.0 - diag[j] * wj) * M[static_cast<long long>(agg[j]) * nc + c];
        for (int k = k0; k < k1; ++k) y -= val[k] * wj * M[static_cast<long long>(agg[col[k]]) * nc + c];
        Y[static_cast<long long>(c) * n + j] = y;
    }
}

// Second pass: the row of rank blockIdx.x, its entries by position.
__global__ void kFoldLines(int n, int npos, const int* __restrict__ pos, const int* __restrict__ row,
                           const int* __restrict__ ptr, const int* __restrict__ col, const double* __restrict__ diag,
                           const double* __restrict__ val, const double* __restrict__ rd, const int* __restrict__ agg,
                           double gamma, const double* __restrict__ Y, const int* __restrict__ at, double* __restrict__ out) {
    extern __shared__ double line[];
    const int i = row[pos[blockIdx.x]];
    const double wi = rd[i];
    const int k0 = ptr[i], k1 = ptr[i + 1];
    for (int p = threadIdx.x; p < npos; p += blockDim.x) {
        const int j = row[p];
        double b = 0.0;
        if (j >= 0) {
            b = (1.0 - diag[i] * wi) * Y[static_cast<long long>(agg[i]) * n + j];
            for (int k = k0; k < k1; ++k) b -= val[k] * wi * Y[static_cast<long long>(agg[col[k]]) * n + j];
            b *= gamma;
        }
        line[p] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {  // a repeated pair has two entries: one thread adds them
        line[at[i]] += 2.0 * wi - wi * diag[i] * wi;
        for (int k = k0; k < k1; ++k) line[at[col[k]]] -= wi * val[k] * rd[col[k]];
    }
    __syncthreads();
    for (int p = threadIdx.x; p < npos; p += blockDim.x)
        out[static_cast<long long>(blockIdx.x) * npos + p] = line[p];
}

__global__ void kDenseSolve(int n, const double* __restrict__ Minv, const double* __restrict__ b, double* __restrict__ x) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int j = 0; j < n; ++j) s += Minv[static_cast<long long>(i) * n + j] * b[j];
        x[i] = s;
    }
}

__global__ void kToFloat(long long n, const double* __restrict__ a, float* __restrict__ out) {
    const long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (e < n) out[e] = static_cast<float>(a[e]);
}

// x = omega D^-1 b (first Jacobi sweep from a zero guess)
__global__ void kSmoothZero(int n, const double* __restrict__ rd, const double* __restrict__ b, double* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = rd[i] * b[i];
}

// x_out = x + omega D^-1 (b - A x)
__global__ void kSmooth(int n, const int* __restrict__ ptr, const int* __restrict__ col, const double* __restrict__ diag,
                        const double* __restrict__ val, const double* __restrict__ rd, const double* __restrict__ b,
                        const double* __restrict__ x, double* __restrict__ xo) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double ax = diag[i] * x[i];
    for (int k = ptr[i]; k < ptr[i + 1]; ++k) ax += val[k] * x[col[k]];
    xo[i] = x[i] + rd[i] * (b[i] - ax);
}

// Post-smoothing sweep fused with prolongation: y = x + P xc, x_out = y + omega D^-1 (b - A y).
__global__ void kProlongSmooth(int n, const int* __restrict__ ptr, const int* __restrict__ col,
                               const double* __restrict__ diag, const double* __restrict__ val,
                               const double* __restrict__ rd, const int* __restrict__ agg,
                               const double* __restrict__ xc, const double* __restrict__ b,
                               const double* __restrict__ x, double* __restrict__ xo) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double yi = x[i] + xc[agg[i]];
    double ay = diag[i] * yi;
    for (int k = ptr[i]; k < ptr[i + 1]; ++k) {
        const int j = col[k];
        ay += val[k] * (x[j] + xc[agg[j]]);
    }
    xo[i] = yi + rd[i] * (b[i] - ay);
}

// b_c[I] = sum over fine rows i of aggregate I of (b - A x)_i
__global__ void kResidualRestrict(int nc, const int* __restrict__ agg_ptr, const int* __restrict__ agg_rows,
                                  const int* __restrict__ ptr, const int* __restrict__ col,
                                  const double* __restrict__ diag, const double* __restrict__ val,
                                  const double* __restrict__ b, const double* __restrict__ x, double* __restrict__ bc) {
    const int I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= nc) return;
    double s = 0.0;
    for (int m = agg_ptr[I]; m < agg_ptr[I + 1]; ++m) {
        const int i = agg_rows[m];
        double ax = diag[i] * x[i];
        for (int k = ptr[i]; k < ptr[i + 1]; ++k) ax += val[k] * x[col[k]];
        s += b[i] - ax;
    }
    bc[I] = s;
}

}  // namespace

namespace {
// Dynamic shared memory of one CTA of the cluster inverse (the rest of the SM's
// 228 KB stays for the driver's reserve).
constexpr std::size_t kInverseSmem = 200 * 1024;

// CTAs of the cluster inverse's cluster, 0 where none can be had.
int inverseCtas() {
    static PerDevice ctas;
    return ctas.get(currentDevice(), [] {
        if (cudaFuncSetAttribute(kDenseInverseBlocked, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kInverseSmem)) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return clusterCtas<kDenseInverseBlocked>(kInvThreads, static_cast<int>(kInverseSmem));
    });
}
}  // namespace

AmgPreconditioner::AmgPreconditioner(DeviceMesh& mesh, const SolverConfig& cfg)
    : mesh_(mesh), ctx_(*mesh.ctx), cfg_(cfg) {
    // Tuning overrides for experiments: Jacobi weight and coarse-correction scale.
    if (const char* w = std::getenv("BSG_AMG_OMEGA")) omega_ = std::atof(w);
    if (const char* g = std::getenv("BSG_AMG_GAMMA")) {
        gamma_ = std::atof(g);
        tuned_ = true;
    }
    if (!(omega_ > 0.0 && omega_ <= 1.0) || !(gamma_ > 0.0 && gamma_ <= 3.0))
        fail(kArgument, "AMG Jacobi weight must be in (0,1] and the correction scale in (0,3]");
    // FP32 V-cycle data on the mixed-precision path (FP64 Krylov vectors and true residual stay FP64)
    fp32_ = cfg.precision == 1 || cfg.precision == 2 || std::getenv("BSG_AMG_FP32") != nullptr;
    if (const char* p = std::getenv("BSG_AMG_PASSES0")) passes0_ = std::max(1, std::min(4, std::atoi(p)));
    if (const char* p = std::getenv("BSG_AMG_PASSES")) passes_ = std::max(1, std::min(4, std::atoi(p)));
}

AmgPreconditioner::~AmgPreconditioner() { clearLevels(); }

void AmgPreconditioner::clearLevels() {
    for (Level* l : levels_) delete l;
    levels_.clear();
    host_ptr_.clear();
    host_agg_.clear();
    cg_ready_ = tree_ = false;
}

int AmgPreconditioner::levels() const { return static_cast<int>(levels_.size()); }
long long AmgPreconditioner::coarseRows(int level) const { return levels_.at(level)->n; }

void AmgPreconditioner::buildStructure(const Dcsr<double>& A) {
    clearLevels();  // what an attempt that failed (stalled coarsening, no memory) left
    HostCsr cur;
    cur.n = A.n;
    cur.ptr.resize(A.n + 1);
    cur.col.resize(A.nnz_off);
    cur.diag.resize(A.n);
    cur.val.resize(A.nnz_off);
    BSG_CUDA(cudaMemcpyAsync(cur.ptr.data(), A.ptr, sizeof(int) * (A.n + 1), cudaMemcpyDeviceToHost, ctx_.stream));
    BSG_CUDA(cudaMemcpyAsync(cur.col.data(), A.col, sizeof(int) * A.nnz_off, cudaMemcpyDeviceToHost, ctx_.stream));
    BSG_CUDA(cudaMemcpyAsync(cur.diag.data(), A.diag, sizeof(double) * A.n, cudaMemcpyDeviceToHost, ctx_.stream));
    BSG_CUDA(cudaMemcpyAsync(cur.val.data(), A.val, sizeof(double) * A.nnz_off, cudaMemcpyDeviceToHost, ctx_.stream));
    ctx_.sync();
    // Coarsening stops at the configured size, at most kAmgCoarsestRows: a coarsest level that
    // size still fits the cluster inverse's distributed shared memory, and every level removed
    // saves the V-cycle its phases, whose cost is latency, not size, on small levels.
    const int coarse_target = std::max(std::min(cfg_.amg_coarse_size, kAmgCoarsestRows), 16);
    const int max_levels = std::max(2, cfg_.amg_max_levels);
    auto* l0 = new Level();
    l0->n = A.n;
    l0->nnz = A.nnz_off;
    l0->buildSell(cur.ptr.data(), A.ptr, A.col, ctx_.stream);
    levels_.push_back(l0);
    while (cur.n > coarse_target && static_cast<int>(levels_.size()) < max_levels) {
        // aggregates from `passes` rounds of pairwise matching (2 by default: up to 4 rows)
        const int passes = levels_.size() == 1 ? passes0_ : passes_;
        int n2 = cur.n;
        std::vector<int> agg(cur.n);
        std::iota(agg.begin(), agg.end(), 0);
        HostCsr work;
        for (int pass = 0; pass < passes; ++pass) {
            int nn = 0;
            const HostCsr& from = pass == 0 ? cur : work;
            const std::vector<int> a = pairwise(from, nn);
            if (pass + 1 < passes) {
                HostCsr coarse = coarsen(from, a, nn, nullptr);
                work = std::move(coarse);
            }
            for (int i = 0; i < cur.n; ++i) agg[i] = a[agg[i]];
            n2 = nn;
        }
        // stop when coarsening stalls (< 1.5x fewer rows): such levels cost a
        // V-cycle their barriers and gathers without shrinking the problem
        if (3 * static_cast<long long>(n2) > 2 * static_cast<long long>(cur.n) && cur.n <= 1024) break;
        if (n2 >= cur.n) break;  // no coarsening possible
        std::vector<int> target, agg_ptr, agg_rows;
        HostCsr next = coarsen(cur, agg, n2, &target);
        aggregateLists(agg, n2, agg_ptr, agg_rows);
        const long long cnnz = static_cast<long long>(next.col.size());
        GalerkinMaps maps = galerkinMaps(cur, target, agg_ptr, agg_rows, static_cast<int>(cnnz));
        if (maps.cintra_src.empty()) maps.cintra_src.push_back(0);
        Level* fine = levels_.back();
        cudaStream_t s = ctx_.stream;
        fine->agg.upload(agg, s);
        fine->agg_ptr.upload(agg_ptr, s);
        fine->agg_rows.upload(agg_rows, s);
        fine->cslot_ptr.upload(maps.cslot_ptr, s);
        fine->cslot_src.upload(maps.cslot_src, s);
        fine->cintra_ptr.upload(maps.cintra_ptr, s);
        fine->cintra_src.upload(maps.cintra_src, s);
        auto* lv = new Level();
        lv->n = n2;
        lv->nnz = cnnz;
        lv->ptr.upload(next.ptr, s);
        if (next.col.empty()) { next.col.push_back(0); next.val.push_back(0.0); }
        lv->col.upload(next.col, s);
        lv->diag.resize(n2);
        lv->val.resize(std::max<long long>(cnnz, 1));
        lv->dptr = lv->ptr.data();
        lv->dcol = lv->col.data();
        lv->ddiag = lv->diag.data();
        lv->dval = lv->val.data();
        lv->buildSell(next.ptr.data(), lv->dptr, lv->dcol, s);
        levels_.push_back(lv);
        ctx_.sync();  // the host arrays go
        host_ptr_.push_back(std::move(cur.ptr));
        host_agg_.push_back(std::move(agg));
        cur = std::move(next);
    }
    host_ptr_.push_back(std::move(cur.ptr));
    for (Level* l : levels_) {
        l->x.resize(l->n);
        l->b.resize(l->n);
        l->t.resize(l->n);
        l->rdiag.resize(l->n);
        const std::size_t e = std::max<long long>(l->sell_entries, 1);
        if (fp32_) {
            for (DeviceArray<float>* a : {&l->diag32, &l->rd32, &l->x32, &l->b32, &l->w32, &l->t32}) a->resize(l->n);
            l->s_val32.resize(e);
            l->s_val32.zero(ctx_.stream);  // padding entries stay zero
        } else {
            l->w.resize(l->n);
        }
        if (!fp32_ || l == levels_.front()) {  // FP64 V-cycle values, and the level-0 Krylov matrix
            l->s_val.resize(e);
            l->s_val.zero(ctx_.stream);
        }
    }
    Level* last = levels_.back();
    if (last->n > 2048)
        fail(kState, "AMG coarsening stalled at " + std::to_string(last->n) +
                         " rows, too many for the dense coarsest solve");
    const std::size_t nn = static_cast<std::size_t>(last->n) * last->n;
    last->dense.resize(nn);
    if (fp32_) dense32_.resize(nn);
    built_ = true;
    if (std::getenv("BSG_AMG_VERBOSE")) {
        long long total = 0;
        for (Level* l : levels_) total += l->nnz + l->n;
        for (std::size_t i = 0; i < levels_.size(); ++i)
            std::fprintf(stderr, "amg level %zu: rows %d, off-diagonal nnz %lld (%.1f per row)\n", i, levels_[i]->n,
                         levels_[i]->nnz, levels_[i]->n ? double(levels_[i]->nnz) / levels_[i]->n : 0.0);
        std::fprintf(stderr, "amg operator complexity %.3f\n", double(total) / double(levels_[0]->nnz + levels_[0]->n));
    }
}

void AmgPreconditioner::prepareCg() {
    if (cg_ready_) return;
    buildTree();
    foldCoarse();
    uploadTree();
    std::vector<std::vector<int>>().swap(host_ptr_);
    std::vector<std::vector<int>>().swap(host_agg_);
    cg_ready_ = true;
}

void AmgPreconditioner::buildTree() {
    const std::vector<std::vector<int>>&ptr = host_ptr_, &agg = host_agg_;
    const int L = static_cast<int>(levels_.size());
    plan_ = TreePlan{};
    tree_ = cfg_.amg_smoothing_steps <= 1 && L <= kMaxTreeLevels && !fp32_;  // (why not in FP32: pcg_tree.cuh)
    if (L < 2 || levels_[0]->n < kTuneRows) tuned_ = true;
    for (int l = 0; tree_ && l + 1 < L; ++l) {
        std::vector<int> size(levels_[l + 1]->n, 0);
        for (int I : agg[l])
            if (++size[I] > 4) tree_ = false;
    }
    if (!tree_) return;
    plan_.slices.assign(L, 0);
    plan_.entries.assign(L, 0.0);
    plan_.rows.assign(L, 0);
    plan_.positions.assign(L, 0);
    plan_.nnz = levels_[0]->nnz;
    // One host image of every level's maps, one allocation, one upload and one clearing: with an array each
    // (nine per level), a synchronisation per level and the trial to its end, a new 4096-cell system's first
    // solve took 4.5 ms, now 3.9 (16x16x16 cells; 4.9 and 4.0 for a 64x64 cavity's first outer iteration).
    constexpr std::size_t kAlign = 64;  // entries
    std::vector<int> image;
    image.reserve(6 * static_cast<std::size_t>(levels_[0]->n));
    const auto room = [&](std::size_t entries) {
        const std::size_t at = image.size();
        image.resize(at + (entries + kAlign - 1) / kAlign * kAlign, -1);
        return at;
    };
    const auto put = [&](const std::vector<int>& v) {
        const std::size_t at = room(v.size());
        std::copy(v.begin(), v.end(), image.begin() + at);
        return at;
    };
    struct Offsets {
        std::size_t row, rank, pos, at, memb, pcol;
    };
    std::vector<Offsets> offsets(L);
    std::vector<int> order;  // rank -> row of the level above
    Members members;         // of the level above
    for (int l = L - 1; l >= 0; --l) {
        Level* lv = levels_[l];
        const int n = lv->n;
        TreeMaps t;
        if (l == L - 1) {
            t.row.resize(n);
            std::iota(t.row.begin(), t.row.end(), 0);
            t.rank = t.pos = t.at = order = t.row;
        } else {
            const long long npos = 4LL * levels_[l + 1]->n;
            if (npos > 2LL * n + 64) break;  // mostly holes: this level and the finer ones keep their numbering
            plan_.slices[l] = (npos + 31) / 32;
            plan_.entries[l] = ptr[l][n];  // without padding
            if (!plan_.fits(l, ctx_.sm_count)) break;  // not even on the whole GPU
            t = treeMaps(n, members, order);
            plan_.entries[l] = paddedEntries(t, ptr[l]);
            if (!plan_.fits(l, ctx_.sm_count)) break;
        }
        plan_.first = l;
        lv->npos = static_cast<int>(t.row.size());
        plan_.rows[l] = n;
        plan_.positions[l] = lv->npos;
        Offsets& o = offsets[l];
        o.row = put(t.row);
        o.rank = put(t.rank);
        o.pos = put(t.pos);
        o.at = put(t.at);
        if (l > 0) {
            members = membersOf(agg[l - 1], n);
            o.memb = room(4 * t.row.size());
            membersByPosition(t, members, image.data() + o.memb);
        }
    }
    // level L - 2 and its V-cycle as one dense matrix (foldCoarse), where that level is small
    plan_.folded = L >= 3 && plan_.first <= L - 2 && levels_[L - 2]->n <= kFoldRows;
    std::size_t bytes = sizeof(int) * image.size();
    const auto take = [&](std::size_t b) {
        const std::size_t at = bytes;
        bytes += (b + 255) / 256 * 256;
        return at;
    };
    for (int l = plan_.first; l < L - 1; ++l) offsets[l].pcol = take(sizeof(int) * ptr[l][levels_[l]->n]);
    const std::size_t vectors = bytes;
    std::vector<std::size_t> vec(L);
    for (int l = plan_.first; l < L; ++l) {
        vec[l] = take(sizeof(double) * levels_[l]->npos);
        take(sizeof(double) * levels_[l]->npos);
        take(sizeof(double) * levels_[l]->npos);
    }
    const std::size_t vectors_end = bytes;
    std::size_t fold_y = 0, folded = 0;
    if (plan_.folded) {
        const std::size_t n = levels_[L - 2]->n;
        fold_y = take(sizeof(double) * levels_[L - 1]->n * n);
        folded = take(sizeof(double) * n * levels_[L - 2]->npos);
    }
    cudaStream_t s = ctx_.stream;
    tree_store_.resize(bytes);
    char* store = tree_store_.data();
    BSG_CUDA(cudaMemcpyAsync(store, image.data(), sizeof(int) * image.size(), cudaMemcpyHostToDevice, s));
    BSG_CUDA(cudaMemsetAsync(store + vectors, 0, vectors_end - vectors, s));  // holes stay zero
    for (int l = plan_.first; l < L; ++l) {
        Level* lv = levels_[l];
        const Offsets& o = offsets[l];
        int* ints = reinterpret_cast<int*>(store);
        lv->t_row = ints + o.row;
        lv->t_rank = ints + o.rank;
        lv->t_pos = ints + o.pos;
        lv->at = ints + o.at;
        lv->t_memb = l > 0 ? reinterpret_cast<int4*>(ints + o.memb) : nullptr;
        if (l < L - 1) {  // the columns' positions
            lv->t_pcol = reinterpret_cast<int*>(store + o.pcol);
            const int nnz = ptr[l][lv->n];
            if (nnz > 0) {
                kGatherInts<<<gridFor(nnz, kBlock), kBlock, 0, s>>>(nnz, lv->dcol, lv->at, lv->t_pcol);
                BSG_CUDA(cudaGetLastError());
                ctx_.launched();
            }
        }
        const std::size_t step = (sizeof(double) * lv->npos + 255) / 256 * 256;
        lv->tb = reinterpret_cast<double*>(store + vec[l]);
        lv->tw = reinterpret_cast<double*>(store + vec[l] + step);
        lv->te = reinterpret_cast<double*>(store + vec[l] + 2 * step);
    }
    if (plan_.folded) {
        fold_y_ = reinterpret_cast<double*>(store + fold_y);
        folded_ = reinterpret_cast<double*>(store + folded);
    }
    ctx_.sync();  // the host image goes
}

// The V-cycle of level f = L - 2 as a matrix.  With W = omega D^-1, piecewise-constant P, the dense
// inverse M of the coarsest level and T = P^T (I - A W), the cycle (one damped-Jacobi sweep
// down and up, coarse correction scaled by gamma) maps b to (2 W - W A W + gamma T^T M T) b, which
// foldCoarse forms in two passes, Y = M T and then its rows, per column of T from the matrix row
// it comes from (A is symmetric).  One product with it replaces the residual, the dense solve
// and the post sweep of that level, two grid barriers of the V-cycle fewer.
void AmgPreconditioner::foldCoarse() {
    if (!plan_.folded) return;
    const int L = static_cast<int>(levels_.size());
    const Level *f = levels_[L - 2], *c = levels_[L - 1];
    kFoldColumns<<<f->n, kBlock, 0, ctx_.stream>>>(f->n, c->n, f->dptr, f->dcol, f->ddiag, f->dval, f->rdiag.data(),
                                                   f->agg.data(), c->dense.data(), fold_y_);
    kFoldLines<<<f->n, kBlock, sizeof(double) * f->npos, ctx_.stream>>>(
        f->n, f->npos, f->t_pos, f->t_row, f->dptr, f->dcol, f->ddiag, f->dval, f->rdiag.data(), f->agg.data(), gamma_,
        fold_y_, f->at, folded_);
    BSG_CUDA(cudaGetLastError());
    ctx_.launches += 2;
}

void AmgPreconditioner::setCorrection(double gamma) {
    gamma_ = gamma;
    foldCoarse();
}

int AmgPreconditioner::treePositions() const {
    return plan_.first == 0 ? std::max(levels_.front()->npos, levels_.front()->n) : levels_.front()->n;
}

TreeView AmgPreconditioner::treeView() const {
    return {static_cast<int>(levels_.size()), plan_.first, gamma_, omega_, d_tree_.data(), d_vl64_.data(),
            d_tvec_.data(), levels_.back()->dense.data(), folded_};
}

void AmgPreconditioner::update(const Dcsr<double>& A, bool numeric) {
    if (!built_) buildStructure(A);
    if (!ready_) numeric = true;
    ready_ = false;
    fine_ = A;
    Level* l0 = levels_[0];
    l0->dptr = A.ptr; l0->dcol = A.col; l0->ddiag = A.diag; l0->dval = A.val;
    if (!numeric) {
        // coarse levels kept; the level-0 matrix and its Jacobi weights always follow the matrix being
        // solved, so a lagged V-cycle smooths the new matrix with its own diagonal (a fresh fine
        // smoother over a lagged coarse correction stays a symmetric positive definite cycle; old
        // weights on a new matrix can stop smoothing when the diagonal moves between versions)
        kRdiag<<<gridFor(l0->n, kBlock), kBlock, 0, ctx_.stream>>>(l0->n, omega_, l0->ddiag, l0->rdiag.data());
        ctx_.launched();
        kCsrToSell<double><<<gridFor(l0->n, kBlock), kBlock, 0, ctx_.stream>>>(
            l0->n, l0->dptr, l0->dval, l0->ddiag, l0->s_ptr.data(), omega_, l0->s_val.data(), nullptr, nullptr);
        ctx_.launched();
        if (fp32_) {
            kCsrToSell<float><<<gridFor(l0->n, kBlock), kBlock, 0, ctx_.stream>>>(
                l0->n, l0->dptr, l0->dval, l0->ddiag, l0->s_ptr.data(), omega_, l0->s_val32.data(), l0->diag32.data(),
                l0->rd32.data());
            ctx_.launched();
        }
        BSG_CUDA(cudaGetLastError());
        uploadViews();
        ready_ = true;
        return;
    }
    for (std::size_t l = 0; l + 1 < levels_.size(); ++l) {
        Level* f = levels_[l];
        Level* c = levels_[l + 1];
        kGalerkin<<<gridFor(c->n, kBlock), kBlock, 0, ctx_.stream>>>(
            c->n, f->agg_ptr.data(), f->agg_rows.data(), f->cintra_ptr.data(), f->cintra_src.data(), c->dptr,
            f->cslot_ptr.data(), f->cslot_src.data(), f->ddiag, f->dval, c->diag.data(), c->val.data());
        ctx_.launched();
    }
    for (Level* l : levels_) {
        kRdiag<<<gridFor(l->n, kBlock), kBlock, 0, ctx_.stream>>>(l->n, omega_, l->ddiag, l->rdiag.data());
        ctx_.launched();
    }
    Level* last = levels_.back();
    const int ctas = inverseCtas();
    const int irows = ctas > 0 ? (last->n + ctas * kInvBlock - 1) / (ctas * kInvBlock) * kInvBlock : 0;
    const std::size_t ismem = sizeof(double) * (static_cast<std::size_t>(irows) + kInvBlock) * last->n;
    if (ctas > 0 && ismem <= kInverseSmem) {
        inv_panel_.resize(2 * static_cast<std::size_t>(kInvBlock) * last->n);
        launchCluster<kDenseInverseBlocked>(ctx_, 1, kInvThreads, static_cast<int>(ismem), static_cast<int>(kInverseSmem),
                                            last->n, irows, last->dptr, last->dcol, last->ddiag, last->dval,
                                            inv_panel_.data(), last->dense.data());
    } else {
        kDenseInverse<<<1, 1024, 2 * sizeof(double) * last->n, ctx_.stream>>>(
            last->n, last->dptr, last->dcol, last->ddiag, last->dval, last->dense.data());
        ctx_.launched();
    }
    BSG_CUDA(cudaGetLastError());
    if (cg_ready_) foldCoarse();
    // SELL-32 values for the persistent solver
    const int nn = last->n * last->n;
    if (fp32_) {
        kToFloat<<<gridFor(nn, kBlock), kBlock, 0, ctx_.stream>>>(nn, last->dense.data(), dense32_.data());
        ctx_.launched();
    }
    for (std::size_t li = 0; li < levels_.size(); ++li) {
        Level* l = levels_[li];
        const unsigned g = gridFor(l->n, kBlock);
        if (fp32_)
            kCsrToSell<float><<<g, kBlock, 0, ctx_.stream>>>(l->n, l->dptr, l->dval, l->ddiag, l->s_ptr.data(), omega_,
                                                              l->s_val32.data(), l->diag32.data(), l->rd32.data());
        if (!fp32_ || li == 0)
            kCsrToSell<double><<<g, kBlock, 0, ctx_.stream>>>(l->n, l->dptr, l->dval, l->ddiag, l->s_ptr.data(), omega_,
                                                               l->s_val.data(), nullptr, nullptr);
        ctx_.launches += (fp32_ && li == 0) ? 2 : 1;
    }
    BSG_CUDA(cudaGetLastError());
    uploadViews();
    ready_ = true;
}

void AmgPreconditioner::uploadViews() {
    // level views for the persistent solver (level 0 borrows the caller's matrix arrays)
    std::vector<AmgLevelView<double>> views(levels_.size());
    for (std::size_t l = 0; l < levels_.size(); ++l) {
        Level* lv = levels_[l];
        const bool coarser = l + 1 < levels_.size();
        views[l] = AmgLevelView<double>{lv->n, lv->dptr, lv->dcol, lv->ddiag, lv->dval, lv->rdiag.data(),
                                        coarser ? lv->agg.data() : nullptr, coarser ? lv->agg_ptr.data() : nullptr,
                                        coarser ? lv->agg_rows.data() : nullptr, lv->x.data(), lv->b.data(),
                                        lv->t.data()};
    }
    d_views_.upload(views, ctx_.stream);
    uploadTree();
    const int L = static_cast<int>(levels_.size());
    if (fp32_) {
        std::vector<VLevel<float>> v(L);
        for (int l = 0; l < L; ++l) {
            Level* lv = levels_[l];
            const bool coarser = l + 1 < L;
            v[l].A = SellMat<float>{lv->n, lv->nslices, lv->s_ptr.data(), lv->s_col.data(), lv->s_val32.data(),
                                    lv->diag32.data(), sellStreams(lv->sell_entries, 4)};
            v[l].rd = lv->rd32.data();
            v[l].agg_ptr = coarser ? lv->agg_ptr.data() : nullptr;
            v[l].agg_rows = coarser ? lv->agg_rows.data() : nullptr;
            v[l].b = lv->b32.data();
            v[l].w = lv->w32.data();
            v[l].x = lv->x32.data();
            v[l].t = lv->t32.data();
        }
        d_vl32_.upload(v, ctx_.stream);
    } else {
        std::vector<VLevel<double>> v(L);
        for (int l = 0; l < L; ++l) {
            Level* lv = levels_[l];
            const bool coarser = l + 1 < L;
            v[l].A = SellMat<double>{lv->n, lv->nslices, lv->s_ptr.data(), lv->s_col.data(), lv->s_val.data(),
                                     lv->ddiag, sellStreams(lv->sell_entries, 8)};
            v[l].rd = lv->rdiag.data();
            v[l].agg_ptr = coarser ? lv->agg_ptr.data() : nullptr;
            v[l].agg_rows = coarser ? lv->agg_rows.data() : nullptr;
            v[l].b = lv->b.data();
            v[l].w = lv->w.data();
            v[l].x = lv->x.data();
            v[l].t = lv->t.data();
        }
        d_vl64_.upload(v, ctx_.stream);
    }
}

void AmgPreconditioner::uploadTree() {
    if (!tree_) return;  // also before prepareCg
    const int L = static_cast<int>(levels_.size());
    std::vector<TreeLevel> t(L);
    std::vector<double*> vec(3 * L, nullptr);
    for (int l = plan_.first; l < L; ++l) {
        Level* lv = levels_[l];
        t[l] = TreeLevel{lv->n, lv->npos, lv->t_row, lv->t_rank, lv->t_pos, lv->t_memb,
                         lv->dptr, lv->t_pcol, lv->dval, lv->ddiag};
        vec[3 * l] = lv->tb;
        vec[3 * l + 1] = lv->tw;
        vec[3 * l + 2] = lv->te;
    }
    d_tree_.upload(t, ctx_.stream);
    d_tvec_.upload(vec, ctx_.stream);
}

SellMat<double> AmgPreconditioner::krylovMatrix() const {
    const Level* l = levels_.front();
    return SellMat<double>{l->n, l->nslices, l->s_ptr.data(), l->s_col.data(), l->s_val.data(), l->ddiag,
                           sellStreams(l->sell_entries, 8)};
}

SellMat<float> AmgPreconditioner::krylovMatrix32() const {
    const Level* l = levels_.front();
    return SellMat<float>{l->n, l->nslices, l->s_ptr.data(), l->s_col.data(), l->s_val32.data(), l->diag32.data(),
                          sellStreams(l->sell_entries, 4)};
}

long long AmgPreconditioner::krylovEntries() const { return levels_.front()->sell_entries; }

VCycleView<double> AmgPreconditioner::sellView64() const {
    VCycleView<double> v;
    v.levels = static_cast<int>(levels_.size());
    v.nu = std::max(1, std::min(2, cfg_.amg_smoothing_steps));
    v.gamma = gamma_;
    v.lv = d_vl64_.data();
    v.dense_inv = levels_.back()->dense.data();
    return v;
}

VCycleView<float> AmgPreconditioner::sellView32() const {
    VCycleView<float> v;
    v.levels = static_cast<int>(levels_.size());
    v.nu = std::max(1, std::min(2, cfg_.amg_smoothing_steps));
    v.gamma = static_cast<float>(gamma_);
    v.lv = d_vl32_.data();
    v.dense_inv = dense32_.data();
    return v;
}

double AmgPreconditioner::sellVcycleBytes() const {
    // One V-cycle of the SELL persistent kernel, every array a phase touches counted once.
    const int L = static_cast<int>(levels_.size());
    const int nu = std::max(1, std::min(2, cfg_.amg_smoothing_steps));
    const double s = fp32_ ? 4.0 : 8.0;  // V-cycle value size
    double bytes = 0.0;
    for (int l = 0; l + 1 < L; ++l) {
        const Level* f = levels_[l];
        const double n = f->n, nc = levels_[l + 1]->n;
        const double sweep = (4.0 + s) * static_cast<double>(f->sell_entries) + 4.0 * (f->nslices + 1) + s * n;  // matrix + diag
        if (nu >= 2) bytes += sweep + 4.0 * s * n;                   // D1: w (gathered), rd, b read; x written
        bytes += sweep + 3.0 * s * n;                                // D2: x, b read; t written
        bytes += 4.0 * (nc + 1) + 4.0 * n + s * n + 3.0 * s * nc;    // D3: lists, t read; b_c, w_c written, rd_c read
        bytes += sweep + 4.0 * s * n;                                // U1: y, rd, b read; t (or output) written
        if (nu >= 2) bytes += sweep + 4.0 * s * n;                   // U2: t, rd, b read; output written
        bytes += 4.0 * n + 4.0 * (nc + 1) + 2.0 * s * n;             // pushes into the finer iterate (l > 0) / z
    }
    const double nc = levels_.back()->n;
    bytes += s * nc * nc + 2.0 * s * nc + 12.0 * (L > 1 ? levels_[L - 2]->n : 0);  // dense solve + push
    return bytes;
}

double AmgPreconditioner::treeSolveBytes(const TreePlan::Place& place, int iterations, bool warm, bool started) const {
    const int levels = place.levels, top = place.top;
    constexpr double s = 8.0, k = 8.0;  // V-cycle and Krylov values
    const double N = levels_[0]->n, it = iterations;
    const double applications = started ? std::max(1.0, it) : 0.0;
    const auto rows = [&](int l) { return static_cast<double>(levels_[l]->n); };
    const auto sweep = [&](int l) {  // one pass over a streamed level's matrix and diagonal
        const Level* f = levels_[l];
        return 12.0 * static_cast<double>(f->sell_entries) + 4.0 * (f->nslices + 1) + 8.0 * f->n;
    };
    double once = 0.0, cycle = 0.0;
    for (int l = top; l < levels - 1; ++l) {  // CSR row, column positions, diagonals and maps, to shared memory
        const Level* f = levels_[l];
        once += 12.0 * static_cast<double>(f->nnz) + 16.0 * f->n + 16.0 * f->npos;
    }
    if (levels == 1) {  // the dense inverse alone
        cycle = s * N * N + (k + s) * N;
    } else {
        for (int l = 0; l < top; ++l) {  // levels streamed in their own numbering
            const double n = rows(l), nc = rows(l + 1);
            if (l > 0) cycle += sweep(l) + 3.0 * s * n;               // w (gathered), b read; t written
            cycle += s * n + (l + 1 < top ? 4.0 * (nc + 1) + 4.0 * n + 3.0 * s * nc   // lists, t, rd read; b, w written
                                          : 16.0 * plan_.positions[l + 1] + 2.0 * s * nc);
            cycle += (l + 1 < top ? 4.0 * (nc + 1) + 4.0 * n : 16.0 * plan_.positions[l + 1]) + 2.0 * s * n;  // pushes
            cycle += l > 0 ? sweep(l) + 4.0 * s * n                   // y (gathered), rd, b read
                           : sweep(0) + 3.0 * s * n + 2.0 * k * n;    // and r for r . z, z written
        }
        for (int l = std::max(top, 1); l < levels - 1; ++l)              // b, w twice, e(coarse) read; b, w(coarse), e written
            cycle += 5.0 * s * rows(l) + 3.0 * s * rows(l + 1);
        const int c = levels - 1;                                        // dense matrix, b read, e written
        cycle += s * (rows(c) * (c + 1 < static_cast<int>(levels_.size()) ? plan_.positions[c] : rows(c)) + 2.0 * rows(c));
        if (top == 0) cycle += (2.0 * k + s) * N + s * rows(1);          // w, e(coarse), r read; z written
    }
    // per iteration: the product ({z, p} read; p, q and omega/d q written) and the update with the next residual
    const double iteration = top == 0 && levels > 1
                                 ? (2.0 + 3.0) * k * N + (4.0 + 2.0 + 3.0) * k * N + s * N + 2.0 * s * rows(1)
                                 : sweep(0) + 4.0 * k * N + (levels > 1 ? sweep(0) + 6.0 * k * N + 4.0 * s * N : 6.0 * k * N);
    const double first = (warm ? (top == 0 && levels > 1 ? 0.0 : sweep(0)) + 4.0 * k * N : 3.0 * k * N) +
                         (started && levels > 1 ? (top == 0 ? k * N : sweep(0)) + 2.0 * s * N : 0.0);
    return once + first + applications * cycle + it * iteration;
}

AmgView<double> AmgPreconditioner::deviceView() const {
    AmgView<double> v;
    v.levels = static_cast<int>(levels_.size());
    v.nu = std::max(1, std::min(2, cfg_.amg_smoothing_steps));
    v.gamma = gamma_;
    v.lv = d_views_.data();
    const Level* last = levels_.back();
    v.dense_inv = last->dense.data();
    v.dense_ld = last->n;
    return v;
}

double AmgPreconditioner::vcycleBytes() const {
    const int L = static_cast<int>(levels_.size());
    const int nu = std::max(1, std::min(2, cfg_.amg_smoothing_steps));
    double bytes = 0.0;
    for (int l = 0; l + 1 < L; ++l) {
        const double n = levels_[l]->n, nc = levels_[l + 1]->n;
        const double matrix = 8.0 * n + 4.0 * (n + 1) + 12.0 * static_cast<double>(levels_[l]->nnz);
        // pre-smoothing: nu == 2 reads the matrix once (first sweep formed on the fly)
        bytes += nu == 2 ? matrix + 24.0 * n : 24.0 * n;
        // residual + restriction: aggregate lists, matrix, x, b; coarse b written
        bytes += 4.0 * (nc + 1) + 4.0 * n + matrix + 16.0 * n + 8.0 * nc;
        // prolongation + first post sweep: matrix, x, agg, rd, b, coarse x; t (or z) written
        bytes += matrix + 36.0 * n + 8.0 * nc;
        if (nu == 2) bytes += matrix + 32.0 * n + (l == 0 ? 8.0 * n : 0.0);  // second sweep (+ r for r.z)
        else bytes += l == 0 ? 8.0 * n : 16.0 * n;                           // r.z, or the t -> x copy
    }
    const double nc = levels_.back()->n;
    bytes += 8.0 * nc * nc + 16.0 * nc;  // dense coarsest solve
    return bytes;
}

void AmgPreconditioner::apply(Context& ctx, const double* r, double* z) {
    const int L = static_cast<int>(levels_.size());
    const int nu = std::max(1, cfg_.amg_smoothing_steps);
    cudaStream_t s = ctx.stream;
    std::vector<double*> xs(L, nullptr);   // buffer holding each level's pre-smoothed iterate
    // Downward leg: damped-Jacobi pre-smoothing from a zero guess, then the
    // fused residual + aggregate restriction.
    for (int l = 0; l < L - 1; ++l) {
        Level* f = levels_[l];
        Level* c = levels_[l + 1];
        const double* b = l == 0 ? r : f->b.data();
        double* cur = f->x.data();
        double* other = f->t.data();
        const unsigned g = gridFor(f->n, kBlock);
        BSG_PROFILE(ctx, l == 0 ? "amg_pre_smooth_restrict_l0" : "amg_coarse_levels");
        kSmoothZero<<<g, kBlock, 0, s>>>(f->n, f->rdiag.data(), b, cur);
        ctx.launched();
        for (int it = 1; it < nu; ++it) {
            kSmooth<<<g, kBlock, 0, s>>>(f->n, f->dptr, f->dcol, f->ddiag, f->dval, f->rdiag.data(), b, cur, other);
            ctx.launched();
            std::swap(cur, other);
        }
        xs[l] = cur;
        kResidualRestrict<<<gridFor(c->n, kBlock), kBlock, 0, s>>>(c->n, f->agg_ptr.data(), f->agg_rows.data(), f->dptr,
                                                                    f->dcol, f->ddiag, f->dval, b, cur, c->b.data());
        ctx.launched();
    }
    Level* last = levels_.back();
    {
        BSG_PROFILE(ctx, "amg_coarse_levels");
        const double* b = L == 1 ? r : last->b.data();
        double* x = L == 1 ? z : last->x.data();
        kDenseSolve<<<gridFor(last->n, 128), 128, 0, s>>>(last->n, last->dense.data(), b, x);
        ctx.launched();
        xs[L - 1] = x;
    }
    // Upward leg: first post-smoothing sweep fused with the prolongation, then
    // further sweeps ping-pong; level 0 ends in z.
    for (int l = L - 2; l >= 0; --l) {
        Level* f = levels_[l];
        const double* b = l == 0 ? r : f->b.data();
        double* x = xs[l];
        double* other = x == f->x.data() ? f->t.data() : f->x.data();
        const unsigned g = gridFor(f->n, kBlock);
        BSG_PROFILE(ctx, l == 0 ? "amg_prolong_post_smooth_l0" : "amg_coarse_levels");
        double* out = (l == 0 && nu == 1) ? z : other;
        kProlongSmooth<<<g, kBlock, 0, s>>>(f->n, f->dptr, f->dcol, f->ddiag, f->dval, f->rdiag.data(), f->agg.data(),
                                            xs[l + 1], b, x, out);
        ctx.launched();
        double* cur = out;
        for (int it = 1; it < nu; ++it) {
            double* dst = (l == 0 && it == nu - 1) ? z : (cur == f->x.data() ? f->t.data() : f->x.data());
            kSmooth<<<g, kBlock, 0, s>>>(f->n, f->dptr, f->dcol, f->ddiag, f->dval, f->rdiag.data(), b, cur, dst);
            ctx.launched();
            cur = dst;
        }
        xs[l] = cur;
    }
    BSG_CUDA(cudaGetLastError());
}

}  // namespace bsg
