// Persistent cooperative BiCGStab on SELL-32 (see bicgstab_sell.cuh).
//
// The iteration is the one of the reference's PETSc KSPBCGS with a point-Jacobi
// (right) preconditioner, per component c with its own rho, alpha, omega, beta:
//   p  = r + beta (p - omega v),  ph = p / d
//   v  = A ph,                    alpha = rho / (r0 . v)
//   s  = r - alpha v,             sh = s / d      (||s|| <= target: x += alpha ph, done)
//   t  = A sh,                    omega = (t . s) / (t . t)
//   x += alpha ph + omega sh,     r = s - omega t, rho' = r0 . r, beta = (rho'/rho)(alpha/omega)
// Phases are separated by group barriers (grid-wide, or per system of a batch),
// and every CTA keeps identical copies of the scalars because every reduction
// gives all CTAs the same fixed-order total.
#include "bicgstab_sell.cuh"

#include <algorithm>
#include <cmath>

namespace bsg {
namespace {

constexpr int BB = 1024;  // threads per CTA, one CTA per SM

// (A x)_i for the C components of row i of slice sl (lane = row within the slice).
template <int C, class T>
__device__ __forceinline__ void sellProduct(const SellMat<T>& S, int sl, int lane, const T* __restrict__ x, T acc[C]) {
    const int beg = S.sptr[sl], w = (S.sptr[sl + 1] - beg) >> 5;
    const int* __restrict__ cp = S.col + beg + lane;
    const T* __restrict__ vp = S.val + beg + lane;
    T a[C];
#pragma unroll
    for (int c = 0; c < C; ++c) a[c] = T(0);
    int k = 0;
    for (; k + 4 <= w; k += 4) {
        int cc[4];
        T vv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            cc[u] = __ldg(cp + 32 * (k + u));
            vv[u] = __ldg(vp + 32 * (k + u));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int c = 0; c < C; ++c) a[c] += vv[u] * x[C * cc[u] + c];
    }
    for (; k < w; ++k) {
        const int j = __ldg(cp + 32 * k);
        const T v = __ldg(vp + 32 * k);
#pragma unroll
        for (int c = 0; c < C; ++c) a[c] += v * x[C * j + c];
    }
    const int i = 32 * sl + lane;
    const T d = i < S.n ? S.diag[i] : T(0);
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = (i < S.n ? d * x[C * i + c] : T(0)) + a[c];
}

// The same row split over K consecutive lanes (see sellRowSplit); every lane of the warp calls it.
template <int C, class T>
__device__ __forceinline__ void sellProductSplit(const SellMat<T>& S, const SplitUnit& u, int K,
                                                 const T* __restrict__ x, T acc[C]) {
    const int beg = S.sptr[u.s], w = (S.sptr[u.s + 1] - beg) >> 5;
    const int* __restrict__ cp = S.col + beg + u.r;
    const T* __restrict__ vp = S.val + beg + u.r;
    const int i = 32 * u.s + u.r;
    const bool own = u.q == 0 && i < S.n;  // this lane takes the diagonal
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = own ? S.diag[i] * x[C * i + c] : T(0);
    for (int k = u.q; k < w; k += K) {
        const int j = __ldg(cp + 32 * k);
        const T v = __ldg(vp + 32 * k);
#pragma unroll
        for (int c = 0; c < C; ++c) acc[c] += v * x[C * j + c];
    }
    for (int o = K >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < C; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
}

// f(i, (A x)_i) for every row i, one thread per row (on a cluster K lanes per row where the
// system has fewer slices than the cluster has warps).
template <int C, class G, class T, class F>
__device__ __forceinline__ void productRows(const SellMat<T>& A, const Lanes& ln, const T* __restrict__ x, F f) {
    if (kInCluster<G>) {
        const int K = splitOf(A.nslices, ln.nwarps);
        if (K > 1) {
            for (int u = ln.gwarp; u < A.nslices * K; u += ln.nwarps) {
                const SplitUnit su = splitUnit(u, K, ln.lane);
                T acc[C];
                sellProductSplit<C, T>(A, su, K, x, acc);
                const int i = 32 * su.s + su.r;
                if (su.q == 0 && i < A.n) f(i, acc);
            }
            return;
        }
    }
    for (int sl = ln.gwarp; sl < A.nslices; sl += ln.nwarps) {
        T acc[C];
        sellProduct<C, T>(A, sl, ln.lane, x, acc);
        const int i = 32 * sl + ln.lane;
        if (i < A.n) f(i, acc);
    }
}

// Products of vector entries are summed in FP64 whatever the vectors' type.
template <class T>
__device__ __forceinline__ double dd(T x) {
    return static_cast<double>(x);
}

template <int C, class T, int BS, class G>
__device__ void bicgBody(G& g, const BicgArgs<C, T>& a) {
    const Lanes ln = lanes<BS>(g);
    const SellMat<T>& A = a.A;
    const int n = A.n;
    BicgState& st = *a.st;
    int buf = 0;
    double rho[C], alpha[C], omega[C], beta[C], target2[C];
    int done[C], iters[C];
    double target2_in[C];
    const int max_iters = st.max_iters;
    // inputs are read before block 0 writes any result into the same struct
#pragma unroll
    for (int c = 0; c < C; ++c) {
        done[c] = st.done[c];
        iters[c] = st.iters[c];
        target2_in[c] = st.target2[c];
        alpha[c] = 1.0;
        omega[c] = 1.0;
        beta[c] = 0.0;
    }
    auto active = [&](int c) { return done[c] == 0 && iters[c] < max_iters; };
    // r = b - A x, r0 = r, p = v = 0; ||r||^2 and ||b||^2 per component
    double nb[2 * C];
#pragma unroll
    for (int j = 0; j < 2 * C; ++j) nb[j] = 0.0;
    productRows<C, G>(A, ln, a.x, [&](int i, const T* acc) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const T bi = a.b[C * i + c], ri = bi - acc[c];
            a.r[C * i + c] = ri;
            a.r0[C * i + c] = ri;
            a.p[C * i + c] = T(0);
            a.v[C * i + c] = T(0);
            nb[c] += dd(ri) * dd(ri);
            nb[C + c] += dd(bi) * dd(bi);
        }
    });
    gridSum<2 * C, BS>(g, nb, a.partial, buf);
#pragma unroll
    for (int c = 0; c < C; ++c) {
        rho[c] = nb[c];
        if (target2_in[c] < 0.0) {
            // the reference's contract: max(atol, rtol * max(||r0||, ||b||)) (solver_control.h:199-210)
            double scale = fmax(sqrt(nb[c]), sqrt(nb[C + c]));
            if (!(scale > 0.0)) scale = 1.0;
            const double tg = fmax(st.atol, st.rtol * scale);
            target2[c] = tg * tg;
        } else {
            target2[c] = target2_in[c];
        }
        if (done[c] == 0 && (!(nb[c] > 0.0) || nb[c] <= target2[c])) done[c] = 1;
    }
    if (g.rank() == 0 && threadIdx.x == 0) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            st.rr0[c] = nb[c];
            st.bb[c] = nb[C + c];
            st.target2[c] = target2[c];
        }
    }
    for (;;) {
        bool any = false;
#pragma unroll
        for (int c = 0; c < C; ++c) any = any || active(c);
        if (!any || g.aborted()) break;
        // p = r + beta (p - omega v), ph = p / d
        for (int i = ln.gthread; i < n; i += ln.nthreads) {
            const T rd = T(1) / A.diag[i];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                if (!active(c)) continue;
                const T pi = a.r[C * i + c] +
                             static_cast<T>(beta[c]) * (a.p[C * i + c] - static_cast<T>(omega[c]) * a.v[C * i + c]);
                a.p[C * i + c] = pi;
                a.ph[C * i + c] = pi * rd;
            }
        }
        g.sync();
        // v = A ph, r0 . v
        double r0v[C];
#pragma unroll
        for (int c = 0; c < C; ++c) r0v[c] = 0.0;
        productRows<C, G>(A, ln, a.ph, [&](int i, const T* acc) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                a.v[C * i + c] = acc[c];
                r0v[c] += dd(a.r0[C * i + c]) * dd(acc[c]);
            }
        });
        gridSum<C, BS>(g, r0v, a.partial, buf);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (!active(c)) continue;
            if (!(fabs(r0v[c]) > 0.0) || !isfinite(r0v[c])) { done[c] = 2; continue; }
            alpha[c] = rho[c] / r0v[c];
        }
        // s = r - alpha v (kept in r), sh = s / d, ||s||^2
        double ss[C];
#pragma unroll
        for (int c = 0; c < C; ++c) ss[c] = 0.0;
        for (int i = ln.gthread; i < n; i += ln.nthreads) {
            const T rd = T(1) / A.diag[i];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                if (!active(c)) continue;
                const T si = a.r[C * i + c] - static_cast<T>(alpha[c]) * a.v[C * i + c];
                a.r[C * i + c] = si;
                a.sh[C * i + c] = si * rd;
                ss[c] += dd(si) * dd(si);
            }
        }
        gridSum<C, BS>(g, ss, a.partial, buf);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (!active(c)) continue;
            if (!isfinite(ss[c])) done[c] = 2;
            else if (ss[c] <= target2[c]) done[c] = 3;  // the half step is accepted
        }
        // t = A sh, t . t and t . s
        double ts[2 * C];
#pragma unroll
        for (int j = 0; j < 2 * C; ++j) ts[j] = 0.0;
        productRows<C, G>(A, ln, a.sh, [&](int i, const T* acc) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                a.t[C * i + c] = acc[c];
                ts[2 * c] += dd(acc[c]) * dd(acc[c]);
                ts[2 * c + 1] += dd(acc[c]) * dd(a.r[C * i + c]);
            }
        });
        gridSum<2 * C, BS>(g, ts, a.partial, buf);
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (active(c)) omega[c] = ts[2 * c] > 0.0 ? ts[2 * c + 1] / ts[2 * c] : 0.0;
        // x += alpha ph + omega sh, r = s - omega t; ||r||^2 and r0 . r (half step: x += alpha ph)
        int mode[C];
#pragma unroll
        for (int c = 0; c < C; ++c) mode[c] = done[c] == 3 ? 2 : (active(c) ? 1 : 0);
        double nr[2 * C];
#pragma unroll
        for (int j = 0; j < 2 * C; ++j) nr[j] = 0.0;
        for (int i = ln.gthread; i < n; i += ln.nthreads) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                if (mode[c] == 0) continue;
                if (mode[c] == 2) {
                    a.x[C * i + c] += static_cast<T>(alpha[c]) * a.ph[C * i + c];
                    continue;
                }
                a.x[C * i + c] += static_cast<T>(alpha[c]) * a.ph[C * i + c] + static_cast<T>(omega[c]) * a.sh[C * i + c];
                const T ri = a.r[C * i + c] - static_cast<T>(omega[c]) * a.t[C * i + c];
                a.r[C * i + c] = ri;
                nr[2 * c] += dd(ri) * dd(ri);
                nr[2 * c + 1] += dd(a.r0[C * i + c]) * dd(ri);
            }
        }
        gridSum<2 * C, BS>(g, nr, a.partial, buf);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (done[c] == 3) { done[c] = 1; iters[c] += 1; continue; }
            if (!active(c)) continue;
            iters[c] += 1;
            const double rr = nr[2 * c], rho_new = nr[2 * c + 1];
            if (!isfinite(rr)) { done[c] = 2; continue; }
            if (rr <= target2[c]) { done[c] = 1; continue; }
            if (omega[c] == 0.0 || !(fabs(rho_new) > 0.0)) { done[c] = 2; continue; }
            beta[c] = (rho_new / rho[c]) * (alpha[c] / omega[c]);
            rho[c] = rho_new;
        }
    }
    // the true residual of every component (the acceptance test's norm)
    double fr[C];
#pragma unroll
    for (int c = 0; c < C; ++c) fr[c] = 0.0;
    g.sync();
    productRows<C, G>(A, ln, a.x, [&](int i, const T* acc) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const T ri = a.b[C * i + c] - acc[c];
            fr[c] += dd(ri) * dd(ri);
        }
    });
    gridSum<C, BS>(g, fr, a.partial, buf);
    if (g.rank() == 0 && threadIdx.x == 0) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            st.done[c] = done[c];
            st.iters[c] = iters[c];
            st.fin2[c] = fr[c];
        }
        st.status = g.failed() ? 3 : 0;
    }
}

template <int C, class T>
__global__ void __launch_bounds__(BB, 1) kBicgSell(const __grid_constant__ BicgArgs<C, T> a, SegmentBarrier* bar) {
    GridGroup g{bar};
    bicgBody<C, T, BB>(g, a);
}

// Up to kBatchArgs systems as one kernel argument (constant bank: no registers for pointers).
constexpr int kBatchArgs = 32;
template <int C>
struct BicgArgsBlock {
    BicgArgs<C> a[kBatchArgs];
    int begin[kBatchArgs + 1];  // CTA ranges
    int count;
};

// A batch: CTAs [begin[s], begin[s+1]) solve system s.
template <int C>
__global__ void __launch_bounds__(BB, 1)
    kBicgSellBatch(const __grid_constant__ BicgArgsBlock<C> batch, SegmentBarrier* bars) {
    int s = 0;  // the system whose CTA range holds this block
    while (s + 1 < batch.count && batch.begin[s + 1] <= static_cast<int>(blockIdx.x)) ++s;
    SegmentGroup g{batch.begin[s], batch.begin[s + 1] - batch.begin[s], bars + s};
    bicgBody<C, double, BB>(g, batch.a[s]);
}

// A small system on one cluster.
template <int C, class T>
__global__ void __launch_bounds__(BB, 1) kBicgCluster(const __grid_constant__ BicgArgs<C, T> a) {
    ClusterGroup g;
    g.sync();  // every CTA's shared memory is live
    bicgBody<C, T, BB>(g, a);
}
// Largest system one cluster solves faster than the grid (barrier 0.3 us instead of 1.3, but 16 SMs'
// gathers).  Three right-hand sides, ms per solve, cluster / grid: 1000-cell Voronoi cube 0.57 / 0.91,
// 4096 cells 0.65 / 0.99, 13824 cells 0.85 / 1.05, 21952 cells 1.44 / 1.08; 2D cavities of 16384
// cells 0.17 / 0.24, 40000 cells 0.34 / 0.25.
constexpr int kClusterRows = 16384;

}  // namespace

template <int C, class T>
void launchBicgstab(Context& ctx, const BicgArgs<C, T>& args) {
    BSG_PROFILE(ctx, sizeof(T) == 4 ? "bicgstab3_persistent_fp32" : "bicgstab3_persistent");
    if (args.A.n <= kClusterRows) {
        launchCluster<kBicgCluster<C, T>>(ctx, 1, BB, 0, 0, args);
        return;
    }
    SegmentBarrier* bar = ctx.grid_barrier;
    const int grid = ctx.sm_count;
    resetBarriers(ctx, bar, 1, grid);
    BicgArgs<C, T> a = args;
    void* params[] = {&a, &bar};
    BSG_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kBicgSell<C, T>), grid, BB, params, 0, ctx.stream));
    ctx.launched();
}

template <int C>
void launchBicgstabBatch(Context& ctx, BicgBatch<C>& batch) {
    BSG_PROFILE(ctx, "bicgstab3_persistent_batch");
    const std::size_t count = batch.args.size();
    if (count == 0) return;
    const std::size_t chunk = std::min(kBatchArgs, ctx.sm_count);
    batch.d_bars.resize(std::max(batch.d_bars.size(), count));
    for (std::size_t k0 = 0; k0 < count; k0 += chunk) {
        BicgArgsBlock<C> block{};
        block.count = static_cast<int>(std::min(chunk, count - k0));
        std::vector<long long> slices(block.count);
        for (int i = 0; i < block.count; ++i) {
            block.a[i] = batch.args[k0 + i];
            slices[i] = block.a[i].A.nslices;
        }
        const std::vector<int> begin = allotCtas(slices, BB / 32, ctx.sm_count);
        std::copy(begin.begin(), begin.end(), block.begin);
        SegmentBarrier* bars = batch.d_bars.data() + k0;
        resetBarriers(ctx, bars, block.count, begin.back(), block.begin);
        void* params[] = {&block, &bars};
        BSG_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kBicgSellBatch<C>), begin.back(), BB, params, 0,
                                             ctx.stream));
        ctx.launched();
    }
    batch.bars_used = static_cast<int>(count);
}

template void launchBicgstab<3, double>(Context&, const BicgArgs<3, double>&);
template void launchBicgstab<1, double>(Context&, const BicgArgs<1, double>&);
template void launchBicgstab<3, float>(Context&, const BicgArgs<3, float>&);
template void launchBicgstab<1, float>(Context&, const BicgArgs<1, float>&);
template void launchBicgstabBatch<3>(Context&, BicgBatch<3>&);
template void launchBicgstabBatch<1>(Context&, BicgBatch<1>&);

}  // namespace bsg
