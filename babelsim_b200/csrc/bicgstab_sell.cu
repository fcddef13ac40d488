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
template <int C, bool STREAM, class T>
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
            cc[u] = entryLoad<STREAM>(cp + 32 * (k + u));
            vv[u] = entryLoad<STREAM>(vp + 32 * (k + u));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int c = 0; c < C; ++c) a[c] += vv[u] * x[C * cc[u] + c];
    }
    for (; k < w; ++k) {
        const int j = entryLoad<STREAM>(cp + 32 * k);
        const T v = entryLoad<STREAM>(vp + 32 * k);
#pragma unroll
        for (int c = 0; c < C; ++c) a[c] += v * x[C * j + c];
    }
    const int i = 32 * sl + lane;
    const T d = i < S.n ? S.diag[i] : T(0);
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = (i < S.n ? d * x[C * i + c] : T(0)) + a[c];
}

// f(i, (A x)_i) for every row i, one thread per row.
template <int C, class T, class F>
__device__ __forceinline__ void productRows(const SellMat<T>& A, const Lanes& ln, const T* __restrict__ x, F f) {
    for (int sl = ln.gwarp; sl < A.nslices; sl += ln.nwarps) {
        T acc[C];
        if (A.stream) sellProduct<C, true>(A, sl, ln.lane, x, acc);
        else sellProduct<C, false>(A, sl, ln.lane, x, acc);
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
    productRows<C>(A, ln, a.x, [&](int i, const T* acc) {
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
        productRows<C>(A, ln, a.ph, [&](int i, const T* acc) {
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
        productRows<C>(A, ln, a.sh, [&](int i, const T* acc) {
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
    productRows<C>(A, ln, a.x, [&](int i, const T* acc) {
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

// ---- the on-chip solver
//
// A small or middling solve is latency: five barriers per iteration, each followed by loads whose
// addresses depend on one another (slice offset -> column -> vector).  Here each CTA owns a range of
// slices and copies its matrix rows into shared memory once; neighbours only ever gather ph and sh, so
// the other vectors, which nobody else reads, live in shared memory too.  The direction and the solution
// update share a phase: rho' = r0 . r is taken as r0 . s - omega r0 . t, whose products ride with those of
// the two phases before, so beta is known when x, r and p are formed and four barriers remain.  ||r|| itself
// is summed as before.  FP64 systems only (see launchBicgstab).

struct ChipSlot {
    int s0, nsl, k, nu;  // slices [s0, s0 + nsl), 2^k lanes per row, nsl << k units
};

// Threads per CTA of the on-chip solver: half as many as the streaming one, for twice the registers.
constexpr int CB = 512;

__host__ __device__ inline int chipLanes(int slices_per_cta) {
    int k = 0;
    while (k < 3 && (slices_per_cta << (k + 1)) <= CB / 32) ++k;
    return k;
}

__device__ __forceinline__ char* chipRows() {
    extern __shared__ __align__(16) char chip_rows[];
    return chip_rows;
}

template <int C, class T, class G>
__device__ void bicgChip(G& g, const BicgArgs<C, T>& a) {
    constexpr int BS = CB;
    constexpr int W = kGatherStride<C>;
    enum { R, R0, P, V, X, TT, kVectors };
    const SellMat<T>& A = a.A;
    const int n = A.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    ChipSlot t;
    {
        const int size = g.size(), rank = g.rank();
        t.s0 = static_cast<int>(static_cast<long long>(A.nslices) * rank / size);
        t.nsl = static_cast<int>(static_cast<long long>(A.nslices) * (rank + 1) / size) - t.s0;
        t.k = chipLanes((A.nslices + size - 1) / size);
        t.nu = t.nsl << t.k;
    }
    const int K = 1 << t.k, rows = 32 >> t.k, q = lane & (K - 1), nloc = 32 * t.nsl, i0 = 32 * t.s0;
    int2* dir = reinterpret_cast<int2*>(chipRows());
    // layout: directory, d and 1/d, own vectors, then the units' rows (values, columns)
    const int own_at = ((8 * t.nu + 15) >> 4) << 4;
    T* own = reinterpret_cast<T*>(chipRows() + own_at);
    const int own_values = (2 + kVectors * C) * nloc;
    const int rows_at = own_at + ((own_values * static_cast<int>(sizeof(T)) + 15) >> 4 << 4);
    for (int u = tid; u < t.nu; u += BS) {
        const int s = t.s0 + (u >> t.k);
        dir[u] = make_int2(0, (((A.sptr[s + 1] - A.sptr[s]) >> 5) + K - 1) >> t.k);
    }
    __syncthreads();
    constexpr int kStepBytes = 32 * (sizeof(T) + sizeof(int));
    if (warp == 0) {  // running sum of the units' sizes
        int base = rows_at;
        for (int u0 = 0; u0 < t.nu; u0 += 32) {
            const int u = u0 + lane;
            const int bytes = u < t.nu ? dir[u].y * kStepBytes : 0;
            int sum = bytes;
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += up;
            }
            if (u < t.nu) dir[u].x = base + sum <= a.chip ? base + sum - bytes : -1;
            base += __shfl_sync(0xffffffffu, sum, 31);
        }
    }
    __syncthreads();
    for (int u = warp; u < t.nu; u += BS / 32) {
        const int2 e = dir[u];
        if (e.x < 0) continue;
        const int s = t.s0 + (u >> t.k), r = (u & (K - 1)) * rows + (lane >> t.k);
        const int beg = A.sptr[s], w = (A.sptr[s + 1] - beg) >> 5;
        T* val = reinterpret_cast<T*>(chipRows() + e.x);
        int* col = reinterpret_cast<int*>(val + 32 * e.y);
        for (int step = 0; step < e.y; ++step) {
            const int k = q + (step << t.k);
            col[32 * step + lane] = k < w ? __ldg(A.col + beg + 32 * k + r) : min(32 * s + r, n - 1);
            val[32 * step + lane] = k < w ? __ldg(A.val + beg + 32 * k + r) : T(0);
        }
    }
    T *dg = own, *rdg = own + nloc;
    for (int l = tid; l < nloc; l += BS) {
        const T d = i0 + l < n ? A.diag[i0 + l] : T(1);
        dg[l] = d;
        rdg[l] = T(1) / d;
    }
    T* vec = own + 2 * nloc;
    // component c of own vector `which`, local row l
    const auto at = [&](int which, int c, int l) -> T& { return vec[(which * C + c) * nloc + l]; };
    __syncthreads();
    // f(l, (A y)_i) for every own row; y is gathered with `stride` entries per row
    const auto product = [&](const T* y, int stride, auto f) {
        for (int u = warp; u < t.nu; u += BS / 32) {
            const int2 e = dir[u];
            const int sub = (u & (K - 1)) * rows + (lane >> t.k), l = 32 * (u >> t.k) + sub, i = i0 + l;
            T acc[C];
            {
                const bool mine = q == 0 && i < n;
                const T d = mine ? dg[l] : T(0);
#pragma unroll
                for (int c = 0; c < C; ++c) acc[c] = mine ? d * y[stride * i + c] : T(0);
            }
            const auto load = [&](int j, T yy[C]) {
                if constexpr (C == 3 && sizeof(T) == 8) {
                    if (stride == 4) {
                        const double2 lo = *reinterpret_cast<const double2*>(y + 4 * static_cast<long long>(j));
                        yy[0] = lo.x;
                        yy[1] = lo.y;
                        yy[2] = y[4 * static_cast<long long>(j) + 2];
                        return;
                    }
                }
#pragma unroll
                for (int c = 0; c < C; ++c) yy[c] = y[static_cast<long long>(stride) * j + c];
            };
            if (e.x >= 0) {
                const T* val = reinterpret_cast<const T*>(chipRows() + e.x) + lane;
                const int* col = reinterpret_cast<const int*>(reinterpret_cast<const T*>(chipRows() + e.x) + 32 * e.y) + lane;
                for (int k = 0; k < e.y; k += 4) {
                    T yy[4][C];
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if (k + m < e.y) load(col[32 * (k + m)], yy[m]);
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if (k + m < e.y) {
                            const T v = val[32 * (k + m)];
#pragma unroll
                            for (int c = 0; c < C; ++c) acc[c] += v * yy[m][c];
                        }
                }
            } else {  // rows that did not fit
                const int s = t.s0 + (u >> t.k);
                const int beg = A.sptr[s], w = (A.sptr[s + 1] - beg) >> 5;
                for (int k = q; k < w; k += K) {
                    const T v = __ldg(A.val + beg + 32 * k + sub);
                    T yy[C];
                    load(__ldg(A.col + beg + 32 * k + sub), yy);
#pragma unroll
                    for (int c = 0; c < C; ++c) acc[c] += v * yy[c];
                }
            }
            for (int o = K >> 1; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < C; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
            if (q == 0 && i < n) f(l, acc);
        }
    };
    BicgState& st = *a.st;
    int buf = 0;
    double rho[C], alpha[C], omega[C], target2[C];
    int done[C], iters[C];
    const int max_iters = st.max_iters;
    double nb[2 * C];
#pragma unroll
    for (int j = 0; j < 2 * C; ++j) nb[j] = 0.0;
    // inputs are read before block 0 writes any result into the same struct
#pragma unroll
    for (int c = 0; c < C; ++c) {
        done[c] = st.done[c];
        iters[c] = st.iters[c];
        target2[c] = st.target2[c];
        omega[c] = 1.0;
    }
    const auto active = [&](int c) { return done[c] == 0 && iters[c] < max_iters; };
    // r = b - A x, r0 = p = r, ph = p / d; ||r||^2 and ||b||^2 per component
    product(a.x, C, [&](int l, const T* acc) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int i = i0 + l;
            const T bi = a.b[C * i + c], ri = bi - acc[c];
            at(R, c, l) = ri;
            at(R0, c, l) = ri;
            at(P, c, l) = ri;
            at(X, c, l) = a.x[C * i + c];
            a.gph[W * static_cast<long long>(i) + c] = ri * rdg[l];
            nb[c] += dd(ri) * dd(ri);
            nb[C + c] += dd(bi) * dd(bi);
        }
    });
    gridSum<2 * C, BS>(g, nb, a.partial, buf);
#pragma unroll
    for (int c = 0; c < C; ++c) {
        rho[c] = nb[c];
        if (target2[c] < 0.0) {
            // the reference's contract: max(atol, rtol * max(||r0||, ||b||)) (solver_control.h:199-210)
            double scale = fmax(sqrt(nb[c]), sqrt(nb[C + c]));
            if (!(scale > 0.0)) scale = 1.0;
            const double tg = fmax(st.atol, st.rtol * scale);
            target2[c] = tg * tg;
        }
        if (done[c] == 0 && (!(nb[c] > 0.0) || nb[c] <= target2[c])) done[c] = 1;
    }
    g.sync();  // every CTA has read the struct
    if (g.rank() == 0 && tid == 0) {
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
        // v = A ph, r0 . v
        double r0v[C];
#pragma unroll
        for (int c = 0; c < C; ++c) r0v[c] = 0.0;
        product(a.gph, W, [&](int l, const T* acc) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                at(V, c, l) = acc[c];
                r0v[c] += dd(at(R0, c, l)) * dd(acc[c]);
            }
        });
        gridSum<C, BS>(g, r0v, a.partial, buf);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (!active(c)) continue;
            if (!(fabs(r0v[c]) > 0.0) || !isfinite(r0v[c])) { done[c] = 2; continue; }
            alpha[c] = rho[c] / r0v[c];
        }
        // s = r - alpha v (kept in r), sh = s / d; ||s||^2 and r0 . s
        double ss[2 * C];
#pragma unroll
        for (int j = 0; j < 2 * C; ++j) ss[j] = 0.0;
        for (int l = tid; l < nloc && i0 + l < n; l += BS) {
            const T rd = rdg[l];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                if (!active(c)) continue;
                const T si = at(R, c, l) - static_cast<T>(alpha[c]) * at(V, c, l);
                at(R, c, l) = si;
                a.gsh[W * static_cast<long long>(i0 + l) + c] = si * rd;
                ss[c] += dd(si) * dd(si);
                ss[C + c] += dd(at(R0, c, l)) * dd(si);
            }
        }
        gridSum<2 * C, BS>(g, ss, a.partial, buf);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (!active(c)) continue;
            if (!isfinite(ss[c])) done[c] = 2;
            else if (ss[c] <= target2[c]) done[c] = 3;  // the half step is accepted
        }
        // t = A sh; t . t, t . s and r0 . t
        double ts[3 * C];
#pragma unroll
        for (int j = 0; j < 3 * C; ++j) ts[j] = 0.0;
        product(a.gsh, W, [&](int l, const T* acc) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                at(TT, c, l) = acc[c];
                ts[3 * c] += dd(acc[c]) * dd(acc[c]);
                ts[3 * c + 1] += dd(acc[c]) * dd(at(R, c, l));
                ts[3 * c + 2] += dd(acc[c]) * dd(at(R0, c, l));
            }
        });
        gridSum<3 * C, BS>(g, ts, a.partial, buf);
        // x += alpha ph + omega sh, r = s - omega t, p = r + beta (p - omega v), ph = p / d; ||r||^2
        // (half step: x += alpha ph)
        int mode[C];
        double beta[C], rho_new[C], rr[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            rr[c] = 0.0;
            beta[c] = rho_new[c] = 0.0;
            mode[c] = done[c] == 3 ? 2 : (active(c) ? 1 : 0);
            if (mode[c] != 1) continue;
            omega[c] = ts[3 * c] > 0.0 ? ts[3 * c + 1] / ts[3 * c] : 0.0;
            rho_new[c] = ss[C + c] - omega[c] * ts[3 * c + 2];
            beta[c] = (rho_new[c] / rho[c]) * (alpha[c] / omega[c]);
        }
        for (int l = tid; l < nloc && i0 + l < n; l += BS) {
            const T rd = rdg[l];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                if (mode[c] == 0) continue;
                const T pi = at(P, c, l);
                if (mode[c] == 2) {
                    at(X, c, l) += static_cast<T>(alpha[c]) * (pi * rd);
                    continue;
                }
                const T si = at(R, c, l);
                at(X, c, l) += static_cast<T>(alpha[c]) * (pi * rd) + static_cast<T>(omega[c]) * (si * rd);
                const T ri = si - static_cast<T>(omega[c]) * at(TT, c, l);
                at(R, c, l) = ri;
                rr[c] += dd(ri) * dd(ri);
                const T pn = ri + static_cast<T>(beta[c]) * (pi - static_cast<T>(omega[c]) * at(V, c, l));
                at(P, c, l) = pn;
                a.gph[W * static_cast<long long>(i0 + l) + c] = pn * rd;
            }
        }
        gridSum<C, BS>(g, rr, a.partial, buf);
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (done[c] == 3) { done[c] = 1; iters[c] += 1; continue; }
            if (!active(c)) continue;
            iters[c] += 1;
            if (!isfinite(rr[c])) { done[c] = 2; continue; }
            if (rr[c] <= target2[c]) { done[c] = 1; continue; }
            if (omega[c] == 0.0 || !(fabs(rho_new[c]) > 0.0)) { done[c] = 2; continue; }
            rho[c] = rho_new[c];
        }
    }
    for (int l = tid; l < nloc && i0 + l < n; l += BS)
#pragma unroll
        for (int c = 0; c < C; ++c) a.x[C * (i0 + l) + c] = at(X, c, l);
    // the true residual of every component (the acceptance test's norm)
    double fr[C];
#pragma unroll
    for (int c = 0; c < C; ++c) fr[c] = 0.0;
    g.sync();
    product(a.x, C, [&](int l, const T* acc) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const T ri = a.b[C * (i0 + l) + c] - acc[c];
            fr[c] += dd(ri) * dd(ri);
        }
    });
    gridSum<C, BS>(g, fr, a.partial, buf);
    if (g.rank() == 0 && tid == 0) {
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
__global__ void __launch_bounds__(CB, 1) kBicgChip(const __grid_constant__ BicgArgs<C, T> a, SegmentBarrier* bar) {
    GridGroup g{bar};
    bicgChip<C, T>(g, a);
}

// A small system on one cluster.
template <int C, class T>
__global__ void __launch_bounds__(CB, 1) kBicgChipCluster(const __grid_constant__ BicgArgs<C, T> a) {
    ClusterGroup g;
    g.sync();  // every CTA's shared memory is live
    bicgChip<C, T>(g, a);
}

template <int C, class T>
__global__ void __launch_bounds__(BB, 1) kBicgSell(const __grid_constant__ BicgArgs<C, T> a, SegmentBarrier* bar) {
    GridGroup g{bar};
    bicgBody<C, T, BB>(g, a);
}

// The systems of a batched launch as one kernel argument.
template <int C>
struct BicgArgsBlock {
    BicgArgs<C> a[kBatchArgs];
    int begin[kBatchArgs + 1];  // CTA ranges
    int count;
};
static_assert(sizeof(BicgArgsBlock<3>) + sizeof(void*) <= kKernelArgumentBytes, "one kernel argument");

// A batch: CTAs [begin[s], begin[s+1]) solve system s.
template <int C>
__global__ void __launch_bounds__(BB, 1)
    kBicgSellBatch(const __grid_constant__ BicgArgsBlock<C> batch, SegmentBarrier* bars) {
    const int s = systemOfBlock(batch.begin, batch.count);
    SegmentGroup g{batch.begin[s], batch.begin[s + 1] - batch.begin[s], bars + s};
    bicgBody<C, double, BB>(g, batch.a[s]);
}

constexpr int kChipSmem = 200 * 1024;
// Largest system that one cluster (barrier 0.3 us instead of 1.3, but 16 SMs) solves on chip faster than
// the grid does.  Three right-hand sides, ms per solve, cluster / grid on chip / grid streamed: 1000-cell
// Voronoi cube 0.25 / 0.52 / 0.92, 4096 cells 0.33 / 0.55 / 1.00, 2D cavity of 4096 cells 0.10 / 0.21 /
// 0.27; grid on chip / streamed: 13824 cells 0.58 / 1.07, 32768 cells 0.61 / 1.05, 64000 cells 0.75 /
// 1.07, 97k hex cells 0.94 / 1.19.
constexpr int kClusterRows = 8192;

// Bytes of shared memory per CTA that hold the system's rows and vectors on `ctas` CTAs; 0 where there
// is no room (keeping the rows alone was tried: 110k-cell Voronoi cube 1.24 ms against 1.06 streamed).
template <int C, class T>
int chipBytes(int nslices, long long entries, int ctas) {
    const int per = (nslices + ctas - 1) / ctas;  // slices of the fullest CTA
    const int k = chipLanes(per);
    const double wide = nslices > 0 ? static_cast<double>(entries) / (32.0 * nslices) : 0.0;
    const double steps = k == 0 ? wide : wide / (1 << k) + 0.5;
    // a few per cent for slices wider than the mean (a unit that does not fit is read from memory)
    const double rows = 1.06 * (per << k) * steps * 32.0 * (sizeof(T) + 4.0) + 2048.0;
    const double vectors = 8.0 * (per << k) + 32.0 * per * (2.0 + 6.0 * C) * sizeof(T) + 64.0;
    const double bytes = std::ceil((rows + vectors) / 1024.0) * 1024.0;
    return bytes <= kChipSmem ? static_cast<int>(bytes) : 0;
}

// Where a system runs on chip: the bytes per CTA of a cluster or of the grid (0: streamed).
struct ChipPlace {
    bool cluster;
    int bytes;
};
template <int C, class T>
ChipPlace chipPlace(Context& ctx, const SellMat<T>& A, long long entries) {
    if (A.n <= kClusterRows) {
        allowSharedMemory<kBicgChipCluster<C, T>>(kChipSmem);
        const int bytes = chipBytes<C, T>(A.nslices, entries, clusterCtas<kBicgChipCluster<C, T>>(CB, kChipSmem));
        if (bytes) return {true, bytes};
    }
    return {false, chipBytes<C, T>(A.nslices, entries, ctx.sm_count)};
}

}  // namespace

template <int C>
bool bicgstabOnChip(Context& ctx, const SellMat<double>& A, long long entries) {
    return chipPlace<C, double>(ctx, A, entries).bytes > 0;
}

template <int C, class T>
void launchBicgstab(Context& ctx, const BicgArgs<C, T>& args) {
    BSG_PROFILE(ctx, C == 3 ? (sizeof(T) == 4 ? "bicgstab3_persistent_fp32" : "bicgstab3_persistent")
                            : (sizeof(T) == 4 ? "bicgstab1_persistent_fp32" : "bicgstab1_persistent"));
    BicgArgs<C, T> a = args;
    // FP32 systems are the inner solves of a refined one, which accepts the first iterate under its target:
    // what the inner iterations round decides which one that is, to a part of the target.  They keep the
    // streaming kernel's arithmetic (r0 . r of the residual that is kept, the diagonal last), at 0.96 against
    // 0.86 ms for three right-hand sides on 110k cells.
    if constexpr (sizeof(T) == 8) {
        const ChipPlace place = chipPlace<C, T>(ctx, a.A, a.entries);
        a.chip = place.bytes;
        if (place.cluster) {
            launchCluster<kBicgChipCluster<C, T>>(ctx, 1, CB, a.chip, kChipSmem, a);
            return;
        }
    }
    SegmentBarrier* bar = ctx.grid_barrier;
    const int grid = ctx.sm_count;
    resetBarriers(ctx, bar, 1, grid);
    void* params[] = {&a, &bar};
    if constexpr (sizeof(T) == 8) {
        if (a.chip) {
            allowSharedMemory<kBicgChip<C, T>>(kChipSmem);
            BSG_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kBicgChip<C, T>), grid, CB, params, a.chip, ctx.stream));
            ctx.launched();
            return;
        }
    }
    BSG_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kBicgSell<C, T>), grid, BB, params, 0, ctx.stream));
    ctx.launched();
}

template <int C>
void launchBicgstabBatch(Context& ctx, BicgBatch<C>& batch) {
    BSG_PROFILE(ctx, "bicgstab3_persistent_batch");
    const std::size_t count = batch.args.size();
    if (count == 0) return;
    batch.d_bars.resize(std::max(batch.d_bars.size(), count));
    std::vector<long long> slices(count);
    for (std::size_t i = 0; i < count; ++i) slices[i] = batch.args[i].A.nslices;
    const std::vector<std::size_t> launches = batchLaunches(slices, BB / 32, ctx.sm_count);
    for (std::size_t l = 0; l + 1 < launches.size(); ++l) {
        const std::size_t k0 = launches[l], k1 = launches[l + 1];
        BicgArgsBlock<C> block{};
        block.count = static_cast<int>(k1 - k0);
        std::copy(batch.args.begin() + k0, batch.args.begin() + k1, block.a);
        const std::vector<int> begin = allotCtas({slices.begin() + k0, slices.begin() + k1}, BB / 32, ctx.sm_count);
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

template bool bicgstabOnChip<3>(Context&, const SellMat<double>&, long long);
template bool bicgstabOnChip<1>(Context&, const SellMat<double>&, long long);
template void launchBicgstab<3, double>(Context&, const BicgArgs<3, double>&);
template void launchBicgstab<1, double>(Context&, const BicgArgs<1, double>&);
template void launchBicgstab<3, float>(Context&, const BicgArgs<3, float>&);
template void launchBicgstab<1, float>(Context&, const BicgArgs<1, float>&);
template void launchBicgstabBatch<3>(Context&, BicgBatch<3>&);  // (scalar systems are not batched)

}  // namespace bsg
