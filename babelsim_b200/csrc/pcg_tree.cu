// Persistent PCG + AMG V-cycle with on-chip coarse levels (see pcg_tree.cuh).
#include "pcg_tree.cuh"

#include <algorithm>
#include <cmath>

namespace bsg {
namespace {

constexpr int TB = 1024;            // threads per CTA, one CTA per SM
constexpr int kTreeLanesLog = 3;       // 8 lanes per row at most: a warp holds whole aggregates of four rows
constexpr int kTreeSmem = 200 * 1024;  // shared memory for matrix rows, at most
// The same while finer levels stream through L1, which shares its 228 KB with shared memory
// (1M cells with 200 KB: 126 us per CG product against 58).
constexpr int kStreamSmem = 112 * 1024;
// Largest level-0 matrix (off-diagonal entries) that one cluster solves faster than the grid: its
// barrier costs 0.3 us instead of 1.3, but it has 16 SMs' shared memory and gathers.  PCG solves in
// ms, cluster / grid: 1000-cell Voronoi cube (14k entries) 0.61 / 0.95, 4096 cells (55k) 1.22 /
// 1.45, 8000 cells (112k) 2.0 / 1.5, 16384-cell 2D cavity (65k) 0.90 / 0.98, 21952 cells 4.5 / 2.1.
constexpr long long kClusterEntries = 100000;
// Largest share of the folded coarse matrix per CTA.
constexpr double kFoldedBytes = 96.0 * 1024.0;
constexpr int kDirBytes = 8;

__device__ __forceinline__ void mark(const PhaseLog& log, int id) {
    if (log.entries && blockIdx.x == 0 && threadIdx.x == 0) {
        const int k = *log.count;
        if (k < log.capacity) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            log.entries[2 * k] = id;
            log.entries[2 * k + 1] = static_cast<long long>(t);
            *log.count = k + 1;
        }
    }
}

// What a row's update needs besides its matrix entries.
struct alignas(8) TreeOwn {
    double d;     // diagonal
    double rd, qrd;   // omega / diagonal of the row, and of the next level's row it belongs to
    int rank;     // -1: a hole
    int qpos;     // position of the next level's row (-1 past the last aggregate)
};

// Lanes per row of a tree level: as many as still give every unit (slice, part) its own warp.
// Returned as a power of two's exponent.
__host__ __device__ inline int treeLanes(int slices, int nwarps) {
    int k = 0;
    while (k < kTreeLanesLog && (static_cast<long long>(slices) << (k + 1)) <= nwarps) ++k;
    return k;
}

struct LevelSlot {
    int u0, nu, k, dir;  // this CTA's units [u0, u0 + nu), 2^k lanes per row, first directory entry
};

struct TreeShared {
    TreeLevel lv[kMaxTreeLevels];
    LevelSlot slot[kMaxTreeLevels];
    double* vec[3 * kMaxTreeLevels];
    int used;
};
__device__ __forceinline__ TreeShared& treeShared() {
    __shared__ TreeShared s;
    return s;
}
__device__ __forceinline__ char* treeRows() {
    extern __shared__ __align__(16) char rows[];
    return rows;
}

// A unit's block: values (T, 32 per step), TreeOwn per row, columns (int, 32 per step).
__device__ __forceinline__ int unitBytes(int steps, int k) {
    return steps * 32 * static_cast<int>(sizeof(double)) + (32 >> k) * static_cast<int>(sizeof(TreeOwn)) + steps * 128;
}

__device__ __forceinline__ TreeOwn ownOf(const TreeLevel& t, const TreeLevel* next, double omega, int p) {
    TreeOwn o;
    const int i = p < t.npos ? t.row[p] : -1;
    o.rank = i >= 0 ? t.rank[p] : -1;
    o.d = i >= 0 ? t.diag[i] : 1.0;
    o.rd = i >= 0 ? omega / o.d : 0.0;
    o.qpos = -1;
    o.qrd = 0.0;
    if (next && (p >> 2) < next->n) {
        o.qpos = next->pos[p >> 2];
        o.qrd = omega / next->diag[next->row[o.qpos]];
    }
    return o;
}

// Copies this CTA's rows of the tree levels into shared memory, coarsest first, until it is
// full; the directory (offset, steps per unit; offset -1: not copied) lies at its start.
template <class G>
__device__ void openTree(const G& g, const TreePcgArgs& a) {
    TreeShared& s = treeShared();
    const int L = a.T.levels, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int l = max(a.top, a.T.first) + threadIdx.x; l < L; l += TB) s.lv[l] = a.T.lv[l];
    for (int k = threadIdx.x; k < 3 * L; k += TB) s.vec[k] = a.T.vec[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        int dir = 0;
        for (int l = L - 2; l >= a.top; --l) {
            const int slices = (s.lv[l].npos + 31) >> 5;
            LevelSlot t;
            t.k = treeLanes(slices, g.size() * (TB / 32));
            const long long units = static_cast<long long>(slices) << t.k;
            t.u0 = static_cast<int>(units * g.rank() / g.size());
            t.nu = static_cast<int>(units * (g.rank() + 1) / g.size()) - t.u0;
            t.dir = dir;
            dir += t.nu;
            s.slot[l] = t;
        }
        s.used = dir;
    }
    __syncthreads();
    int2* dir = reinterpret_cast<int2*>(treeRows());
    const int ndir = s.used;
    if (ndir * kDirBytes > a.smem) {  // no room for the directory: every unit is read from memory
        __syncthreads();
        if (threadIdx.x == 0) s.used = -1;
        __syncthreads();
        return;
    }
    for (int l = L - 2; l >= a.top; --l) {
        const LevelSlot t = s.slot[l];
        const TreeLevel& v = s.lv[l];
        for (int u = warp; u < t.nu; u += TB / 32) {
            const int p = (t.u0 + u) * (32 >> t.k) + (lane >> t.k);
            const int i = p < v.npos ? v.row[p] : -1;
            int w = i >= 0 ? v.ptr[i + 1] - v.ptr[i] : 0;
            for (int o = 16; o > 0; o >>= 1) w = max(w, __shfl_xor_sync(0xffffffffu, w, o));
            if (lane == 0) dir[t.dir + u] = make_int2(0, (w + (1 << t.k) - 1) >> t.k);
        }
    }
    __syncthreads();
    if (warp == 0) {  // offsets: running sum of the units' sizes, coarsest level first
        int base = ((ndir * kDirBytes + 15) >> 4) << 4;
        for (int l = L - 2; l >= a.top; --l) {
            const LevelSlot t = s.slot[l];
            for (int u0 = 0; u0 < t.nu; u0 += 32) {
                const int u = u0 + lane;
                int bytes = 0;
                if (u < t.nu) {
                    const int steps = dir[t.dir + u].y;
                    bytes = unitBytes(steps, t.k);
                }
                int sum = bytes;
                for (int o = 1; o < 32; o <<= 1) {
                    const int up = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += up;
                }
                if (u < t.nu) dir[t.dir + u].x = base + sum <= a.smem ? base + sum - bytes : -1;
                base += __shfl_sync(0xffffffffu, sum, 31);
            }
        }
    }
    __syncthreads();
    for (int l = L - 2; l >= a.top; --l) {
        const LevelSlot t = s.slot[l];
        const TreeLevel& v = s.lv[l];
        const TreeLevel* next = &s.lv[l + 1];
        for (int u = warp; u < t.nu; u += TB / 32) {
            const int2 e = dir[t.dir + u];
            if (e.x < 0) continue;
            char* block = treeRows() + e.x;
            const int vb = e.y * 32 * static_cast<int>(sizeof(double));
            TreeOwn* own = reinterpret_cast<TreeOwn*>(block + vb);
            int* col = reinterpret_cast<int*>(own + (32 >> t.k));
            const int rows = 32 >> t.k, p0 = (t.u0 + u) * rows;
            if (lane < rows) own[lane] = ownOf(v, next, a.T.omega, p0 + lane);
            const int p = p0 + (lane >> t.k), q = lane & ((1 << t.k) - 1);
            const int i = p < v.npos ? v.row[p] : -1;
            const int k0 = i >= 0 ? v.ptr[i] : 0, len = i >= 0 ? v.ptr[i + 1] - k0 : 0;
            for (int step = 0; step < e.y; ++step) {
                const int k = q + (step << t.k);
                const bool on = k < len;
                col[32 * step + lane] = on ? v.pcol[k0 + k] : min(p, v.npos - 1);  // padding: its own value, times zero
                reinterpret_cast<double*>(block)[32 * step + lane] = on ? v.val[k0 + k] : 0.0;
            }
        }
    }
    __syncthreads();
}

// f(p, q, own, sum) for every unit of tree level l, with sum = sum_k a_pk y(col) (all K lanes of
// a row hold it); pre(p, own) runs before the gathers and its result is passed on, so the
// row's own vector entries travel together with them.
template <class Y, class P, class F>
__device__ __forceinline__ void sweepTree(int l, bool stored, double omega, Y y, P pre, F f) {
    const TreeShared& s = treeShared();
    const LevelSlot t = s.slot[l];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int K = 1 << t.k, rows = 32 >> t.k, sub = lane >> t.k, q = lane & (K - 1);
    const int2* dir = reinterpret_cast<const int2*>(treeRows()) + t.dir;
    for (int u = warp; u < t.nu; u += TB / 32) {
        const int p = (t.u0 + u) * rows + sub;
        const int2 e = stored ? dir[u] : make_int2(-1, 0);
        if (e.x >= 0) {
            const char* block = treeRows() + e.x;
            const double* v = reinterpret_cast<const double*>(block) + lane;
            const TreeOwn& o = *(reinterpret_cast<const TreeOwn*>(block + e.y * 32 * sizeof(double)) + sub);
            const int* c = reinterpret_cast<const int*>(reinterpret_cast<const TreeOwn*>(block + e.y * 32 * sizeof(double)) + rows) + lane;
            const auto mine = pre(p, o);
            double a0 = 0.0, a1 = 0.0;
            int k = 0;
            for (; k + 8 <= e.y; k += 8) {
                double yy[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) yy[i] = y(c[32 * (k + i)]);
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    a0 += v[32 * (k + i)] * yy[i];
                    a1 += v[32 * (k + i + 1)] * yy[i + 1];
                }
            }
            for (; k < e.y; k += 4) {  // the last one to seven steps, still gathered four at a time
                double yy[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) yy[i] = k + i < e.y ? y(c[32 * (k + i)]) : 0.0;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (k + i < e.y) a0 += v[32 * (k + i)] * yy[i];
            }
            double sum = a0 + a1;
            for (int o2 = K >> 1; o2 > 0; o2 >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o2);
            f(p, q, K, o, mine, sum);
        } else {  // rows that did not fit
            const TreeLevel& v = s.lv[l];
            const TreeOwn o = ownOf(v, &s.lv[l + 1], omega, p);
            const auto mine = pre(p, o);
            double sum = 0.0;
            if (o.rank >= 0)
                for (int i = v.row[p], k = v.ptr[i] + q; k < v.ptr[i + 1]; k += K)
                    sum += v.val[k] * y(v.pcol[k]);
            for (int o2 = K >> 1; o2 > 0; o2 >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o2);
            f(p, q, K, o, mine, sum);
        }
    }
}

// Sum over the four rows of an aggregate (K lanes each hold their row's value).
__device__ __forceinline__ double quadSum(double t, int K) {
    t += __shfl_xor_sync(0xffffffffu, t, K);
    t += __shfl_xor_sync(0xffffffffu, t, 2 * K);
    return t;
}

// f(p, own) for every position of tree level l that holds a row, one lane each.
template <class F>
__device__ __forceinline__ void treeRowsOf(int l, bool stored, double omega, F f) {
    const TreeShared& s = treeShared();
    const LevelSlot t = s.slot[l];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rows = 32 >> t.k;
    const int2* dir = reinterpret_cast<const int2*>(treeRows()) + t.dir;
    for (int u = warp; u < t.nu; u += TB / 32) {
        if (lane >= rows) continue;
        const int p = (t.u0 + u) * rows + lane;
        const int2 e = stored ? dir[u] : make_int2(-1, 0);
        if (e.x >= 0) {
            const TreeOwn& o = reinterpret_cast<const TreeOwn*>(treeRows() + e.x + e.y * 32 * sizeof(double))[lane];
            if (o.rank >= 0) f(p, o);
        } else {
            const TreeOwn o = ownOf(s.lv[l], &s.lv[l + 1], omega, p);
            if (o.rank >= 0) f(p, o);
        }
    }
}

__device__ __forceinline__ double memberSum(const double* t, int4 m) {
    const double t0 = m.x >= 0 ? t[m.x] : 0.0, t1 = m.y >= 0 ? t[m.y] : 0.0;
    const double t2 = m.z >= 0 ? t[m.z] : 0.0, t3 = m.w >= 0 ? t[m.w] : 0.0;
    return ((t0 + t1) + t2) + t3;
}

// Coarsest level: e_I = sum_J inv_IJ b_J, I < n, J < cols.  A CTA's rows are split over its warps, so
// that each lane has a few loads in flight instead of a long chain.  emit(I, value) runs on one
// thread per row.
template <class G, class B, class F>
__device__ __forceinline__ void denseRows(const G& g, int n, int cols, const double* __restrict__ inv, B b, F emit) {
    __shared__ double part[TB / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int size = g.size(), r0 = static_cast<int>(static_cast<long long>(n) * g.rank() / size);
    const int mine = static_cast<int>(static_cast<long long>(n) * (g.rank() + 1) / size) - r0;
    int lw = 0;  // 2^lw warps per row
    while (lw < 5 && (mine << (lw + 1)) <= TB / 32) ++lw;
    const int per = (TB / 32) >> lw, step = 32 << lw;
    for (int first = 0; first < mine; first += per) {
        const int r = first + (warp >> lw);
        double s = 0.0;
        if (r < mine) {
            const double* row = inv + static_cast<long long>(r0 + r) * cols;
            for (int J = ((warp & ((1 << lw) - 1)) << 5) + lane; J < cols; J += 8 * step) {
                double x[8], y[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const bool on = J + k * step < cols;
                    x[k] = on ? __ldg(row + J + k * step) : 0.0;
                    y[k] = on ? b(J + k * step) : 0.0;
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) s += x[k] * y[k];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) part[warp] = s;
        __syncthreads();
        if (threadIdx.x < per && first + static_cast<int>(threadIdx.x) < mine) {
            double v = 0.0;
            for (int k = 0; k < (1 << lw); ++k) v += part[(threadIdx.x << lw) + k];
            emit(r0 + first + static_cast<int>(threadIdx.x), v);
        }
        if (first + per < mine) __syncthreads();
    }
}

// The V-cycle below the finest level: on entry the residual of level 0 has been restricted
// (top = 0: level 1's b and w are set) or is in nat[0].t (top > 0); on return level 1's result is in
// its e (top = 0) or has been pushed into nat[0].x.
template <bool TREE0, class G>
__device__ __forceinline__ void treeCoarse(G& g, const TreePcgArgs& a, bool stored) {
    TreeShared& s = treeShared();
    const int L = a.T.levels, top = TREE0 ? 0 : a.top;
    const Lanes c = lanes<TB>(g);
    const double gamma = a.T.gamma;
    const double omega = a.T.omega;
    // ---- down, levels in their own numbering
    for (int l = 0; l < top; ++l) {
        const VLevel<double> f = a.T.nat[l];
        if (l > 0) {
            const double* w = f.w;
            for (int sl = c.gwarp; sl < f.A.nslices; sl += c.nwarps) {
                const int i = 32 * sl + c.lane;
                const double ax = sellRow(f.A, sl, c.lane, [&](int j) { return w[j]; });
                if (i < f.A.n) f.t[i] = f.b[i] - (f.A.diag[i] * w[i] + ax);
            }
            g.sync();
            mark(a.log, 30 + l);
        }
        const double* t = f.t;
        if (l + 1 < top) {
            const VLevel<double> cl = a.T.nat[l + 1];
            for (int I = c.gthread; I < cl.A.n; I += c.nthreads) {
                double x = 0.0;
                for (int m = f.agg_ptr[I]; m < f.agg_ptr[I + 1]; ++m) x += t[f.agg_rows[m]];
                cl.b[I] = x;
                cl.w[I] = cl.rd[I] * x;
            }
        } else if (top == L - 1) {
            double* b = s.vec[3 * top];
            const TreeLevel& v = s.lv[top];
            for (int p = c.gthread; p < v.npos; p += c.nthreads) b[p] = memberSum(t, v.memb[p]);  // zero in holes
        } else {
            double *b = s.vec[3 * top], *w = s.vec[3 * top + 1];
            const int4* memb = s.lv[top].memb;
            treeRowsOf(top, stored, omega, [&](int p, const TreeOwn& o) {
                const double x = memberSum(t, memb[p]);
                b[p] = x;
                w[p] = o.rd * x;
            });
        }
        g.sync();
        mark(a.log, 100 + l);
    }
    // ---- down, tree levels: residual and restriction in one phase
    for (int l = max(top, 1); l < L - 1; ++l) {
        const double *b = s.vec[3 * l], *w = s.vec[3 * l + 1];
        double *cb = s.vec[3 * l + 3], *cw = s.vec[3 * l + 4];
        struct Own {
            double b, w;
        };
        sweepTree(
            l, stored, omega, [&](int j) { return w[j]; },
            [&](int p, const TreeOwn& o) { return o.rank >= 0 ? Own{b[p], w[p]} : Own{0.0, 0.0}; },
            [&](int p, int q, int K, const TreeOwn& o, const Own& m, double sum) {
                const double x = quadSum(o.rank >= 0 ? m.b - (o.d * m.w + sum) : 0.0, K);
                if (q == 0 && (p & 3) == 0 && o.qpos >= 0) {
                    cb[o.qpos] = x;
                    cw[o.qpos] = o.qrd * x;
                }
            });
        g.sync();
        mark(a.log, 100 + l);
    }
    // ---- coarsest level
    {
        const double* b = s.vec[3 * (L - 1)];
        double* e = s.vec[3 * (L - 1) + 2];
        const TreeLevel& v = s.lv[L - 1];
        if (top == L - 1) {
            const VLevel<double> f = a.T.nat[L - 2];
            denseRows(g, v.n, v.npos, a.T.dense_inv, [&](int J) { return b[J]; }, [&](int I, double x) {
                const int4 m = v.memb[v.pos[I]];
                if (m.x >= 0) f.x[m.x] = f.w[m.x] + gamma * x;
                if (m.y >= 0) f.x[m.y] = f.w[m.y] + gamma * x;
                if (m.z >= 0) f.x[m.z] = f.w[m.z] + gamma * x;
                if (m.w >= 0) f.x[m.w] = f.w[m.w] + gamma * x;
            });
        } else {
            denseRows(g, v.n, v.npos, a.T.dense_inv, [&](int J) { return b[J]; }, [&](int I, double x) { e[I] = x; });
        }
        g.sync();
        mark(a.log, 50);
    }
    // ---- up, tree levels: the iterate is w + gamma e(coarse) of its rank
    for (int l = L - 2; l >= max(top, 1); --l) {
        const double *b = s.vec[3 * l], *w = s.vec[3 * l + 1], *ce = s.vec[3 * l + 5];
        double* e = s.vec[3 * l + 2];
        const auto y = [&](int j) { return w[j] + gamma * ce[j >> 2]; };
        if (l > top || top == 0) {
            struct Own {
                double b, y;
            };
            sweepTree(
                l, stored, omega, y,
                [&](int p, const TreeOwn& o) { return o.rank >= 0 ? Own{b[p], y(p)} : Own{0.0, 0.0}; },
                [&](int p, int q, int K, const TreeOwn& o, const Own& m, double sum) {
                    if (q == 0 && o.rank >= 0) e[o.rank] = m.y + o.rd * (m.b - (o.d * m.y + sum));
                });
        } else {
            // the last tree level pushes into the streamed level above it
            const VLevel<double> f = a.T.nat[l - 1];
            const int4* memb = s.lv[l].memb;
            struct Own {
                double b, y, w[4];
                int4 m;
            };
            const int K0 = 1 << s.slot[l].k, q0 = threadIdx.x & (K0 - 1);  // lane q takes members q, q + K, ...
            sweepTree(
                l, stored, omega, y,
                [&](int p, const TreeOwn& o) {
                    Own m{0.0, 0.0, {0.0, 0.0, 0.0, 0.0}, make_int4(-1, -1, -1, -1)};
                    if (o.rank >= 0) {
                        m.m = memb[p];
                        m.b = b[p];
                        m.y = y(p);
                        if ((0 & (K0 - 1)) != q0) m.m.x = -1;
                        if ((1 & (K0 - 1)) != q0) m.m.y = -1;
                        if ((2 & (K0 - 1)) != q0) m.m.z = -1;
                        if ((3 & (K0 - 1)) != q0) m.m.w = -1;
                        if (m.m.x >= 0) m.w[0] = f.w[m.m.x];
                        if (m.m.y >= 0) m.w[1] = f.w[m.m.y];
                        if (m.m.z >= 0) m.w[2] = f.w[m.m.z];
                        if (m.m.w >= 0) m.w[3] = f.w[m.m.w];
                    }
                    return m;
                },
                [&](int p, int q, int K, const TreeOwn& o, const Own& m, double sum) {
                    const double add = gamma * (m.y + o.rd * (m.b - (o.d * m.y + sum)));
                    if (m.m.x >= 0) f.x[m.m.x] = m.w[0] + add;
                    if (m.m.y >= 0) f.x[m.m.y] = m.w[1] + add;
                    if (m.m.z >= 0) f.x[m.m.z] = m.w[2] + add;
                    if (m.m.w >= 0) f.x[m.m.w] = m.w[3] + add;
                });
        }
        g.sync();
        mark(a.log, 80 + l);
    }
    // ---- up, streamed levels
    for (int l = top - 1; l >= 1; --l) {
        const VLevel<double> f = a.T.nat[l], fin = a.T.nat[l - 1];
        if (l == L - 1) continue;  // the coarsest level is the dense one
        const double* x = f.x;
        for (int sl = c.gwarp; sl < f.A.nslices; sl += c.nwarps) {
            const int i = 32 * sl + c.lane;
            const double ax = sellRow(f.A, sl, c.lane, [&](int j) { return x[j]; });
            if (i < f.A.n) {
                const double yi = x[i];
                const double add = gamma * (yi + f.rd[i] * (f.b[i] - (f.A.diag[i] * yi + ax)));
                for (int m = fin.agg_ptr[i]; m < fin.agg_ptr[i + 1]; ++m) {
                    const int ii = fin.agg_rows[m];
                    fin.x[ii] = fin.w[ii] + add;
                }
            }
        }
        g.sync();
        mark(a.log, 80 + l);
    }
}

// The CG iteration; see pcgBody in pcg_sell.cu for the recurrences and the fused update.
template <bool TREE0, class G>
__device__ void treeSolve(G& g, const TreePcgArgs& a) {
    openTree(g, a);
    TreeShared& s = treeShared();
    const bool stored = s.used >= 0;
    const Lanes c = lanes<TB>(g);
    const int L = a.T.levels, n = a.n;
    constexpr bool tree0 = TREE0;           // level 0 in tree numbering too
    const bool flat = !TREE0 && L == 1;     // the preconditioner is the dense inverse
    const double omega = a.T.omega;
    const double gamma = a.T.gamma;
    const SellMat<double>& A = a.A;
    VLevel<double> f0{};
    if (!tree0 && !flat) f0 = a.T.nat[0];
    double* w0 = tree0 ? s.vec[1] : f0.w;  // omega / diagonal * r on level 0
    double *b1 = L > 1 ? s.vec[3] : nullptr, *w1 = L > 1 ? s.vec[4] : nullptr;
    const double* e1 = L > 1 ? s.vec[5] : nullptr;
    const int* row0 = tree0 ? s.lv[0].row : nullptr;
    double* x = tree0 ? a.xt : a.x;
    int buf = 0;
    PcgState& st = *a.st;
    const int warm = st.warm;
    const int max_iterations = st.max_iterations;
    const double target2_in = st.target2, atol = st.atol, rtol = st.rtol;
    // the residual of the vector w on level 0 and its restriction, after w and r are set everywhere
    const auto firstResidual = [&] {
        if (tree0) {
            const double* r = a.r;
            struct Own {
                double b, w;
            };
            sweepTree(
                0, stored, omega, [&](int j) { return w0[j]; },
                [&](int p, const TreeOwn& o) {
                    return o.rank >= 0 ? Own{r[p], w0[p]} : Own{0.0, 0.0};
                },
                [&](int p, int q, int K, const TreeOwn& o, const Own& m, double sum) {
                    const double t = quadSum(o.rank >= 0 ? m.b - (o.d * m.w + sum) : 0.0, K);
                    if (q == 0 && (p & 3) == 0 && o.qpos >= 0) {
                        b1[o.qpos] = t;
                        w1[o.qpos] = o.qrd * t;
                    }
                });
        } else {
            const double* w = f0.w;
            for (int sl = c.gwarp; sl < f0.A.nslices; sl += c.nwarps) {
                const int i = 32 * sl + c.lane;
                const double aw = sellRow(f0.A, sl, c.lane, [&](int j) { return w[j]; });
                if (i < n) f0.t[i] = f0.b[i] - (f0.A.diag[i] * w[i] + aw);
            }
        }
        g.sync();
        mark(a.log, 30);
    };
    // z = M r; this thread's share of r . z
    const auto precondition = [&](const double* r, double2* zp) -> double {
        double rz = 0.0;
        double* z = reinterpret_cast<double*>(a.zp0);  // level 0 in its own numbering
        if (flat) {
            denseRows(g, n, n, a.T.dense_inv, [&](int J) { return r[J]; }, [&](int I, double v) {
                z[I] = v;
                rz += r[I] * v;
            });
            return rz;
        }
        treeCoarse<TREE0>(g, a, stored);
        if (tree0) {
            const auto y = [&](int j) { return w0[j] + gamma * e1[j >> 2]; };
            struct Own {
                double r, y;
            };
            sweepTree(
                0, stored, omega, y,
                [&](int p, const TreeOwn& o) { return o.rank >= 0 ? Own{r[p], y(p)} : Own{0.0, 0.0}; },
                [&](int p, int q, int K, const TreeOwn& o, const Own& m, double sum) {
                    if (q != 0 || o.rank < 0) return;
                    const double zi = m.y + o.rd * (m.r - (o.d * m.y + sum));
                    zp[p].x = zi;
                    rz += m.r * zi;
                });
        } else {
            const double* y = f0.x;
            for (int sl = c.gwarp; sl < f0.A.nslices; sl += c.nwarps) {
                const int i = 32 * sl + c.lane;
                const double ay = sellRow(f0.A, sl, c.lane, [&](int j) { return y[j]; });
                if (i < n) {
                    const double yi = y[i];
                    const double zi = yi + f0.rd[i] * (f0.b[i] - (f0.A.diag[i] * yi + ay));
                    z[i] = zi;
                    rz += r[i] * zi;
                }
            }
        }
        return rz;
    };
    // r = b - A x (x = 0 unless warm), ||r0||^2, ||b||^2, w = omega / diagonal * r on level 0
    double v[2] = {0.0, 0.0};
    if (tree0) {
        if (warm) {
            treeRowsOf(0, stored, omega, [&](int p, const TreeOwn& o) { x[p] = a.x[row0[p]]; });
            g.sync();
        }
        const auto seed = [&](int p, const TreeOwn& o, double bi, double ri) {
            a.r[p] = ri;
            const double wi = o.rd * ri;
            w0[p] = wi;
            a.wq0[p].x = wi;
            v[0] += ri * ri;
            v[1] += bi * bi;
        };
        if (warm) {
            const double* xx = x;
            sweepTree(
                0, stored, omega, [&](int j) { return xx[j]; },
                [&](int p, const TreeOwn& o) { return o.rank >= 0 ? a.b[row0[p]] : 0.0; },
                [&](int p, int q, int K, const TreeOwn& o, double bi, double sum) {
                    if (q == 0 && o.rank >= 0) seed(p, o, bi, bi - (o.d * xx[p] + sum));
                });
        } else {
            treeRowsOf(0, stored, omega, [&](int p, const TreeOwn& o) {
                x[p] = 0.0;
                const double bi = a.b[row0[p]];
                seed(p, o, bi, bi);
            });
        }
    } else {
        for (int sl = c.gwarp; sl < A.nslices; sl += c.nwarps) {
            const int i = 32 * sl + c.lane;
            double ri = 0.0;
            if (warm) {
                const double* xx = x;
                const double ax = sellRow(A, sl, c.lane, [&](int j) { return xx[j]; });
                if (i < n) ri = a.b[i] - (A.diag[i] * xx[i] + ax);
            } else if (i < n) {
                ri = a.b[i];
                x[i] = 0.0;
            }
            if (i < n) {
                a.r[i] = ri;
                if (!flat) {
                    f0.b[i] = ri;
                    f0.w[i] = f0.rd[i] * ri;
                }
                v[0] += ri * ri;
                v[1] += a.b[i] * a.b[i];
            }
        }
    }
    gridSum<2, TB>(g, v, a.partial, buf);
    mark(a.log, 1);
    double target2 = target2_in;
    if (target2 < 0.0) {
        // the reference's contract: max(atol, rtol * max(||r0||, ||b||)) (solver_control.h:199-210)
        double scale = fmax(sqrt(v[0]), sqrt(v[1]));
        if (!(scale > 0.0)) scale = 1.0;
        const double t = fmax(atol, rtol * scale);
        target2 = t * t;
    }
    if (g.rank() == 0 && threadIdx.x == 0) {
        st.rr0 = v[0];
        st.bb = v[1];
        st.target2 = target2;
        st.rr = v[0];
        st.iterations = 0;
        st.status = 1;
    }
    const auto finish = [&](int status, int it, double rr) {
        if (tree0)
            treeRowsOf(0, stored, omega, [&](int p, const TreeOwn& o) { a.x[row0[p]] = x[p]; });
        if (g.rank() == 0 && threadIdx.x == 0) {
            st.rr = rr;
            st.iterations = it;
            st.status = status;
        }
    };
    if (isfinite(v[0]) && v[0] <= target2) {
        finish(0, 0, v[0]);
        return;
    }
    if (!flat) firstResidual();
    double rz = 0.0, beta = 0.0;
    double2 *zp = a.zp0, *zpn = a.zp1;  // {z, p} of this iteration, and of the next
    double2 *wq = a.wq0, *wqn = a.wq1;  // {w, omega / diagonal * q}
    double *r = a.r, *q = a.q;
    // level 0 in its own numbering keeps each vector apart (see TreePcgArgs)
    double *zs = reinterpret_cast<double*>(a.zp0), *pold = zs + n, *pnew = reinterpret_cast<double*>(a.zp1), *rn = pnew + n;
    int it = 0;
    int status = 1;
    double rr = v[0];
    while (it < max_iterations) {
        double zr[1] = {precondition(r, zp)};
        gridSum<1, TB>(g, zr, a.partial, buf);
        mark(a.log, 4);
        if (g.aborted()) { status = 3; break; }
        if (it > 0) beta = zr[0] / rz;
        rz = zr[0];
        if (!isfinite(rz) || rz == 0.0) { status = 2; break; }
        // p_new = z + beta p_old and q = A p_new in one sweep (neighbours' p_new formed on the fly)
        const bool first = beta == 0.0;
        const auto pj = [&](int j) {
            const double2 v2 = zp[j];
            return first ? v2.x : v2.x + beta * v2.y;
        };
        double pq[1] = {0.0};
        if (tree0) {
            sweepTree(
                0, stored, omega, pj, [&](int p, const TreeOwn& o) { return o.rank >= 0 ? pj(p) : 0.0; },
                [&](int p, int sub, int K, const TreeOwn& o, double pi, double sum) {
                    if (sub != 0 || o.rank < 0) return;
                    const double qi = o.d * pi + sum;
                    zpn[p].y = pi;
                    q[p] = qi;
                    wq[p].y = o.rd * qi;
                    pq[0] += pi * qi;
                });
        } else {
            const double* zz = zs;
            const double* po = pold;
            for (int sl = c.gwarp; sl < A.nslices; sl += c.nwarps) {
                const int i = 32 * sl + c.lane;
                const double ap = first ? sellRow(A, sl, c.lane, [&](int j) { return zz[j]; })
                                    : sellRow(A, sl, c.lane, [&](int j) { return zz[j] + beta * po[j]; });
                if (i < n) {
                    const double pi = first ? zz[i] : zz[i] + beta * po[i];
                    const double qi = A.diag[i] * pi + ap;
                    pnew[i] = pi;
                    q[i] = qi;
                    pq[0] += pi * qi;
                }
            }
        }
        gridSum<1, TB>(g, pq, a.partial, buf);
        mark(a.log, 2);
        if (!(fabs(pq[0]) > 0.0) || !isfinite(pq[0])) { status = 2; break; }
        const double alpha = rz / pq[0];
        const auto wj = [&](int j) {
            const double2 v2 = wq[j];
            return v2.x - alpha * v2.y;
        };
        double nr[1] = {0.0};
        if (tree0) {
            // x += alpha p, r_new = r - alpha q, w = rd r_new, and the residual of w (neighbours' w
            // formed from their pairs) restricted to level 1, all in this phase
            struct Own {
                double r, x;
            };
            sweepTree(
                0, stored, omega, wj,
                [&](int p, const TreeOwn& o) {
                    return o.rank >= 0 ? Own{r[p] - alpha * q[p], x[p] + alpha * zpn[p].y} : Own{0.0, 0.0};
                },
                [&](int p, int sub, int K, const TreeOwn& o, const Own& m, double sum) {
                    const double wi = o.rd * m.r;
                    if (sub == 0 && o.rank >= 0) {
                        x[p] = m.x;
                        r[p] = m.r;
                        w0[p] = wi;
                        wqn[p].x = wi;
                        nr[0] += m.r * m.r;
                    }
                    const double t = quadSum(o.rank >= 0 ? m.r - (o.d * wi + sum) : 0.0, K);
                    if (sub == 0 && (p & 3) == 0 && o.qpos >= 0) {
                        b1[o.qpos] = t;
                        w1[o.qpos] = o.qrd * t;
                    }
                });
        } else if (!flat) {
            const double* rd = f0.rd;
            const double *rc = r, *qq = q;
            for (int sl = c.gwarp; sl < f0.A.nslices; sl += c.nwarps) {
                const int i = 32 * sl + c.lane;
                const double aw = sellRow(f0.A, sl, c.lane, [&](int j) { return rd[j] * (rc[j] - alpha * qq[j]); });
                if (i < n) {
                    x[i] += alpha * pnew[i];
                    const double ri = rc[i] - alpha * qq[i];
                    rn[i] = ri;
                    const double wi = rd[i] * ri;
                    f0.b[i] = ri;
                    f0.w[i] = wi;
                    f0.t[i] = ri - (f0.A.diag[i] * wi + aw);
                    nr[0] += ri * ri;
                }
            }
        } else {
            for (int i = c.gthread; i < n; i += c.nthreads) {
                x[i] += alpha * pnew[i];
                const double ri = r[i] - alpha * q[i];
                rn[i] = ri;
                nr[0] += ri * ri;
            }
        }
        gridSum<1, TB>(g, nr, a.partial, buf);
        mark(a.log, 3);
        rr = nr[0];
        ++it;
        if (!isfinite(rr)) { status = 2; break; }
        if (rr <= target2) { status = 0; break; }
        if (!tree0) {
            double* t1 = r;
            r = rn;
            rn = t1;
        }
        double* t1 = pold;
        pold = pnew;
        pnew = t1;
        double2* tmp = zp;
        zp = zpn;
        zpn = tmp;
        tmp = wq;
        wq = wqn;
        wqn = tmp;
    }
    finish(g.failed() ? 3 : status, it, rr);
}

template <class G>
__device__ __forceinline__ void treeBody(G& g, const TreePcgArgs& a) {
    if (a.top == 0 && a.T.levels > 1) treeSolve<true>(g, a);
    else treeSolve<false>(g, a);
}

__global__ void __launch_bounds__(TB, 1) kPcgTree(const __grid_constant__ TreePcgArgs a, SegmentBarrier* bar) {
    GridGroup g{bar};
    treeBody(g, a);
}

// The systems of a batched launch as one kernel argument.
struct TreeArgsBlock {
    TreePcgArgs a[kBatchArgs];
    int begin[kBatchArgs + 1];  // CTA ranges
    int count;
};
static_assert(sizeof(TreeArgsBlock) + sizeof(void*) <= kKernelArgumentBytes, "one kernel argument");

// A batch: CTAs [begin[s], begin[s+1]) solve system s.
__global__ void __launch_bounds__(TB, 1)
    kPcgTreeBatch(const __grid_constant__ TreeArgsBlock batch, SegmentBarrier* bars) {
    const int s = systemOfBlock(batch.begin, batch.count);
    SegmentGroup g{batch.begin[s], batch.begin[s + 1] - batch.begin[s], bars + s};
    treeBody(g, batch.a[s]);
}

// A small system on one cluster.
__global__ void __launch_bounds__(TB, 1) kPcgTreeCluster(const __grid_constant__ TreePcgArgs a) {
    ClusterGroup g;
    g.sync();  // every CTA's shared memory is live
    treeBody(g, a);
}
TreePlan::Place place(const TreePlan& plan, TreePcgArgs& a, int ctas) {
    const TreePlan::Place p = plan.place(ctas);
    a.top = p.top;
    a.smem = p.smem;
    if (p.levels < a.T.levels) {
        a.T.levels = p.levels;
        a.T.dense_inv = a.T.folded;
    }
    return p;
}

}  // namespace

double TreePlan::bytes(int from, int levels, int ctas) const {
    const double own = sizeof(TreeOwn);
    double total = 64.0;
    for (int l = from; l < levels - 1; ++l) {
        const int K = 1 << treeLanes(static_cast<int>(slices[l]), ctas * (TB / 32));
        const double wide = slices[l] > 0 ? entries[l] / (32.0 * slices[l]) : 0.0;
        const double steps = K == 1 ? wide : wide / K + 0.5 * (K - 1) / K;
        constexpr double entry = sizeof(double) + sizeof(int);
        // a few per cent for uneven slices, and the unit a CTA may have more than its share
        total += 1.04 * slices[l] * (K * (steps * 32.0 * entry + kDirBytes) + 32.0 * own) / ctas + steps * 32.0 * entry +
                 32.0 / K * own;
    }
    return total;
}

bool TreePlan::fits(int from, int ctas) const {
    return bytes(from, static_cast<int>(slices.size()), ctas) <= (from == 0 ? kTreeSmem : kStreamSmem);
}

TreePlan::Place TreePlan::place(int ctas) const {
    const int L = static_cast<int>(slices.size());
    Place p{L - 1, L, 0};
    if (folded && static_cast<double>(rows[L - 2]) * positions[L - 2] * sizeof(double) <= kFoldedBytes * static_cast<double>(ctas))
        p.levels = L - 1;
    p.top = p.levels - 1;
    if (first == 0 && p.levels > 1 && bytes(0, p.levels, ctas) <= kTreeSmem) p.top = 0;
    else
        while (p.top > std::max(first, 1) && bytes(p.top - 1, p.levels, ctas) <= kStreamSmem) --p.top;
    p.smem = static_cast<int>(std::min<double>(kTreeSmem, std::ceil((1.05 * bytes(p.top, p.levels, ctas) + 2048.0) / 1024.0) * 1024.0));
    return p;
}

TreePlan::Place launchTreePcg(Context& ctx, const TreePlan& plan, TreePcgArgs a) {
    a.log = PhaseLog{ctx.phase_entries, ctx.phase_capacity, ctx.phase_count};
    if (plan.nnz <= kClusterEntries) {
        allowSharedMemory<kPcgTreeCluster>(kTreeSmem);
        const TreePlan::Place at = place(plan, a, clusterCtas<kPcgTreeCluster>(TB, kTreeSmem));
        BSG_PROFILE(ctx, "pcg_amg_persistent");
        launchCluster<kPcgTreeCluster>(ctx, 1, TB, a.smem, kTreeSmem, a);
        return at;
    }
    allowSharedMemory<kPcgTree>(kTreeSmem);
    const int grid = ctx.sm_count;
    const TreePlan::Place at = place(plan, a, grid);
    SegmentBarrier* bar = ctx.grid_barrier;
    resetBarriers(ctx, bar, 1, grid);
    void* params[] = {&a, &bar};
    BSG_PROFILE(ctx, "pcg_amg_persistent");
    BSG_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kPcgTree), grid, TB, params, a.smem, ctx.stream));
    ctx.launched();
    return at;
}

void launchTreePcgBatch(Context& ctx, TreeBatch& batch) {
    const std::size_t count = batch.args.size();
    if (count == 0) return;
    allowSharedMemory<kPcgTreeBatch>(kTreeSmem);
    batch.d_bars.resize(std::max(batch.d_bars.size(), count));
    const std::vector<long long> slices(batch.slices.begin(), batch.slices.end());
    const std::vector<std::size_t> launches = batchLaunches(slices, TB / 32, ctx.sm_count);
    for (std::size_t l = 0; l + 1 < launches.size(); ++l) {
        const std::size_t k0 = launches[l], k1 = launches[l + 1];
        TreeArgsBlock block{};
        const int m = block.count = static_cast<int>(k1 - k0);
        const std::vector<int> begin = allotCtas({slices.begin() + k0, slices.begin() + k1}, TB / 32, ctx.sm_count);
        std::copy(begin.begin(), begin.end(), block.begin);
        int smem = 0;
        for (int i = 0; i < m; ++i) {
            block.a[i] = batch.args[k0 + i];
            place(*batch.plans[k0 + i], block.a[i], begin[i + 1] - begin[i]);
            smem = std::max(smem, block.a[i].smem);
        }
        SegmentBarrier* bars = batch.d_bars.data() + k0;
        resetBarriers(ctx, bars, m, begin.back(), block.begin);
        void* params[] = {&block, &bars};
        BSG_PROFILE(ctx, "pcg_amg_persistent_batch");
        BSG_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kPcgTreeBatch), begin.back(), TB, params,
                                             smem, ctx.stream));
        ctx.launched();
    }
    batch.bars_used = static_cast<int>(count);
}

}  // namespace bsg
