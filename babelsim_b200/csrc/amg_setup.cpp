// See amg_setup.h.  Every loop over rows that do not depend on one another runs on several
// threads; each thread owns a contiguous range of coarse rows and adds in the same order as one
// thread would, so the result does not depend on their number.
#include "amg_setup.h"

#include <algorithm>
#include <exception>
#include <numeric>
#include <thread>

namespace bsg {

int hostThreads() {
    static const int n = std::max(1, std::min(8, static_cast<int>(std::thread::hardware_concurrency())));
    return n;
}

void parallelRanges(int n, int grain, const std::function<void(int, int, int)>& f) {
    const int threads = std::max(1, std::min(hostThreads(), n / std::max(grain, 1)));
    if (threads == 1) {
        f(0, n, 0);
        return;
    }
    std::vector<std::thread> pool;
    std::vector<std::exception_ptr> failed(threads);
    const auto run = [&](int t) {
        try {
            f(static_cast<int>(static_cast<long long>(n) * t / threads),
              static_cast<int>(static_cast<long long>(n) * (t + 1) / threads), t);
        } catch (...) {
            failed[t] = std::current_exception();
        }
    };
    pool.reserve(threads - 1);
    int started = 1;
    try {
        for (; started < threads; ++started) pool.emplace_back(run, started);
    } catch (...) {  // no more threads to be had: the caller does their share
    }
    run(0);
    for (int t = started; t < threads; ++t) run(t);
    for (std::thread& t : pool) t.join();
    for (const std::exception_ptr& e : failed)
        if (e) std::rethrow_exception(e);
}

std::vector<int> pairwise(const HostCsr& a, int& n_coarse) {
    std::vector<int> agg(a.n, -1);
    int next = 0;
    for (int i = 0; i < a.n; ++i) {
        if (agg[i] >= 0) continue;
        int best = -1;
        double bs = 0.0;
        for (int k = a.ptr[i]; k < a.ptr[i + 1]; ++k) {
            const double s = -a.val[k];
            if (!(s > bs)) continue;
            const int j = a.col[k];
            if (j == i || agg[j] >= 0) continue;
            bs = s;
            best = j;
        }
        agg[i] = next;
        if (best >= 0) agg[best] = next;
        ++next;
    }
    n_coarse = next;
    return agg;
}

void aggregateLists(const std::vector<int>& agg, int nc, std::vector<int>& ptr, std::vector<int>& rows) {
    const int n = static_cast<int>(agg.size());
    ptr.assign(nc + 1, 0);
    rows.resize(n);
    for (int i = 0; i < n; ++i) ++ptr[agg[i] + 1];
    for (int I = 0; I < nc; ++I) ptr[I + 1] += ptr[I];
    std::vector<int> fill(ptr.begin(), ptr.end() - 1);
    for (int i = 0; i < n; ++i) rows[fill[agg[i]]++] = i;
}

namespace {
constexpr int kGrain = 4096;  // rows per thread at least
}

HostCsr coarsen(const HostCsr& a, const std::vector<int>& agg, int nc, std::vector<int>* slot_target) {
    std::vector<int> mptr, mrow;
    aggregateLists(agg, nc, mptr, mrow);
    HostCsr c;
    c.n = nc;
    c.ptr.assign(nc + 1, 0);
    c.diag.assign(nc, 0.0);
    if (slot_target) slot_target->resize(a.ptr[a.n]);
    struct Part {
        int begin = 0, end = 0;
        std::vector<int> col;
        std::vector<double> val;
    };
    std::vector<Part> parts(hostThreads());
    parallelRanges(nc, kGrain, [&](int I0, int I1, int t) {
        Part& p = parts[t];
        p.begin = I0;
        p.end = I1;
        std::vector<int> marker(nc, -1), place(nc), cols;
        for (int I = I0; I < I1; ++I) {
            cols.clear();
            double d = 0.0;
            for (int m = mptr[I]; m < mptr[I + 1]; ++m) {
                const int i = mrow[m];
                d += a.diag[i];
                for (int k = a.ptr[i]; k < a.ptr[i + 1]; ++k) {
                    const int J = agg[a.col[k]];
                    if (J == I) {
                        d += a.val[k];
                    } else if (marker[J] != I) {
                        marker[J] = I;
                        cols.push_back(J);
                    }
                }
            }
            c.diag[I] = d;
            std::sort(cols.begin(), cols.end());
            const int base = static_cast<int>(p.col.size());
            for (std::size_t q = 0; q < cols.size(); ++q) place[cols[q]] = base + static_cast<int>(q);
            p.col.insert(p.col.end(), cols.begin(), cols.end());
            p.val.resize(p.col.size(), 0.0);
            c.ptr[I + 1] = static_cast<int>(cols.size());
            for (int m = mptr[I]; m < mptr[I + 1]; ++m) {
                const int i = mrow[m];
                for (int k = a.ptr[i]; k < a.ptr[i + 1]; ++k) {
                    const int J = agg[a.col[k]];
                    if (J != I) p.val[place[J]] += a.val[k];
                    if (slot_target) (*slot_target)[k] = J == I ? -1 : place[J];
                }
            }
        }
    });
    for (int I = 0; I < nc; ++I) c.ptr[I + 1] += c.ptr[I];
    c.col.resize(c.ptr[nc]);
    c.val.resize(c.ptr[nc]);
    parallelRanges(static_cast<int>(parts.size()), 1, [&](int t0, int t1, int) {
        for (int t = t0; t < t1; ++t) {
            const Part& p = parts[t];
            if (p.end == p.begin) continue;
            const int base = c.ptr[p.begin];
            std::copy(p.col.begin(), p.col.end(), c.col.begin() + base);
            std::copy(p.val.begin(), p.val.end(), c.val.begin() + base);
            if (!slot_target || base == 0) continue;
            for (int m = mptr[p.begin]; m < mptr[p.end]; ++m)
                for (int k = a.ptr[mrow[m]]; k < a.ptr[mrow[m] + 1]; ++k)
                    if ((*slot_target)[k] >= 0) (*slot_target)[k] += base;
        }
    });
    return c;
}

GalerkinMaps galerkinMaps(const HostCsr& a, const std::vector<int>& target, const std::vector<int>& agg_ptr,
                          const std::vector<int>& agg_rows, int cnnz) {
    const int nc = static_cast<int>(agg_ptr.size()) - 1;
    GalerkinMaps g;
    g.cslot_ptr.assign(static_cast<std::size_t>(cnnz) + 1, 0);
    g.cslot_src.resize(a.ptr[a.n]);
    g.cintra_ptr.assign(nc + 1, 0);
    // a coarse row's entries are its own, so ranges of coarse rows touch disjoint counters
    parallelRanges(nc, kGrain, [&](int I0, int I1, int) {
        for (int I = I0; I < I1; ++I)
            for (int m = agg_ptr[I]; m < agg_ptr[I + 1]; ++m)
                for (int k = a.ptr[agg_rows[m]]; k < a.ptr[agg_rows[m] + 1]; ++k) {
                    if (target[k] >= 0) ++g.cslot_ptr[target[k] + 1];
                    else ++g.cintra_ptr[I + 1];
                }
    });
    for (int c = 0; c < cnnz; ++c) g.cslot_ptr[c + 1] += g.cslot_ptr[c];
    for (int I = 0; I < nc; ++I) g.cintra_ptr[I + 1] += g.cintra_ptr[I];
    g.cintra_src.resize(g.cintra_ptr[nc]);
    std::vector<int> fill(g.cslot_ptr.begin(), g.cslot_ptr.end() - 1);
    parallelRanges(nc, kGrain, [&](int I0, int I1, int) {
        for (int I = I0; I < I1; ++I) {
            int q = g.cintra_ptr[I];
            for (int m = agg_ptr[I]; m < agg_ptr[I + 1]; ++m)
                for (int k = a.ptr[agg_rows[m]]; k < a.ptr[agg_rows[m] + 1]; ++k) {
                    if (target[k] >= 0) g.cslot_src[fill[target[k]]++] = k;
                    else g.cintra_src[q++] = k;
                }
        }
    });
    return g;
}

Members membersOf(const std::vector<int>& agg, int nc) {
    Members m(nc, {-1, -1, -1, -1});
    for (std::size_t i = 0; i < agg.size(); ++i) {
        std::array<int, 4>& q = m[agg[i]];
        for (int j = 0; j < 4; ++j)
            if (q[j] < 0) {
                q[j] = static_cast<int>(i);
                break;
            }
    }
    return m;
}

TreeMaps treeMaps(int n, const Members& members, std::vector<int>& order) {
    TreeMaps t;
    const std::size_t npos = 4 * order.size();
    t.row.assign(npos, -1);
    t.rank.assign(npos, -1);
    t.pos.resize(n);
    t.at.resize(n);
    std::vector<int> next(n);
    int k = 0;
    for (std::size_t c = 0; c < order.size(); ++c)
        for (int j = 0; j < 4; ++j) {
            const int i = members[order[c]][j];
            if (i < 0) break;
            const int p = static_cast<int>(4 * c) + j;
            t.row[p] = i;
            t.rank[p] = k;
            t.pos[k] = p;
            t.at[i] = p;
            next[k++] = i;
        }
    order = std::move(next);
    return t;
}

double paddedEntries(const TreeMaps& t, const std::vector<int>& ptr) {
    const int npos = static_cast<int>(t.row.size()), slices = (npos + 31) / 32;
    std::vector<long long> sums(hostThreads(), 0);
    parallelRanges(slices, kGrain / 32, [&](int s0, int s1, int thread) {
        long long sum = 0;
        for (int s = s0; s < s1; ++s) {
            int w = 0;
            for (int p = 32 * s; p < std::min(npos, 32 * (s + 1)); ++p)
                if (t.row[p] >= 0) w = std::max(w, ptr[t.row[p] + 1] - ptr[t.row[p]]);
            sum += w;
        }
        sums[thread] = sum;
    });
    return 32.0 * static_cast<double>(std::accumulate(sums.begin(), sums.end(), 0LL));
}

void membersByPosition(const TreeMaps& t, const Members& members, int* out) {
    parallelRanges(static_cast<int>(t.row.size()), kGrain, [&](int p0, int p1, int) {
        for (int p = p0; p < p1; ++p)
            if (t.row[p] >= 0) std::copy(members[t.row[p]].begin(), members[t.row[p]].end(), out + 4 * static_cast<std::size_t>(p));
    });
}

}  // namespace bsg
