// Host setup of the multilevel preconditioner (multilevel.cu): the coarse
// levels of a 3-D mesh, built once per mesh from its unit-resistivity matrix.
//
// Level k -> k + 1 (smoothed aggregation; Vanek, Mandel & Brezina, Computing 56,
// 1996): two passes of pairwise matching by strongest negative coupling
// (Notay, ETNA 37, 2010) make aggregates of about four rows, whose indicator
// vectors T get one damped Jacobi step, P = (I - 4/3 D^-1 U) T
// with D the rows' absolute sums.  Entries below
// kDrop of their row's largest are dropped (the row's own aggregate is kept)
// and the row is rescaled to its sum, so P holds about 2.5 entries per row.
// P depends on the geometry only: the model enters through the Galerkin
// products A_{k+1} = P^T A_k P on the device.  Patterns of A P and P^T A P are
// built here once.
#include <algorithm>
#include <cmath>
#include <exception>
#include <thread>

#include "ertgb_internal.cuh"

namespace ertgb {

namespace {

constexpr double kStrong = 0.25;  // a pair's coupling against the row's strongest
constexpr int64_t kSmall = 1024;  // rows of a level that is paired whatever the coupling (dense rows, few free partners)
constexpr int64_t kTail = 4096;   // rows of a level that is paired three times (x8): launches, not work, are its cost
constexpr double kDrop = 0.15;    // smoothed entries kept, against the row's largest

struct Csr {
    int64_t n = 0, m = 0;  // rows, columns
    std::vector<int32_t> rp, ci;
    std::vector<double> v;
};

// one pass of pairwise matching in row order; returns the number of
// aggregates.  A row without couplings (a fixed potential) joins none (-1): the
// smoother alone solves it
int64_t match(const Csr &A, double strong, std::vector<int32_t> &agg) {
    agg.assign((size_t)A.n, -1);
    int64_t na = 0;
    for (int64_t i = 0; i < A.n; i++) {
        if (agg[i] >= 0) continue;
        double strongest = 0.0, best = 0.0, off = 0.0;
        int32_t with = -1;
        for (int32_t q = A.rp[i]; q < A.rp[i + 1]; q++) {
            const int32_t j = A.ci[q];
            if (j == i) continue;
            const double c = -A.v[q];
            off += std::fabs(c);
            strongest = std::max(strongest, c);
            if (agg[j] < 0 && c > best) {
                best = c;
                with = j;
            }
        }
        if (off == 0.0) continue;
        agg[i] = (int32_t)na;
        if (with >= 0 && best >= strong * strongest) agg[with] = (int32_t)na;
        na++;
    }
    return na;
}

Csr transpose(const Csr &A) {
    Csr T;
    T.n = A.m;
    T.m = A.n;
    T.rp.assign((size_t)A.m + 1, 0);
    for (int32_t c : A.ci) T.rp[c + 1]++;
    for (int64_t i = 0; i < A.m; i++) T.rp[i + 1] += T.rp[i];
    T.ci.resize(A.ci.size());
    T.v.resize(A.v.size());
    std::vector<int32_t> pos(T.rp.begin(), T.rp.end() - 1);
    for (int64_t i = 0; i < A.n; i++)
        for (int32_t q = A.rp[i]; q < A.rp[i + 1]; q++) {
            const int32_t p = pos[A.ci[q]]++;
            T.ci[p] = (int32_t)i;
            T.v[p] = A.v[q];
        }
    return T;
}

// f(first row, last row, part) over contiguous row ranges on a few host
// threads (one for a small matrix); an exception of a part is rethrown here
template <class F> int by_rows(int64_t n, F f) {
    const int parts = (int)std::max<int64_t>(1, std::min<int64_t>({(int64_t)std::thread::hardware_concurrency(), 16,
                                                                  n / 2048}));
    if (parts == 1) {
        f((int64_t)0, n, 0);
        return 1;
    }
    std::vector<std::thread> th;
    std::vector<std::exception_ptr> errs((size_t)parts);
    for (int p = 0; p < parts; p++)
        th.emplace_back([&, p] {
            try {
                f(n * p / parts, n * (p + 1) / parts, p);
            } catch (...) {
                errs[(size_t)p] = std::current_exception();
            }
        });
    for (auto &t : th) t.join();
    for (auto &e : errs)
        if (e) std::rethrow_exception(e);
    return parts;
}

// row-wise construction: row(i, cols, acc) fills the columns of row i
// (ascending in the result) and their values; scratch of m columns per thread
template <class Row> Csr build_rows(int64_t n, int64_t m, Row row) {
    Csr C;
    C.n = n;
    C.m = m;
    C.rp.assign((size_t)n + 1, 0);
    std::vector<std::vector<int32_t>> ci(16);
    std::vector<std::vector<double>> v(16);
    const int parts = by_rows(n, [&](int64_t i0, int64_t i1, int p) {
        std::vector<int32_t> at((size_t)m, -1), cols;
        std::vector<double> acc((size_t)m, 0.0);
        for (int64_t i = i0; i < i1; i++) {
            cols.clear();
            row(i, at, acc, cols);
            for (int32_t c : cols) {
                ci[p].push_back(c);
                v[p].push_back(acc[c]);
            }
            C.rp[i + 1] = (int32_t)cols.size();
        }
    });
    for (int64_t i = 0; i < n; i++) C.rp[i + 1] += C.rp[i];
    C.ci.reserve((size_t)C.rp[n]);
    C.v.reserve((size_t)C.rp[n]);
    for (int p = 0; p < parts; p++) {
        C.ci.insert(C.ci.end(), ci[p].begin(), ci[p].end());
        C.v.insert(C.v.end(), v[p].begin(), v[p].end());
    }
    return C;
}

// C = A B, columns ascending (B's rows may repeat a column)
Csr multiply(const Csr &A, const Csr &B) {
    return build_rows(A.n, B.m, [&](int64_t i, std::vector<int32_t> &at, std::vector<double> &acc,
                                    std::vector<int32_t> &cols) {
        for (int32_t q = A.rp[i]; q < A.rp[i + 1]; q++)
            for (int32_t p = B.rp[A.ci[q]]; p < B.rp[A.ci[q] + 1]; p++) {
                const int32_t c = B.ci[p];
                if (at[c] != (int32_t)i) {
                    at[c] = (int32_t)i;
                    acc[c] = 0.0;
                    cols.push_back(c);
                }
                acc[c] += A.v[q] * B.v[p];
            }
        std::sort(cols.begin(), cols.end());
    });
}

// sum of A's entries over aggregates of rows and columns: T^T (A T), the
// columns renamed
Csr collapse(const Csr &A, const std::vector<int32_t> &agg, int64_t na) {
    Csr T, AT;
    T.n = AT.n = A.n;
    T.m = AT.m = na;
    T.rp.assign((size_t)A.n + 1, 0);
    AT.rp.assign((size_t)A.n + 1, 0);
    AT.ci.reserve(A.ci.size());
    AT.v.reserve(A.ci.size());
    for (int64_t i = 0; i < A.n; i++) {
        if (agg[i] >= 0) {
            T.ci.push_back(agg[i]);
            T.v.push_back(1.0);
            for (int32_t q = A.rp[i]; q < A.rp[i + 1]; q++)
                if (agg[A.ci[q]] >= 0) {
                    AT.ci.push_back(agg[A.ci[q]]);
                    AT.v.push_back(A.v[q]);
                }
        }
        T.rp[i + 1] = (int32_t)T.ci.size();
        AT.rp[i + 1] = (int32_t)AT.ci.size();
    }
    return multiply(transpose(T), AT);
}

// smoothed, filtered prolongation of the aggregates
Csr prolongation(const Csr &U, const std::vector<int32_t> &agg, int64_t na) {
    // D = the rows' absolute sums: D^-1 U has its spectrum in [0, 1]
    std::vector<double> l1((size_t)U.n, 0.0);
    for (int64_t i = 0; i < U.n; i++)
        for (int32_t q = U.rp[i]; q < U.rp[i + 1]; q++) l1[i] += std::fabs(U.v[q]);
    const double w = 4.0 / 3.0;
    Csr P = build_rows(U.n, na, [&](int64_t i, std::vector<int32_t> &at, std::vector<double> &acc,
                                    std::vector<int32_t> &cols) {
        const int32_t own = agg[i];
        if (own < 0) return;
        cols.push_back(own);
        at[own] = (int32_t)i;
        acc[own] = 1.0;
        if (l1[i] > 0.0)
            for (int32_t q = U.rp[i]; q < U.rp[i + 1]; q++) {
                const int32_t c = agg[U.ci[q]];
                if (c < 0) continue;
                if (at[c] != (int32_t)i) {
                    at[c] = (int32_t)i;
                    acc[c] = 0.0;
                    cols.push_back(c);
                }
                acc[c] -= w * U.v[q] / l1[i];
            }
        double big = 0.0, sum = 0.0, kept = 0.0;
        for (int32_t c : cols) {
            big = std::max(big, std::fabs(acc[c]));
            sum += acc[c];
        }
        size_t k = 0;
        for (int32_t c : cols)
            if (c == own || std::fabs(acc[c]) >= kDrop * big) {
                cols[k++] = c;
                kept += acc[c];
            }
        cols.resize(k);
        std::sort(cols.begin(), cols.end());
        const double scale = std::fabs(kept) > 0.3 * std::fabs(sum) ? sum / kept : 1.0;
        for (int32_t c : cols) acc[c] = (double)(float)(acc[c] * scale);  // as the device holds it
    });
    return P;
}

}  // namespace

bool build_levels(const std::vector<int32_t> &rowptr, const std::vector<int32_t> &colidx,
                  const std::vector<double> &unit, int64_t coarsest, int max_levels, std::vector<HostLevel> &out) {
    out.clear();
    Csr U;
    U.n = U.m = (int64_t)rowptr.size() - 1;
    U.rp = rowptr;
    U.ci = colidx;
    U.v = unit;
    while (U.n > coarsest) {
        if ((int)out.size() >= max_levels) return false;
        const double strong = U.n > kSmall ? kStrong : 0.0;
        const int passes = U.n > kTail ? 2 : 3;
        std::vector<int32_t> a1, a2;
        int64_t n2 = match(U, strong, a1);
        Csr W = collapse(U, a1, n2);
        for (int p = 1; p < passes; p++) {
            n2 = match(W, strong, a2);
            for (auto &a : a1)
                if (a >= 0) a = a2[a];
            if (p + 1 < passes) W = collapse(W, a2, n2);
        }
        if (n2 < 1 || n2 * 10 > U.n * 6) return false;  // the matching stalls: no useful hierarchy
        const Csr P = prolongation(U, a1, n2), PT = transpose(P), AP = multiply(U, P);
        Csr C = multiply(PT, AP);
        HostLevel l;
        l.n = U.n;
        l.nc = n2;
        l.rp = U.rp;
        l.ci = U.ci;
        l.P_rp = P.rp;
        l.P_ci = P.ci;
        l.P_v.assign(P.v.begin(), P.v.end());
        l.PT_rp = PT.rp;
        l.PT_ci = PT.ci;
        l.PT_v.assign(PT.v.begin(), PT.v.end());
        l.AP_rp = AP.rp;
        l.AP_ci = AP.ci;
        out.push_back(std::move(l));
        U = std::move(C);
    }
    if (out.empty()) return false;
    HostLevel last;  // the coarsest level: its pattern only
    last.n = U.n;
    last.rp = U.rp;
    last.ci = U.ci;
    out.push_back(std::move(last));
    return true;
}

}  // namespace ertgb
