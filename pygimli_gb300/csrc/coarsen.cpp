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
#include <condition_variable>
#include <exception>
#include <functional>
#include <mutex>
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
// smoother alone solves it.  join: a row whose partners are all taken goes to the
// strongest one's aggregate instead of staying alone
int64_t match(const Csr &A, double strong, bool join, std::vector<int32_t> &agg) {
    agg.assign((size_t)A.n, -1);
    int64_t na = 0;
    for (int64_t i = 0; i < A.n; i++) {
        if (agg[i] >= 0) continue;
        double strongest = 0.0, best = 0.0, off = 0.0;
        int32_t with = -1, first = -1;
        for (int32_t q = A.rp[i]; q < A.rp[i + 1]; q++) {
            const int32_t j = A.ci[q];
            if (j == i) continue;
            const double c = -A.v[q];
            off += std::fabs(c);
            if (c > strongest) {
                strongest = c;
                first = j;
            }
            if (agg[j] < 0 && c > best) {
                best = c;
                with = j;
            }
        }
        if (off == 0.0) continue;
        if (join && with < 0 && first >= 0) {
            agg[i] = agg[first];
            continue;
        }
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

// Host threads of one hierarchy: started once (about 25 passes over rows follow,
// and starting 16 threads for each took longer than a pass), joined at the end.
// On 16 cores, against threads per pass over 2048 rows each at least: 23k nodes
// 20.3 -> 9.8 ms, 88k nodes 48 -> 30 ms.
class Team {
  public:
    static constexpr int kMost = 16;
    struct Part {  // what a part keeps from one construction to the next
        std::vector<int32_t> at, cols, ci;
        std::vector<double> acc, v;
    };
    Part part[kMost];

    explicit Team(int64_t n) {
        const int want = (int)std::min<int64_t>({(int64_t)std::thread::hardware_concurrency(), kMost, n / kRows});
        th_.reserve(kMost);
        try {
            for (int p = 1; p < want; p++) th_.emplace_back([this, p] { work(p); });
        } catch (const std::exception &) {  // no more threads or memory: those that started do
        }
    }
    ~Team() {
        {
            std::lock_guard<std::mutex> g(m_);
            stop_ = true;
        }
        start_.notify_all();
        for (auto &t : th_) t.join();
    }
    Team(const Team &) = delete;
    Team &operator=(const Team &) = delete;

    // f(first row, last row, part) over contiguous row ranges, kRows rows each at
    // least (a coarse level's rows are the long ones); returns the number of
    // parts.  An exception of a part is rethrown here
    template <class F> int by_rows(int64_t n, F f) {
        const int parts = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)th_.size() + 1, n / kRows));
        if (parts == 1) {
            f((int64_t)0, n, 0);
            return 1;
        }
        const std::function<void(int)> job = [&](int p) {
            try {
                f(n * p / parts, n * (p + 1) / parts, p);
            } catch (...) {
                errs_[p] = std::current_exception();
            }
        };
        {
            std::lock_guard<std::mutex> g(m_);
            for (auto &e : errs_) e = nullptr;
            job_ = &job;
            parts_ = parts;
            left_ = parts - 1;
            turn_++;
        }
        start_.notify_all();
        job(0);
        {
            std::unique_lock<std::mutex> g(m_);
            done_.wait(g, [&] { return left_ == 0; });
            job_ = nullptr;
        }
        for (auto &e : errs_)
            if (e) std::rethrow_exception(e);
        return parts;
    }

  private:
    static constexpr int64_t kRows = 256;
    std::vector<std::thread> th_;
    std::mutex m_;
    std::condition_variable start_, done_;
    const std::function<void(int)> *job_ = nullptr;
    int parts_ = 0, left_ = 0;
    uint64_t turn_ = 0;
    bool stop_ = false;
    std::exception_ptr errs_[kMost];

    void work(int p) {
        uint64_t seen = 0;
        std::unique_lock<std::mutex> g(m_);
        for (;;) {
            start_.wait(g, [&] { return stop_ || turn_ != seen; });
            if (stop_) return;
            seen = turn_;
            if (p >= parts_) continue;
            const std::function<void(int)> *job = job_;
            g.unlock();
            (*job)(p);
            g.lock();
            if (--left_ == 0) done_.notify_one();
        }
    }
};

// row-wise construction: row(i, at, acc, cols) fills the columns of row i
// (ascending in the result) and their values; scratch of m columns per part
template <class Row> Csr build_rows(Team &team, int64_t n, int64_t m, Row row) {
    Csr C;
    C.n = n;
    C.m = m;
    C.rp.assign((size_t)n + 1, 0);
    const int parts = team.by_rows(n, [&](int64_t i0, int64_t i1, int p) {
        Team::Part &w = team.part[p];
        w.at.assign((size_t)m, -1);
        w.acc.resize((size_t)m);
        w.ci.clear();
        w.v.clear();
        for (int64_t i = i0; i < i1; i++) {
            w.cols.clear();
            row(i, w.at, w.acc, w.cols);
            w.ci.insert(w.ci.end(), w.cols.begin(), w.cols.end());
            for (int32_t c : w.cols) w.v.push_back(w.acc[c]);
            C.rp[i + 1] = (int32_t)w.cols.size();
        }
    });
    for (int64_t i = 0; i < n; i++) C.rp[i + 1] += C.rp[i];
    C.ci.resize((size_t)C.rp[n]);
    C.v.resize((size_t)C.rp[n]);
    auto gather = [&](int64_t i0, int64_t, int p) {  // the same parts
        std::copy(team.part[p].ci.begin(), team.part[p].ci.end(), C.ci.begin() + C.rp[i0]);
        std::copy(team.part[p].v.begin(), team.part[p].v.end(), C.v.begin() + C.rp[i0]);
    };
    if (parts == 1) gather(0, n, 0);
    else team.by_rows(n, gather);
    return C;
}

// C = A B, columns ascending (B's rows may repeat a column)
Csr multiply(Team &team, const Csr &A, const Csr &B) {
    return build_rows(team, A.n, B.m, [&](int64_t i, std::vector<int32_t> &at, std::vector<double> &acc,
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

// sum of A's entries over aggregates of rows and columns (T^T A T), an
// aggregate's rows in ascending order
Csr collapse(Team &team, const Csr &A, const std::vector<int32_t> &agg, int64_t na) {
    std::vector<int32_t> first((size_t)na + 1, 0), rows((size_t)A.n);
    for (int32_t a : agg)
        if (a >= 0) first[a + 1]++;
    for (int64_t a = 0; a < na; a++) first[a + 1] += first[a];
    std::vector<int32_t> pos(first.begin(), first.end() - 1);
    for (int64_t i = 0; i < A.n; i++)
        if (agg[i] >= 0) rows[pos[agg[i]]++] = (int32_t)i;
    return build_rows(team, na, na, [&](int64_t a, std::vector<int32_t> &at, std::vector<double> &acc,
                                        std::vector<int32_t> &cols) {
        for (int32_t r = first[a]; r < first[a + 1]; r++)
            for (int32_t q = A.rp[rows[r]]; q < A.rp[rows[r] + 1]; q++) {
                const int32_t c = agg[A.ci[q]];
                if (c < 0) continue;
                if (at[c] != (int32_t)a) {
                    at[c] = (int32_t)a;
                    acc[c] = 0.0;
                    cols.push_back(c);
                }
                acc[c] += A.v[q];
            }
        std::sort(cols.begin(), cols.end());
    });
}

// smoothed, filtered prolongation of the aggregates
Csr prolongation(Team &team, const Csr &U, const std::vector<int32_t> &agg, int64_t na) {
    // D = the rows' absolute sums: D^-1 U has its spectrum in [0, 1]
    std::vector<double> l1((size_t)U.n, 0.0);
    for (int64_t i = 0; i < U.n; i++)
        for (int32_t q = U.rp[i]; q < U.rp[i + 1]; q++) l1[i] += std::fabs(U.v[q]);
    const double w = 4.0 / 3.0;
    Csr P = build_rows(team, U.n, na, [&](int64_t i, std::vector<int32_t> &at, std::vector<double> &acc,
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
    Team team(U.n);
    while (U.n > coarsest) {
        if ((int)out.size() >= max_levels) return false;
        const int passes = U.n > kTail ? 2 : 3;
        std::vector<int32_t> a1, a2;
        auto pair_up = [&](double strong, bool join) {
            int64_t n2 = match(U, strong, join, a1);
            Csr W = collapse(team, U, a1, n2);
            for (int p = 1; p < passes; p++) {
                n2 = match(W, strong, join, a2);
                for (auto &a : a1)
                    if (a >= 0) a = a2[a];
                if (p + 1 < passes) W = collapse(team, W, a2, n2);
            }
            return n2;
        };
        int64_t n2 = pair_up(U.n > kSmall ? kStrong : 0.0, false);
        auto stalls = [&] { return n2 < 1 || n2 * 10 > U.n * 6; };
        // H2 and P2 refinements end in stars (rows that couple to one hub only, from
        // some 1700 rows downwards), which pairs cannot collapse.  With the hierarchy given
        // up there its construction was lost: first responses on the H2 mesh of a
        // 16.6k-node box, 12 electrodes, FSAI, took 166 ms, 118 without coarse levels, 99
        // so (P2: 273, 214, 128), repeated ones 115 and 43 (185 and 41).
        if (stalls()) n2 = pair_up(0.0, true);
        if (stalls()) return false;  // no useful hierarchy
        Csr P = prolongation(team, U, a1, n2), PT = transpose(P), AP = multiply(team, U, P);
        Csr C = multiply(team, PT, AP);
        HostLevel l;
        l.n = U.n;
        l.nc = n2;
        l.rp = std::move(U.rp);
        l.ci = std::move(U.ci);
        l.P_rp = std::move(P.rp);
        l.P_ci = std::move(P.ci);
        l.P_v.assign(P.v.begin(), P.v.end());
        l.PT_rp = std::move(PT.rp);
        l.PT_ci = std::move(PT.ci);
        l.PT_v.assign(PT.v.begin(), PT.v.end());
        l.AP_rp = std::move(AP.rp);
        l.AP_ci = std::move(AP.ci);
        out.push_back(std::move(l));
        U = std::move(C);
    }
    if (out.empty()) return false;
    HostLevel last;  // the coarsest level: its pattern only
    last.n = U.n;
    last.rp = std::move(U.rp);
    last.ci = std::move(U.ci);
    out.push_back(std::move(last));
    return true;
}

}  // namespace ertgb
