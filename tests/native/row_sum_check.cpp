// CPU check of the segmented serial sum (row_sum.h): the warp algorithm of warp_row_sum
// replayed lane by lane, in calls of up to 32 x 36 terms, against the plain serial loop
// acc = acc + t_k, on the row families of serial_sum_cases.h; and the offset rules
// (rs::row_mark, rs::row_code, rs::row_apply) against chains actually added from shifted starts.
//
//   row_sum_check ROWS  ->  "rows R terms T bad B serial S rules N rbad M"
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../red.cuda.closeencounter_gb300/csrc/row_sum.h"
#include "serial_sum_cases.h"

using namespace redgb;
using xf::bitsd;
using xf::dbits;

static long long g_serial = 0;

// one call of warp_row_sum over m <= 32 seg terms
static double call_emulated(double acc, const double* T, int seg, int m)
{
    double p[32], g[32];
    uint64_t end[32], tend[32];
    std::vector<uint32_t> codes[32];
    bool hard[32], loose[32], done[32];
    int n[32], P[32];
    int d[32];
    for (int l = 0; l < 32; l++) {
        n[l] = std::max(0, std::min(seg, m - l * seg));
    }
    int top = (int)((dbits(acc) >> 52) & 0x7ff);
    for (int k = 0; k < m; k++) top = std::max(top, (int)((dbits(T[k]) >> 52) & 0x7ff));
    int64_t u = rs::row_units(dbits(acc), top);
    for (int l = 0; l < 32; l++) {
        p[l] = bitsd(rs::row_from_units(u, top));
        for (int k = 0; k < n[l]; k++) u += rs::row_units(dbits(T[l * seg + k]), top);
    }
    bool any = false;
    for (int l = 0; l < 32; l++) {
        g[l] = l ? p[l] : acc;
        hard[l] = rs::near_edge(dbits(g[l]));
        double a = g[l];
        for (int k = 0; k < n[l]; k++) {
            const double t = T[l * seg + k], s = a + t;
            const uint32_t rec = rs::row_mark(dbits(a), dbits(t), dbits(s), k, &hard[l]);
            if (rec) codes[l].push_back(rs::row_code(rec, dbits(t)));
            a = s;
        }
        end[l] = tend[l] = dbits(a);
        d[l] = 0;
        loose[l] = l > 0 && !rs::row_diff(end[l - 1], dbits(g[l]), &d[l]);
        if (l == 0 || loose[l]) d[l] = 0;
        any = any || loose[l] || d[l] != 0;
        P[l] = (l ? P[l - 1] : 0) + d[l];
        done[l] = l == 0;
    }
    if (!any) return bitsd(end[31]);
    const int LIM = (int)(rs::MAX_OFF / 2);
    unsigned todo = 0, slows = 0;
    for (int l = 1; l < 32; l++) {
        const bool slow = hard[l] || loose[l] || P[l] >= LIM || P[l] <= -LIM;
        if (!codes[l].empty() || slow) todo |= 1u << l;
        if (slow) slows |= 1u << l;
    }
    int off = 0;
    auto mine = [&](int l) { return done[l] ? tend[l] : rs::row_shift(end[l], P[l] + off); };
    while (todo) {
        const int L = __builtin_ctz(todo);
        todo &= todo - 1;
        const bool is_slow = slows >> L & 1;
        uint64_t start = is_slow ? mine(L - 1) : rs::row_shift(dbits(g[L]), P[L] + off);
        int dl = P[L] + off;
        bool serial = false, force = false;
        if (is_slow) serial = !rs::row_diff(start, dbits(g[L]), &dl) || (hard[L] && dl != 0);
        if (!serial && dl != 0)
            for (size_t q = 0; q < codes[L].size(); q++) {
                dl = rs::row_apply(codes[L][q], dl);
                if ((dl ^ (dl >> 31)) >= (int)rs::MAX_OFF) {
                    serial = true;
                    break;
                }
            }
        if (serial) {
            double b = bitsd(start);
            for (int q = 0; q < n[L]; q++) b = b + T[L * seg + q];
            g_serial += n[L];
            tend[L] = dbits(b);
            force = !rs::row_diff(tend[L], end[L], &dl);
        } else {
            tend[L] = rs::row_shift(end[L], dl);
        }
        done[L] = true;
        off = dl - P[L];
        if (force || off >= LIM || off <= -LIM) {
            if (L < 31) {
                todo |= 1u << (L + 1);
                slows |= 1u << (L + 1);
            }
            off = 0;
        }
    }
    return bitsd(mine(31));
}

static bool same(double a, double b) { return (std::isnan(a) && std::isnan(b)) || dbits(a) == dbits(b); }

int main(int argc, char** argv)
{
    const long long rows = argc > 1 ? atoll(argv[1]) : 2000;
    std::vector<double> t(SC_MAX_LEN + 64);
    long long terms = 0, bad = 0;
    for (int fam = 0; fam < 5; fam++) {
        const long long s0 = g_serial, t0 = terms;
        for (long long row = 0; row < rows; row++) {
            double acc0;
            const int n = sc_row(4711, fam, (uint64_t)row, &acc0, t.data());
            double ref = acc0;
            for (int k = 0; k < n; k++) ref = ref + t[k];
            // whole rows and rows in short calls (segments of 1 to 36 terms)
            for (int form = 0; form < 2; form++) {
                const int most = form ? 32 * (1 + (int)(row % 7)) : 32 * 36;
                double got = acc0;
                for (int b = 0; b < n; b += most) {
                    const int m = std::min(most, n - b);
                    got = call_emulated(got, t.data() + b, (m + 31) / 32, m);
                }
                if (!same(ref, got)) {
                    if (bad < 5) printf("mismatch family %d row %lld form %d: %a vs %a\n", fam, row, form, got, ref);
                    bad++;
                }
            }
            terms += 2 * n;
        }
        printf("family %d terms %lld serial %lld\n", fam, terms - t0, g_serial - s0);
    }
    // the rules: a chain of additions from a start shifted by d ulps ends where the codes say
    long long rules = 0, rbad = 0;
    ScRng g{99};
    for (long long k = 0; k < 50 * rows; k++) {
        const double a0 = (g.below(2) ? -1.0 : 1.0) * sc_random_mag(g, -2, 2);
        const int d0 = g.below(2001) - 1000;
        if (rs::near_edge(dbits(a0))) continue;
        double a = a0, b = bitsd(rs::row_shift(dbits(a0), d0));
        int d = d0;
        bool use = true;
        for (int q = 0; q < 12 && use; q++) {
            double tq = (g.below(2) ? -1.0 : 1.0) * sc_random_mag(g, -12, 1);
            if (g.below(3) == 0) tq = bitsd(dbits(tq) & ~((1ull << g.below(50)) - 1));  // short significands: ties
            const double s = a + tq;
            bool hard = false;
            const uint32_t rec = rs::row_mark(dbits(a), dbits(tq), dbits(s), q, &hard);
            use = !hard;
            if (use && rec) d = rs::row_apply(rs::row_code(rec, dbits(tq)), d);
            if (d >= rs::MAX_OFF || d <= -rs::MAX_OFF) use = false;
            if (!use) break;
            a = s;
            b = b + tq;
            rules++;
            if (rs::row_shift(dbits(a), d) != dbits(b)) {
                rbad++;
                break;
            }
        }
    }
    printf("rows %lld terms %lld bad %lld serial %lld rules %lld rbad %lld\n", 5 * rows, terms, bad, g_serial, rules, rbad);
    return bad || rbad ? 1 : 0;
}
