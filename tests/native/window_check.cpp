// window_check.cpp -- host test of build_window_plan (ccd_b200/csrc/window_plan.cpp),
// built with sanitizers by tests/test_window_plan.py: on random matrices of all
// four column formats, with fixed columns and 1 to 16 CTAs, the conflict masks
// and the CTAs' slices must be those of a plain pairwise comparison.  Exit
// status 0 when every case agrees.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <set>
#include <vector>

#include "window.h"

using namespace ccdb;

int main(int argc, char** argv) {
    const int cases = argc > 1 ? std::atoi(argv[1]) : 200;
    std::mt19937_64 rng(4711);
    int failures = 0;
    for (int c = 0; c < cases; ++c) {
        // every twentieth matrix is tall enough for medium and long columns
        const int64_t K = c % 20 == 0 ? 1200 + rng() % 1200 : 1 + rng() % 200;
        const int32_t J = 1 + rng() % 60;
        const int C = 1 << rng() % 5;
        std::vector<uint8_t> fmt(J), fixed(J);
        std::vector<int64_t> cs(J + 1, 0), vs(J + 1, 0);
        std::vector<int32_t> rows;
        for (int j = 0; j < J; ++j) {
            const int f = rng() % 20;
            fmt[j] = f == 0 ? F_INTERCEPT : f == 1 ? F_DENSE : f < 8 ? F_SPARSE : F_INDICATOR;
            fixed[j] = rng() % 8 == 0;
            const bool dense = fmt[j] == F_DENSE || fmt[j] == F_INTERCEPT;
            if (!dense) {
                const unsigned dens = rng() % 3 ? 2 + rng() % 4 : rng() % 100;
                for (int64_t k = 0; k < K; ++k)
                    if (rng() % 100 < dens) rows.push_back((int32_t)k);
            }
            cs[j + 1] = (int64_t)rows.size();
            vs[j + 1] = vs[j] + (fmt[j] == F_DENSE ? K : fmt[j] == F_SPARSE ? cs[j + 1] - cs[j] : 0);
        }
        const bool no_fixed = rng() % 4 == 0;
        const WindowPlan w = build_window_plan(K, J, cs.data(), rows.data(), vs.data(), fmt.data(),
                                               no_fixed ? nullptr : fixed.data(), C);
        auto fail = [&](const char* what, int q) {
            if (failures++ < 10) std::printf("case %d position %d: %s\n", c, q, what);
        };
        std::vector<int> active;
        for (int j = 0; j < J; ++j)
            if (no_fixed || !fixed[j]) active.push_back(j);
        if (w.cols.size() != active.size() || w.slices.size() != active.size() * C) {
            fail("sizes", -1);
            continue;
        }
        std::vector<std::set<int64_t>> held(active.size());
        std::vector<bool> is_long(active.size());
        for (size_t q = 0; q < active.size(); ++q) {
            const int j = active[q];
            const bool dense = fmt[j] == F_DENSE || fmt[j] == F_INTERCEPT;
            if (dense)
                for (int64_t k = 0; k < K; ++k) held[q].insert(k);
            else
                held[q].insert(rows.begin() + cs[j], rows.begin() + cs[j + 1]);
            int64_t most = 0, at = 0;
            for (int r = 0; r < C; ++r) {
                const int64_t k0 = K * r / C, k1 = K * (r + 1) / C;
                int64_t n = 0;
                for (int64_t k : held[q]) n += k >= k0 && k < k1;
                const WinSlice s = w.slices[(size_t)r * active.size() + q];
                if (dense ? (s.lo != k0 || s.hi != k1) : (s.lo != at || s.hi != at + n)) fail("slice", (int)q);
                at += n;
                most = std::max(most, n);
            }
            is_long[q] = most > kWindowLong;
            const WinCol& m = w.cols[q];
            if (m.j != j || m.n != (int64_t)held[q].size() || m.cb != cs[j] || m.vb != vs[j]) fail("record", (int)q);
            if (((m.flags & 8) != 0) != is_long[q] || ((m.flags & 16) != 0) != (most > kWindowShort)) fail("length", (int)q);
        }
        for (size_t q = 0; q < active.size(); ++q) {
            if (is_long[q]) continue;
            for (int d = 1; d < kWindow && d <= (int)q; ++d) {
                if (is_long[q - d]) continue;
                bool meet = false;
                for (int64_t k : held[q]) meet |= held[q - d].count(k) > 0;
                if (((w.cols[q].conflict >> (kWindow - 1 - d)) & 1) != (meet ? 1 : 0)) fail("conflict", (int)q);
            }
        }
    }
    if (failures) return 1;
    std::printf("%d plans identical\n", cases);
    return 0;
}
