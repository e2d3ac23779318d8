// exit_check.cpp -- host test of on_the_way (ccd_b200/csrc/sweep_exit.h), run by
// tests/test_sweep_exit.py.  CTAs that exchange messages of random delays, each wait
// with a random bound, are stepped through one cycle by an event queue; a CTA's two
// barriers count announced and landed bytes as the hardware's do.  Whatever runs
// out, every CTA must reach the end of the cycle, and one that gave up must see its
// corrected barriers complete exactly when the last byte sent to it has landed.
#include <cstdio>
#include <cstdlib>
#include <queue>
#include <random>
#include <vector>

#include "sweep_exit.h"

using namespace ccdb;

namespace {

struct Barrier {
    int phase = 0;
    bool announced = false;
    long tx = 0;
    void settle() {
        if (announced && tx == 0) {
            ++phase;
            announced = false;
        }
    }
    void announce(long bytes) {
        announced = true;
        tx += bytes;
        settle();
    }
    void land(long bytes) {
        tx -= bytes;
        settle();
    }
};

struct Event {
    double at;
    int kind, cta, from, exchange;  // 0: a message lands; 1: the CTA acts; 2: its wait runs out
    bool operator<(const Event& o) const { return at > o.at; }
};

}  // namespace

int main(int argc, char** argv) {
    const int cases = argc > 1 ? std::atoi(argv[1]) : 2000;
    std::mt19937_64 rng(99);
    long gave_up_cases = 0, ahead_seen = 0, missing_seen = 0, mixed_end = 0;
    for (int i = 0; i < cases; ++i) {
        const int C = 1 + (int)(rng() % 16), R = 1 + (int)(rng() % 6);
        std::vector<uint32_t> bytes(R + 1);
        for (auto& b : bytes) b = 8 * (1 + rng() % 20);
        auto unit = [&] { return (rng() % 100000) / 100000.0; };
        const double limit = 0.5 + 2.0 * unit(), slow = i % 3 ? 0.03 : 0.0;
        std::priority_queue<Event> q;
        std::vector<CycleReport> rep(C);
        std::vector<Barrier> bar(2 * C);
        std::vector<int> at_end(C, 0), waiting(C, -1), in_flight(C, 0);
        auto act = [&](int c, double t) {  // send for the next exchange, or be at the end of the cycle
            CycleReport& r = rep[c];
            if ((int)r.sent == R) {
                at_end[c] = 1;
                return;
            }
            const int e = (int)r.sent++;
            r.bytes[e & 1] = bytes[e];
            bar[2 * c + (e & 1)].announce((long)C * bytes[e]);
            for (int to = 0; to < C; ++to) {
                const double d = 0.1 * unit() + (unit() < slow ? 4.0 * unit() : 0.0);
                q.push({t + d, 0, to, c, e});
                ++in_flight[to];
            }
            waiting[c] = e;
            q.push({t + limit, 2, c, 0, e});
        };
        for (int c = 0; c < C; ++c) q.push({0.3 * unit() + (unit() < slow ? 3.0 * unit() : 0.0), 1, c, 0, 0});
        std::vector<Event> late;  // what lands after the end of the cycle
        while (!q.empty()) {
            int done = 0;
            for (int c = 0; c < C; ++c) done += at_end[c];
            if (done == C) break;
            const Event v = q.top();
            q.pop();
            if (v.kind == 0) {
                --in_flight[v.cta];
                Barrier& b = bar[2 * v.cta + (v.exchange & 1)];
                const int before = b.phase;
                b.land(bytes[v.exchange]);
                if (b.phase != before && waiting[v.cta] >= 0 && (waiting[v.cta] & 1) == (v.exchange & 1)) {
                    waiting[v.cta] = -1;
                    q.push({v.at + 0.02 * unit(), 1, v.cta, 0, 0});
                }
            } else if (v.kind == 1) {
                if (!rep[v.cta].gave_up) act(v.cta, v.at);
            } else if (waiting[v.cta] == v.exchange) {
                rep[v.cta].gave_up = 1;
                at_end[v.cta] = 1;
                waiting[v.cta] = -1;
            }
        }
        int up = 0;
        for (int c = 0; c < C; ++c) {
            if (!at_end[c]) {
                std::printf("case %d: CTA %d never reaches the end of the cycle\n", i, c);
                return 1;
            }
            up += (int)rep[c].gave_up;
        }
        gave_up_cases += up > 0;
        mixed_end += up > 0 && up < C;
        for (; !q.empty(); q.pop())
            if (q.top().kind == 0) late.push_back(q.top());
        for (int c = 0; c < C; ++c) {
            if (!rep[c].gave_up) {
                if (in_flight[c] != 0) {
                    std::printf("case %d: CTA %d did not give up and bytes are on their way to it\n", i, c);
                    return 1;
                }
                continue;
            }
            const OnTheWay w = on_the_way(rep.data(), C, c);
            ahead_seen += w.ahead > 0;
            missing_seen += w.missing > 0;
            const int e = (int)rep[c].sent - 1;
            Barrier &a = bar[2 * c + (e & 1)], &n = bar[2 * c + (~e & 1)];
            const int want_a = (e >> 1) + 1, want_n = ((e + 1) >> 1) + 1;
            if (w.missing) a.land((long)w.missing);
            if (w.ahead) n.announce((long)w.ahead);
            for (const Event& v : late) {
                if (v.cta != c) continue;
                if (in_flight[c] > 0 && a.phase == want_a && (!w.ahead || n.phase == want_n)) {
                    std::printf("case %d: CTA %d leaves while bytes are on their way to it\n", i, c);
                    return 1;
                }
                bar[2 * c + (v.exchange & 1)].land(bytes[v.exchange]);
                --in_flight[c];
            }
            if (a.phase != want_a || (w.ahead && n.phase != want_n) || a.tx != 0 || n.tx != 0) {
                std::printf("case %d: CTA %d waits for bytes that nobody sent\n", i, c);
                return 1;
            }
        }
    }
    std::printf("%d cycles, %ld with a wait that ran out (%ld with CTAs that did not), %ld missing, %ld ahead: all left in order\n",
                cases, gave_up_cases, mixed_end, missing_seen, ahead_seen);
    return gave_up_cases && mixed_end && ahead_seen && missing_seen ? 0 : 2;
}
