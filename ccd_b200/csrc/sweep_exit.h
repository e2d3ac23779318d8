// sweep_exit.h -- how the CTAs of a cluster leave a windowed sweep together when a
// bounded wait has run out in one of them (window.cu, group_window.cu).
//
// Exchanges are numbered; a CTA sends for exchange e + 1 only when every byte of
// exchange e has come to it.  A CTA whose wait for exchange e runs out sends no
// more, so the others run out of exchange e or e + 1 in their turn, and all of them
// meet at the end of the cycle.  There each tells the others whether it gave up,
// for how many exchanges it has sent, and the bytes that it sent to each CTA in the
// last two.  One that gave up makes all of them leave, and from these reports a CTA
// knows what may still be on its way to its shared memory, which it awaits before
// it leaves.
#pragma once

#include <cstdint>

#include "step.h"

namespace ccdb {

struct CycleReport {
    uint32_t gave_up;
    uint32_t sent;      // exchanges that this CTA has sent for
    uint32_t bytes[2];  // to each CTA, in the last even and the last odd one
};
static_assert(sizeof(CycleReport) == 16, "sent as one word");

// What a CTA that gave up has to put right on its barriers before it can wait for
// what is on its way: exchange sent - 1 was announced to its barrier with the bytes
// of all CTAs, `missing` of which nobody sent; exchange `sent` was not announced,
// and `ahead` bytes of it have been sent.
struct OnTheWay {
    uint32_t missing, ahead;
};

CCDB_HD OnTheWay on_the_way(const CycleReport* all, int C, int me) {
    OnTheWay w{0, 0};
    const uint32_t n = all[me].sent;
    for (int c = 0; c < C; ++c) {
        if (all[c].sent < n) w.missing += all[me].bytes[(n - 1) & 1];
        if (all[c].sent > n) w.ahead += all[c].bytes[n & 1];
    }
    return w;
}

}  // namespace ccdb
