// window_device.cuh -- device pieces that the two windowed sweeps share
// (window.cu, group_window.cu): sixteen warps with a column each, four helper
// warps that copy ahead, and the exchange between the CTAs of a cluster.
#pragma once

#include <cstdint>

#include "common.cuh"
#include "sweep_exit.h"
#include "window_sweep.h"

namespace ccdb {
namespace win {

constexpr int kHelpers = 4;             // warps that look ahead for the others, one per scheduler
constexpr int kWorkers = kWindow * 32;  // threads that hold columns
constexpr int kT = kWorkers + 32 * kHelpers;
constexpr int kWarps = kT / 32;
constexpr int kE = 4;            // staged entries per lane
constexpr int kStage = 32 * kE;  // a warp's column: its first entries, copied ahead
constexpr unsigned kFull = 0xffffffffu;
constexpr long long kLookNs = 1000 * 1000;  // an attempt to wait sleeps in hardware for less
static_assert(kHelpers * 4 == kWindow, "eight lanes of a helper copy for a slot");

// The record of one position, copied ahead of its use.
struct __align__(16) Rec {
    WinCol c;
    WinScal s;
    double2 bh;
    WinSlice e;
    int64_t pad;
};
static_assert(sizeof(WinScal) == 48 && sizeof(Rec) == 112, "copied in 16-byte pieces");

// What the helpers decide between two rounds.
struct __align__(16) Turn {
    int base;   // the first position in flight
    int limit;  // positions below it are in flight
    int alone;  // base's column is the only one
    int stop;   // a wait for the other CTAs ran out
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned peer_u32(const void* p, int rank) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the threads that hold columns
__device__ __forceinline__ void workers_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kWorkers) : "memory"); }

// st.async of 8 or 16 bytes to shared memory `at` of a CTA of the cluster, counted
// by the mbarrier `bar` there (addresses of the cluster's window).
__device__ __forceinline__ void send8(unsigned at, unsigned bar, double v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(at), "d"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void send16(unsigned at, unsigned bar, double a, double b) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(at), "d"(a), "d"(b), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void expect_bytes(const uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// whether the bytes have come: a look, then one that sleeps in hardware for a while
__device__ __forceinline__ bool landed(const uint64_t* bar, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool arrived(const uint64_t* bar, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
// false when the bytes have not all come within limit_ns, by looks that sleep
__device__ __forceinline__ bool wait_sleeping(const uint64_t* bar, unsigned parity, long long limit_ns) {
    unsigned long long t0 = 0;
    for (unsigned n = 0; !arrived(bar, parity); ++n)
        if ((n & 15u) == 15u) {
            const unsigned long long t = global_ns();
            if (t0 == 0) t0 = t;
            if ((long long)(t - t0) > limit_ns) return false;
        }
    return true;
}
// the same for a bound below one sleep
__device__ __forceinline__ bool wait_looking(const uint64_t* bar, unsigned parity, long long limit_ns) {
    const unsigned long long t0 = global_ns();
    while (!landed(bar, parity))
        if ((long long)(global_ns() - t0) > limit_ns) return false;
    return true;
}
__device__ __forceinline__ bool wait_bytes(const uint64_t* bar, unsigned parity, long long limit_ns) {
    const bool brief = limit_ns < kLookNs;
    if (!brief && arrived(bar, parity)) return true;  // nearly always; without this line a Poisson fit took 1.2 % longer
    return brief ? wait_looking(bar, parity, limit_ns) : wait_sleeping(bar, parity, limit_ns);
}
__device__ __forceinline__ void init_bars(uint64_t* bars, int n) {
    for (int i = 0; i < n; ++i)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bars + i)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// A copy of `bytes` (a multiple of 16, from and to 16-byte boundaries) to this CTA's
// shared memory by the copy engine, counted by `bar`.
__device__ __forceinline__ void bulk_copy(void* to, const void* from, unsigned bytes, const uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(to)),
                 "l"(from), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// What was sent to a CTA that gave up an exchange lands before it leaves (bounded).
__device__ __forceinline__ void drain(const uint64_t* bar, unsigned parity) {
    const unsigned long long t0 = global_ns();
    while (!arrived(bar, parity) && global_ns() - t0 < 1000000000ull) __nanosleep(200);
}
// `bytes` that were announced to this CTA's `bar` and that nobody sends.
__device__ __forceinline__ void forgo_bytes(const uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// A CTA's report of the cycle into `to` (by CTA) of CTA `peer`.
__device__ __forceinline__ void tell(const CycleReport* to, int peer, const CycleReport& r) {
    asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(peer_u32(to, peer)), "r"(r.gave_up), "r"(r.sent),
                 "r"(r.bytes[0]), "r"(r.bytes[1])
                 : "memory");
}
// One thread of a CTA that gave up, once all reports are here: every byte that was
// sent to this CTA has landed (sweep_exit.h).
__device__ __forceinline__ void land_all(const uint64_t* bars, const CycleReport* all, int C, int me) {
    const OnTheWay w = on_the_way(all, C, me);
    const unsigned e = all[me].sent - 1, n = e + 1;  // the last announced exchange, and the one after it
    if (w.missing) forgo_bytes(&bars[e & 1], w.missing);
    if (w.ahead) expect_bytes(&bars[n & 1], w.ahead);
    drain(&bars[e & 1], (e >> 1) & 1);
    if (w.ahead) drain(&bars[n & 1], (n >> 1) & 1);
}

// Copies made ahead of use by eight lanes (l8) of a helper.
struct Ahead {
    const WinCol* cols;
    const WinScal* scal;
    const double2* bh;
    const WinSlice* slices;  // this CTA's
    const int32_t* rows;
    const double* vals;
    int n_active;

    // the record of the column at a position
    __device__ __forceinline__ void record(int at, Rec& r, int l8) const {
        if (at >= n_active) return;
        const char* from = reinterpret_cast<const char*>(l8 < 2   ? (const void*)(cols + at)
                                                         : l8 < 5 ? (const void*)(scal + at)
                                                                  : (const void*)(bh + at));
        if (l8 < 6) cp_async16(reinterpret_cast<char*>(&r) + 16 * l8, from + 16 * (l8 < 2 ? l8 : l8 < 5 ? l8 - 2 : 0));
        else if (l8 == 6) cp_async8(&r.e, slices + at);
    }
    // its first STAGE entries, by LANES lanes
    template <int STAGE = kStage, int LANES = 8>
    __device__ __forceinline__ void entries(int at, const Rec& r, int32_t* to, double* vto, int l8) const {
        if (at >= n_active || (r.c.flags & 8)) return;
        const int n = min(r.e.hi - r.e.lo, STAGE);
        const int32_t* from = rows + r.c.cb + r.e.lo;
        const double* vfrom = vals + r.c.vb + r.e.lo;
#pragma unroll 2
        for (int p = l8; p < n; p += LANES) {
            if (r.c.flags & 1) cp_async4(to + p, from + p);
            else to[p] = r.e.lo + p;
            if (r.c.flags & 2) cp_async8(vto + p, vfrom + p);
        }
    }
    // every copy that this thread began has landed
    __device__ __forceinline__ void done() const {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
    }
};

// The stamps of a traced sweep, by one lane of a helper that has little else to do.  A
// traced sweep is another compilation of the same code: a pointer that is tested
// each round cost a fit 1.5 %.
#ifdef CCDB_TRACE_ROUNDS
struct Tracer {
    RoundStamp* to;
    bool mine;
    const volatile int* gate;  // a word of shared memory, not below 0
    int n = 0;
    RoundStamp s{};
    // the clock behind the last barrier: its reading depends on a word that is read there
    // (by itself it moved in front of the barrier)
    __device__ long long now() const { return *gate >= 0 ? clock64() : 0; }
    __device__ void begin(int base, int flying, int alone) {
        s.begin = now();
        s.base = base;
        s.flying = flying;
        s.alone = alone;
    }
    __device__ void steps() { s.steps = now(); }
    __device__ void end(int taken, int moved) {
        s.end = now();
        s.taken = taken;
        s.moved = moved;
        if (mine && n < kTracedRounds) to[n] = s;
        ++n;
    }
};
#else
struct Tracer {
    RoundStamp* to;
    bool mine;
    const volatile int* gate;
    __device__ __forceinline__ void begin(int, int, int) {}
    __device__ __forceinline__ void steps() {}
    __device__ __forceinline__ void end(int, int) {}
};
#endif

// where the staged entries of a position lie
template <int STAGE = kStage, int WINDOW = kWindow>
__device__ __forceinline__ int stage_at(int pos) { return (((pos / WINDOW) & 1) * WINDOW + (pos & (WINDOW - 1))) * STAGE; }

}  // namespace win
}  // namespace ccdb
