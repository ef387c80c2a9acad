// What the kernels with resident anatomy (rd_lanes.cu, adj_lanes.cu) share: the
// division of an SM into lanes, their barrier and the row arithmetic.
#pragma once
#include "gbg_internal.cuh"

#include "arrivals.cuh"

namespace gbg {
namespace lanes {

constexpr int kWps = 4;                    // warps per scheduler: 16 warps of up to 128 registers
constexpr int kThreads = 128 * kWps;
// Samples a team has in flight. More lanes hide more of the barrier (4: 205 ms on
// the 512-sample population, 8: 164 ms, both with rows moved between planes; in
// register rings 8 take 150); beyond 8 the states of a 128^3 population outgrow L2.
constexpr int kMaxLanes = 8;
// a unit's table, one float4 per lane and slot: cxs (2 rows), cy (rows y-1,
// y, y+1), cz (2 rows)
constexpr int kSlots = 7;
constexpr size_t kUnitBytes = (size_t)kSlots * 32 * sizeof(float4);
constexpr int kMaxUnits = 64;              // units a CTA can own
// The tables' room in a CTA; the rest of the 227 KB is the kernels' static shared
// memory. A kernel's limit is the function's, not a handle's: it is always set to
// this, as a smaller one would fail the launch another thread is about to make.
constexpr int kTableBytes = 224 * 1024;
static_assert(kMaxUnits * kUnitBytes <= kTableBytes, "the most units fit");
// Planes loaded ahead: one plane's arithmetic does not cover an L2 load (170
// against 164 ms, before the rings), a third plane spills registers (207 ms).
constexpr int kAhead = 2;
constexpr int kSyncStride = 32;            // words per lane of the barrier array

__device__ __forceinline__ int wrapm(int i, int n) { return i == 0 ? n - 1 : i - 1; }
__device__ __forceinline__ int wrapp(int i, int n) { return i == n - 1 ? 0 : i + 1; }

// what a lane's warps share of its samples and its barrier
struct Lane {
    int next, ok;            // sample to take next (sorted order), no timeout so far
    unsigned target, slot;   // arrivals the next barrier waits for, slot of the next sample number
};

__device__ __forceinline__ bool span_hits(int lo, int hi, int grow, int a, int b, int n) {
    lo -= grow;
    hi += grow;
    if (lo < 0 || hi > n - 1) return true;
    return lo <= b && a <= hi;
}

__device__ __forceinline__ void group_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

struct V4 {
    float v[4];
};
__device__ __forceinline__ V4 v4(const float4 &a) { return V4{{a.x, a.y, a.z, a.w}}; }
__device__ __forceinline__ V4 ldp(const float *p) { return v4(*reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ V4 ldg4(const float *p) { return v4(__ldg(reinterpret_cast<const float4 *>(p))); }
__device__ __forceinline__ V4 lds(const float4 *p) { return v4(*p); }
__device__ __forceinline__ V4 sub(const V4 &a, const V4 &b) {
    return V4{{a.v[0] - b.v[0], a.v[1] - b.v[1], a.v[2] - b.v[2], a.v[3] - b.v[3]}};
}

// The number of the lane's next sample: drawn from `queue` by rank 0 on the way into
// the barrier of the last step, and read by everyone after it. Two slots in turn,
// as a CTA may still have to read one when the next is written.
__device__ __forceinline__ void draw_next(const Lane &ln, unsigned *sync, unsigned *queue, int lanes) {
    *(volatile unsigned *)(sync + 1 + ln.slot) = atomicAdd(queue, 1u) + (unsigned)lanes;
}
__device__ __forceinline__ void read_next(Lane &ln, const unsigned *sync) {
    ln.next = (int)*(volatile const unsigned *)(sync + 1 + ln.slot);
    ln.slot ^= 1u;
}

// Barrier of a team's T CTAs on one lane, by one thread of the lane after its
// warps have met: sync[0] counts arrivals. last: the sample's last step.
// Bounded (seconds); on a timeout the status word is set and every lane leaves
// at its next barrier.
__device__ __forceinline__ void lane_barrier(Lane &ln, unsigned *sync, unsigned *queue, int T, int rank, int lanes, bool last,
                                             int *status) {
    if (last && rank == 0) draw_next(ln, sync, queue, lanes);
    arrive(sync);
    ln.target += T;
    if (!wait_for_arrivals(sync, ln.target, status)) ln.ok = 0;
    if (last) read_next(ln, sync);
}

// lane_barrier where the team is a cluster: a CTA arrives at the shared-memory
// barrier `bar` of every CTA and waits at its own (target counts its phases). A
// CTA may arrive for phase j + 1 where another's arrival for phase j is still on
// its way, but no phase ends early: when the first wait for phase j ends anywhere,
// its barrier has (j + 1) T arrivals, of which none came from a CTA more than j +
// 1 times, so every CTA has released its step j; the fence before the arrivals
// carries that on.
__device__ __forceinline__ void cluster_barrier(Lane &ln, unsigned long long *bar, unsigned *sync, unsigned *queue, int T, int rank,
                                                int lanes, bool last, int *status) {
    if (last && rank == 0) draw_next(ln, sync, queue, lanes);
    const unsigned own = (unsigned)__cvta_generic_to_shared(bar), parity = ln.target & 1u;
    asm volatile("fence.acq_rel.cluster;" ::: "memory");
    for (int r = 0; r < T; ++r) {
        unsigned at;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(own), "r"(r));
        asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(at) : "memory");
    }
    unsigned done = 0;
    for (long long spins = 0; !done;) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(own), "r"(parity)
            : "memory");
        if (done) break;
        if (++spins > (1ll << 27)) {  // a test is shorter than a load from L2: seconds too
            atomicExch(status, (int)DEV_BARRIER_TIMEOUT);
            ln.ok = 0;
            break;
        }
        if ((spins & 16383) == 0 && *(volatile int *)status != DEV_OK) {
            ln.ok = 0;
            break;
        }
    }
    ++ln.target;
    if (last) read_next(ln, sync);
}

}  // namespace lanes
}  // namespace gbg
