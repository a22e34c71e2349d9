// cluster_max.cuh -- the argmax of CLEAN's minor cycles: candidates as 64-bit keys, their maximum
// over a warp, and over a thread-block cluster by remote stores.
#pragma once
#include <stdint.h>

struct Cand {
    float a;      // |value|
    int32_t idx;  // flat 0-based index, INT32_MAX if none
    float v;      // signed value
};

// A candidate as a 64-bit key whose unsigned order is better()'s: |value| bits (|value| >= 0
// and not NaN here, so the bits order as the values do), then INT32_MAX - index (the first
// index wins a tie), then the value's sign bit.  One atomicMax per CTA finds the maximum.
__device__ __forceinline__ unsigned long long cand_key(Cand c) {
    return ((unsigned long long)__float_as_uint(c.a) << 32) |
           ((unsigned long long)(uint32_t)(INT32_MAX - c.idx) << 1) | (__float_as_uint(c.v) >> 31);
}
// the largest key of a warp's lanes: the largest high word, then the largest low word among
// the lanes that hold it
__device__ __forceinline__ unsigned long long warp_key_max(unsigned long long k) {
    const unsigned hi = (unsigned)(k >> 32), lo = (unsigned)k;
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    return ((unsigned long long)mhi << 32) | mlo;
}
__device__ __forceinline__ Cand key_cand(unsigned long long k) {
    Cand c;
    c.a = __uint_as_float((uint32_t)(k >> 32));
    c.idx = INT32_MAX - (int32_t)((uint32_t)k >> 1);
    c.v = (k & 1ull) ? -c.a : c.a;
    return c;
}

constexpr int CM_SPIN = 1 << 20;  // polls of a cluster wait before it gives up
inline int cm_spin(int wait_limit) { return wait_limit < 0 ? CM_SPIN : wait_limit; }

__device__ __forceinline__ uint32_t cl_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// The cluster's maxima of one round: slot r holds CTA r's key.
template <int C>
struct ClusterMax {
    unsigned long long slot[2][C];
    unsigned long long bar[2];
};

// Waits that run out.  A warp whose wait of round n runs out takes note (CM_LATE) and goes to the
// top of round n + 1.  Other warps of its CTA may have had the keys in time, so between a wait and
// the top of the next round no warp takes a CTA-wide barrier or leaves the loop; at the top the CTA
// votes.  There the warp waits once more, as long: the other CTAs' stores to this one must land
// before it may leave, and their keys say whether round n was the last, where all stop as they
// would have.  If not, the CTA sends CM_ABORT in place of its key, which is above every key (|value|
// has no sign bit): all CTAs find it in the round's maximum and stop together, with no store on
// its way.  Only when the second wait runs out as well does a CTA leave without the others.
// The states share one word and the loops count in rounds alone: a register each for a flag or a
// counter cost 1-4 % of an iteration where the residual fills the registers.
constexpr unsigned CM_LATE = 1, CM_LAST = 2, CM_GAVE_UP = 4;  // a warp's state: see above; the loop ends; failed
constexpr unsigned long long CM_ABORT = ~0ull;

template <int C>
__device__ __forceinline__ void cluster_max_init(ClusterMax<C> *m) {
    if (threadIdx.x == 0) {
#pragma unroll
        for (int p = 0; p < 2; p++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cl_smem(&m->bar[p])));
        asm volatile("fence.mbarrier_init.release.cluster;");
#pragma unroll
        for (int p = 0; p < 2; p++)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(cl_smem(&m->bar[p])),
                         "r"((uint32_t)(8 * C)));
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Called by the first C lanes of one warp: the CTA's key of round n to slot `rank` of CTA
// `lane`.  A slot is written again two rounds later, by a CTA that has this CTA's key of the
// round between, which is sent after every warp here has read the slot.
template <int C>
__device__ __forceinline__ void cluster_max_send(ClusterMax<C> *m, int n, int rank, int lane,
                                                 unsigned long long key) {
    uint32_t dst, bar;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(cl_smem(&m->slot[n & 1][rank])), "r"(lane));
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(cl_smem(&m->bar[n & 1])), "r"(lane));
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
                 "l"(key), "r"(bar)
                 : "memory");
}

// The warp's wait for round n's keys of all CTAs.
template <int C>
__device__ __forceinline__ bool cluster_max_arrived(ClusterMax<C> *m, int n, int polls) {
    const uint32_t bar = cl_smem(&m->bar[n & 1]);
    const uint32_t parity = (uint32_t)(n >> 1) & 1u;
    uint32_t done = 0;
    for (int spin = 0; spin < polls && !done; spin++)
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;"
            " selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
    return __all_sync(0xffffffffu, done);
}
template <int C>
__device__ __forceinline__ unsigned long long cluster_max_keys(ClusterMax<C> *m, int n, bool ok) {
    const int lane = threadIdx.x & 31;
    return warp_key_max(ok && lane < C ? *(volatile unsigned long long *)&m->slot[n & 1][lane] : 0ull);
}
// Called by every thread: round n's keys of all CTAs, reduced; ok is cleared when they were not
// there after `limit` polls.
template <int C>
__device__ __forceinline__ unsigned long long cluster_max_wait(ClusterMax<C> *m, int n, bool &ok, int limit) {
    ok = cluster_max_arrived(m, n, limit);
    return cluster_max_keys(m, n, ok);
}
__device__ __forceinline__ bool cluster_max_aborts(unsigned long long key) { return (long long)key < 0; }

// At the top of round n, when some warp's wait ran out or found the end: whether the CTA leaves.
// If not, CM_ABORT is its key of the round (one of skey's, which the first warp reduces).
// stops(key, n): whether round n's maximum is the last (CM_ABORT is).
template <int C, class F>
__device__ __forceinline__ bool cluster_max_ends(ClusterMax<C> *m, int n, unsigned &state, unsigned long long *skey,
                                                 F stops) {
    if (__syncthreads_or(state & (CM_LATE | CM_GAVE_UP))) state |= CM_GAVE_UP;
    if ((state & CM_LATE) &&
        (!cluster_max_arrived(m, n - 1, CM_SPIN) || stops(cluster_max_keys(m, n - 1, true), n - 1)))
        state |= CM_LAST;
    state &= ~CM_LATE;
    if (__syncthreads_or(state & CM_LAST)) return true;
    if (threadIdx.x == 0) skey[0] = CM_ABORT;
    __syncthreads();
    return false;
}

// One thread, after its CTA has passed round n's wait: the barrier's next phase expects C keys.
template <int C>
__device__ __forceinline__ void cluster_max_rearm(ClusterMax<C> *m, int n) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(cl_smem(&m->bar[n & 1])),
                 "r"((uint32_t)(8 * C))
                 : "memory");
}
