// lookback.cuh -- single-pass prefix sums over tiles by decoupled look-back (Merrill and
// Garland, "Single-pass parallel prefix scan with decoupled look-back", 2016): a tile
// publishes its own sum, then adds the sums published by the tiles before it back to the
// first complete prefix, and publishes its own.  A tile's word holds sum and state, so one
// 64-bit store publishes both and no fence is needed.  Words start at 0 (cleared before the
// launch); tiles take their numbers from a counter, so every tile waited for has started.
#pragma once
#include "common.cuh"

constexpr unsigned long long LB_AGG = 1ull << 62, LB_PREFIX = 2ull << 62, LB_FLAGS = 3ull << 62;
constexpr int LB_SPIN = 1 << 22;  // polls of one word before giving up (about a second)
inline int lb_spin(const sde_ctx *ctx) { return ctx->wait_limit < 0 ? LB_SPIN : ctx->wait_limit; }

__device__ __forceinline__ void lb_publish(unsigned long long *w, unsigned long long flag, unsigned long long v) {
    *reinterpret_cast<volatile unsigned long long *>(w) = flag | v;
}

// Sum of the tiles before `tile` (one thread; the words of consecutive tiles are `stride`
// apart).  Eight words are read at a time, in flight together (four: 2 % slower in a sort pass of
// 64.7 million pairs, 12 % at 1.3 million).  *fail is set and 0 returned when a word does not
// arrive in `limit` polls; what was made from the sum is then wrong, and whatever reads it has to
// look at *fail first.
__device__ __forceinline__ unsigned long long lb_sum_before(const unsigned long long *words, int64_t tile,
                                                            int64_t stride, unsigned long long *fail, int limit) {
    constexpr int A = 8;
    unsigned long long sum = 0;
    int64_t p = tile - 1;
    for (int spin = 0; spin < limit; spin++) {
        unsigned long long w[A];
#pragma unroll
        for (int a = 0; a < A; a++)
            w[a] = p - a >= 0 ? *reinterpret_cast<const volatile unsigned long long *>(words + (p - a) * stride) : LB_PREFIX;
#pragma unroll
        for (int a = 0; a < A; a++) {
            if (!(w[a] & LB_FLAGS)) break;  // not there yet: read again from here
            sum += w[a] & ~LB_FLAGS;
            if (w[a] & LB_PREFIX) return sum;
            p--;
            spin = 0;
        }
    }
    atomicExch(fail, 1ull);
    return 0;
}

// Exclusive sums of in(i) over i < n in tiles of T * R items, handed to out(i, value, sum
// before) in the calling block's own order; the total goes to *total (written by the last
// tile).  Values are below 2^62 in sum (two counts of 31 bits, say).
template <int T, int R, class In, class Out>
__device__ __forceinline__ void lb_scan_tile(int64_t n, unsigned long long *words, uint32_t *next,
                                             unsigned long long *total, unsigned long long *fail, int limit, In in,
                                             Out out) {
    __shared__ unsigned long long sv[T * R * 17 / 16];  // padded: a thread reads its R consecutive items
    __shared__ unsigned long long wsum[T / 32], sbefore;
    __shared__ uint32_t stile;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    auto at = [](int i) { return i + (i >> 4); };
    if (t == 0) stile = atomicAdd(next, 1u);
    __syncthreads();
    const int64_t tile = stile, base = tile * (T * R);
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int64_t i = base + r * T + t;
        sv[at(r * T + t)] = i < n ? in(i) : 0ull;
    }
    __syncthreads();
    unsigned long long v[R], sum = 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
        v[r] = sv[at(t * R + r)];
        sum += v[r];
    }
    unsigned long long x = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    unsigned long long pre = 0, all = 0;
#pragma unroll
    for (int w = 0; w < T / 32; w++) {
        pre += w < warp ? wsum[w] : 0ull;
        all += wsum[w];
    }
    if (t == 0) {
        unsigned long long b = 0;
        if (tile > 0) {
            lb_publish(&words[tile], LB_AGG, all);
            b = lb_sum_before(words, tile, 1, fail, limit);
        }
        lb_publish(&words[tile], LB_PREFIX, b + all);
        sbefore = b;
        if (base + T * R >= n) *total = b + all;
    }
    __syncthreads();
    unsigned long long run = sbefore + pre + x - sum;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int64_t i = base + t * R + r;
        if (i < n) out(i, v[r], run);
        run += v[r];
    }
}
