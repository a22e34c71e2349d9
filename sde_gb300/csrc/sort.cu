// sort.cu -- a stable LSD radix sort of (key, value) pairs, 8-bit digits, one sweep a digit.
//
// Stability matters: the weight-density counts of GRDUWT2D/GRDRUW2D are sequential FP32
// sums in visibility order (grd/grduwt2d.f:114), so the per-cell sums are reproduced
// bit-exactly by sorting (cell, weight) pairs stably and summing each cell's run in order.
//
// k_rs_hist counts every digit of every pass in one read of the keys.  A pass is then one
// kernel: a block ranks a tile of items in shared memory, publishes its count of each digit,
// sums the counts of the tiles before it by look-back (lookback.cuh) and writes each digit's
// run of the tile to consecutive addresses.  Separate count, scan and scatter kernels read
// the keys twice a pass and took five launches: 64.7 million pairs, three passes 1.75 ms, here
// 1.27 ms; 84 240 pairs 0.11 ms, here 0.04 ms.
#include <algorithm>

#include "common.cuh"
#include "lookback.cuh"

namespace {

constexpr int RS_HT = 256;       // threads of the counting kernel
constexpr int RS_MAXPASS = 4;

// What a sort needs zeroed, followed by the passes' look-back words.
struct SortCtl {
    uint32_t hist[RS_MAXPASS][256];   // digit counts, then the digits' first positions
    uint32_t tile[RS_MAXPASS];        // next tile of each pass
    uint32_t done, pad[11];
};

__global__ void __launch_bounds__(RS_HT) k_rs_hist(const uint32_t *__restrict__ keys, int64_t n, int passes,
                                                    SortCtl *ctl) {
    // one count table per warp: items of one digit arrive together in sorted stretches
    __shared__ uint32_t h[RS_MAXPASS][RS_HT / 32][256];
    __shared__ uint32_t wsum[8];
    __shared__ bool last;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int p = 0; p < passes; p++)
        for (int w = 0; w < RS_HT / 32; w++) h[p][w][t] = 0;
    __syncthreads();
    constexpr int R = 8;
    for (int64_t base = (int64_t)blockIdx.x * RS_HT * R; base < n; base += (int64_t)gridDim.x * RS_HT * R) {
        uint32_t k[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int64_t i = base + r * RS_HT + t;
            k[r] = i < n ? keys[i] : 0u;
        }
#pragma unroll
        for (int r = 0; r < R; r++)
            if (base + r * RS_HT + t < n)
                for (int p = 0; p < passes; p++) atomicAdd(&h[p][warp][(k[r] >> (8 * p)) & 255u], 1u);
    }
    __syncthreads();
    for (int p = 0; p < passes; p++) {
        uint32_t c = 0;
        for (int w = 0; w < RS_HT / 32; w++) c += h[p][w][t];
        if (c) atomicAdd(&ctl->hist[p][t], c);
    }
    // the last block turns the counts into first positions
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicAdd(&ctl->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int p = 0; p < passes; p++) {
        const uint32_t c = __ldcg(&ctl->hist[p][t]);
        uint32_t x = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        uint32_t pre = 0;
        for (int w = 0; w < warp; w++) pre += wsum[w];
        ctl->hist[p][t] = pre + x - c;
        __syncthreads();
    }
}

// One pass: T threads rank R items each (warp w takes 32 R consecutive items, round by round;
// item order is (warp, round, lane)).  vin == NULL: the values are the items' indices.  The
// lanes of a round with the same digit find each other through a word per digit in shared
// memory, whose bits they set by atomics (64.7 million pairs a pass: match.any 670 us, eight
// ballots 660 us, this 390 us, at 6144 items a tile of 256 threads).  Bound by the latency of
// ranking and of the loads, so by the warps resident: three passes of 64.7 million pairs take
// 1.52 ms with tiles of 256 x 24, 1.39 of 384 x 12, 1.37 of 320 x 16 and of 256 x 16 (four an
// SM), 1.58 of 512 x 12 (two an SM), 1.27 of 384 x 16; one buffer for keys and values in turn,
// for a fourth CTA, spills (1.54).
template <int T, int R>
struct SweepSmem {
    uint32_t wcnt[T / 32][256];  // per-warp digit counts, then the warp's offsets
    uint32_t peers[T / 32][256]; // lanes of the round that hold the digit
    uint32_t dstart[256];        // the digit's first position in the tile
    uint32_t gbase[256];         // the digit's first position in the output
    uint32_t wtot[8];
    uint32_t tile;
    uint32_t kbuf[T * R], vbuf[T * R];  // the tile's items in (digit, item) order
};

template <int T, int R>
__global__ void __launch_bounds__(T, 3) k_rs_sweep(const uint32_t *__restrict__ kin, const uint32_t *__restrict__ vin,
                                                uint32_t *__restrict__ kout, uint32_t *__restrict__ vout, int64_t n,
                                                int pass, SortCtl *ctl, unsigned long long *state,
                                                unsigned long long *fail, int limit) {
    extern __shared__ __align__(16) unsigned char rs_smem[];
    SweepSmem<T, R> &S = *reinterpret_cast<SweepSmem<T, R> *>(rs_smem);
    constexpr int TILE = T * R;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, shift = 8 * pass;
    const uint32_t lt = (1u << lane) - 1u;
    // tiles are taken in order, so the tiles before this one are running or done
    if (t == 0) S.tile = atomicAdd(&ctl->tile[pass], 1u);
    for (int i = t; i < T / 32 * 256; i += T) (&S.wcnt[0][0])[i] = (&S.peers[0][0])[i] = 0;
    __syncthreads();
    const int64_t tile = S.tile, base = tile * TILE, wbase = base + (int64_t)warp * 32 * R;
    uint32_t key[R], pos[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int64_t i = wbase + r * 32 + lane;
        key[r] = i < n ? kin[i] : 0u;
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
        const bool valid = wbase + r * 32 + lane < n;
        const uint32_t digit = (key[r] >> shift) & 255u;
        if (valid) atomicOr(&S.peers[warp][digit], 1u << lane);
        __syncwarp();
        const uint32_t peers = S.peers[warp][digit], before = S.wcnt[warp][digit];
        pos[r] = before + __popc(peers & lt);
        __syncwarp();
        if (valid && (peers & lt) == 0) {
            S.wcnt[warp][digit] = before + __popc(peers);
            S.peers[warp][digit] = 0;
        }
        __syncwarp();
    }
    __syncthreads();
    // digit t: offsets of the warps' runs within the digit, and the digit's total, published
    uint32_t total = 0, x = 0;
    if (t < 256) {
#pragma unroll
        for (int w = 0; w < T / 32; w++) {
            const uint32_t c = S.wcnt[w][t];
            S.wcnt[w][t] = total;
            total += c;
        }
        lb_publish(&state[tile * 256 + t], tile == 0 ? LB_PREFIX : LB_AGG, total);
        x = total;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) S.wtot[warp] = x;
    }
    __syncthreads();
    if (t < 256) {
        uint32_t pre = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) pre += w < warp ? S.wtot[w] : 0u;
        S.dstart[t] = pre + x - total;
    }
    __syncthreads();
    // (the values are read only now: the ranking needs their registers for more warps)
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int64_t i = wbase + r * 32 + lane;
        if (i < n) {
            const uint32_t digit = (key[r] >> shift) & 255u;
            const uint32_t p = S.dstart[digit] + S.wcnt[warp][digit] + pos[r];
            S.kbuf[p] = key[r];
            S.vbuf[p] = vin ? vin[i] : (uint32_t)i;
        }
    }
    if (t < 256) {
        unsigned long long before = 0;
        if (tile > 0) {
            before = lb_sum_before(state + t, tile, 256, fail, limit);
            lb_publish(&state[tile * 256 + t], LB_PREFIX, before + total);
        }
        S.gbase[t] = ctl->hist[pass][t] + (uint32_t)before;
    }
    __syncthreads();
    const int ntile = (int)min((int64_t)TILE, n - base);
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int p = r * T + t;
        if (p < ntile) {
            const uint32_t k = S.kbuf[p];
            const uint32_t digit = (k >> shift) & 255u;
            // (a look-back that gave up leaves a wrong position, kept inside the arrays, and places
            // that nothing is written to: the sorted arrays then hold what the scratch held)
            const uint32_t d = S.gbase[digit] + (uint32_t)p - S.dstart[digit];
            if (d < (uint64_t)n) {
                kout[d] = k;
                vout[d] = S.vbuf[p];
            }
        }
    }
}

template <int T, int R>
int sweep(sde_ctx *ctx, const uint32_t *kin, const uint32_t *vin, uint32_t *kout, uint32_t *vout, int64_t n, int pass,
          SortCtl *ctl, unsigned long long *state, unsigned long long *fail) {
    const int sm = (int)sizeof(SweepSmem<T, R>);
    SDE_CUDA_TRY(cudaFuncSetAttribute(k_rs_sweep<T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
    k_rs_sweep<T, R><<<ceil_div(n, T * R), T, sm, ctx->stream>>>(kin, vin, kout, vout, n, pass, ctl, state, fail,
                                                               lb_spin(ctx));
    SDE_CHECK_LAUNCH();
    return SDE_OK;
}

}  // namespace

// Sorts pairs by the low `bits` bits of the keys, stably.  *keys: the keys; first_vals: their
// values, NULL for the items' indices; keys_tmp, *vals and vals_tmp: scratch.  On return *keys
// and *vals are whichever of the arrays hold the result.  *fail (device, zeroed by the caller)
// is set when a bounded wait gave up: the result then holds any keys and values at all, and a
// kernel that uses them as indexes looks at *fail first.
int launch_radix_sort_u32(sde_ctx *ctx, uint32_t **keys, const uint32_t *first_vals, uint32_t **vals, int64_t n,
                          int bits, uint32_t *keys_tmp, uint32_t *vals_tmp, unsigned long long *fail) {
    if (n < 1) return SDE_OK;
    if (n >= (int64_t)0xFFFFFFFF) {
        sde_set_error("radix sort: %lld items exceeds 32-bit offsets", (long long)n);
        return SDE_EINVAL;
    }
    // Tiles of 6144 items write runs of about 24 per digit; with fewer than two of them an SM
    // the smaller tiles fill the chip (84 240 items: 41 tiles instead of 14).
    const bool small = n < (int64_t)ctx->num_sms * 2 * 6144;
    const int passes = (bits + 7) / 8, ntile = ceil_div(n, small ? 2048 : 6144);
    const size_t per_pass = sizeof(unsigned long long) * 256 * (size_t)ntile;
    SortCtl *ctl;
    const size_t bytes = sizeof(SortCtl) + per_pass * passes;
    SDE_TRY(ctx_scratch(ctx, "rs_ctl", bytes, (void **)&ctl));
    SDE_CUDA_TRY(cudaMemsetAsync(ctl, 0, bytes, ctx->stream));
    unsigned long long *state = reinterpret_cast<unsigned long long *>(ctl + 1);
    const int hb = std::min(ceil_div(n, RS_HT * 8), ctx->num_sms * 4);
    k_rs_hist<<<hb, RS_HT, 0, ctx->stream>>>(*keys, n, passes, ctl);
    SDE_CHECK_LAUNCH();
    uint32_t *sk = *keys, *sv = *vals, *dk = keys_tmp, *dv = vals_tmp;
    for (int p = 0; p < passes; p++) {
        const uint32_t *vin = p == 0 ? first_vals : sv;
        unsigned long long *st = state + per_pass / sizeof(unsigned long long) * p;
        SDE_TRY(small ? (sweep<256, 8>(ctx, sk, vin, dk, dv, n, p, ctl, st, fail))
                      : (sweep<384, 16>(ctx, sk, vin, dk, dv, n, p, ctl, st, fail)));
        std::swap(sk, dk);
        std::swap(sv, dv);
    }
    *keys = sk;
    *vals = sv;
    return SDE_OK;
}
