// weights.cu -- uniform (GRDUWT2D) and robust (GRDRUW2D) weighting, bit-exact.
//
// Pass 1 of the reference (grd/grduwt2d.f:90-115, grd/grdruw2d.f:132-159) adds WT into the
// density grid GWT(UCEN,VCEN) sequentially in FP32, in visibility order.  Here each
// visibility's cell key is computed with the reference's exact FP32/FP64 operations (no
// FMA contraction), the (key, WT) pairs are sorted stably, and one thread sums each
// cell's run in order: the same additions in the same order, so GWT is bit-identical.
// Pass 2 (grd/grduwt2d.f:118-160, grd/grdruw2d.f:196-242) is an element-wise gather.
#include <math.h>
#include <string.h>

#include "common.cuh"

namespace {

struct WParams {
    float uscale, uoffset, vscale, voffset;
    int uorigin, vorigin, nu, nv;
    double s[9];
};

// FP32 uv -> cell of the weighting routines (grd/grduwt2d.f:92-111, grd/grdruw2d.f:198-217).
// ROT: the rotation is applied, and W read, at all.
template <bool ROT>
__device__ __forceinline__ bool wcell(const WParams &p, float u, float v, const float *w, int64_t i, int &uc,
                                      int &vc, float &ul, float &vl) {
    float ucell, vcell;
    // With SHIFT(2,1) = SHIFT(3,1) = SHIFT(1,2) = SHIFT(3,2) = 0 and the diagonal within
    // 2^-40 of 1 (CRDSHIFT without a shift: sin^2 + cos^2 can miss 1 by an ulp), the DOUBLE
    // ULOCAL = SHIFT(1,1)*U + 0*V + 0*W and VLOCAL lie within |U|*2^-39 of U and V, far
    // inside half a REAL ulp, so the REAL ULOCAL, VLOCAL are U and V themselves.
    if (ROT) {
        double du = (double)u, dv = (double)v, dw = (double)w[i];
        ul = __double2float_rn(__dadd_rn(__dadd_rn(__dmul_rn(p.s[0], du), __dmul_rn(p.s[1], dv)),
                                         __dmul_rn(p.s[2], dw)));
        vl = __double2float_rn(__dadd_rn(__dadd_rn(__dmul_rn(p.s[3], du), __dmul_rn(p.s[4], dv)),
                                         __dmul_rn(p.s[5], dw)));
    } else {
        ul = u;
        vl = v;
    }
    ucell = __fadd_rn(__fmul_rn(p.uscale, ul), p.uoffset);
    vcell = __fadd_rn(__fmul_rn(p.vscale, vl), p.voffset);
    if (ucell > 0.0f) {
        ucell = __fadd_rn(ucell, (float)p.uorigin);
        vcell = __fadd_rn(vcell, (float)p.vorigin);
    } else {
        ucell = __fadd_rn(-ucell, (float)p.uorigin);
        vcell = __fadd_rn(-vcell, (float)p.vorigin);
    }
    uc = nint_f(ucell);
    vc = nint_f(vcell);
    return !(uc < 1 || uc > p.nu || vc < 1 || vc > p.nv);
}

// W_PER visibilities a thread, their loads in flight together (64.7 million: one a thread 337
// us, here 148)
constexpr int W_T = 256, W_PER = 4;
template <bool ROT>
__global__ void __launch_bounds__(W_T) k_wkey(WParams p, const float *__restrict__ wt, const float *__restrict__ u,
                                              const float *__restrict__ v, const float *__restrict__ w, int64_t n,
                                              uint32_t *keys, unsigned long long *counts) {
    const int64_t i0 = (int64_t)blockIdx.x * (W_T * W_PER) + threadIdx.x;
    uint32_t valid = 0, drop = 0;
    float wi[W_PER], ui[W_PER], vi[W_PER];
#pragma unroll
    for (int j = 0; j < W_PER; j++) {
        const int64_t i = i0 + j * W_T;
        wi[j] = i < n ? wt[i] : 0.0f;
        ui[j] = i < n ? u[i] : 0.0f;
        vi[j] = i < n ? v[i] : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < W_PER; j++) {
        const int64_t i = i0 + j * W_T;
        if (i >= n) break;
        uint32_t key = KEY_INVALID;
        if (wi[j] > 0.0f) {
            int uc, vc;
            float ul, vl;
            if (wcell<ROT>(p, ui[j], vi[j], w, i, uc, vc, ul, vl)) {
                key = (uint32_t)(vc - 1) * (uint32_t)p.nu + (uint32_t)(uc - 1);
                valid++;
            } else {
                drop++;
            }
        }
        keys[i] = key;
    }
    // block-aggregated counters: [0] on-grid, [1] dropped (one atomic per block and counter)
    __shared__ uint32_t sum[2];
    if (threadIdx.x < 2) sum[threadIdx.x] = 0;
    __syncthreads();
    valid = __reduce_add_sync(0xffffffffu, valid);
    drop = __reduce_add_sync(0xffffffffu, drop);
    if ((threadIdx.x & 31) == 0) {
        if (valid) atomicAdd(&sum[0], valid);
        if (drop) atomicAdd(&sum[1], drop);
    }
    __syncthreads();
    if (threadIdx.x < 2 && sum[threadIdx.x]) atomicAdd(&counts[threadIdx.x], (unsigned long long)sum[threadIdx.x]);
}

// GWT(cell) = ((0 + w1) + w2) + ... in visibility order: FP32 additions in the reference's
// order, so every cell's sum is one sequential chain.  A block stages SEG_TILE sorted entries
// (plus the one before and SEG_SHORT after) in shared memory and lists its run heads, so that
// every thread has a run; a run of at most SEG_SHORT entries is summed from there, SEG_U
// values in flight.  A longer run (dense cells hold up to ~2e5 visibilities) is put on a list
// for k_segsum_long, which costs microseconds a run to find and fetch: with SEG_SHORT = 32 the
// two kernels took 0.56 + 0.53 ms on 64.7 million visibilities, now 0.30 + 0.09.
constexpr int SEG_SHORT = 512;
constexpr int SEG_TILE = 2048;
constexpr int SEG_T = 256;
constexpr int SEG_U = 8;
__global__ void __launch_bounds__(SEG_T) k_segsum(const uint32_t *__restrict__ keys,
                                                  const uint32_t *__restrict__ vals,
                                                  unsigned long long *counts, float *gwt, uint32_t *longq) {
    __shared__ uint32_t sk[SEG_TILE + SEG_SHORT + SEG_U + 1];  // keys[base - 1 ...]
    __shared__ float sv[SEG_TILE + SEG_SHORT + SEG_U];          // vals[base ...]
    __shared__ uint16_t head[SEG_TILE];
    __shared__ int nhead;
    if (counts[7]) return;  // the sort gave up: its keys index nothing
    const int64_t nvalid = (int64_t)counts[0];
    const int64_t base = (int64_t)blockIdx.x * SEG_TILE;
    if (base >= nvalid) return;
    if (threadIdx.x == 0) nhead = 0;
    for (int i = threadIdx.x; i < SEG_TILE + SEG_SHORT + SEG_U + 1; i += SEG_T) {
        const int64_t q = base - 1 + i;
        sk[i] = q >= 0 && q < nvalid ? keys[q] : KEY_INVALID;  // valid keys are below KEY_INVALID
    }
    for (int i = threadIdx.x; i < SEG_TILE + SEG_SHORT + SEG_U; i += SEG_T) {
        const int64_t q = base + i;
        sv[i] = q < nvalid ? __uint_as_float(vals[q]) : 0.0f;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < SEG_TILE; j += SEG_T)
        if (sk[j + 1] != KEY_INVALID && sk[j] != sk[j + 1]) head[atomicAdd(&nhead, 1)] = (uint16_t)j;
    __syncthreads();
    for (int e = threadIdx.x; e < nhead; e += SEG_T) {
        const int j = head[e];
        const uint32_t k = sk[j + 1];
        if (sk[j + 1 + SEG_SHORT] == k) {
            const unsigned long long slot = atomicAdd(&counts[2], 1ull);
            longq[slot] = (uint32_t)(base + j);
            continue;
        }
        float s = 0.0f;
        bool more = true;
        for (int q = j; more; q += SEG_U) {
            uint32_t kq[SEG_U];
            float x[SEG_U];
#pragma unroll
            for (int a = 0; a < SEG_U; a++) {
                kq[a] = sk[q + 1 + a];
                x[a] = sv[q + a];
            }
#pragma unroll
            for (int a = 0; a < SEG_U; a++) {
                more = more && kq[a] == k;
                if (more) s = __fadd_rn(s, x[a]);
            }
        }
        gwt[k] = s;
    }
}

// The sequential FP32 sum of a long run, SEG_BLK entries at a time in parallel.  While the sum s
// stays in one binade, s = m u with u its spacing and m in [2^23, 2^24), and an addition of
// w > 0 rounds to s + i u: i is the integer nearest w / u, except that a fraction of exactly
// one half goes to the even m + i, so there i depends on m's parity alone.  An entry is
// therefore a pair of increments, one for each parity of m, and two in a row compose to
// another such pair; a warp composes its lanes' entries in order.  If m and the block's whole
// increment stay below 2^24 no addition has left the binade and s = (m + i) u is the
// sequence's own result; otherwise (about twice a doubling of s, and for weights too large or
// small for this) lane 0 adds the block one by one.  The longest run bounds the kernel: 184 000
// entries 0.36 ms by one addition latency each, below 0.1 here.
struct ParInc {
    uint32_t i0, i1;  // increments of m for an even and an odd m
};
__device__ __forceinline__ ParInc par_then(ParInc a, ParInc b) {
    return ParInc{a.i0 + ((a.i0 & 1u) ? b.i1 : b.i0), a.i1 + ((a.i1 & 1u) ? b.i0 : b.i1)};
}

constexpr int SEG_BLK = 512;
constexpr int SEG_RING = 4;   // blocks in shared memory: three of them on their way
constexpr int SEG_WARPS = 4;  // warps per block of k_segsum_long
__global__ void __launch_bounds__(SEG_WARPS * 32) k_segsum_long(
    const uint32_t *__restrict__ keys, const uint32_t *__restrict__ vals,
    unsigned long long *counts, const uint32_t *__restrict__ longq, float *gwt) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int PER = SEG_BLK / 32;
    __shared__ __align__(16) float buf[SEG_WARPS][SEG_RING][SEG_BLK];
    if (counts[7]) return;  // the sort gave up
    const int64_t nvalid = (int64_t)counts[0];
    const int64_t nlong = (int64_t)counts[2];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    // runs are taken from a counter, so the warp that holds the longest run takes no other
    for (;;) {
        int64_t r = 0;
        if (lane == 0) r = (int64_t)atomicAdd(&counts[3], 1ull);
        r = __shfl_sync(FULL, r, 0);
        if (r >= nlong) break;
        const int64_t p = longq[r];
        const uint32_t k = keys[p];
        int64_t end = 0;
        if (lane == 0) {
            // keys[p + SEG_SHORT] == k (why the run is here); find the first index past the run
            int64_t lo = p + SEG_SHORT, step = 64;
            while (lo + step < nvalid && keys[lo + step] == k) {
                lo += step;
                step *= 2;
            }
            int64_t hi = lo + step < nvalid ? lo + step : nvalid;  // keys[hi] != k or hi = nvalid
            while (hi - lo > 1) {
                const int64_t mid = lo + (hi - lo) / 2;
                if (keys[mid] == k) lo = mid; else hi = mid;
            }
            end = hi;
        }
        end = __shfl_sync(FULL, end, 0);
        const int64_t len = end - p;
        const int nblk = (int)((len + SEG_BLK - 1) / SEG_BLK);
        // block b to its place in the ring, zeros past the run
        auto fetch = [&](int b) {
            if (b < nblk) {
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&buf[wib][b % SEG_RING][lane]);
#pragma unroll
                for (int j = 0; j < PER; j++) {
                    const int64_t q = p + (int64_t)b * SEG_BLK + j * 32 + lane;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + j * 128),
                                 "l"(vals + (q < end ? q : p)), "r"(q < end ? 4 : 0)
                                 : "memory");
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        for (int b = 0; b < SEG_RING - 1; b++) fetch(b);
        float s = 0.0f;
        for (int b = 0; b < nblk; b++) {
            float *cur = buf[wib][b % SEG_RING];
            __syncwarp();  // every lane has read the block whose place is taken now
            fetch(b + SEG_RING - 1);
            asm volatile("cp.async.wait_group %0;" ::"n"(SEG_RING - 1) : "memory");
            __syncwarp();
            // lane l composes entries PER l .. PER l + PER - 1 (zeros past the run add nothing)
            const uint32_t e = (__float_as_uint(s) >> 23) & 255u;
            bool done = false;
            if (e >= 64u && e <= 190u) {  // u and 1/u are normal, as is every w / u that counts
                const float iu = __uint_as_float((277u - e) << 23);  // 1 / u = 2^(150 - e)
                const uint32_t m = (__float_as_uint(s) & 0x7FFFFFu) | 0x800000u;
                float x[PER];
#pragma unroll
                for (int j = 0; j < PER; j += 4)
                    *reinterpret_cast<float4 *>(&x[j]) = reinterpret_cast<const float4 *>(cur)[(PER * lane + j) / 4];
                ParInc c{0u, 0u};
                bool fits = true;
#pragma unroll
                for (int j = 0; j < PER; j++) {
                    const float y = __fmul_rn(x[j], iu);  // exact: a power of two
                    fits = fits && y < 32768.f;           // (512 of them stay below 2^24)
                    const float f = floorf(y), fr = __fsub_rn(y, f);
                    const uint32_t i = (uint32_t)f + (fr > 0.5f ? 1u : 0u);
                    const uint32_t tie = fr == 0.5f ? 1u : 0u;
                    c = par_then(c, ParInc{i + (tie & i), i + (tie & ~i)});
                }
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    ParInc o;
                    o.i0 = __shfl_down_sync(FULL, c.i0, d);
                    o.i1 = __shfl_down_sync(FULL, c.i1, d);
                    c = par_then(c, o);  // (lanes past 31 - d compose a wrong tail; lane 0 never uses it)
                }
                const uint32_t sum = m + ((m & 1u) ? c.i1 : c.i0);
                done = __all_sync(FULL, fits) && __shfl_sync(FULL, sum, 0) < 0x1000000u;
                if (done && lane == 0) s = __uint_as_float((e << 23) | (sum & 0x7FFFFFu));
            }
            if (!done && lane == 0) {
                const int cnt = (int)(len - (int64_t)b * SEG_BLK < SEG_BLK ? len - (int64_t)b * SEG_BLK : SEG_BLK);
                const float4 *c4 = reinterpret_cast<const float4 *>(cur);
                if (cnt == SEG_BLK) {
#pragma unroll 8
                    for (int j = 0; j < SEG_BLK / 4; j++) {
                        const float4 x = c4[j];
                        s = __fadd_rn(s, x.x);
                        s = __fadd_rn(s, x.y);
                        s = __fadd_rn(s, x.z);
                        s = __fadd_rn(s, x.w);
                    }
                } else {
                    for (int j = 0; j < cnt; j++) s = __fadd_rn(s, cur[j]);
                }
            }
            s = __shfl_sync(FULL, s, 0);
        }
        if (lane == 0) gwt[k] = s;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
    }
}

// Deterministic FP64 sums (block partials in a fixed order).
constexpr int RED_THREADS = 256;
__device__ __forceinline__ double block_sum_d(double x) {
    __shared__ double sh[RED_THREADS / 32];
    for (int d = 16; d > 0; d >>= 1) x = __dadd_rn(x, __shfl_down_sync(0xffffffffu, x, d));
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh[warp] = x;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < RED_THREADS / 32; k++) r = __dadd_rn(r, sh[k]);
    return r;
}

// hi + mid + lo += x without a rounding error that a DOUBLE sum of a few terms would see (two
// TwoSums; FP64 additions and conversions run at 1/64 of the FP32 rate)
__device__ __forceinline__ void sum3(float &hi, float &mid, float &lo, float x) {
    const float s = __fadd_rn(hi, x), bb = __fsub_rn(s, hi);
    const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(x, bb));
    const float m = __fadd_rn(mid, e), mb = __fsub_rn(m, mid);
    lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(mid, __fsub_rn(m, mb)), __fsub_rn(e, mb)));
    hi = s;
    mid = m;
}

// partial[b] = sum of weights of sorted valid entries in block b's range
__global__ void __launch_bounds__(RED_THREADS) k_sumwt_part(const uint32_t *vals,
                                                             const unsigned long long *counts,
                                                             int per_thread, double *partial) {
    int64_t nvalid = (int64_t)counts[0];
    int64_t base = ((int64_t)blockIdx.x * RED_THREADS + threadIdx.x) * per_thread;
    float hi = 0.0f, mid = 0.0f, lo = 0.0f;
    if (base + per_thread <= nvalid) {  // 16-byte reads: the bases are multiples of per_thread = 4 k
        for (int k = 0; k < per_thread; k += 4) {
            const uint4 x = *reinterpret_cast<const uint4 *>(vals + base + k);
            sum3(hi, mid, lo, __uint_as_float(x.x));
            sum3(hi, mid, lo, __uint_as_float(x.y));
            sum3(hi, mid, lo, __uint_as_float(x.z));
            sum3(hi, mid, lo, __uint_as_float(x.w));
        }
    } else {
        for (int k = 0; k < per_thread; k++)
            if (base + k < nvalid) sum3(hi, mid, lo, __uint_as_float(vals[base + k]));
    }
    double s;
    if (isfinite(hi)) {
        s = __dadd_rn((double)hi, __dadd_rn((double)mid, (double)lo));
    } else {  // weights whose sum leaves the REALs: SUMWT is DOUBLE (grd/grdruw2d.f:132-159)
        s = 0.0;
        for (int k = 0; k < per_thread; k++)
            if (base + k < nvalid) s = __dadd_rn(s, (double)__uint_as_float(vals[base + k]));
    }
    double r = block_sum_d(s);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
}

// partial[b] = sum over cells in block b's range of (double)(g*g), g > 0 (grd/grdruw2d.f:168-175)
__global__ void __launch_bounds__(RED_THREADS) k_sumlocwt_part(const float *gwt, int64_t ncell,
                                                                int per_thread, double *partial) {
    int64_t base = ((int64_t)blockIdx.x * RED_THREADS + threadIdx.x) * per_thread;
    double s = 0.0;
    for (int k = 0; k < per_thread; k++) {
        int64_t q = base + k;
        if (q < ncell) {
            float g = gwt[q];
            if (g > 0.0f) s = __dadd_rn(s, (double)__fmul_rn(g, g));
        }
    }
    double r = block_sum_d(s);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
}

// The partials in a fixed order: thread t adds partials t, t + RED_THREADS, ..., then a
// fixed tree over the threads (deterministic for a given partial count).
__global__ void __launch_bounds__(RED_THREADS) k_sum_partials(const double *partial, int n, double *out) {
    __shared__ double sh[RED_THREADS];
    double s = 0.0;
    for (int k = threadIdx.x; k < n; k += RED_THREADS) s = __dadd_rn(s, partial[k]);
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int h = RED_THREADS / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) sh[threadIdx.x] = __dadd_rn(sh[threadIdx.x], sh[threadIdx.x + h]);
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sh[0];
}

struct AzParams {
    int doaz;
    float r1, rbscale, rpa, pi;
    double ratio;  // SUMLOCWT / SUMWT
};

// Pass 2.  uniform: grd/grduwt2d.f:146-158; robust: grd/grdruw2d.f:225-240.
// NEWWT of one on-grid visibility of weight wi in a cell of density g.
__device__ __forceinline__ float new_weight(const WParams &p, int robust, float f2, float d2, const AzParams &az,
                                            float wi, float g, int uc, int vc, float ul, float vl) {
    float out;
    if (!robust) {
        if (g > 0.0f) {
            if (uc == p.uorigin && vc != p.vorigin)
                out = __fdiv_rn(__fmul_rn(0.5f, wi), g);
            else
                out = __fdiv_rn(wi, g);
        } else {
            out = -1.0f;
        }
    } else {
        float ff2 = f2;
        if (az.doaz) {  // CUDA atan2f/fmodf/powf: within the CUDA math library's ulp bounds
            float t = atan2f(vl, ul);
            t = __fsub_rn(fmodf(__fadd_rn(__fsub_rn(t, az.rpa), __fmul_rn(2.5f, az.pi)), az.pi),
                          __fdiv_rn(az.pi, 2.0f));
            float r = __fsub_rn(az.r1, __fmul_rn(fabsf(t), az.rbscale));
            float tt = __fmul_rn(5.0f, powf(10.0f, -r));
            ff2 = __double2float_rn(__ddiv_rn((double)__fmul_rn(tt, tt), az.ratio));
        }
        if (g > 0.0f) {
            float den = __fadd_rn(__fmul_rn(g, ff2), d2);
            if (uc == p.uorigin && vc != p.vorigin)
                out = __fdiv_rn(__fmul_rn(0.5f, wi), den);
            else
                out = __fdiv_rn(wi, den);
        } else {
            out = -1.0f;
        }
    }
    return out;
}

// W_PER visibilities a thread: their loads, then their density reads, in flight together (64.7
// million: one a thread 428 us, here 314).  When the sort gave up (*fail) there are no densities:
// NEWWT is left alone and the context's time-out word set, for callers that read no counts.
template <bool ROT>
__global__ void __launch_bounds__(W_T) k_newwt(WParams p, int robust, float f2, float d2, AzParams az,
                        const float *wt, const float *__restrict__ u, const float *__restrict__ v,
                        const float *__restrict__ w, const float *__restrict__ gwt, int64_t n,
                        float *newwt, const unsigned long long *__restrict__ fail, int *status) {
    const int64_t i0 = (int64_t)blockIdx.x * (W_T * W_PER) + threadIdx.x;
    const bool failed = *fail != 0;
    float wi[W_PER], ui[W_PER], vi[W_PER], g[W_PER], ul[W_PER], vl[W_PER];
    int uc[W_PER], vc[W_PER];
    bool on[W_PER];
#pragma unroll
    for (int j = 0; j < W_PER; j++) {
        const int64_t i = i0 + j * W_T;
        wi[j] = i < n ? wt[i] : 0.0f;
        ui[j] = i < n ? u[i] : 0.0f;
        vi[j] = i < n ? v[i] : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < W_PER; j++) {
        on[j] = !(wi[j] <= 0.0f) && wcell<ROT>(p, ui[j], vi[j], w, i0 + j * W_T, uc[j], vc[j], ul[j], vl[j]);
        g[j] = on[j] ? gwt[(int64_t)(vc[j] - 1) * p.nu + (uc[j] - 1)] : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < W_PER; j++)
        if (!(wi[j] <= 0.0f) && i0 + j * W_T < n && !failed)
            newwt[i0 + j * W_T] = on[j] ? new_weight(p, robust, f2, d2, az, wi[j], g[j], uc[j], vc[j], ul[j], vl[j])
                                        : -1.0f;
    if (failed && i0 == 0) atomicExch(&status[STATUS_TIMEOUT], 1);
}

int key_bits(int64_t maxkey) {
    int b = 1;
    while (b < 32 && ((int64_t)1 << b) <= maxkey) b++;
    return b;
}

}  // namespace

// sde_weights up to its last wait: the new weights may still be on their way on the stream.
int weights_queue(sde_ctx *ctx, int rmode, const float robust[3], float ds, const float *wt, const float *u,
                  const float *v, const float *w, int64_t nvis, float uscale, float uoffset, float vscale,
                  float voffset, int uorigin, int vorigin, int nu, int nv, const double shift[9], float *newwt,
                  float *gwt, sde_wstats *stats) {
    if (!ctx || nvis < 0 || nu <= 0 || nv <= 0 || !shift) {
        sde_set_error("sde_weights: bad arguments");
        return SDE_EINVAL;
    }
    if (rmode < 0 || rmode > 4) {
        sde_set_error("sde_weights: unrecognized RMODE %d", rmode);
        return SDE_EBADMODE;
    }
    if ((int64_t)nu * nv >= (int64_t)KEY_INVALID) {
        sde_set_error("sde_weights: grid too large");
        return SDE_EINVAL;
    }
    SDE_CUDA_TRY(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    WParams p;
    p.uscale = uscale; p.uoffset = uoffset; p.vscale = vscale; p.voffset = voffset;
    p.uorigin = uorigin; p.vorigin = vorigin; p.nu = nu; p.nv = nv;
    memcpy(p.s, shift, sizeof p.s);
    const bool doshift = (shift[0] != 1.0) || (shift[4] != 1.0) || (shift[8] != 1.0);
    const bool near_identity = shift[1] == 0.0 && shift[2] == 0.0 && shift[3] == 0.0 && shift[5] == 0.0 &&
                               fabs(shift[0] - 1.0) <= 0x1p-40 && fabs(shift[4] - 1.0) <= 0x1p-40;
    const bool rot = doshift && !near_identity;  // see wcell
    const int64_t ncell = (int64_t)nu * nv;
    if (!gwt) SDE_TRY(ctx_scratch(ctx, "w_gwt", sizeof(float) * (size_t)ncell, (void **)&gwt));
    SDE_CUDA_TRY(cudaMemsetAsync(gwt, 0, sizeof(float) * (size_t)ncell, st));
    uint32_t *keys, *vals, *ktmp, *vtmp;
    unsigned long long *counts;
    size_t nb4 = sizeof(uint32_t) * (size_t)(nvis > 0 ? nvis : 1);
    SDE_TRY(ctx_scratch(ctx, "w_keys", nb4, (void **)&keys));
    SDE_TRY(ctx_scratch(ctx, "w_vals", nb4, (void **)&vals));
    SDE_TRY(ctx_scratch(ctx, "w_ktmp", nb4, (void **)&ktmp));
    SDE_TRY(ctx_scratch(ctx, "w_vtmp", nb4, (void **)&vtmp));
    SDE_TRY(ctx_scratch(ctx, "w_counts", 64 + 2 * sizeof(double), (void **)&counts));
    double *sums = reinterpret_cast<double *>(counts + 8);  // [0] sumwt [1] sumlocwt
    SDE_CUDA_TRY(cudaMemsetAsync(counts, 0, 64 + 2 * sizeof(double), st));
    if (nvis > 0) {
        (rot ? k_wkey<true> : k_wkey<false>)<<<ceil_div(nvis, W_T * W_PER), W_T, 0, st>>>(p, wt, u, v, w, nvis, keys, counts);
        SDE_CHECK_LAUNCH();
        SDE_TRY(launch_radix_sort_u32(ctx, &keys, reinterpret_cast<const uint32_t *>(wt), &vals, nvis, key_bits(ncell), ktmp, vtmp,
                                      &counts[7]));
        uint32_t *longq;
        SDE_TRY(ctx_scratch(ctx, "w_longq", sizeof(uint32_t) * (size_t)(nvis / (SEG_SHORT + 1) + 1),
                            (void **)&longq));
        k_segsum<<<ceil_div(nvis, SEG_TILE), SEG_T, 0, st>>>(keys, vals, counts, gwt, longq);
        SDE_CHECK_LAUNCH();
        k_segsum_long<<<ctx->num_sms * 4, SEG_WARPS * 32, 0, st>>>(keys, vals, counts, longq, gwt);
        SDE_CHECK_LAUNCH();
    }
    float f2 = 1.0f, d2 = 0.0f;
    AzParams az;
    memset(&az, 0, sizeof az);
    unsigned long long hcounts[8] = {0};
    double hs[2] = {0.0, 0.0};
    const int robust_mode = rmode >= 1;
    const bool need_sums = robust_mode || stats;
    if (need_sums) {
        const int per = 16;
        int nbw = ceil_div(nvis > 0 ? nvis : 1, (int64_t)RED_THREADS * per);
        int nbc = ceil_div(ncell, (int64_t)RED_THREADS * per);
        double *part;
        SDE_TRY(ctx_scratch(ctx, "w_part", sizeof(double) * (size_t)(nbw > nbc ? nbw : nbc),
                            (void **)&part));
        k_sumwt_part<<<nbw, RED_THREADS, 0, st>>>(vals, counts, per, part);
        SDE_CHECK_LAUNCH();
        k_sum_partials<<<1, RED_THREADS, 0, st>>>(part, nbw, sums);
        SDE_CHECK_LAUNCH();
        if (rmode == 1 || rmode == 3) {
            k_sumlocwt_part<<<nbc, RED_THREADS, 0, st>>>(gwt, ncell, per, part);
            SDE_CHECK_LAUNCH();
            k_sum_partials<<<1, RED_THREADS, 0, st>>>(part, nbc, sums + 1);
            SDE_CHECK_LAUNCH();
        }
        // counts and sums lie together: one copy
        unsigned char both[sizeof hcounts + sizeof hs];
        SDE_TRY(ctx_read_small(ctx, st, both, counts, sizeof both));
        memcpy(hcounts, both, sizeof hcounts);
        memcpy(hs, both + sizeof hcounts, sizeof hs);
        if (hcounts[7]) {
            sde_set_error("sde_weights: a device wait timed out");
            return SDE_ETIMEDOUT;
        }
    }
    // robust parameters on the host, with the reference's REAL/DOUBLE mix (grd/grdruw2d.f:106-193)
    float rob = robust ? robust[0] : 0.0f;
    if (rmode == 3) {
        rob = (robust[0] + robust[1]) / 2.0f;
        float rpa = -robust[2] + 90.0f - 90.0f;
        while (rpa < -90.0f) rpa = rpa + 180.0f;
        while (rpa > 90.0f) rpa = rpa - 180.0f;
        float pi = 4.0f * atanf(1.0f);
        rpa = rpa * pi / 180.0f;
        az.doaz = 1;
        az.r1 = robust[0];
        az.rpa = rpa;
        az.pi = pi;
        az.rbscale = (robust[0] - robust[1]) / (pi / 2.0f);
        az.ratio = hs[1] / hs[0];
    }
    if (rmode == 1 || rmode == 3) {
        float t = 5.0f * powf(10.0f, -rob);
        f2 = (float)((double)(t * t) / (hs[1] / hs[0]));
        d2 = 1.0f;
    } else if (rmode == 2) {
        f2 = rob * rob;
        d2 = 2.0f * (ds * ds);
    } else {
        f2 = 1.0f;
        d2 = 0.0f;
    }
    if (nvis > 0) {
        (rot ? k_newwt<true> : k_newwt<false>)<<<ceil_div(nvis, W_T * W_PER), W_T, 0, st>>>(
            p, robust_mode, f2, d2, az, wt, u, v, w, gwt, nvis, newwt, &counts[7], ctx->d_status);
        SDE_CHECK_LAUNCH();
    }
    if (stats) {
        stats->ndrop = (int64_t)hcounts[1];
        stats->sumwt = hs[0];
        stats->sumlocwt = hs[1];
        stats->f2 = f2;
        stats->d2 = d2;
    }
    return SDE_OK;
}

int sde_weights(sde_ctx *ctx, int rmode, const float robust[3], float ds, const float *wt,
                const float *u, const float *v, const float *w, int64_t nvis, float uscale,
                float uoffset, float vscale, float voffset, int uorigin, int vorigin, int nu,
                int nv, const double shift[9], float *newwt, float *gwt, sde_wstats *stats) {
    SDE_TRY(weights_queue(ctx, rmode, robust, ds, wt, u, v, w, nvis, uscale, uoffset, vscale, voffset, uorigin, vorigin,
                          nu, nv, shift, newwt, gwt, stats));
    if (stats) SDE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return SDE_OK;
}
