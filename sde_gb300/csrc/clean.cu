// clean.cu -- Hogbom CLEAN minor cycle (PIX2DRCL), PIXISAMA, and the uvmap PSF-peak
// normalisation (ARRSTAT max + ARRSCALE by 1/max).
//
// PIX2DRCL (pix/pix2drcl.f:67-130): RES = DRT*BOX; per iteration the first index of the
// strictly largest |RES| (PIXISAMA, pix/pixisama.f:45-53), stop tests, component record,
// then RES -= (PNTSUB*PSF(OFFX-IX,OFFY-IY))*BOX over the whole window in FP32.  Here one
// cooperative persistent launch runs every iteration: each CTA owns a contiguous slice of
// the window, applies the previous component's subtraction to it with the same FP32
// operations (no FMA), finds its slice's first maximum, and that maximum joins a global one
// (a packed key, one atomicMax per CTA) inside a grid barrier (bounded spin); every CTA then
// reads the same global (max, first index), so component positions are identical to the
// reference's.  Windows that fit one thread-block cluster run in k_hogbom_cluster,
// those that fit the registers of the chip in k_hogbom_regs.
#include <cooperative_groups.h>
#include <math.h>
#include <string.h>

#include <mutex>

#include "cluster_max.cuh"
#include "common.cuh"

namespace {

constexpr int CL_THREADS = 512;
constexpr size_t CL_SMEM_SLICE_MAX = 100 * 1024;  // largest RES slice kept in shared memory
constexpr int CL_BATCH = 4;                        // pixels per thread with PSF loads in flight
constexpr unsigned SPIN_LIMIT = 1u << 26;

__device__ __forceinline__ Cand better(Cand x, Cand y) {
    // larger |a| wins; ties go to the smaller index (first occurrence)
    if (y.a > x.a || (y.a == x.a && y.idx < x.idx)) return y;
    return x;
}

__device__ Cand block_best(Cand c) {
    __shared__ Cand sh[32];
    for (int d = 16; d > 0; d >>= 1) {
        Cand o;
        o.a = __shfl_down_sync(0xffffffffu, c.a, d);
        o.idx = __shfl_down_sync(0xffffffffu, c.idx, d);
        o.v = __shfl_down_sync(0xffffffffu, c.v, d);
        c = better(c, o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[warp] = c;
    __syncthreads();
    if (warp == 0) {
        c = lane < (int)(blockDim.x >> 5) ? sh[lane] : Cand{-1.0f, INT32_MAX, 0.0f};
        for (int d = 16; d > 0; d >>= 1) {
            Cand o;
            o.a = __shfl_down_sync(0xffffffffu, c.a, d);
            o.idx = __shfl_down_sync(0xffffffffu, c.idx, d);
            o.v = __shfl_down_sync(0xffffffffu, c.v, d);
            c = better(c, o);
        }
        if (lane == 0) sh[0] = c;
    }
    __syncthreads();
    Cand r = sh[0];
    __syncthreads();
    return r;
}

struct Barrier {
    unsigned count;  // arrivals since the launch (grid_sync)
    int stopreq[2];  // cancel requests published by CTA 0 before each barrier
    unsigned long long best[3];  // each iteration's maximum, as a packed key (cand_key)
};

// Grid-wide barrier on a monotonic arrival count: barrier number `epoch` (0, 1, ...) is passed
// when the count reaches (epoch + 1) * nblocks, so the last CTA's arrival releases the others
// (no reset, no second word) and that CTA does not wait.  Gives up after SPIN_LIMIT polls and
// reports through *timeout.  The count is cleared before each launch.
__device__ bool grid_sync(Barrier *b, unsigned nblocks, unsigned epoch, int *timeout,
                          unsigned long long *pub = nullptr, const unsigned long long *key = nullptr) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        const unsigned target = (epoch + 1u) * nblocks;
        // the CTA's maximum (a key, 0 for none) joins the global one before the CTA arrives
        if (pub && *key) atomicMax(pub, *key);
        __threadfence();
        const unsigned arrived = atomicAdd(&b->count, 1u) + 1u;
        if ((int)(arrived - target) < 0) {
            volatile unsigned *vc = &b->count;
            unsigned spins = 0;
            while ((int)(*vc - target) < 0) {
                if (++spins > SPIN_LIMIT) {
                    atomicExch(timeout, 1);
                    ok = 0;
                    break;
                }
                if (*(volatile int *)timeout) {
                    ok = 0;
                    break;
                }
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

struct CleanArgs {
    const float *drt, *psf, *box;
    float *cln, *res, *cflux;
    int *cx, *cy;
    int nx, ny, pnx, pny, pmpx, pmpy;
    float gain, flux, tflux_in;
    int nsub, bsub;
    volatile int *cancel;
    Barrier *bar;
    int *status;     // [STATUS_TIMEOUT]
    float *out;      // [0] maxres [1] tflux [2] ansub (as int bits)
    int limit;       // polls of k_hogbom_cluster's and k_hogbom_regs' waits
};

// SMEM: the CTA's slice of RES lives in shared memory for all iterations (dynamic shared
// memory of one slice) and goes to A.res once at the end; otherwise RES is read and written
// in global memory every iteration.  The arithmetic is the same either way.
template <bool SMEM>
__global__ void __launch_bounds__(CL_THREADS) k_hogbom(CleanArgs A) {
    extern __shared__ float sres[];
    const int64_t npix = (int64_t)A.nx * A.ny;
    const int64_t per = (npix + gridDim.x - 1) / gridDim.x;
    const int64_t lo = per * blockIdx.x;
    const int64_t hi = lo + per < npix ? lo + per : npix;
    const int64_t pnpix = (int64_t)A.pnx * A.pny;
    auto R = [&](int64_t k) -> float & { return SMEM ? sres[k - lo] : A.res[k]; };
    __shared__ int stop_sh;
    // the CTA's maximum of a pass as a key (cand_key; 0 for none): warps add theirs with
    // atomicMax, thread 0 adds it to the global word inside the next grid barrier
    __shared__ unsigned long long s_key;
    if (threadIdx.x == 0) s_key = 0ull;
    __syncthreads();
    // RES = DRT * BOX, and the first maximum of the slice
    Cand c{-1.0f, INT32_MAX, 0.0f};
    for (int64_t k = lo + threadIdx.x; k < hi; k += blockDim.x) {
        float r = A.box ? __fmul_rn(A.drt[k], A.box[k]) : __fmul_rn(A.drt[k], 1.0f);
        R(k) = r;
        c = better(c, Cand{fabsf(r), (int32_t)k, r});
    }
    {
        const unsigned long long wk = warp_key_max(c.a >= 0.0f ? cand_key(c) : 0ull);
        if ((threadIdx.x & 31) == 0 && wk) atomicMax(&s_key, wk);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) A.bar->stopreq[0] = (A.cancel && *A.cancel) ? 1 : 0;
    unsigned epoch = 0;
    if (!grid_sync(A.bar, gridDim.x, epoch++, &A.status[STATUS_TIMEOUT], &A.bar->best[0], &s_key)) return;
    // the maxima of successive passes take best[0], best[1], best[2] in turn: a word is read
    // after the barrier that follows its pass, and cleared by CTA 0 one pass before it is
    // used again (after every CTA has read it, before any CTA adds to it)
    int ph = 0;
    int cur = 0;
    float tflux = A.tflux_in;
    const int nabs = A.nsub < 0 ? -A.nsub : A.nsub;
    int isub;
    int stopped = 0;
    float maxres = 0.0f;
    for (isub = A.bsub; isub <= nabs; isub++) {
        // global first maximum of the last pass
        const Cand g = key_cand(__ldcg(&A.bar->best[ph % 3]));
        if (blockIdx.x == 0 && threadIdx.x == 0) A.bar->best[(ph + 2) % 3] = 0ull;
        if (threadIdx.x == 0) s_key = 0ull;  // (ordered before the warps' additions by the barrier below)
        // PIXISAMA returns 1 (index 0) when no |value| exceeds 0
        // every |value| >= 0 beats the -1 sentinel, so when nothing exceeds 0 the winner
        // is index 0 -- PIXISAMA's default of 1 (pix/pixisama.f:45)
        const int32_t ip = g.idx;
        const int pmx = 1 + ip % A.nx, pmy = 1 + ip / A.nx;
        maxres = g.v;
        if (threadIdx.x == 0) {
            int s = 0;
            if (A.nsub < 0 && maxres < 0.0f) s = 1;
            if (fabsf(maxres) <= A.flux) s = 1;
            if (((volatile int *)A.bar->stopreq)[cur]) s = 2;
            stop_sh = s;
        }
        __syncthreads();
        if (stop_sh) {
            stopped = stop_sh;
            break;
        }
        const float pntsub = __fmul_rn(A.gain, maxres);
        tflux = __fadd_rn(tflux, pntsub);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            const int64_t ci = (int64_t)(pmy - 1) * A.nx + (pmx - 1);
            A.cln[ci] = __fadd_rn(A.cln[ci], pntsub);
            A.cflux[isub - 1] = pntsub;
            A.cx[isub - 1] = pmx;
            A.cy[isub - 1] = pmy;
        }
        const int offx = A.pmpx + pmx, offy = A.pmpy + pmy;
        Cand lc{-1.0f, INT32_MAX, 0.0f};
        // RES -= (PNTSUB*PSF(OFFX-IX, OFFY-IY))*BOX over the slice.  PSF is addressed as the
        // reference's array is, by its flat index (OFFX-IX-1) + (OFFY-IY-1)*PNX (0-based IX,
        // IY here: -2), which steps by -1 per pixel and by NX-PNX per row; when the whole
        // window's indices lie in the PSF no per-pixel check is made.  A thread visits its
        // pixels in increasing order, so a strictly larger |RES| is its first maximum.
        {
            const int nslice = (int)(hi - lo);
            int sidx = threadIdx.x;
            const int64_t k0 = lo + sidx;
            int ix0 = (int)(k0 % A.nx);
            const int iy0 = (int)(k0 / A.nx);
            int64_t flat = (int64_t)(offx - ix0 - 2) + (int64_t)(offy - iy0 - 2) * A.pnx;
            const int64_t fmin = (int64_t)(offx - (A.nx - 1) - 2) + (int64_t)(offy - (A.ny - 1) - 2) * A.pnx;
            const int64_t fmax = (int64_t)(offx - 2) + (int64_t)(offy - 2) * A.pnx;
            const bool inside = fmin >= 0 && fmax < pnpix;
            const int step = blockDim.x;
            const int64_t wrap = (int64_t)A.nx - A.pnx;
            float la = -1.0f, lv = 0.0f;
            int li = INT32_MAX;
            // CL_BATCH pixels at a time: their PSF and RES loads are issued before any is used
            for (; sidx < nslice; sidx += CL_BATCH * step) {
                float p[CL_BATCH], r0[CL_BATCH];
#pragma unroll
                for (int j = 0; j < CL_BATCH; j++) {
                    const bool in = sidx + j * step < nslice;
                    p[j] = !in ? 0.0f
                               : inside ? A.psf[flat]
                                        : ((flat >= 0 && flat < pnpix) ? A.psf[flat] : 0.0f);
                    r0[j] = in ? R(lo + sidx + j * step) : 0.0f;
                    ix0 += step;
                    flat -= step;
                    while (ix0 >= A.nx) {
                        ix0 -= A.nx;
                        flat += wrap;
                    }
                }
#pragma unroll
                for (int j = 0; j < CL_BATCH; j++) {
                    const int sj = sidx + j * step;
                    if (sj < nslice) {
                        float sub = __fmul_rn(pntsub, p[j]);
                        if (A.box) sub = __fmul_rn(sub, A.box[lo + sj]);
                        const float r = __fsub_rn(r0[j], sub);
                        R(lo + sj) = r;
                        if (fabsf(r) > la) {
                            la = fabsf(r);
                            li = (int)(lo + sj);
                            lv = r;
                        }
                    }
                }
            }
            lc = Cand{la, li, lv};
        }
        {
            const unsigned long long wk = warp_key_max(lc.a >= 0.0f ? cand_key(lc) : 0ull);
            if ((threadIdx.x & 31) == 0 && wk) atomicMax(&s_key, wk);
        }
        cur ^= 1;
        if (blockIdx.x == 0 && threadIdx.x == 0) A.bar->stopreq[cur] = (A.cancel && *A.cancel) ? 1 : 0;
        if (!grid_sync(A.bar, gridDim.x, epoch++, &A.status[STATUS_TIMEOUT], &A.bar->best[(ph + 1) % 3], &s_key))
            return;
        ph++;
    }
    if (SMEM)
        for (int64_t k = lo + threadIdx.x; k < hi; k += blockDim.x) A.res[k] = R(k);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        int ansub;
        if (!stopped) {
            ansub = A.nsub;
        } else {
            ansub = isub - 1;
        }
        A.out[1] = tflux;
        A.out[2] = __int_as_float(ansub);
        A.out[3] = __int_as_float(stopped);
        if (stopped) A.out[0] = maxres;
    }
    if (!stopped) {
        // final PIXISAMA over the residual (pix/pix2drcl.f:134-138): the last pass's maximum
        if (blockIdx.x == 0 && threadIdx.x == 0) A.out[0] = key_cand(__ldcg(&A.bar->best[ph % 3])).v;
    }
}


// ---------------------------------------------------------------------------------------
// Small windows: the whole minor cycle in one thread-block cluster.  A window of up to
// HC_MAXPIX pixels is spread over the cluster's threads, PER pixels each (residual and
// component image in registers for all iterations), so an iteration needs no grid-wide
// barrier: every CTA sends its maximum to every CTA with one remote store that also counts
// on the receiver's mbarrier (st.async), and waits for the others' on its own.  The
// arithmetic and the pick (largest |RES|, then the first index) are k_hogbom's.
// An iteration is a latency chain: PSF load, warp maximum, CTA barrier, remote store, slot
// maximum.  Measured a component, k_hogbom -> here: 127^2 3.5 -> 0.9 us, 255^2 3.4 -> 1.1,
// 361^2 3.5 -> 1.6, 511^2 3.7 -> 2.25.  Few warps a CTA: every warp repeats the scalar part of
// the chain, and with 1024 threads those instructions queue for issue slots (255^2 1.3 us).
constexpr int HC_CTAS = 16;   // cluster size (above the portable 8: opted in at launch)
constexpr int64_t HC_MAXPIX = (int64_t)512 * HC_CTAS * 32;
constexpr int HC_RING = 256;  // components kept before they go into CLN

// Row of pixel idx in rows of nx pixels, by the reciprocal ceil(2^32 / nx): the product can
// only reach the next row's first pixel early.
__device__ __forceinline__ uint32_t row_recip(int nx) { return nx > 1 ? 0xFFFFFFFFu / (uint32_t)nx + 1u : 0u; }
__device__ __forceinline__ int row_of(int idx, int nx, uint32_t recip) {
    if (nx == 1) return idx;
    const int q = (int)__umulhi((uint32_t)idx, recip);
    return q * nx > idx ? q - 1 : q;
}

// PSF peak (1-based) from PIXISAMA's index (pix/pix2drcl.f:73-80)
__host__ __device__ inline void psf_peak(int64_t ip1, int pnx, int pny, int *pmpx, int *pmpy) {
    const int ipeak = (int)((ip1 > 0 ? ip1 : 1) - 1);  // PIXISAMA's default I = 1
    int px = 1 + ipeak % pnx;
    int py = 1 + (ipeak - px + 1) / pnx;
    if (px >= pnx) px = pnx / 2;
    if (py >= pny) py = pny / 2;
    *pmpx = px;
    *pmpy = py;
}

// Every shift of the window by a component lies inside the PSF array, axis by axis: no PSF
// read is out of range or wraps into another row.
__host__ __device__ inline bool psf_covers(int pmpx, int pmpy, int nx, int ny, int pnx, int pny) {
    return pmpx - (nx - 1) >= 1 && pmpx + (nx - 1) <= pnx && pmpy - (ny - 1) >= 1 && pmpy + (ny - 1) <= pny;
}

// A.psf_ip: the PSF's peak index on the device (k_isamax_final).  When the PSF does not cover
// every shift nothing is done and A.out[3] is HC_NOTCOVERED (the caller runs k_hogbom).
constexpr int HC_NOTCOVERED = 3;
template <int T, int PER>
__global__ void __launch_bounds__(T, 1) k_hogbom_cluster(CleanArgs A, const int64_t *psf_ip) {
    __shared__ __align__(16) ClusterMax<HC_CTAS> cm;
    __shared__ unsigned long long skey[T / 32];
    __shared__ int ring_idx[HC_RING];
    __shared__ float ring_f[HC_RING];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t rank;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    int pmpx, pmpy;
    psf_peak(*psf_ip, A.pnx, A.pny, &pmpx, &pmpy);
    if (!psf_covers(pmpx, pmpy, A.nx, A.ny, A.pnx, A.pny)) {
        if (rank == 0 && t == 0) A.out[3] = __int_as_float(HC_NOTCOVERED);
        return;
    }
    cluster_max_init(&cm);
    const int npix = A.nx * A.ny, base = (int)rank * PER * T;
    float r[PER];
    int rel[PER];  // the pixel's PSF offset from the component's: -ix - iy * pnx
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int k = base + j * T + t;
        const bool in = k < npix;
        const int iy = in ? k / A.nx : 0, ix = in ? k - iy * A.nx : 0;
        rel[j] = -ix - iy * A.pnx;
        r[j] = in ? __fmul_rn(A.drt[k], A.box ? A.box[k] : 1.0f) : 0.f;
    }
    // NaN pixels (and the padding past the window) never win
    auto best = [&]() {
        float la = -1.0f, lv = 0.f;
        int li = 0;
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const int k = base + j * T + t;
            if (k < npix && fabsf(r[j]) > la) {
                la = fabsf(r[j]);
                li = k;
                lv = r[j];
            }
        }
        return warp_key_max(la >= 0.0f ? cand_key(Cand{la, li, lv}) : 0ull);
    };
    // n components of the ring into CLN, each by its pixel's thread in order
    auto drain = [&](int n) {
        __syncthreads();
        for (int i = 0; i < n; i++) {
            const int own = ring_idx[i] - base - t;
            if (own >= 0 && own < PER * T && own % T == 0)
                A.cln[ring_idx[i]] = __fadd_rn(A.cln[ring_idx[i]], ring_f[i]);
        }
        __syncthreads();
    };
    float tflux = A.tflux_in, maxres = 0.f;
    const int nabs = A.nsub < 0 ? -A.nsub : A.nsub;
    const uint32_t rnx = row_recip(A.nx);
    unsigned state = 0;
    // (a key of 0: no pixel is a number, so there is nothing to subtract)
    auto stops = [&](unsigned long long gk, int n) {
        const float v = key_cand(gk).v;
        return A.bsub + n > nabs || (A.nsub < 0 && v < 0.0f) || fabsf(v) <= A.flux || gk == 0ull || cluster_max_aborts(gk);
    };
    int n = 0;  // rounds, and the components subtracted
    for (;; n++) {
        const unsigned long long wk = best();
        if (lane == 0) skey[warp] = wk;
        if (__syncthreads_or(state & (CM_LATE | CM_LAST)) && cluster_max_ends(&cm, n, state, skey, stops)) break;
        if (warp == 0) {
            const unsigned long long ck = warp_key_max(lane < T / 32 ? skey[lane] : 0ull);
            if (lane < HC_CTAS) cluster_max_send(&cm, n, (int)rank, lane, ck);
        }
        // (after a wait that ran out the ring may lack a component)
        if (n > 0 && n % HC_RING == 0 && !(state & CM_GAVE_UP)) drain(HC_RING);
        bool ok;
        const unsigned long long gk = cluster_max_wait(&cm, n, ok, A.limit);
        if (!ok) {
            state |= CM_LATE;
            continue;
        }
        if (t == 0) cluster_max_rearm(&cm, n);
        const Cand g = key_cand(gk);
        maxres = g.v;
        if (stops(gk, n)) {
            state |= cluster_max_aborts(gk) ? CM_LAST | CM_GAVE_UP : CM_LAST;
            continue;
        }
        const float pntsub = __fmul_rn(A.gain, maxres);
        tflux = __fadd_rn(tflux, pntsub);
        const int gy = row_of(g.idx, A.nx, rnx), gx = g.idx - gy * A.nx;
        // PSF(OFFX-IX, OFFY-IY), flat: (pmpx-1 + gx - ix) + (pmpy-1 + gy - iy) * pnx
        const float *p0 = A.psf + (pmpx - 1 + gx) + (int64_t)(pmpy - 1 + gy) * A.pnx;
        float p[PER];
#pragma unroll
        for (int j = 0; j < PER; j++) p[j] = __ldg(p0 + rel[j]);
        if (t == 0) {
            ring_idx[n % HC_RING] = g.idx;
            ring_f[n % HC_RING] = pntsub;
            if (rank == 0) {
                const int c = A.bsub + n - 1;
                A.cflux[c] = pntsub;
                A.cx[c] = gx + 1;
                A.cy[c] = gy + 1;
            }
        }
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const float sub = __fmul_rn(pntsub, p[j]);
            r[j] = __fsub_rn(r[j], A.box ? __fmul_rn(sub, A.box[min(base + j * T + t, npix - 1)]) : sub);
        }
    }
    if (state & CM_GAVE_UP) {
        if (t == 0) atomicExch(&A.status[STATUS_TIMEOUT], 1);
    } else {
        n--;  // the loop ends one round after the one that stopped it
        drain(n % HC_RING);
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const int k = base + j * T + t;
            if (k < npix) A.res[k] = r[j];
        }
        if (rank == 0 && t == 0) {
            const bool stopped = A.bsub + n <= nabs;
            A.out[0] = maxres;
            A.out[1] = tflux;
            A.out[2] = __int_as_float(stopped ? A.bsub + n - 1 : A.nsub);
            A.out[3] = __int_as_float(stopped ? 1 : 0);
        }
    }
    // no CTA leaves while another's stores to it may be in flight
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---------------------------------------------------------------------------------------
// Windows above one cluster's: the residual stays in the registers of one CTA per SM for all
// iterations (HR_T threads x HR_PER pixels), and an iteration reads only the PSF (and the box).
// The pixels of a thread are HR_T apart in the CTA's contiguous slice; a bit per pixel says
// whether the step to it starts a new row, so the PSF offset is carried by two integer adds.
// The next group's PSF loads are in flight while one is subtracted.
// The maximum of a pass: a maximum per group, then only the warp that holds the CTA's searches
// its group for the first pixel, and the key goes to a slot of every mailbox, which one warp of
// each of its HR_SHARE CTAs polls.  A 64-bit store carries key and round together (bit 63, the
// spare sign of |value|), so there is no counter, no atomic and no fence in the chain.  Slots
// alternate: one written in round n is written again in round n + 2, whose writer has seen every
// key of round n + 1, each sent after its CTA had read round n.
// Bound by the L2's rate for the PSF at large windows (2047^2: 4600 cycles of an iteration's
// 10500, 18 or 27 loads ahead alike) and by the exchange (3000) at small ones: with one mailbox
// polled by all CTAs it took 8000, with 1, 2, 4, 8, 16 CTAs a mailbox 723^2 takes 2.75, 2.66,
// 2.73, 2.80, 2.97 us an iteration.  k_hogbom -> here, us an iteration without and with a box:
// 723^2 4.85 -> 2.66 and 5.34 -> 3.06, 1023^2 5.6 -> 3.0 and 6.5 -> 3.5, 1447^2 7.2 -> 3.75 and
// 8.8 -> 4.7, 2047^2 9.7 -> 5.4 and 12.8 -> 7.9.
constexpr int HR_T = 256, HR_PER = 108;
static_assert(HR_PER % 27 == 0, "whole words of row bits");
constexpr int HR_MAXCTAS = 160;  // a mailbox: 5 slots a polling lane, all in flight
constexpr int HR_SHARE = 2;      // CTAs that poll one mailbox
constexpr int HR_SPIN = 1 << 22;
constexpr size_t HR_SLOTS = (size_t)HR_MAXCTAS / HR_SHARE * 2 * HR_MAXCTAS;  // [mailbox][round & 1][writer]
constexpr unsigned long long HR_TAG = 1ull << 63;

template <bool BOX>
__global__ void __launch_bounds__(HR_T, 1) k_hogbom_regs(CleanArgs A, unsigned long long *slots) {
    constexpr int HR_G = BOX ? 9 : 18, HR_NG = HR_PER / HR_G;  // (a box value is loaded with each PSF value)
    __shared__ unsigned s_max[HR_T / 32];
    __shared__ unsigned s_low;
    __shared__ unsigned long long s_key;
    __shared__ int s_ok;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nb = gridDim.x;
    const int npix = A.nx * A.ny;
    const int slice = (npix + nb - 1) / nb;
    const int64_t lo64 = (int64_t)slice * blockIdx.x;
    const int lo = (int)(lo64 < npix ? lo64 : npix);
    const int mine = min(slice, npix - lo);                         // the CTA's pixels
    const int nj = mine > t ? (mine - t + HR_T - 1) / HR_T : 0;     // the thread's
    const int ncta = (mine + HR_T - 1) / HR_T;                      // the CTA's largest nj
    const int nbox = (nb + HR_SHARE - 1) / HR_SHARE;
    const int wrap = A.pnx - A.nx;
    const uint32_t rnx = row_recip(A.nx);
    float r[HR_PER];
    unsigned cross[HR_PER / 27];  // bit j % 27 of word j / 27: pixel j starts a new row
    int rel0;                     // PSF offset of the first pixel: -ix - iy * pnx
    {
        const int k0 = min(lo + t, npix - 1);
        const int iy = k0 / A.nx;
        int ix = k0 - iy * A.nx;
        rel0 = -ix - iy * A.pnx;
#pragma unroll
        for (int j = 0; j < HR_PER; j++) {
            if (j % 27 == 0) cross[j / 27] = 0u;
            if (j > 0) {
                ix += HR_T;
                if (ix >= A.nx) {
                    ix -= A.nx;
                    cross[j / 27] |= 1u << (j % 27);
                }
            }
            r[j] = __int_as_float(0x7FC00000);  // no pixel: a NaN, which no maximum takes
            if (j < nj) {
                const int k = lo + j * HR_T + t;
                r[j] = __fmul_rn(A.drt[k], BOX ? A.box[k] : 1.0f);
            }
        }
    }
    float gmax[HR_NG];  // largest |residual| of a group; NaN pixels never win
    auto group_max = [&](int g) {
        float m = -1.0f;
#pragma unroll
        for (int i = 0; i < HR_G; i++) m = fmaxf(m, fabsf(r[g * HR_G + i]));
        gmax[g] = m;
    };
#pragma unroll
    for (int g = 0; g < HR_NG; g++) group_max(g);
    float tflux = A.tflux_in, maxres = 0.f;
    const int nabs = A.nsub < 0 ? -A.nsub : A.nsub;
    int isub = A.bsub, stopped = 0;
    for (int n = 0;; n++) {
        // the CTA's maximum: 0 for none, else the bits of |value| plus one
        float m = gmax[0];
#pragma unroll
        for (int g = 1; g < HR_NG; g++) m = fmaxf(m, gmax[g]);
        const unsigned code = m >= 0.0f ? __float_as_uint(m) + 1u : 0u;
        const unsigned wcode = __reduce_max_sync(0xffffffffu, code);
        if (lane == 0) s_max[warp] = wcode;
        if (t == 0) s_low = 0u;
        __syncthreads();
        const unsigned ccode = __reduce_max_sync(0xffffffffu, s_max[lane & (HR_T / 32 - 1)]);
        if (wcode == ccode && code == ccode && code) {
            int first = INT32_MAX;
            float v = 0.f;
#pragma unroll
            for (int g = HR_NG - 1; g >= 0; g--)
                if (gmax[g] == m) {
#pragma unroll
                    for (int i = HR_G - 1; i >= 0; i--)
                        if (fabsf(r[g * HR_G + i]) == m) {
                            first = g * HR_G + i;
                            v = r[g * HR_G + i];
                        }
                }
            atomicMax(&s_low, (unsigned)cand_key(Cand{m, lo + first * HR_T + t, v}));
        }
        __syncthreads();
        if (warp == 0) {
            const unsigned long long tag = (n >> 1) & 1 ? 0ull : HR_TAG;
            const unsigned long long out = (ccode ? (unsigned long long)(ccode - 1u) << 32 : 0ull) | s_low | tag;
#pragma unroll
            for (int b = 0; b < (HR_MAXCTAS / HR_SHARE + 31) / 32; b++)
                if (b * 32 + lane < nbox)
                    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(
                                     slots + ((size_t)(b * 32 + lane) * 2 + (n & 1)) * HR_MAXCTAS + blockIdx.x),
                                 "l"(out)
                                 : "memory");
            const unsigned long long *row = slots + ((size_t)(blockIdx.x % nbox) * 2 + (n & 1)) * HR_MAXCTAS;
            unsigned long long best = 0ull;
            bool done = false;
            for (int spin = 0; spin < A.limit && !done; spin++) {
                unsigned long long k[HR_MAXCTAS / 32];
#pragma unroll
                for (int b = 0; b < HR_MAXCTAS / 32; b++) {
                    k[b] = tag;
                    if (b * 32 + lane < nb)
                        asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(k[b]) : "l"(row + b * 32 + lane) : "memory");
                }
                bool all = true;
                best = 0ull;
#pragma unroll
                for (int b = 0; b < HR_MAXCTAS / 32; b++) {
                    all = all && (k[b] & HR_TAG) == tag;
                    k[b] &= ~HR_TAG;
                    best = k[b] > best ? k[b] : best;
                }
                done = __all_sync(0xffffffffu, all);
            }
            best = warp_key_max(best);
            if (lane == 0) {
                s_key = best;
                s_ok = done;
            }
        }
        __syncthreads();
        if (!s_ok) {
            if (t == 0) atomicExch(&A.status[STATUS_TIMEOUT], 1);
            return;
        }
        const Cand g = key_cand(s_key);
        maxres = g.v;
        if (isub > nabs) break;
        // (a key of 0: no pixel is a number, so there is nothing to subtract)
        if ((A.nsub < 0 && maxres < 0.0f) || fabsf(maxres) <= A.flux || s_key == 0ull) {
            stopped = 1;
            break;
        }
        const float pntsub = __fmul_rn(A.gain, maxres);
        tflux = __fadd_rn(tflux, pntsub);
        const int gy = row_of(g.idx, A.nx, rnx), gx = g.idx - gy * A.nx;
        // the component's pixel, in its thread (the add waits until the PSF loads are issued)
        const int own = g.idx - lo - t;
        const bool owner = own >= 0 && own < mine - t && own % HR_T == 0;
        float cln = 0.f;
        if (owner) cln = A.cln[g.idx];
        if (blockIdx.x == 0 && t == 0) {
            A.cflux[isub - 1] = pntsub;
            A.cx[isub - 1] = gx + 1;
            A.cy[isub - 1] = gy + 1;
        }
        // PSF(OFFX-IX, OFFY-IY), flat: (pmpx-1 + gx - ix) + (pmpy-1 + gy - iy) * pnx
        const float *p0 = A.psf + (A.pmpx - 1 + gx) + (int64_t)(A.pmpy - 1 + gy) * A.pnx;
        float p[2][HR_G], bx[2][BOX ? HR_G : 1];
        int o = rel0;
        auto load = [&](int q) {
#pragma unroll
            for (int i = 0; i < HR_G; i++) {
                const int j = q * HR_G + i;
                if (j > 0) {
                    o -= HR_T;
                    if (cross[j / 27] >> (j % 27) & 1u) o -= wrap;
                }
                p[q & 1][i] = j < nj ? __ldg(p0 + o) : 0.f;
                if (BOX) bx[q & 1][i] = j < nj ? __ldg(A.box + lo + j * HR_T + t) : 0.f;
            }
        };
        load(0);
#pragma unroll
        for (int q = 0; q < HR_NG; q++) {
            if (q * HR_G < ncta) {
                if (q + 1 < HR_NG) {
                    if ((q + 1) * HR_G < ncta) load(q + 1);
                }
#pragma unroll
                for (int i = 0; i < HR_G; i++) {
                    const int j = q * HR_G + i;
                    float sub = __fmul_rn(pntsub, p[q & 1][i]);
                    if (BOX) sub = __fmul_rn(sub, bx[q & 1][i]);
                    r[j] = __fsub_rn(r[j], sub);
                }
                group_max(q);
            }
        }
        if (owner) A.cln[g.idx] = __fadd_rn(cln, pntsub);
        isub++;
    }
#pragma unroll
    for (int j = 0; j < HR_PER; j++)
        if (j < nj) A.res[lo + j * HR_T + t] = r[j];
    if (blockIdx.x == 0 && t == 0) {
        A.out[0] = maxres;
        A.out[1] = tflux;
        A.out[2] = __int_as_float(stopped ? isub - 1 : A.nsub);
        A.out[3] = __int_as_float(stopped);
    }
}

// first strictly-largest |a| (PIXISAMA), two-level
// (16-byte loads, four in flight a thread, from the first aligned element on; 4096^2: 51 -> 14 us)
__global__ void __launch_bounds__(CL_THREADS) k_isamax_part(const float *a, int64_t n, Cand *part) {
    // a thread's indices rise, so a strictly larger |a| is its first maximum (NaN never is)
    float la = -1.0f, lv = 0.0f;
    int li = INT32_MAX;
    auto take = [&](float v, int64_t k) {
        if (fabsf(v) > la) {
            la = fabsf(v);
            li = (int)k;
            lv = v;
        }
    };
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    const int64_t head = min(n, (int64_t)((16 - ((uintptr_t)a & 15)) & 15) / 4), n4 = (n - head) / 4;
    const float4 *a4 = reinterpret_cast<const float4 *>(a + head);
    if (g < head) take(a[g], g);
    int64_t k = g;
    for (; k + 3 * step < n4; k += 4 * step) {
        float4 x[4];
#pragma unroll
        for (int i = 0; i < 4; i++) x[i] = __ldg(a4 + k + i * step);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t e = head + 4 * (k + i * step);
            take(x[i].x, e);
            take(x[i].y, e + 1);
            take(x[i].z, e + 2);
            take(x[i].w, e + 3);
        }
    }
    for (; k < n4; k += step) {
        const float4 x = __ldg(a4 + k);
        const int64_t e = head + 4 * k;
        take(x.x, e);
        take(x.y, e + 1);
        take(x.z, e + 2);
        take(x.w, e + 3);
    }
    if (head + 4 * n4 + g < n) take(a[head + 4 * n4 + g], head + 4 * n4 + g);
    const Cand c = block_best(Cand{la, li, lv});
    if (threadIdx.x == 0) part[blockIdx.x] = c;
}

__global__ void __launch_bounds__(CL_THREADS) k_isamax_final(const Cand *part, int nb, int64_t *out) {
    Cand c{-1.0f, INT32_MAX, 0.0f};
    for (int b = threadIdx.x; b < nb; b += blockDim.x) c = better(c, part[b]);
    c = block_best(c);
    // 1-based index of the first largest |a|, or 0 when no |a| exceeds 0
    if (threadIdx.x == 0) *out = c.a > 0.0f ? (int64_t)c.idx + 1 : 0;
}

// max value (ARRSTAT's ARRMAX) over an image
__global__ void __launch_bounds__(CL_THREADS) k_max_part(const float *a, int64_t n, float *part) {
    __shared__ float sh[32];
    float m = -INFINITY;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        m = fmaxf(m, a[k]);
    for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, d));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : -INFINITY;
        for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, d));
        if (threadIdx.x == 0) part[blockIdx.x] = m;
    }
}

__global__ void k_max_final(const float *part, int nb, float *out) {
    float m = -INFINITY;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) m = fmaxf(m, part[b]);
    for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, d));
    if (threadIdx.x == 0) *out = m;
}

// OUT = (1/max) * IN + 0.0 (task/uvmap.f:440 with pix/pixrscal.f)
__global__ void k_scale_inv(float *a, int64_t n, const float *maxp) {
    const float s = 1.0f / *maxp;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        a[k] = __fadd_rn(__fmul_rn(s, a[k]), 0.0f);
}

}  // namespace

int sde_isamax(sde_ctx *ctx, const float *a, int64_t n, int64_t *index_out) {
    SDE_TRY(sde_isamax0(ctx, a, n, index_out));
    if (*index_out == 0) *index_out = 1;  // PIXISAMA's default I = 1
    return SDE_OK;
}

// PIXISAMA's index (0 when no |a| exceeds 0) left on the device
static int isamax_dev(sde_ctx *ctx, const float *a, int64_t n, int64_t **dev) {
    if (!ctx || !a || n <= 0 || n > INT32_MAX) return SDE_EINVAL;
    SDE_CUDA_TRY(cudaSetDevice(ctx->device));
    int nb = ctx->num_sms * 2;
    Cand *part;
    int64_t *d;
    SDE_TRY(ctx_scratch(ctx, "isa_part", sizeof(Cand) * (size_t)nb, (void **)&part));
    SDE_TRY(ctx_scratch(ctx, "isa_out", sizeof(int64_t), (void **)&d));
    k_isamax_part<<<nb, CL_THREADS, 0, ctx->stream>>>(a, n, part);
    SDE_CHECK_LAUNCH();
    k_isamax_final<<<1, CL_THREADS, 0, ctx->stream>>>(part, nb, d);
    SDE_CHECK_LAUNCH();
    *dev = d;
    return SDE_OK;
}

int sde_isamax0(sde_ctx *ctx, const float *a, int64_t n, int64_t *index_out) {
    if (!index_out) return SDE_EINVAL;
    int64_t *d;
    SDE_TRY(isamax_dev(ctx, a, n, &d));
    return ctx_read_small(ctx, ctx->stream, index_out, d, sizeof(int64_t));
}

int sde_image_max(sde_ctx *ctx, const float *image, int64_t n, float *max_dev) {
    if (!ctx || !image || n <= 0 || !max_dev) return SDE_EINVAL;
    int nb = ctx->num_sms * 2;
    float *part;
    SDE_TRY(ctx_scratch(ctx, "max_part", sizeof(float) * (size_t)nb, (void **)&part));
    KTimer kt(ctx, "image_max");
    k_max_part<<<nb, CL_THREADS, 0, ctx->stream>>>(image, n, part);
    SDE_CHECK_LAUNCH();
    k_max_final<<<1, 32, 0, ctx->stream>>>(part, nb, max_dev);
    SDE_CHECK_LAUNCH();
    return SDE_OK;
}

int sde_image_scale_by_inverse(sde_ctx *ctx, float *image, int64_t n, const float *max_dev) {
    if (!ctx || !image || n <= 0 || !max_dev) return SDE_EINVAL;
    KTimer kt(ctx, "scale_inv");
    k_scale_inv<<<ctx->num_sms * 4, 256, 0, ctx->stream>>>(image, n, max_dev);
    SDE_CHECK_LAUNCH();
    return SDE_OK;
}

// The CLEAN kernels are loaded when the context is created (with CUDA's lazy module
// loading a kernel's first launch would otherwise load it, ~18 ms measured on the first
// sde_hogbom of a process), and the cooperative launch's occupancy is queried once.
int clean_preload(sde_ctx *ctx) {
    cudaFuncAttributes a;
    SDE_CUDA_TRY(cudaFuncGetAttributes(&a, k_isamax_part));
    SDE_CUDA_TRY(cudaFuncGetAttributes(&a, k_isamax_final));
    SDE_CUDA_TRY(cudaFuncGetAttributes(&a, k_max_part));
    SDE_CUDA_TRY(cudaFuncGetAttributes(&a, k_max_final));
    SDE_CUDA_TRY(cudaFuncGetAttributes(&a, k_scale_inv));
    SDE_CUDA_TRY(cudaFuncGetAttributes(&a, k_hogbom_regs<false>));
    SDE_CUDA_TRY(cudaFuncGetAttributes(&a, k_hogbom_regs<true>));
    int per_sm = 0;
    SDE_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_hogbom<false>, CL_THREADS, 0));
    ctx->hogbom_per_sm = per_sm;
    SDE_CUDA_TRY(cudaFuncSetAttribute(k_hogbom<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)CL_SMEM_SLICE_MAX));
    // the cluster kernels: larger clusters than the portable size, if they can be resident
    struct {
        const void *k;
        int threads;
    } hc[] = {{(const void *)k_hogbom_cluster<256, 4>, 256},
              {(const void *)k_hogbom_cluster<256, 16>, 256},
              {(const void *)k_hogbom_cluster<256, 32>, 256},
              {(const void *)k_hogbom_cluster<512, 32>, 512}};
    ctx->hogbom_cluster = true;
    for (const auto &h : hc) {
        SDE_CUDA_TRY(cudaFuncSetAttribute(h.k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = HC_CTAS;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(HC_CTAS);
        cfg.blockDim = dim3(h.threads);
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        SDE_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, h.k, &cfg));
        if (n < 1) ctx->hogbom_cluster = false;
    }
    return SDE_OK;
}

// a minor cycle's scalars after the work queued on the context's stream
static int clean_result(sde_ctx *ctx, const float *dout, sde_clean_result *out, int *stopped) {
    float *h = reinterpret_cast<float *>(ctx->h_small);
    SDE_CUDA_TRY(cudaMemcpyAsync(h, dout, 4 * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    SDE_CUDA_TRY(cudaMemcpyAsync(ctx->h_status, ctx->d_status, sizeof(int) * STATUS_COUNT,
                                 cudaMemcpyDeviceToHost, ctx->stream));
    SDE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    if (ctx->h_status[STATUS_TIMEOUT]) {
        sde_set_error("sde_hogbom: a device wait timed out");
        return SDE_ETIMEDOUT;
    }
    memcpy(stopped, &h[3], 4);
    if (*stopped == HC_NOTCOVERED) return SDE_OK;
    out->maxres = h[0];
    out->tflux = h[1];
    memcpy(&out->ansub, &h[2], 4);
    return SDE_OK;
}

static int launch_hogbom_cluster(const CleanArgs &A, const int64_t *psf_ip, cudaStream_t st) {
    const int64_t npix = (int64_t)A.nx * A.ny;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = HC_CTAS;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(HC_CTAS);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const int64_t per = ceil_div(npix, (int64_t)256 * HC_CTAS);
    cudaError_t e;
    if (per <= 4) {
        e = cudaLaunchKernelEx(&cfg, k_hogbom_cluster<256, 4>, A, psf_ip);
    } else if (per <= 16) {
        e = cudaLaunchKernelEx(&cfg, k_hogbom_cluster<256, 16>, A, psf_ip);
    } else if (per <= 32) {
        e = cudaLaunchKernelEx(&cfg, k_hogbom_cluster<256, 32>, A, psf_ip);
    } else {
        cfg.blockDim = dim3(512);
        e = cudaLaunchKernelEx(&cfg, k_hogbom_cluster<512, 32>, A, psf_ip);
    }
    SDE_CUDA_TRY(e);
    return SDE_OK;
}

int sde_hogbom(sde_ctx *ctx, const float *drt, const float *psf, const float *box, int nx, int ny,
               int pnx, int pny, float gain, int nsub, int bsub, float flux, float tflux_in,
               float *cln, float *res, float *cflux, int *cx, int *cy, volatile int *cancel_flag,
               sde_clean_result *out) {
    if (!ctx || !drt || !psf || !cln || !res || nx < 1 || ny < 1 || pnx < 1 || pny < 1 || !out ||
        (int64_t)nx * ny > INT32_MAX || bsub < 1) {
        sde_set_error("sde_hogbom: bad arguments");
        return SDE_EINVAL;
    }
    const int nabs = nsub < 0 ? -nsub : nsub;
    if (nabs >= bsub && (!cflux || !cx || !cy)) {
        sde_set_error("sde_hogbom: component arrays required");
        return SDE_EINVAL;
    }
    SDE_CUDA_TRY(cudaSetDevice(ctx->device));
    float *dout;
    SDE_TRY(ctx_scratch(ctx, "cl_out", 4 * sizeof(float), (void **)&dout));
    SDE_CUDA_TRY(cudaMemsetAsync(ctx->d_status, 0, sizeof(int) * STATUS_COUNT, ctx->stream));
    CleanArgs A;
    A.drt = drt; A.psf = psf; A.box = box; A.cln = cln; A.res = res; A.cflux = cflux;
    A.cx = cx; A.cy = cy; A.nx = nx; A.ny = ny; A.pnx = pnx; A.pny = pny;
    A.pmpx = A.pmpy = 0; A.gain = gain; A.flux = flux; A.tflux_in = tflux_in;
    A.nsub = nsub; A.bsub = bsub; A.cancel = cancel_flag; A.bar = nullptr;
    A.status = ctx->d_status; A.out = dout; A.limit = cm_spin(ctx->wait_limit);
    // PSF peak (pix/pix2drcl.f:73-80)
    int64_t *psf_ip;
    SDE_TRY(isamax_dev(ctx, psf, (int64_t)pnx * pny, &psf_ip));
    // a window that one cluster holds, and no interrupt flag to poll
    if (ctx->hogbom_cluster && !cancel_flag && (int64_t)nx * ny <= HC_MAXPIX) {
        {
            KTimer kt(ctx, "hogbom");
            SDE_TRY(launch_hogbom_cluster(A, psf_ip, ctx->stream));
        }
        int stopped;
        SDE_TRY(clean_result(ctx, dout, out, &stopped));
        if (stopped != HC_NOTCOVERED) return SDE_OK;
    }
    int64_t ip1;
    SDE_TRY(ctx_read_small(ctx, ctx->stream, &ip1, psf_ip, sizeof ip1));
    psf_peak(ip1, pnx, pny, &A.pmpx, &A.pmpy);
    // a window that the registers hold, rows no shorter than a thread's step, the PSF covering it
    if (!cancel_flag && nx >= HR_T && ctx->num_sms <= HR_MAXCTAS &&
        (int64_t)nx * ny <= (int64_t)ctx->num_sms * HR_T * HR_PER && psf_covers(A.pmpx, A.pmpy, nx, ny, pnx, pny)) {
        if (ctx->wait_limit < 0) A.limit = HR_SPIN;
        unsigned long long *slots;
        SDE_TRY(ctx_scratch(ctx, "cl_slots", HR_SLOTS * sizeof(*slots), (void **)&slots));
        SDE_CUDA_TRY(cudaMemsetAsync(slots, 0, HR_SLOTS * sizeof(*slots), ctx->stream));
        void *args[] = {&A, &slots};
        {
            KTimer kt(ctx, "hogbom");
            SDE_CUDA_TRY(cudaLaunchCooperativeKernel(
                box ? (const void *)k_hogbom_regs<true> : (const void *)k_hogbom_regs<false>,
                dim3(ctx->num_sms), dim3(HR_T), args, 0, ctx->stream));
        }
        int stopped;
        return clean_result(ctx, dout, out, &stopped);
    }
    int per_sm = ctx->hogbom_per_sm;
    if (per_sm < 1) SDE_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_hogbom<false>, CL_THREADS, 0));
    if (per_sm < 1) {
        sde_set_error("sde_hogbom: kernel cannot be resident");
        return SDE_ECUDA;
    }
    int64_t npix = (int64_t)nx * ny;
    int nblocks = ctx->num_sms * (per_sm > 2 ? 2 : per_sm);
    int64_t want = (npix + 4 * CL_THREADS - 1) / (4 * CL_THREADS);  // small windows: fewer CTAs
    if (want < nblocks) nblocks = (int)(want < 1 ? 1 : want);
    // the residual in shared memory when every CTA's slice fits there and the launch stays
    // co-resident with it (windows up to ~2800^2 on GB300, two CTAs per SM)
    const size_t slice = sizeof(float) * (size_t)((npix + nblocks - 1) / nblocks);
    bool smem_res = false;
    if (slice <= CL_SMEM_SLICE_MAX) {
        int fit = 0;
        SDE_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_hogbom<true>, CL_THREADS, slice));
        smem_res = (int64_t)fit * ctx->num_sms >= nblocks;
    }
    SDE_TRY(ctx_scratch(ctx, "cl_bar", sizeof(Barrier), (void **)&A.bar));
    SDE_CUDA_TRY(cudaMemsetAsync(A.bar, 0, sizeof(Barrier), ctx->stream));
    void *args[] = {&A};
    KTimer kt(ctx, "hogbom");
    if (smem_res)
        SDE_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_hogbom<true>, dim3(nblocks), dim3(CL_THREADS),
                                                 args, slice, ctx->stream));
    else
        SDE_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_hogbom<false>, dim3(nblocks), dim3(CL_THREADS),
                                                 args, 0, ctx->stream));
    int stopped;
    SDE_TRY(clean_result(ctx, dout, out, &stopped));
    if (stopped == 2) return SDE_ECANCELLED;
    return SDE_OK;
}

// ---------------------------------------------------------------------------------------
// Hogbom CLEAN without any device allocation.
//
// Some callers cannot call cudaMalloc: code that owns all device memory through its own
// allocator or a fixed arena, embedded/real-time hosts that forbid allocation after start-up,
// and serving loops that must not block on the allocator.  For them this entry point runs the
// same minor cycle as sde_hogbom on arrays the caller already holds, keeping its scratch --
// the per-CTA partial maxima of the PSF-peak search, the grid barrier with the iterations'
// maxima, the status words and the result scalars -- in one file-scope device array of fixed
// size.  That array exists on every GPU that loads the library, for the life of the process.
namespace {
constexpr int NOALLOC_MAX_CTAS = 1024;  // CTAs of the PSF-peak search and of CLEAN (~12 KB in all)
struct NoAllocScratch {
    Cand isa_part[NOALLOC_MAX_CTAS];
    int64_t isa_out;
    Barrier bar;
    int status[STATUS_COUNT];
    float out[4];
};
}  // namespace

static __device__ __align__(256) NoAllocScratch g_clean_scratch;

// Host-side copies of g_clean_scratch's device address, one per device.  The array's name in
// host code only stands in for the symbol; the address every kernel receives comes from
// cudaGetSymbolAddress, taken with that device current the first time the device is used.
// It is taken again when the device's current context has changed since (a caller's
// cudaDeviceReset destroys the primary context, and the next one loads the module, and with
// it the array, anew -- possibly at another address).
static NoAllocScratch *g_clean_scratch_dev[64];
static unsigned long long g_clean_scratch_ctx[64];
static std::mutex g_clean_scratch_mu;

// unique ID of the calling thread's current CUDA context (driver API, resolved at run time)
static int current_context_id(unsigned long long *id) {
    typedef CUresult (*GetCurrentFn)(CUcontext *);
    typedef CUresult (*GetIdFn)(CUcontext, unsigned long long *);
    static GetCurrentFn get_current = nullptr;
    static GetIdFn get_id = nullptr;
    if (!get_current || !get_id) {
        void *a = nullptr, *b = nullptr;
        cudaDriverEntryPointQueryResult qa, qb;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &a, 12000, cudaEnableDefault, &qa) !=
                cudaSuccess ||
            cudaGetDriverEntryPointByVersion("cuCtxGetId", &b, 12000, cudaEnableDefault, &qb) !=
                cudaSuccess ||
            qa != cudaDriverEntryPointSuccess || qb != cudaDriverEntryPointSuccess || !a || !b) {
            sde_set_error("sde_hogbom_noalloc: driver context queries unavailable");
            return SDE_ECUDA;
        }
        get_current = (GetCurrentFn)a;
        get_id = (GetIdFn)b;
    }
    CUcontext c = nullptr;
    if (get_current(&c) != CUDA_SUCCESS || !c || get_id(c, id) != CUDA_SUCCESS) {
        sde_set_error("sde_hogbom_noalloc: no current CUDA context");
        return SDE_ECUDA;
    }
    return SDE_OK;
}

static int clean_scratch_address(int dev, NoAllocScratch **out) {
    if (dev < 0 || dev >= 64) {
        sde_set_error("sde_hogbom_noalloc: device %d out of range", dev);
        return SDE_EINVAL;
    }
    // make the device's primary context current on this thread (no allocation)
    SDE_CUDA_TRY(cudaSetDevice(dev));
    unsigned long long id = 0;
    SDE_TRY(current_context_id(&id));
    std::lock_guard<std::mutex> lk(g_clean_scratch_mu);
    if (!g_clean_scratch_dev[dev] || g_clean_scratch_ctx[dev] != id) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_clean_scratch);
        if (e != cudaSuccess || !p) {
            sde_set_error("sde_hogbom_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            return e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver ? SDE_ENODEV : SDE_ECUDA;
        }
        g_clean_scratch_dev[dev] = (NoAllocScratch *)p;
        g_clean_scratch_ctx[dev] = id;
    }
    *out = g_clean_scratch_dev[dev];
    return SDE_OK;
}

extern "C" int sde_hogbom_noalloc(void *stream, const float *drt, const float *psf,
                                  const float *box, int nx, int ny, int pnx, int pny, float gain,
                                  int nsub, int bsub, float flux, float tflux_in, float *cln,
                                  float *res, float *cflux, int *cx, int *cy,
                                  volatile int *cancel_flag, sde_clean_result *out) {
    if (!drt || !psf || !cln || !res || !out || nx < 1 || ny < 1 || pnx < 1 || pny < 1 || bsub < 1) {
        sde_set_error("sde_hogbom_noalloc: bad arguments");
        return SDE_EINVAL;
    }
    if ((int64_t)nx * ny > INT32_MAX || (int64_t)pnx * pny > INT32_MAX) {
        sde_set_error("sde_hogbom_noalloc: window %dx%d or PSF %dx%d exceeds 2^31-1 pixels", nx, ny,
                      pnx, pny);
        return SDE_EINVAL;
    }
    const int nabs = nsub < 0 ? -nsub : nsub;
    if (nabs >= bsub && (!cflux || !cx || !cy)) {
        sde_set_error("sde_hogbom_noalloc: component arrays required");
        return SDE_EINVAL;
    }
    cudaStream_t st = (cudaStream_t)stream;
    int dev = 0, nsm = 0;
    SDE_CUDA_TRY(cudaGetDevice(&dev));
    SDE_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    NoAllocScratch *S = nullptr;
    SDE_TRY(clean_scratch_address(dev, &S));
    // PSF peak (pix/pix2drcl.f:73-80) with the partials in the static array
    int nbi = nsm * 2;
    if (nbi > NOALLOC_MAX_CTAS) nbi = NOALLOC_MAX_CTAS;
    k_isamax_part<<<nbi, CL_THREADS, 0, st>>>(psf, (int64_t)pnx * pny, S->isa_part);
    SDE_CHECK_LAUNCH();
    k_isamax_final<<<1, CL_THREADS, 0, st>>>(S->isa_part, nbi, &S->isa_out);
    SDE_CHECK_LAUNCH();
    int64_t ip1 = 0;
    SDE_CUDA_TRY(cudaMemcpyAsync(&ip1, &S->isa_out, sizeof ip1, cudaMemcpyDeviceToHost, st));
    SDE_CUDA_TRY(cudaStreamSynchronize(st));
    if (ip1 == 0) ip1 = 1;  // PIXISAMA's default I = 1
    const int ipeak = (int)(ip1 - 1);
    int pmpx = 1 + ipeak % pnx;
    int pmpy = 1 + (ipeak - pmpx + 1) / pnx;
    if (pmpx >= pnx) pmpx = pnx / 2;
    if (pmpy >= pny) pmpy = pny / 2;
    int per_sm = 0;
    SDE_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_hogbom<false>, CL_THREADS, 0));
    if (per_sm < 1) {
        sde_set_error("sde_hogbom_noalloc: kernel cannot be resident");
        return SDE_ECUDA;
    }
    const int64_t npix = (int64_t)nx * ny;
    int nblocks = nsm * (per_sm > 2 ? 2 : per_sm);
    const int64_t want = (npix + 4 * CL_THREADS - 1) / (4 * CL_THREADS);
    if (want < nblocks) nblocks = (int)(want < 1 ? 1 : want);
    if (nblocks > NOALLOC_MAX_CTAS) nblocks = NOALLOC_MAX_CTAS;
    // the array keeps the previous call's contents: clear what must start at zero
    SDE_CUDA_TRY(cudaMemsetAsync(&S->bar, 0, sizeof(Barrier), st));
    SDE_CUDA_TRY(cudaMemsetAsync(S->status, 0, sizeof(S->status), st));
    SDE_CUDA_TRY(cudaMemsetAsync(S->out, 0, sizeof(S->out), st));
    CleanArgs A;
    A.drt = drt; A.psf = psf; A.box = box; A.cln = cln; A.res = res; A.cflux = cflux;
    A.cx = cx; A.cy = cy; A.nx = nx; A.ny = ny; A.pnx = pnx; A.pny = pny;
    A.pmpx = pmpx; A.pmpy = pmpy; A.gain = gain; A.flux = flux; A.tflux_in = tflux_in;
    A.nsub = nsub; A.bsub = bsub; A.cancel = cancel_flag; A.bar = &S->bar;
    A.status = S->status; A.out = S->out;
    void *args[] = {&A};
    SDE_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_hogbom<false>, dim3(nblocks), dim3(CL_THREADS),
                                             args, 0, st));
    float h[4];
    int hs[STATUS_COUNT];
    SDE_CUDA_TRY(cudaMemcpyAsync(h, S->out, sizeof h, cudaMemcpyDeviceToHost, st));
    SDE_CUDA_TRY(cudaMemcpyAsync(hs, S->status, sizeof hs, cudaMemcpyDeviceToHost, st));
    SDE_CUDA_TRY(cudaStreamSynchronize(st));
    if (hs[STATUS_TIMEOUT]) {
        sde_set_error("sde_hogbom_noalloc: grid barrier timed out");
        return SDE_ETIMEDOUT;
    }
    int ansub, stopped;
    memcpy(&ansub, &h[2], 4);
    memcpy(&stopped, &h[3], 4);
    out->maxres = h[0];
    out->tflux = h[1];
    out->ansub = ansub;
    if (stopped == 2) return SDE_ECANCELLED;
    return SDE_OK;
}
