// plan.cu -- builds a resident, tile- and chunk-sorted visibility set (sde_plan).
//
// For every visibility the plan evaluates, once, the cell placement that GRDH2D uses (FP64,
// grd/grdh2d.f:114-166) and the one GRDDEH2D uses (FP32 cell from FP64 coordinates,
// grd/grddeh2d.f:92-118), with the reference's results: its exact operations, or FP32
// arithmetic whose error bound decides the same roundings (geom.cuh).  Visibilities are
// then sorted by (uv tile, cell), split into same-cell chunks of <= CHUNK_MAX, and the
// chunks of each work item are ordered by (length, 7x7 colour class, chunk index, place) so that
// the 32 chunks a warp flushes at once never overlap; the plan stores the visibilities in
// that chunk order, so a team's concurrent chunks read one contiguous range.  The observed
// visibilities are stored already rotated/conjugated into the gridding frame (FVIS of
// grd/grdh2d.f:125-143), so the per-cycle kernels carry no FP64 or trigonometric work.
#include <math.h>
#include <string.h>

#include "common.cuh"
#include "geom.cuh"
#include "lookback.cuh"

namespace {

using namespace sde_geom;

constexpr int LENBIN_BITS = 3;  // coarse length bins above the colour class in the chunk order

// Bit 0 of a caller-order degridding word (a table byte offset, a multiple of 128, is even
// there) carries the gridding-frame conjugation (the plan's own words leave it clear).
constexpr uint32_t GDD_GCONJ_U = 1u;
static_assert(TAPROW_BYTES % 2 == 0, "bit 0 of a degridding word is free");

// A visibility's plan data in caller order, one 32-byte sector: the plan record {WT, the
// gridder's tap-table offsets, observed value in the gridding frame}, the degridding word
// (with the gridding-frame conjugation in bit 0), the rotation and, for an exception, its
// place in the exception list.  The gather into sorted
// order reads one sector per visibility.
struct __align__(32) PlanRecU {
    float4 rec;
    uint32_t gdd;
    float rc, rs;
    uint32_t exc_slot;  // the visibility's place in the exception list (exceptions only)
};

// What the build reads back and what must start at zero: the visibility counts, the control
// words of the two scans below, and (following this) their tiles' look-back words.
struct ScanCtl {
    unsigned long long total;
    uint32_t next, pad;
};
struct PlanCounts {
    unsigned long long ngrid, nexc, npos, exc_next;  // gridded, exceptions, WT > 0, list slots taken
    unsigned long long fail;                         // a device wait gave up
    ScanCtl runs, emit;                              // totals: runs; chunks | items << 31
    unsigned long long pad;
};
constexpr int SC_T = 256, SC_R = 4;  // 1024 entries a scan tile
int64_t scan_tiles(int64_t n) { return n / (SC_T * SC_R) + 1; }

// Per visibility (caller order): gridding key, the PlanRecU sector and, for an exception, its
// entry in the exception list, from both routines' geometry (geom_vis).  GE_PER visibilities a
// thread, their loads in flight together (64.7 million: one a thread, its value and coordinates
// read once its weight was known, 1.19 ms; here 0.91).
constexpr int GE_T = 256, GE_PER = 2;
__device__ __forceinline__ void store_rec(PlanRecU *r, const PlanRecU &v) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(r), "f"(v.rec.x), "f"(v.rec.y),
                 "f"(v.rec.z), "f"(v.rec.w), "r"(v.gdd), "f"(v.rc), "f"(v.rs), "r"(v.exc_slot)
                 : "memory");
}
__global__ void __launch_bounds__(GE_T) k_plan_geom(GParams p, const float *__restrict__ u, const float *__restrict__ v,
                            const float *__restrict__ w, const float2 *__restrict__ vis,
                            const float *__restrict__ wt, int64_t n, uint32_t *keys,
                            PlanRecU *rec_u, uint32_t *exc_list,
                            PlanCounts *counts) {
    const int64_t i0 = (int64_t)blockIdx.x * (GE_T * GE_PER) + threadIdx.x;
    uint32_t nvalid = 0, nexc = 0, npos = 0;
    float wts[GE_PER], us[GE_PER], vs[GE_PER], ws[GE_PER];
    float2 vals[GE_PER];
#pragma unroll
    for (int j = 0; j < GE_PER; j++) {
        const int64_t i = min(i0 + j * GE_T, n - 1);
        wts[j] = wt[i];
        us[j] = u[i];
        vs[j] = v[i];
        ws[j] = w[i];
        vals[j] = vis[i];
    }
#pragma unroll
    for (int j = 0; j < GE_PER; j++) {
        const int64_t i = i0 + j * GE_T;
        if (i >= n) break;
        const float wi = wts[j];
        uint32_t key = KEY_INVALID, pdd = 0, tw = 0;
        float2 f = make_float2(0.f, 0.f), r = make_float2(1.f, 0.f);
        uint8_t gc = 0;
        if (wi > 0.0f) {
            npos++;
            const GGeo g = geom_vis(p, us[j], vs[j], ws[j], vals[j].x, vals[j].y);
            const DGeo &dg = g.dg;
            gc = g.gc ? 1 : 0;
            r = make_float2(g.rc, g.rs);
            const int nuc = g.nuc, nvc = g.nvc;
            const bool gvalid = g.sane && !(nuc + 2 * p.supp > p.nu) && !(nvc + p.supp > p.nv) && !(nvc - p.supp < 1);
            if (gvalid) {
                const int dug = g.dug, dvg = g.dvg;
                int ucen = nuc + p.supp, vcen = nvc;  // 1-based, gridding frame
                int tu = (ucen - 1) >> TILE_LOG2, lu = (ucen - 1) & (TILE - 1);
                int tv = (vcen - 1) >> TILE_LOG2, lv = (vcen - 1) & (TILE - 1);
                key = ((uint32_t)(tv * p.ntu + tu) << 12) | ((uint32_t)lv << 6) | (uint32_t)lu;
                // GRDDEH2D's reflection branch (NUD <= SUPP) reads conj(G(-u, 2*VORIGIN - v))
                // left of the v axis; the tiled degridder holds those values in the u = 0
                // tile's halo, so the branch stays in the tiled path when every mirrored
                // row lies inside the grid (else the reference skips taps: exception)
                const bool refl_tiled = p.uorigin == 1 && 2 * p.vorigin - (dg.nvd + p.supp) >= 1 &&
                                        2 * p.vorigin - (dg.nvd - p.supp) <= p.nv;
                bool exc = !dg.valid || dg.nud != nuc || dg.nvd != nvc ||
                           (dg.nud <= p.supp && !refl_tiled) || dg.conj != (gc != 0);
                // column of the cell within its chunk's cell pair (chunks start on even lu)
                const uint32_t off = (uint32_t)lu & 1u;
                tw = taps_word(dug, dvg, off);
                pdd = exc ? (taps_word(0, 0, off) | GDD_EXCEPTION) : taps_word(dg.dui, dg.dvi, off);
                nvalid++;
                nexc += exc;
                f = make_float2(g.fr, g.fi);
            } else {
                nexc++;  // degrid-only or degrid-invalid: exception path
            }
        }
        keys[i] = key;
        PlanRecU pr;
        pr.rec = make_float4(wi, __uint_as_float(tw), f.x, f.y);
        pr.gdd = pdd | (gc ? GDD_GCONJ_U : 0u);
        pr.rc = r.x;
        pr.rs = r.y;
        pr.exc_slot = 0;
        // GRDDEH2D's exception path takes the visibilities with WT > 0 that do not grid or
        // whose degridding cell is not the gridding cell: appended to the list (a few in 10^4;
        // the list's order does not matter, each is degridded on its own)
        if (wi > 0.0f && (key == KEY_INVALID || (pdd & GDD_EXCEPTION) != 0)) {
            pr.exc_slot = (uint32_t)atomicAdd(&counts->exc_next, 1ull);
            exc_list[pr.exc_slot] = (uint32_t)i;
        }
        store_rec(rec_u + i, pr);
    }
    // block-aggregated counters (one atomic per block and counter: per-warp atomics on three
    // addresses serialise in L2 at this visibility count)
    __shared__ uint32_t sum[3];
    if (threadIdx.x < 3) sum[threadIdx.x] = 0;
    __syncthreads();
    nvalid = __reduce_add_sync(0xffffffffu, nvalid);
    nexc = __reduce_add_sync(0xffffffffu, nexc);
    npos = __reduce_add_sync(0xffffffffu, npos);
    if ((threadIdx.x & 31) == 0) {
        if (nvalid) atomicAdd(&sum[0], nvalid);
        if (nexc) atomicAdd(&sum[1], nexc);
        if (npos) atomicAdd(&sum[2], npos);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (sum[0]) atomicAdd(&counts->ngrid, (unsigned long long)sum[0]);
        if (sum[1]) atomicAdd(&counts->nexc, (unsigned long long)sum[1]);
        if (sum[2]) atomicAdd(&counts->npos, (unsigned long long)sum[2]);
    }
}

// Gather the per-visibility data into the plan's order (one 32-byte sector read per
// visibility): a block takes GA_CHUNKS consecutive chunks, whose visibilities are one
// contiguous range of the output, and its threads take the range's positions, finding the
// chunk of a position by bisection of the chunks' starts; the reads of GA_BATCH positions are
// in flight together (64.7 million visibilities: 1.80 ms by a warp per chunk, whose 27
// visibilities are one round, here 1.61).  An exception that also grids learns its
// position here.
__device__ __forceinline__ PlanRecU load_rec(const PlanRecU *r) {
    PlanRecU v;  // one 32-byte load
    asm("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v.rec.x), "=f"(v.rec.y), "=f"(v.rec.z), "=f"(v.rec.w), "=r"(v.gdd), "=f"(v.rc), "=f"(v.rs),
          "=r"(v.exc_slot)
        : "l"(r));
    return v;
}
constexpr int GA_CHUNKS = 64, GA_BATCH = 4, GA_T = 256;
__global__ void __launch_bounds__(GA_T) k_plan_gather(const uint32_t *__restrict__ perm,
                                                      const uint2 *__restrict__ chunks,
                                                      const uint32_t *__restrict__ csrc, int64_t nchunks,
                                                      const PlanRecU *__restrict__ rec_u, float2 *fobs,
                                                      float4 *rec, float *wt, uint32_t *gdd, uint32_t *orig,
                                                      float2 *rot, uint8_t *gconj, DegridExc *exc) {
    __shared__ uint32_t to[GA_CHUNKS + 1], from[GA_CHUNKS];
    const int t = threadIdx.x;
    const int64_t c0 = (int64_t)blockIdx.x * GA_CHUNKS;
    const int nc = (int)min((int64_t)GA_CHUNKS, nchunks - c0);
    if (t < nc) {
        const uint2 ch = chunks[c0 + t];
        to[t] = ch.x;
        from[t] = csrc[c0 + t];
        if (t == nc - 1) to[nc] = ch.x + (ch.y >> 16);
    }
    __syncthreads();
    const uint32_t end = to[nc];
    for (uint32_t p0 = to[0] + t; p0 < end; p0 += GA_BATCH * GA_T) {
        uint32_t src[GA_BATCH];
#pragma unroll
        for (int j = 0; j < GA_BATCH; j++) {
            const uint32_t p = p0 + j * GA_T;
            if (p >= end) break;
            int lo = 0, hi = nc;  // the last chunk that starts at or before p
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (to[mid] <= p) lo = mid; else hi = mid;
            }
            src[j] = perm[from[lo] + (p - to[lo])];
        }
        PlanRecU pr[GA_BATCH];
#pragma unroll
        for (int j = 0; j < GA_BATCH; j++)
            if (p0 + j * GA_T < end) pr[j] = load_rec(rec_u + src[j]);
#pragma unroll
        for (int j = 0; j < GA_BATCH; j++) {
            const uint32_t p = p0 + j * GA_T;
            if (p >= end) break;
            const float4 r = pr[j].rec;
            const uint32_t d = pr[j].gdd;
            rec[p] = r;
            fobs[p] = make_float2(r.z, r.w);
            wt[p] = r.x;
            gdd[p] = d & ~GDD_GCONJ_U;
            orig[p] = src[j];
            gconj[p] = (d & GDD_GCONJ_U) ? 1 : 0;
            if (rot) rot[p] = make_float2(pr[j].rc, pr[j].rs);
            if ((d & GDD_EXCEPTION) && exc) exc[pr[j].exc_slot].pos = (int32_t)p;
        }
    }
}

// The exception list's entries, one thread per exception (pos is set by k_plan_gather for the
// exceptions that also grid).
__global__ void k_exc_write(GParams p, const float *__restrict__ u, const float *__restrict__ v,
                            const float *__restrict__ w, const float *__restrict__ wt,
                            const PlanRecU *__restrict__ rec_u, const uint32_t *__restrict__ exc_list,
                            int64_t nexc, DegridExc *exc, float *exc_wt, float2 *exc_rot) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nexc) return;
    const uint32_t i = exc_list[s];
    DGeo g = p.fast ? degrid_geom_fast(p, u[i], v[i]) : degrid_geom(p, u[i], v[i], w[i]);
    DegridExc e;
    e.orig = i;
    e.pos = -1;
    e.nuc = g.nud;
    e.nvc = g.nvd;
    e.delui = (int16_t)g.dui;
    e.delvi = (int16_t)g.dvi;
    e.conj = g.conj;
    e.valid = g.valid;
    e.gconj = (rec_u[i].gdd & GDD_GCONJ_U) ? 1 : 0;
    e.pad = 0;
    exc[s] = e;
    exc_wt[s] = wt[i];
    exc_rot[s] = make_float2(g.rc, g.rs);
}

// Runs, work items and chunks from the sorted keys.  A run is one cell pair of one tile
// (equal key >> 1); a tile's visibilities split into work items at every item_max from the
// tile's first one; a run's part within one item (a piece) splits into chunks of chunk_max
// from the piece's start.  Chunks and items are numbered in position order.
//
// The runs' starts, compacted, and the first visibility of every tile that has one.  A warp
// takes RU_R rounds of 32 consecutive keys; heads are counted by ballots, so the keys stay in
// registers.
constexpr int RU_T = 512, RU_R = 16;  // 8192 keys a scan tile
__global__ void __launch_bounds__(RU_T) k_runs(const uint32_t *__restrict__ keys, PlanCounts *counts, int64_t n,
                                               unsigned long long *words, uint32_t *rstart, uint32_t *tstart,
                                               int limit) {
    __shared__ uint32_t wsum[RU_T / 32];
    __shared__ unsigned long long before;
    __shared__ uint32_t stile;
    __shared__ bool failed;
    const int64_t nv = (int64_t)counts->ngrid;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) {
        stile = atomicAdd(&counts->runs.next, 1u);
        failed = *(volatile unsigned long long *)&counts->fail != 0;
    }
    __syncthreads();
    // the sort gave up: its keys index nothing (one thread reads the word for the block, as
    // another block's look-back may set it at any moment)
    if (failed) return;
    const int64_t tile = stile, base = tile * (RU_T * RU_R), w0 = base + (int64_t)warp * 32 * RU_R;
    uint32_t key[RU_R], mask[RU_R];
#pragma unroll
    for (int r = 0; r < RU_R; r++) {
        const int64_t q = w0 + r * 32 + lane;
        key[r] = q < nv ? keys[q] : 0u;
    }
    uint32_t prev = w0 > 0 && w0 <= nv ? keys[w0 - 1] : 0u;  // (lane 0's) the key before the round
    uint32_t sum = 0;
#pragma unroll
    for (int r = 0; r < RU_R; r++) {
        const int64_t q = w0 + r * 32 + lane;
        uint32_t p = __shfl_up_sync(0xffffffffu, key[r], 1);
        if (lane == 0) p = prev;
        prev = __shfl_sync(0xffffffffu, key[r], 31);
        mask[r] = __ballot_sync(0xffffffffu, q < nv && (q == 0 || (p >> 1) != (key[r] >> 1)));
        sum += __popc(mask[r]);
    }
    if (lane == 0) wsum[warp] = sum;
    __syncthreads();
    uint32_t pre = 0, all = 0;
#pragma unroll
    for (int w = 0; w < RU_T / 32; w++) {
        pre += w < warp ? wsum[w] : 0u;
        all += wsum[w];
    }
    if (t == 0) {
        unsigned long long b = 0;
        if (tile > 0) {
            lb_publish(&words[tile], LB_AGG, all);
            b = lb_sum_before(words, tile, 1, &counts->fail, limit);
        }
        lb_publish(&words[tile], LB_PREFIX, b + all);
        before = b;
        if (base + RU_T * RU_R >= n) counts->runs.total = b + all;
    }
    __syncthreads();
    uint32_t at = (uint32_t)before + pre;
#pragma unroll
    for (int r = 0; r < RU_R; r++) {
        const int64_t q = w0 + r * 32 + lane;
        if ((mask[r] >> lane) & 1u) {
            const uint32_t o = at + __popc(mask[r] & ((1u << lane) - 1u));
            if (o < (uint64_t)n) rstart[o] = (uint32_t)q;
            if (q == 0 || (keys[q - 1] >> 12) != (key[r] >> 12)) tstart[key[r] >> 12] = (uint32_t)q;
        }
        at += __popc(mask[r]);
    }
}

// A run's pieces: piece(a, b, starts_item) for each.
template <class F>
__device__ __forceinline__ void run_pieces(int64_t rs, int64_t re, int64_t ts, int item_max, F piece) {
    for (int64_t a = rs; a < re;) {
        const int64_t is = ts + (a - ts) / item_max * item_max;
        const int64_t b = min(re, is + item_max);
        piece(a, b, is == a);
        a = b;
    }
}

// The runs' chunks and the items that start in them, numbered by a scan of both counts (31
// bits each).  A chunk's entry: where its visibilities are in the sort's order, its even cell
// and length, and its sort key within the item, in bits from the top: a coarse length bin
// (LENBIN_BITS, longest first), the colour class, the length class, the chunk index, the window's
// place among its colour's and (16 bits) its number in the item.  The 8 chunks that a warp of the gridder or degridder takes
// together then have similar lengths (the warp runs to its longest) and mostly one colour.  On
// the large single field the lanes do useful work in 94% of the warps' visibility slots with 8
// bins, 81% with the colour class alone above the length (a simulation of both orders on its
// chunks; measured: gridder 0.82 -> 0.75 ms).
__global__ void __launch_bounds__(SC_T) k_run_emit(const uint32_t *__restrict__ keys, PlanCounts *counts,
                                                   const uint32_t *__restrict__ rstart,
                                                   const uint32_t *__restrict__ tstart, int64_t nruns,
                                                   int item_max, int chunk_max, int lbits, int jbits,
                                                   int64_t max_items, int64_t max_chunks, int limit,
                                                   unsigned long long *words,
                                                   uint64_t *ckey, uint2 *craw, WorkItem *items) {
    const int64_t nvalid = (int64_t)counts->ngrid;
    auto run_end = [&](int64_t r) { return r + 1 < nruns ? (int64_t)rstart[r + 1] : nvalid; };
    auto in = [&](int64_t r) -> unsigned long long {
        const int64_t rs = rstart[r];
        unsigned long long c = 0, h = 0;
        run_pieces(rs, run_end(r), tstart[keys[rs] >> 12], item_max, [&](int64_t a, int64_t b, bool starts) {
            h += starts;
            c += (unsigned long long)((b - a + chunk_max - 1) / chunk_max);
        });
        return c | (h << 31);
    };
    // a piece's chunks step threads at a time from the first-th; bits above the chunk index
    auto piece_chunks = [&](uint32_t cell, int64_t c, int64_t a, int64_t b, int first, int step) {
        const uint32_t lu = cell & 63u, lv = cell >> 6;
        const uint64_t color = ((lu >> 1) & 3u) * 7u + (lv % 7u);
        // the windows of a colour, so that neighbours differ in banks (TROW, grid.cu): four in a
        // row cover n mod 2 and m mod 2, eight n mod 4 as well (64.7 million visibilities, gridding:
        // 704 -> 689 us with the row stride; 10 million on 2048^2 197 -> 191)
        const uint32_t n = lu >> 3, m = lv / 7u;
        const uint64_t place = (m >> 1) << 4 | (n >> 2) << 3 | (n >> 1 & 1u) << 2 | (m & 1u) << 1 | (n & 1u);
        const int nc = (int)((b - a + chunk_max - 1) / chunk_max);
        for (int j = first; j < nc; j += step) {
            const int64_t q = a + (int64_t)j * chunk_max;
            const int len = (int)min((int64_t)chunk_max, b - q), cls = chunk_max - len;
            const int bin = min(cls * (1 << LENBIN_BITS) / chunk_max, (1 << LENBIN_BITS) - 1);
            ckey[c + j] = (((((((uint64_t)bin << 6) | color) << lbits) | (uint64_t)cls) << jbits) | (uint64_t)j) << 7 | place;
            craw[c + j] = make_uint2((uint32_t)q, cell | ((uint32_t)len << 16));
        }
        return nc;
    };
    // A run of more than EM_LONG chunks is left to a warp (a dense cell's has thousands).
    constexpr int EM_LONG = 4;
    struct LongRun {
        uint32_t rs, re, ts, cell, chunk;
    };
    __shared__ LongRun lrun[SC_T * SC_R];
    __shared__ int nlong;
    if (threadIdx.x == 0) nlong = 0;
    auto out = [&](int64_t r, unsigned long long cnt, unsigned long long before) {
        const int64_t rs = rstart[r];
        const uint32_t k = keys[rs];
        int64_t c = (int64_t)(before & 0x7FFFFFFFull), nit = (int64_t)(before >> 31);
        const int64_t nc = (int64_t)(cnt & 0x7FFFFFFFull);
        // (sums of a look-back that gave up: nothing is written outside the arrays)
        if (c + nc > max_chunks || nit + (int64_t)(cnt >> 31) > max_items) return;
        const bool is_long = nc > EM_LONG;
        const int64_t re = run_end(r), ts = tstart[k >> 12];
        if (is_long)
            lrun[atomicAdd(&nlong, 1)] = LongRun{(uint32_t)rs, (uint32_t)re, (uint32_t)ts, k & 4094u, (uint32_t)c};
        run_pieces(rs, re, ts, item_max, [&](int64_t a, int64_t b, bool starts) {
            if (starts) {
                WorkItem wi;
                wi.tile = (int32_t)(k >> 12);
                wi.cbeg = (int32_t)c;
                wi.vbeg = (int32_t)a;
                wi.cend = wi.vend = wi.dense = wi.r0 = 0;
                wi.rstep = 1;
                items[nit++] = wi;
            }
            c += is_long ? (b - a + chunk_max - 1) / chunk_max : piece_chunks(k & 4094u, c, a, b, 0, 1);
        });
    };
    lb_scan_tile<SC_T, SC_R>(nruns, words, &counts->emit.next, &counts->emit.total, &counts->fail, limit, in,
                             out);
    __syncthreads();
    for (int e = threadIdx.x >> 5; e < nlong; e += SC_T / 32) {
        const LongRun r = lrun[e];
        int64_t c = r.chunk;
        run_pieces(r.rs, r.re, r.ts, item_max,
                   [&](int64_t a, int64_t b, bool) { c += piece_chunks(r.cell, c, a, b, threadIdx.x & 31, 32); });
    }
}

// Raw-grid cores of the compensation plane: the footprint of a tile (tu, tv) (its 64x64
// cells and 3-cell halo, raw rows [64 tv - 3, 64 tv + 67), raw indices [64 tu - 2,
// 64 tu + 68)) lies in cores (tu, tv), (tu+1, tv), (tu, tv+1), (tu+1, tv+1), where core
// (cu, cv) is raw rows [64 cv - 3, 64 cv + 61) x raw indices [64 cu - 2, 64 cu + 62).
// (core starts on a 4-byte boundary, and its last word is the plan's)
__device__ __forceinline__ void mark_cores(int tile, int ntu, uint8_t *core, unsigned mark) {
    const int tu = tile % ntu, tv = tile / ntu, ncu = ntu + 1;
    uint32_t *words = reinterpret_cast<uint32_t *>(core);
    const int at[4] = {tv * ncu + tu, tv * ncu + tu + 1, (tv + 1) * ncu + tu, (tv + 1) * ncu + tu + 1};
#pragma unroll
    for (int k = 0; k < 4; k++) atomicOr(&words[at[k] >> 2], mark << (8 * (at[k] & 3)));
}

// Each item's ends, its dense flag (its tile's items, contiguous, hold >= DENSE_TILE_VIS
// visibilities together), the cores of a dense tile, and its entries of the launch list:
// every item once, or once per part with its rounds dealt out.  Where no item is larger than a
// part the list is the items in their own order, neighbouring tiles together (64.7 million
// visibilities, gridding in an order that the blocks' timing made: 700 -> 727 us); smaller
// plans' entries are appended in any order.
__global__ void k_item_finish(WorkItem *items, int64_t nitems, int64_t nchunks, int64_t nvalid, int ntu, uint8_t *core,
                              int item_max, int part, WorkItem *parts,
                              unsigned long long *nparts) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nitems) return;
    const int32_t tile = items[t].tile;
    int64_t lo = 0, hi = t;  // first item of the tile
    while (lo < hi) {
        const int64_t mid = (lo + hi) / 2;
        if (items[mid].tile < tile) lo = mid + 1; else hi = mid;
    }
    const int64_t first = lo;
    lo = t;
    hi = nitems;  // one past the last item of the tile
    while (lo < hi) {
        const int64_t mid = (lo + hi) / 2;
        if (items[mid].tile <= tile) lo = mid + 1; else hi = mid;
    }
    const int64_t end = lo < nitems ? items[lo].vbeg : nvalid;
    WorkItem it = items[t];
    it.cend = t + 1 < nitems ? items[t + 1].cbeg : (int32_t)nchunks;
    it.vend = t + 1 < nitems ? items[t + 1].vbeg : (int32_t)nvalid;
    it.dense = end - items[first].vbeg >= DENSE_TILE_VIS;
    items[t].cend = it.cend;
    items[t].vend = it.vend;
    items[t].dense = it.dense;
    // parts add to the same cells as items of a dense tile do: their sums are compensated too
    // (84 240 visibilities on 512^2, two runs' PSFs apart: 2.4e-4 without, 8e-5 with, 1.6e-4 with
    // whole items; gridding 27.6 -> 28.1 us)
    const int np = item_max <= part ? 1 : item_parts(it, part);
    if (it.dense || np > 1) mark_cores(tile, ntu, core, it.dense ? CORE_DENSE : CORE_PARTS);
    if (np > 1) it.dense = 1;
    const unsigned long long at =
        item_max <= part ? (unsigned long long)t : atomicAdd(nparts, (unsigned long long)np);
    if (item_max <= part && t == 0) *nparts = (unsigned long long)nitems;
    it.rstep = np;
    for (int k = 0; k < np; k++) {
        it.r0 = k;
        parts[at + k] = it;
    }
}

// One block per work item: its chunks sorted by their keys in shared memory (bitonic), and
// their places in the plan, which follow one another from the item's first visibility.  An
// item has at most 2048 cell pairs and item_max / chunk_max longer runs' chunks, so with the
// default sizes every item fits; one with more than OR_MAX chunks keeps position order.  The
// device-wide radix sort of 64-bit keys that this replaces took 7 passes of 5 launches.
constexpr int OR_MAX = 4096, OR_T = 256;
__global__ void __launch_bounds__(OR_T) k_item_order(const WorkItem *__restrict__ items, int64_t nitems,
                                                     const uint64_t *__restrict__ ckey,
                                                     const uint2 *__restrict__ craw, uint2 *chunks, uint32_t *csrc) {
    __shared__ uint64_t sk[OR_MAX];
    __shared__ uint32_t wsum[OR_T / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const WorkItem it = items[blockIdx.x];
    const int m = it.cend - it.cbeg;
    const bool sorted = m <= OR_MAX;
    if (sorted) {
        int n = 2;
        while (n < m) n <<= 1;
        for (int i = t; i < n; i += OR_T) sk[i] = i < m ? (ckey[it.cbeg + i] << 16) | (uint32_t)i : ~0ull;
        __syncthreads();
        for (int k = 2; k <= n; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = t; i < n / 2; i += OR_T) {
                    const int a = 2 * i - (i & (j - 1)), b = a + j;  // the pair (a, a ^ j), a's bit j clear
                    const uint64_t x = sk[a], y = sk[b];
                    if ((x > y) == ((a & k) == 0)) {
                        sk[a] = y;
                        sk[b] = x;
                    }
                }
                // pairs closer than a warp's span stay in the warp's own stretch
                if (j > 32 || (j == 1 && k < n)) __syncthreads(); else __syncwarp();
            }
        __syncthreads();
    }
    uint32_t at = (uint32_t)it.vbeg;
    for (int base = 0; base < m; base += OR_T) {
        const int p = base + t;
        uint2 c = make_uint2(0u, 0u);
        if (p < m) c = craw[it.cbeg + (sorted ? (int)(sk[p] & 0xFFFFu) : p)];
        const uint32_t len = c.y >> 16;
        uint32_t x = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        uint32_t pre = 0, all = 0;
#pragma unroll
        for (int w = 0; w < OR_T / 32; w++) {
            pre += w < warp ? wsum[w] : 0u;
            all += wsum[w];
        }
        if (p < m) {
            chunks[it.cbeg + p] = make_uint2(at + pre + x - len, c.y);
            csrc[it.cbeg + p] = c.x;
        }
        at += all;
        __syncthreads();
    }
}

int bits_for(int64_t maxval) {
    int b = 1;
    while (b < 63 && ((int64_t)1 << b) <= maxval) b++;
    return b;
}

}  // namespace

int sde_grid_pitch(int nu) { return (nu + 3) & ~3; }

int64_t sde_plan_nvis(const sde_plan *plan) { return plan ? plan->nvis : 0; }
int64_t sde_plan_bytes(const sde_plan *plan) { return plan ? plan->bytes : 0; }
int sde_plan_stats(const sde_plan *plan, int64_t *nitems, int64_t *nchunks, int64_t *nexc) {
    if (!plan) return SDE_EINVAL;
    if (nitems) *nitems = plan->nitems;
    if (nchunks) *nchunks = plan->nchunks;
    if (nexc) *nexc = plan->nexc;
    return SDE_OK;
}

// Several arrays in one allocation, each on a 256-byte boundary.
struct Slab {
    size_t bytes = 0;
    struct Part {
        void **p;
        size_t off;
    };
    std::vector<Part> parts;
    template <class T>
    void add(T **p, size_t n) {
        parts.push_back({reinterpret_cast<void **>(p), bytes});
        bytes += (n + 255) & ~(size_t)255;
    }
    // The size is rounded up by at most 1/16, so that plans of about the same number of
    // visibilities take each other's blocks from the pool: mapping new ones costs milliseconds
    // at 65 M visibilities.
    int alloc(sde_plan *pl, void **base) {
        size_t step = 256;
        while (step * 32 <= bytes) step *= 2;
        bytes = (bytes + step - 1) / step * step;
        SDE_TRY(ctx_alloc(pl->ctx, base, bytes));
        pl->bytes += (int64_t)bytes;
        for (const Part &q : parts) *q.p = static_cast<char *>(*base) + q.off;
        return SDE_OK;
    }
};

int sde_plan_destroy(sde_plan *pl) {
    if (!pl) return SDE_OK;
    sde_ctx *ctx = pl->ctx;
    cudaSetDevice(ctx->device);
    // stream-ordered frees: after the plan's last use on the context's stream
    void *ptrs[] = {pl->slab[0], pl->slab[1], pl->table, pl->wt_all, pl->inv};
    for (void *p : ptrs) ctx_free(ctx, p, 0);
    ctx->bytes -= pl->bytes;
    delete pl;
    return SDE_OK;
}

static int read_counts(sde_ctx *ctx, const PlanCounts *dev, PlanCounts *host) {
    static_assert(sizeof(PlanCounts) <= H_SMALL_BYTES, "counts fit the pinned buffer");
    SDE_TRY(ctx_read_small(ctx, ctx->stream, host, dev, sizeof *host));
    if (host->fail) {
        sde_set_error("plan: a device wait timed out");
        return SDE_ETIMEDOUT;
    }
    return SDE_OK;
}

// Upload (or alias) caller arrays; builds everything described at the top of the file.
int sde_plan_create(sde_ctx *ctx, const sde_gridspec *spec, int64_t nvis, const float *u,
                    const float *v, const float *w, const float *vis, const float *wt,
                    int where, sde_plan **out) {
    return sde_plan_create_opts(ctx, spec, nvis, u, v, w, vis, wt, where, nullptr, out);
}

int sde_plan_create_opts(sde_ctx *ctx, const sde_gridspec *spec, int64_t nvis, const float *u,
                         const float *v, const float *w, const float *vis, const float *wt,
                         int where, const sde_plan_opts *opts, sde_plan **out) {
    if (!ctx || !spec || !out || nvis < 0 || (nvis > 0 && (!u || !v || !w || !vis || !wt))) {
        sde_set_error("sde_plan_create: bad arguments");
        return SDE_EINVAL;
    }
    const int item_max = opts && opts->item_max > 0 ? opts->item_max : ITEM_MAX;
    const int chunk_max = opts && opts->chunk_max > 0 ? opts->chunk_max : CHUNK_MAX;
    if (item_max > ITEM_LIMIT || chunk_max > CHUNK_LIMIT || chunk_max > item_max) {
        sde_set_error("sde_plan_create: work item %d / chunk %d out of range (item <= %d, "
                      "chunk <= %d, chunk <= item)", item_max, chunk_max, ITEM_LIMIT, CHUNK_LIMIT);
        return SDE_EINVAL;
    }
    if (spec->supp != SUPP || spec->osamp != OSAMP) {
        sde_set_error("sde_plan_create: support %d / oversampling %d unsupported (SF needs 3/128)",
                      spec->supp, spec->osamp);
        return SDE_EINVAL;
    }
    if (spec->nu < 2 * SUPP + 1 || spec->nv < 2 * SUPP + 1 || nvis >= (int64_t)0x7FFFFFFF) {
        sde_set_error("sde_plan_create: grid %dx%d / %lld visibilities out of range", spec->nu,
                      spec->nv, (long long)nvis);
        return SDE_EINVAL;
    }
    SDE_CUDA_TRY(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    sde_plan *pl = new sde_plan();
    pl->ctx = ctx;
    pl->spec = *spec;
    pl->doshift = (spec->shift[0] != 1.0) || (spec->shift[4] != 1.0) || (spec->shift[8] != 1.0);
    pl->pitch = plan_pitch(spec->nu);
    pl->ntu = (spec->nu + TILE - 1) / TILE;
    pl->ntv = (spec->nv + TILE - 1) / TILE;
    pl->nvis_in = nvis;
    pl->item_max = item_max;
    pl->chunk_max = chunk_max;
    int rc = SDE_OK;
#define PL_TRY(x)                      \
    do {                               \
        rc = (x);                      \
        if (rc != SDE_OK) goto fail;   \
    } while (0)
#define PL_CUDA(x)                                                                   \
    do {                                                                             \
        cudaError_t _e = (x);                                                        \
        if (_e != cudaSuccess) {                                                     \
            sde_set_error("plan: %s: %s", #x, cudaGetErrorString(_e));               \
            rc = _e == cudaErrorMemoryAllocation ? SDE_ENOMEM : SDE_ECUDA;           \
            goto fail;                                                               \
        }                                                                            \
    } while (0)
    {
        const size_t n = (size_t)(nvis > 0 ? nvis : 1);
        const float *du = u, *dv = v, *dw = w, *dwt = wt;
        const float2 *dvis = (const float2 *)vis;
        if (where == SDE_HOST && nvis > 0) {
            float *bu, *bv, *bw, *bwt;
            float2 *bvis;
            PL_TRY(ctx_scratch(ctx, "pl_u", 4 * n, (void **)&bu));
            PL_TRY(ctx_scratch(ctx, "pl_v", 4 * n, (void **)&bv));
            PL_TRY(ctx_scratch(ctx, "pl_w", 4 * n, (void **)&bw));
            PL_TRY(ctx_scratch(ctx, "pl_wt", 4 * n, (void **)&bwt));
            PL_TRY(ctx_scratch(ctx, "pl_vis", 8 * n, (void **)&bvis));
            PL_CUDA(cudaMemcpyAsync(bu, u, 4 * n, cudaMemcpyHostToDevice, st));
            PL_CUDA(cudaMemcpyAsync(bv, v, 4 * n, cudaMemcpyHostToDevice, st));
            PL_CUDA(cudaMemcpyAsync(bw, w, 4 * n, cudaMemcpyHostToDevice, st));
            PL_CUDA(cudaMemcpyAsync(bwt, wt, 4 * n, cudaMemcpyHostToDevice, st));
            PL_CUDA(cudaMemcpyAsync(bvis, vis, 8 * n, cudaMemcpyHostToDevice, st));
            du = bu; dv = bv; dw = bw; dwt = bwt; dvis = bvis;
        }
        GParams gp;
        gp.uscale = spec->uscale; gp.uoffset = spec->uoffset;
        gp.vscale = spec->vscale; gp.voffset = spec->voffset;
        gp.uorigin = spec->uorigin; gp.vorigin = spec->vorigin;
        gp.nu = spec->nu; gp.nv = spec->nv; gp.supp = spec->supp; gp.osamp = spec->osamp;
        memcpy(gp.s, spec->shift, sizeof gp.s);
        gp.doshift = pl->doshift;
        gp.identity = 1;
        for (int k = 0; k < 9; k++)
            if (spec->shift[k] != ((k % 4) == 0 ? 1.0 : 0.0)) gp.identity = 0;
        gp.diagonal = 1;
        for (int k = 0; k < 9; k++)
            if (k % 4 != 0 && spec->shift[k] != 0.0) gp.diagonal = 0;
        gp.fast = gp.identity && spec->uoffset == 0.0f && spec->voffset == 0.0f;
        gp.near_id = gp.diagonal && fabs(spec->shift[0] - 1.0) <= 0x1p-50 && fabs(spec->shift[4] - 1.0) <= 0x1p-50 &&
                     spec->uoffset == 0.0f && spec->voffset == 0.0f && spec->osamp >= 1 && spec->osamp <= 65536;
        gp.ntu = pl->ntu;
        gp.twopi = (double)(8.0f * atanf(1.0f));  // TWOPI = 8 * ATAN(1.0), REAL (grdh2d.f:91)

        uint32_t *keys, *vals, *ktmp, *vtmp, *exc_list, *rstart, *tstart;
        PlanRecU *rec_u;
        PlanCounts *counts;
        PL_TRY(ctx_scratch(ctx, "pl_keys", 4 * n, (void **)&keys));
        PL_TRY(ctx_scratch(ctx, "pl_vals", 4 * n, (void **)&vals));
        PL_TRY(ctx_scratch(ctx, "pl_ktmp", 4 * n, (void **)&ktmp));
        PL_TRY(ctx_scratch(ctx, "pl_vtmp", 4 * n, (void **)&vtmp));
        PL_TRY(ctx_scratch(ctx, "pl_exclist", 4 * n, (void **)&exc_list));
        PL_TRY(ctx_scratch(ctx, "pl_rec", sizeof(PlanRecU) * n, (void **)&rec_u));
        const int64_t ntiles = (int64_t)pl->ntu * pl->ntv, nscan = scan_tiles((int64_t)n);
        const size_t count_bytes = sizeof(PlanCounts) + 2 * 8 * (size_t)nscan;
        PL_TRY(ctx_scratch(ctx, "pl_counts", count_bytes, (void **)&counts));
        unsigned long long *words = reinterpret_cast<unsigned long long *>(counts + 1);
        PL_TRY(ctx_scratch(ctx, "pl_rstart", 4 * n, (void **)&rstart));
        PL_TRY(ctx_scratch(ctx, "pl_tstart", 4 * (size_t)ntiles, (void **)&tstart));
        PL_CUDA(cudaMemsetAsync(counts, 0, count_bytes, st));
        const int T = 256;
        if (nvis > 0) {
            k_plan_geom<<<ceil_div(nvis, GE_T * GE_PER), GE_T, 0, st>>>(gp, du, dv, dw, dvis, dwt, nvis, keys, rec_u, exc_list,
                                                       counts);
            PL_CUDA(cudaGetLastError());
        }
        int kbits = bits_for((ntiles << 12) + 1);
        if (kbits > 32) {
            sde_set_error("plan: grid too large for 32-bit tile keys");
            rc = SDE_EINVAL;
            goto fail;
        }
        if (nvis > 0) {
            PL_TRY(launch_radix_sort_u32(ctx, &keys, nullptr, &vals, nvis, kbits, ktmp, vtmp, &counts->fail));
            k_runs<<<ceil_div(nvis, RU_T * RU_R), RU_T, 0, st>>>(keys, counts, nvis, words, rstart, tstart,
                                                                 lb_spin(ctx));
            PL_CUDA(cudaGetLastError());
        }
        // the counts and the number of runs: one wait for both
        PlanCounts hc;
        PL_TRY(read_counts(ctx, counts, &hc));
        const int64_t nvalid = (int64_t)hc.ngrid, nexc = (int64_t)hc.nexc;
        pl->nuntouched = nvis - (int64_t)hc.npos;
        pl->nvis = nvalid;
        pl->nexc = nexc;
        const size_t nv1 = (size_t)(nvalid > 0 ? nvalid : 1);
        // at most one item per tile that has a run and one more per item_max visibilities; a
        // chunk per run, per item inside a run, and per chunk_max visibilities
        const int64_t nruns = nvalid > 0 ? (int64_t)hc.runs.total : 0;
        const int64_t max_items = std::min(ntiles, nruns) + nvalid / pl->item_max;
        const int64_t max_chunks = nruns + max_items + nvalid / pl->chunk_max;
        const size_t ne1 = (size_t)(nexc > 0 ? nexc : 1);
        Slab a;
        a.add(&pl->fobs, 8 * nv1);
        a.add(&pl->rec, 16 * nv1);
        a.add(&pl->wt, 4 * nv1);
        a.add(&pl->gdd, 4 * nv1);
        a.add(&pl->orig, 4 * nv1);
        a.add(&pl->gconj, nv1);
        if (pl->doshift) a.add(&pl->rot, 8 * nv1);
        a.add(&pl->d_sums, 4 * sizeof(double));
        a.add(&pl->exc, exc_bytes(ne1));
        if (nvalid > 0) a.add(&pl->items, sizeof(WorkItem) * (size_t)max_items);
        PL_TRY(a.alloc(pl, &pl->slab[0]));
        // exception list (also carries the GRDDEH2D geometry of non-gridding visibilities);
        // the gather below fills in the sorted positions
        if (nexc > 0) {
            float *exc_wt = (float *)((char *)pl->exc + exc_wt_off(ne1));
            float2 *exc_rot = (float2 *)((char *)pl->exc + exc_rot_off(ne1));
            k_exc_write<<<ceil_div(nexc, T), T, 0, st>>>(gp, du, dv, dw, dwt, rec_u, exc_list, nexc, pl->exc,
                                                       exc_wt, exc_rot);
            PL_CUDA(cudaGetLastError());
        }
        // runs, chunks, work items
        if (nvalid > 0) {
            uint64_t *ckey;
            uint2 *craw;
            uint32_t *csrc;
            PL_TRY(ctx_scratch(ctx, "pl_ckey", 8 * (size_t)max_chunks, (void **)&ckey));
            PL_TRY(ctx_scratch(ctx, "pl_craw", 8 * (size_t)max_chunks, (void **)&craw));
            PL_TRY(ctx_scratch(ctx, "pl_csrc", 4 * (size_t)max_chunks, (void **)&csrc));
            const int jbits = bits_for(pl->item_max / pl->chunk_max);
            const int lbits = bits_for(pl->chunk_max - 1);
            k_run_emit<<<ceil_div(nruns, SC_T * SC_R), SC_T, 0, st>>>(
                keys, counts, rstart, tstart, nruns, pl->item_max, pl->chunk_max, lbits, jbits, max_items, max_chunks,
                lb_spin(ctx), words + nscan, ckey, craw, pl->items);
            PL_CUDA(cudaGetLastError());
            PL_TRY(read_counts(ctx, counts, &hc));
            const int64_t nitems = (int64_t)(hc.emit.total >> 31), nchunks = (int64_t)(hc.emit.total & 0x7FFFFFFFull);
            pl->nitems = nitems;
            pl->nchunks = nchunks;
            // an item has at most ceil(visibilities / part) entries
            const int part = part_size(nvis);
            pl->parts_max = nitems + nvalid / part;
            const size_t ncore = (size_t)(pl->ntu + 1) * (pl->ntv + 1);
            uint8_t *zero;  // the entries' count, then the cores
            Slab b;
            b.add(&pl->chunks, sizeof(uint2) * (size_t)nchunks);
            b.add(&pl->parts, sizeof(WorkItem) * (size_t)pl->parts_max);
            b.add(&zero, sizeof(unsigned long long) + ncore);
            PL_TRY(b.alloc(pl, &pl->slab[1]));
            pl->nparts = reinterpret_cast<unsigned long long *>(zero);
            pl->core_lo = zero + sizeof(unsigned long long);
            PL_CUDA(cudaMemsetAsync(zero, 0, sizeof(unsigned long long) + ncore, st));
            k_item_finish<<<ceil_div(nitems, T), T, 0, st>>>(pl->items, nitems, nchunks, nvalid, pl->ntu, pl->core_lo,
                                                           pl->item_max, part, pl->parts, pl->nparts);
            PL_CUDA(cudaGetLastError());
            k_item_order<<<(unsigned)nitems, OR_T, 0, st>>>(pl->items, nitems, ckey, craw, pl->chunks, csrc);
            PL_CUDA(cudaGetLastError());
            k_plan_gather<<<ceil_div(nchunks, GA_CHUNKS), GA_T, 0, st>>>(vals, pl->chunks, csrc, nchunks, rec_u,
                                                                       pl->fobs, pl->rec, pl->wt, pl->gdd, pl->orig,
                                                                       pl->rot, pl->gconj,
                                                                       nexc > 0 ? pl->exc : nullptr);
            PL_CUDA(cudaGetLastError());
        }
        // gridding function: the context's 'SF' table
        pl->cf = ctx->d_cf;
        pl->cft = ctx->d_cft;
    }
    ctx->bytes += pl->bytes;
    *out = pl;
    return SDE_OK;
fail:
    ctx->bytes += pl->bytes;
    sde_plan_destroy(pl);
    return rc;
#undef PL_TRY
#undef PL_CUDA
}
