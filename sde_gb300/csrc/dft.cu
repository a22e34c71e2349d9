// dft.cu -- the direct Fourier transforms of uvmap's and vismodel's DFT options:
//   VISDFT3D (vis/visdft3d.f, 2-D): dirty(ix,iy) = RNORM sum_k WT_k Re(V_k E_k(ix,iy)),
//            psf(ix,iy) = RNORM sum_k WT_k Re(E_k(ix,iy)), E = exp(-i CF (u DX (ix-RX) + v DY (iy-RY)))
//   IMGDFT2D (img/imgdft2d.f): V_k = sum_{ix,iy} I(ix,iy) conj(E_k(ix,iy)) for WT_k > 0
// with CF = 2 pi^2/180 (DX, DY in degrees), RNORM = 1/sum WT over WT > 0.
// Both are dense contractions over visibilities x pixels.  E separates into a row factor and
// a column factor, so a CTA tile stages, per chunk of visibilities, the factors of its columns
// and rows in shared memory and accumulates the tile in registers (2 FMA per visibility, pixel
// and output, packed FP32x2).  Phases are exact to FP32 rounding: the turns per pixel, g, are
// split into two 8-bit heads and a tail (a head times a pixel offset of at most 16 bits is
// exact in FP32, so is its fractional part; the tail's product is 2^-15 of the phase); the
// reference's rotation recurrence, whose error grows along each row, is not used.  Offsets are
// taken from the half pixel nearest the reference pixel; what is left of it, on both axes, is
// one phase per visibility, computed in 64 bits and added to the row factor's.  Sums over
// chunks are compensated (TwoSum).
#include <algorithm>

#include "common.cuh"

namespace {

constexpr int DT = 64;       // tile: 64 x 64 pixels (image) or 64 visibilities (vis)
constexpr int DK = 32;       // visibilities (or columns) per staged chunk
constexpr int DTHR = 128;

// per visibility: turns per pixel along x and y, each as two 8-bit heads and a tail, and
// the weights
struct DftVis {
    float4 gx;  // h1, h2, tail, 0
    float4 gy;  // h1, h2, tail, turns of the reference pixel's rest on both axes (k_dft_prep)
    float4 w;   // (RNORM WT V) re, im; RNORM WT; 0     (zero for WT <= 0)
};

__device__ __forceinline__ double head8(double x) {
    if (x == 0.0) return 0.0;
    int e;
    frexp(x, &e);
    const double q = ldexp(1.0, e - 8);
    return rint(x / q) * q;  // at most 8 significant bits
}

// whole turns per half pixel (offsets are multiples of 1/2) change no phase
__device__ __forceinline__ float4 split3(double g, float rest) {
    g -= 2.0 * rint(0.5 * g);
    const double h1 = head8(g), r = g - h1, h2 = head8(r);
    return make_float4((float)h1, (float)h2, (float)(r - h2), rest);
}

// exp(2 pi i s t), t = (h1 + h2 + l) n + t0 for a pixel offset n (|n| < 2^15, a multiple of 1/2):
// h n is exact for both heads, so are their fractional parts (rounding to an integer by adding
// 1.5 * 2^23; |h n| < 2^16 since split3's turns lie in [-1, 1]).  |t| <= 1.6 or so: the
// quarter turn nearest t is taken off exactly, and sine and cosine of the rest, |r| <= 1/8
// turn, are polynomials in r^2 (least maximum error, fitted to the functions by iteratively
// reweighted least squares; 3.3e-9 relative and 5e-11).  Against the functions in 64 bits the
// result's rms error is 1.5e-8 (correctly rounded values: 1.4e-8), its largest 5.9e-8.  A
// third of the instructions of sincospif with its own reduction of t.
// (t0 = -0 adds nothing, and the compiler leaves it out.)
__device__ __forceinline__ float2 cis_turns(float4 g, float n, float s, float t0 = -0.f) {
    constexpr float M = 12582912.f;  // 1.5 * 2^23
    const float a1 = __fsub_rn(__fmaf_rn(g.x, n, M), M), a2 = __fsub_rn(__fmaf_rn(g.y, n, M), M);
    const float f = __fadd_rn(__fmaf_rn(g.x, n, -a1), __fmaf_rn(g.y, n, -a2));
    const float t = __fmaf_rn(g.z, n, f) + t0;
    const float qm = __fmaf_rn(t, 4.f, M);
    const int q = __float_as_int(qm);  // its low bits: the quarter turns
    const float r = __fmaf_rn(__fsub_rn(qm, M), -0.25f, t), r2 = __fmul_rn(r, r);
    float sp = __fmaf_rn(r2, -75.39141845703125f, 81.5923080444336f);
    sp = __fmaf_rn(r2, sp, -41.34165954589844f);
    sp = __fmaf_rn(r2, sp, -1.9532846806669113e-07f);
    const float sn = __fmaf_rn(r, 6.2831854820251465f, __fmul_rn(r, sp));
    float cp = __fmaf_rn(r2, 59.244354248046875f, -85.4437026977539f);
    cp = __fmaf_rn(r2, cp, 64.93932342529297f);
    cp = __fmaf_rn(r2, cp, -19.739208221435547f);
    const float cs = __fmaf_rn(r2, cp, 1.f);
    const bool odd = (q & 1) != 0;
    const float c = odd ? sn : cs, d = odd ? cs : sn;
    return make_float2(__int_as_float(__float_as_int(c) ^ (((q + 1) & 2) << 30)),
                       s * __int_as_float(__float_as_int(d) ^ ((q & 2) << 30)));
}

__device__ __forceinline__ void two_sum(float &hi, float &lo, float x) {
    const float s = __fadd_rn(hi, x);
    const float bp = __fsub_rn(s, hi);
    const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(x, bp));
    hi = s;
    lo = __fadd_rn(lo, err);
}

__global__ void k_dft_sumwt(const float *__restrict__ wt, int64_t n, double *sum) {
    double s = 0.0;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        if (wt[k] > 0.f) s += wt[k];
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if ((threadIdx.x & 31) == 0) atomicAdd(sum, s);
}

// CF u DX / (2 pi) = u DX pi/180 turns per pixel; (fx, fy): the reference pixel beyond the half
// pixel that the offsets count from (ref_half)
__global__ void k_dft_prep(const float *__restrict__ u, const float *__restrict__ v, const float2 *__restrict__ vis,
                           const float *__restrict__ wt, int64_t n, double dx, double dy, double fx, double fy,
                           const double *sumwt, DftVis *out) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const double d2r = 3.14159265358979323846 / 180.0;
    DftVis r;
    const double gx = (double)u[k] * dx * d2r, gy = (double)v[k] * dy * d2r, rest = -(gx * fx + gy * fy);
    r.gx = split3(gx, 0.f);
    r.gy = split3(gy, (float)(rest - rint(rest)));
    const float w = wt ? wt[k] : 1.f;
    if (w > 0.f) {
        const float c = sumwt ? (float)((double)w / *sumwt) : 1.f;
        const float2 vv = vis ? vis[k] : make_float2(0.f, 0.f);
        r.w = make_float4(c * vv.x, c * vv.y, c, 0.f);
    } else {
        r.w = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    out[k] = r;
}

// hi + lo += x, each half on its own: TwoSum by packed operations (a - b is the FMA a + b * -1)
__device__ __forceinline__ void two_sum2(float2 &hi, float2 &lo, float2 x) {
    const float2 m1 = make_float2(-1.f, -1.f);
    const float2 s = __fadd2_rn(hi, x);
    const float2 bp = __ffma2_rn(hi, m1, s);
    const float2 e1 = __ffma2_rn(__ffma2_rn(bp, m1, s), m1, hi), e2 = __ffma2_rn(bp, m1, x);
    hi = s;
    lo = __fadd2_rn(lo, __fadd2_rn(e1, e2));
}

// VISDFT3D tile, dirty image and PSF together: the factors of a visibility (two cis_turns per
// row or column) cost as much as the FMAs of 30 pixels, so one pass makes both images from
// them.  Thread (tx, ty) of 8 x 16 owns columns 4 tx + {0..3} and 32 + 4 tx + {0..3} (a
// quarter-warp's 16-byte reads are contiguous) of rows 4 ty + {0..3}, as column pairs.  The
// visibilities are split over blockIdx.z (kper each, a multiple of DK) into partial images
// (hi, lo) that k_dft_reduce adds in split order.  FP32 pipe bound; registers (two images of
// 32 pixels as chunk sum, hi and lo) allow two CTAs an SM, one of which can stage factors
// while the other multiplies.  84 240 visibilities on 300 x 277, both images:
// 1.83 ms (34 TFLOP/s with the padding); one image a pass, 4 x 4 pixels a thread, sincospif:
// 3.12 ms.
struct DftTile {
    float exr[DK][DT], exi[DK][DT];  // column factors, the imaginary part negated
    float2 by[2][DK][DT];            // row factors times WT V (dirty), times WT (PSF)
    float4 pv[2][DK * 3];            // the chunk's DftVis, and the next one's
};
template <bool DIRTY, bool PSF>
__global__ void __launch_bounds__(DTHR, 2) k_dft_image(const DftVis *__restrict__ pv, int64_t nvis, int nx, int ny,
                                                       float rx, float ry, int64_t kper, float2 *part_d,
                                                       float2 *part_p) {
    extern __shared__ __align__(16) unsigned char dft_smem[];
    DftTile &S = *reinterpret_cast<DftTile *>(dft_smem);
    constexpr int NO = (DIRTY ? 1 : 0) + (PSF ? 1 : 0);
    const int t = threadIdx.x, tx = t & 7, ty = t >> 3;
    const int x0 = blockIdx.x * DT, y0 = blockIdx.y * DT;
    float2 hi[NO][4][4], lo[NO][4][4];  // [image][column pair][row]
#pragma unroll
    for (int o = 0; o < NO; o++)
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) hi[o][a][b] = lo[o][a][b] = make_float2(0.f, 0.f);
    const int64_t kb = (int64_t)blockIdx.z * kper, ke = min(nvis, kb + kper);
    // a chunk's records, zero (no weight) past the last
    auto record = [&](int64_t k0) {
        return t < DK * 3 && k0 + t / 3 < ke ? reinterpret_cast<const float4 *>(pv + k0)[t]
                                             : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    if (t < DK * 3) S.pv[0][t] = record(kb);
    int buf = 0;
    for (int64_t k0 = kb; k0 < ke; k0 += DK, buf ^= 1) {
        const float4 next = record(k0 + DK);
        __syncthreads();
        // factors of the chunk: exp(-2 pi i gx (x0+i+1-RX)), w exp(-2 pi i gy (y0+j+1-RY))
        for (int e = t; e < DK * DT; e += DTHR) {
            const int k = e / DT, i = e % DT;
            const float4 gx = S.pv[buf][3 * k], gy = S.pv[buf][3 * k + 1], w = S.pv[buf][3 * k + 2];
            const float2 fx = cis_turns(gx, (float)(x0 + i + 1) - rx, -1.f);
            const float2 c = cis_turns(gy, (float)(y0 + i + 1) - ry, -1.f, gy.w);
            const float2 fp = make_float2(w.z * c.x, w.z * c.y);
            const float2 fd = make_float2(__fsub_rn(__fmul_rn(w.x, c.x), __fmul_rn(w.y, c.y)),
                                          __fadd_rn(__fmul_rn(w.x, c.y), __fmul_rn(w.y, c.x)));
            S.exr[k][i] = fx.x;
            S.exi[k][i] = -fx.y;
            if (DIRTY) S.by[0][k][i] = fd;
            if (PSF) S.by[NO - 1][k][i] = fp;
        }
        __syncthreads();
        float2 acc[NO][4][4];
#pragma unroll
        for (int o = 0; o < NO; o++)
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 4; b++) acc[o][a][b] = make_float2(0.f, 0.f);
#pragma unroll 2
        for (int k = 0; k < DK; k++) {
            const float4 r0 = *reinterpret_cast<const float4 *>(&S.exr[k][4 * tx]);
            const float4 r1 = *reinterpret_cast<const float4 *>(&S.exr[k][32 + 4 * tx]);
            const float4 i0 = *reinterpret_cast<const float4 *>(&S.exi[k][4 * tx]);
            const float4 i1 = *reinterpret_cast<const float4 *>(&S.exi[k][32 + 4 * tx]);
            const float2 xr[4] = {make_float2(r0.x, r0.y), make_float2(r0.z, r0.w), make_float2(r1.x, r1.y),
                                  make_float2(r1.z, r1.w)};
            const float2 xi[4] = {make_float2(i0.x, i0.y), make_float2(i0.z, i0.w), make_float2(i1.x, i1.y),
                                  make_float2(i1.z, i1.w)};
#pragma unroll
            for (int o = 0; o < NO; o++) {
                const float4 *pb = reinterpret_cast<const float4 *>(&S.by[o][k][4 * ty]);
                const float4 y0_ = pb[0], y1_ = pb[1];
                const float2 yb[4] = {make_float2(y0_.x, y0_.y), make_float2(y0_.z, y0_.w), make_float2(y1_.x, y1_.y),
                                      make_float2(y1_.z, y1_.w)};
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    const float2 yr = make_float2(yb[b].x, yb[b].x), yi = make_float2(yb[b].y, yb[b].y);
#pragma unroll
                    for (int a = 0; a < 4; a++)
                        acc[o][a][b] = __ffma2_rn(xr[a], yr, __ffma2_rn(xi[a], yi, acc[o][a][b]));
                }
            }
        }
#pragma unroll
        for (int o = 0; o < NO; o++)
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 4; b++) two_sum2(hi[o][a][b], lo[o][a][b], acc[o][a][b]);
        if (t < DK * 3) S.pv[buf ^ 1][t] = next;
    }
#pragma unroll
    for (int o = 0; o < NO; o++) {
        float2 *part = DIRTY && o == 0 ? part_d : part_p;
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const int ix = x0 + (a < 2 ? 0 : 32) + 4 * tx + 2 * (a & 1), iy = y0 + 4 * ty + b;
                if (iy >= ny) continue;
                float2 *p = &part[((size_t)blockIdx.z * ny + iy) * nx + ix];
                if (ix < nx) p[0] = make_float2(hi[o][a][b].x, lo[o][a][b].x);
                if (ix + 1 < nx) p[1] = make_float2(hi[o][a][b].y, lo[o][a][b].y);
            }
    }
}

// the partial images of the visibility splits, added in split order (compensated)
__global__ void k_dft_reduce(const float2 *__restrict__ part, int nsplit, int64_t npix, float *out) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += (int64_t)gridDim.x * blockDim.x) {
        float hi = 0.f, lo = 0.f;
        for (int s = 0; s < nsplit; s++) {
            const float2 q = part[(size_t)s * npix + p];
            two_sum(hi, lo, q.x);
            lo = __fadd_rn(lo, q.y);
        }
        out[p] = __fadd_rn(hi, lo);
    }
}

// IMGDFT2D: a CTA takes 64 visibilities and a band of 16 R rows: T(k, row) = sum_x I(x, row)
// exp(2 pi i gx (x+1-RX)) over chunks of 32 columns, then the band's share of V_k, sum_rows
// exp(2 pi i gy (row+1-RY)) T(k, row), which k_dft_vis_sum adds in band order.  Thread (tk, tr)
// of 8 x 16 owns visibilities 2 tk + {0, 1} + 16 j (a quarter-warp's 16-byte reads are
// contiguous) and rows R tr + {0..R-1}; a column's factors are made once for all rows of the
// band, so a taller band makes fewer, and a band too tall for the image is padding: R is
// chosen by dft_rows.  A single band's share is V_k itself: out is then the visibilities (the sum's
// launch is 5 us of the 33 that 1000 visibilities of 16 x 16 take).  84 240 visibilities, 300 x 277: 0.65 ms (43 TFLOP/s);
// 4 x 4 per thread over all rows with sincospif: 1.18 ms.
template <int R>
__global__ void __launch_bounds__(DTHR, R == 8 ? 2 : 3) k_dft_vis(const float *__restrict__ image, int nx, int ny,
                                                                  float rx, float ry, const DftVis *__restrict__ pv,
                                                                  int64_t nvis, float2 *out) {
    constexpr int RB = 16 * R;
    __shared__ __align__(16) float2 ex[DK][DT];      // [column][visibility]
    __shared__ __align__(16) float img[DK][RB + 2];  // [column][row], padded: the row-wise fill has 2-way conflicts
    __shared__ float2 psum[16][DT];                  // per row group, per visibility
    __shared__ float4 gx[DT];
    const int t = threadIdx.x, tk = t & 7, tr = t >> 3;
    const int64_t v0 = (int64_t)blockIdx.x * DT;
    const int y0 = blockIdx.y * RB;
    if (t < DT) gx[t] = v0 + t < nvis ? pv[v0 + t].gx : make_float4(0.f, 0.f, 0.f, 0.f);
    float2 acc[8][R];
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
        for (int b = 0; b < R; b++) acc[a][b] = make_float2(0.f, 0.f);
    for (int c0 = 0; c0 < nx; c0 += DK) {
        __syncthreads();
        for (int e = t; e < DK * DT; e += DTHR) {
            const int c = e / DT, i = e % DT;
            ex[c][i] = cis_turns(gx[i], (float)(c0 + c + 1) - rx, 1.f);  // (the image is 0 past its columns)
        }
        for (int e = t; e < DK * RB; e += DTHR) {
            // image rows along the warp's columns: coalesced reads
            const int ic = e % DK, ir = e / DK;
            img[ic][ir] = (c0 + ic < nx && y0 + ir < ny) ? image[(size_t)(y0 + ir) * nx + c0 + ic] : 0.f;
        }
        __syncthreads();
#pragma unroll 2
        for (int c = 0; c < DK; c++) {
            float2 xa[8];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float4 q = *reinterpret_cast<const float4 *>(&ex[c][2 * tk + 16 * j]);
                xa[2 * j] = make_float2(q.x, q.y);
                xa[2 * j + 1] = make_float2(q.z, q.w);
            }
            float ib[R];
#pragma unroll
            for (int b = 0; b < R; b += 2) {
                const float2 q = *reinterpret_cast<const float2 *>(&img[c][R * tr + b]);
                ib[b] = q.x;
                ib[b + 1] = q.y;
            }
#pragma unroll
            for (int b = 0; b < R; b++) {
                const float2 i2 = make_float2(ib[b], ib[b]);
#pragma unroll
                for (int a = 0; a < 8; a++) acc[a][b] = __ffma2_rn(i2, xa[a], acc[a][b]);
            }
        }
    }
    // the row factors, and the sum over the thread's rows
#pragma unroll
    for (int a = 0; a < 8; a++) {
        const int v = 2 * tk + (a & 1) + 16 * (a >> 1);
        const float4 gy = v0 + v < nvis ? pv[v0 + v].gy : make_float4(0.f, 0.f, 0.f, 0.f);
        float2 s = make_float2(0.f, 0.f);
#pragma unroll
        for (int b = 0; b < R; b++) {
            const int row = y0 + R * tr + b;
            if (row >= ny) continue;
            const float2 f = cis_turns(gy, (float)(row + 1) - ry, 1.f, gy.w);
            s.x = fmaf(f.x, acc[a][b].x, fmaf(-f.y, acc[a][b].y, s.x));
            s.y = fmaf(f.x, acc[a][b].y, fmaf(f.y, acc[a][b].x, s.y));
        }
        psum[tr][v] = s;
    }
    __syncthreads();
    if (t < DT && v0 + t < nvis) {
        float2 band = make_float2(0.f, 0.f);
        for (int g = 0; g < 16; g++) {
            band.x += psum[g][t].x;
            band.y += psum[g][t].y;
        }
        if (gridDim.y > 1 || pv[v0 + t].w.z > 0.f) out[(size_t)blockIdx.y * nvis + v0 + t] = band;
    }
}

// the bands' shares, added in band order (compensated)
__global__ void k_dft_vis_sum(const float2 *__restrict__ part, int nband, const DftVis *__restrict__ pv, int64_t nvis,
                              float2 *vis) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nvis || !(pv[k].w.z > 0.f)) return;
    float2 hi = make_float2(0.f, 0.f), lo = hi;
    for (int b = 0; b < nband; b++) two_sum2(hi, lo, part[(size_t)b * nvis + k]);
    vis[k] = __fadd2_rn(hi, lo);
}

// Rows per thread of k_dft_vis: the cheapest cover of ny rows by bands of 16 R, a band costing
// its FMAs (128 a column and row) and its column factors (64, about 40 instructions each).
int dft_rows(int ny) {
    int best = 4;
    int64_t cost = INT64_MAX;
    for (int r : {4, 6, 8}) {
        const int64_t c = (int64_t)ceil_div(ny, 16 * r) * (16 * r * 128 + 64 * 40);
        if (c < cost) {
            cost = c;
            best = r;
        }
    }
    return best;
}

// bytes of the bands' shares that sde_dft_vis keeps (all of them would be 33 GB for 64.7 million
// visibilities of an 8192-row image)
constexpr int64_t VIS_PART = 256 << 20;

// the half pixel nearest a reference pixel
double ref_half(double ref) { return 0.5 * rint(2.0 * ref); }

int fail(const char *m) {
    sde_set_error("%s", m);
    return SDE_EINVAL;
}

}  // namespace

extern "C" int sde_dft_image(sde_ctx *ctx, int64_t nvis, const float *u, const float *v, const float *vis,
                             const float *wt, int nx, int ny, double refx, double deltx, double refy,
                             double delty, float *dirty, float *psf) {
    if (!ctx || nvis < 1 || !u || !v || !wt || nx < 1 || ny < 1 || (!dirty && !psf) || (dirty && !vis))
        return fail("sde_dft_image: bad arguments");
    // pixel offsets |ix - REF| < 2^14 keep the split phases exact
    if (nx > 8192 || ny > 8192 || fabs(refx) > 8192 || fabs(refy) > 8192)
        return fail("sde_dft_image: image over 8192 pixels or reference pixel outside +-8192");
    SDE_CUDA_TRY(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    const double hx = ref_half(refx), hy = ref_half(refy);
    double *sw;
    DftVis *pv;
    SDE_TRY(ctx_scratch(ctx, "dft_sumwt", sizeof(double), (void **)&sw));
    SDE_TRY(ctx_scratch(ctx, "dft_vis", sizeof(DftVis) * (size_t)nvis, (void **)&pv));
    SDE_CUDA_TRY(cudaMemsetAsync(sw, 0, sizeof(double), st));
    k_dft_sumwt<<<ctx->num_sms * 4, 256, 0, st>>>(wt, nvis, sw);
    k_dft_prep<<<(unsigned)ceil_div(nvis, (int64_t)256), 256, 0, st>>>(
        u, v, reinterpret_cast<const float2 *>(vis), wt, nvis, deltx, delty, refx - hx, refy - hy, sw, pv);
    SDE_CHECK_LAUNCH();
    double h = 0.0;
    SDE_CUDA_TRY(cudaMemcpyAsync(&h, sw, sizeof h, cudaMemcpyDeviceToHost, st));
    SDE_CUDA_TRY(cudaStreamSynchronize(st));
    if (!(h > 0.0)) {
        sde_set_error("No valid data");  // vis/visdft3d.f:44
        return SDE_EINVAL;
    }
    // the visibilities split over blockIdx.z: tiles x splits fill the SMs' two CTAs twice over
    const int tiles = (int)(ceil_div(nx, DT) * ceil_div(ny, DT));
    const int64_t chunks = ceil_div(nvis, (int64_t)DK);
    const int64_t kper = ceil_div(chunks, std::max<int64_t>(1, std::min<int64_t>(chunks, ctx->num_sms * 4 / tiles))) * DK;
    const int nsplit = ceil_div(nvis, kper);
    const int64_t npix = (int64_t)nx * ny;
    float2 *part;
    SDE_TRY(ctx_scratch(ctx, "dft_part", sizeof(float2) * (size_t)nsplit * npix * (dirty && psf ? 2 : 1), (void **)&part));
    float2 *part_p = dirty ? part + (size_t)nsplit * npix : part;
    const dim3 grid((unsigned)ceil_div(nx, DT), (unsigned)ceil_div(ny, DT), (unsigned)nsplit);
    KTimer kt(ctx, "dft_image");
    auto kern = dirty && psf ? k_dft_image<true, true> : dirty ? k_dft_image<true, false> : k_dft_image<false, true>;
    SDE_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DftTile)));
    kern<<<grid, DTHR, sizeof(DftTile), st>>>(pv, nvis, nx, ny, (float)hx, (float)hy, kper, part, part_p);
    SDE_CHECK_LAUNCH();
    if (dirty) k_dft_reduce<<<ctx->num_sms * 4, 256, 0, st>>>(part, nsplit, npix, dirty);
    if (psf) k_dft_reduce<<<ctx->num_sms * 4, 256, 0, st>>>(part_p, nsplit, npix, psf);
    SDE_CHECK_LAUNCH();
    return SDE_OK;
}

extern "C" int sde_dft_vis(sde_ctx *ctx, const float *image, int nx, int ny, double refx, double deltx,
                           double refy, double delty, int64_t nvis, const float *u, const float *v,
                           const float *wt, float *vis) {
    if (!ctx || !image || nx < 1 || ny < 1 || nvis < 1 || !u || !v || !wt || !vis)
        return fail("sde_dft_vis: bad arguments");
    if (nx > 8192 || ny > 8192 || fabs(refx) > 8192 || fabs(refy) > 8192)
        return fail("sde_dft_vis: image over 8192 pixels or reference pixel outside +-8192");
    SDE_CUDA_TRY(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    const double hx = ref_half(refx), hy = ref_half(refy);
    DftVis *pv;
    SDE_TRY(ctx_scratch(ctx, "dft_vis", sizeof(DftVis) * (size_t)nvis, (void **)&pv));
    k_dft_prep<<<(unsigned)ceil_div(nvis, (int64_t)256), 256, 0, st>>>(u, v, nullptr, wt, nvis, deltx, delty,
                                                                      refx - hx, refy - hy, nullptr, pv);
    SDE_CHECK_LAUNCH();
    // the bands' shares of a slice of visibilities at a time: a slice of VIS_PART bytes is at least
    // 524288 visibilities (64 bands of an 8192-row image), 8192 CTAs a band
    const int r = dft_rows(ny), nband = ceil_div(ny, 16 * r);
    const int64_t slice = nband == 1 ? nvis : std::min<int64_t>(nvis, VIS_PART / (int64_t)sizeof(float2) / nband / DT * DT);
    float2 *out = reinterpret_cast<float2 *>(vis), *part = out;
    if (nband > 1)
        SDE_TRY(ctx_scratch(ctx, "dft_part", sizeof(float2) * (size_t)nband * (size_t)slice, (void **)&part));
    KTimer kt(ctx, "dft_vis");
    auto kern = r == 4 ? k_dft_vis<4> : r == 6 ? k_dft_vis<6> : k_dft_vis<8>;
    for (int64_t k0 = 0; k0 < nvis; k0 += slice) {
        const int64_t n = std::min(slice, nvis - k0);
        kern<<<dim3((unsigned)ceil_div(n, (int64_t)DT), (unsigned)nband), DTHR, 0, st>>>(
            image, nx, ny, (float)hx, (float)hy, pv + k0, n, part);
        SDE_CHECK_LAUNCH();
        if (nband == 1) break;
        k_dft_vis_sum<<<(unsigned)ceil_div(n, (int64_t)256), 256, 0, st>>>(part, nband, pv + k0, n, out + k0);
        SDE_CHECK_LAUNCH();
    }
    return SDE_OK;
}
