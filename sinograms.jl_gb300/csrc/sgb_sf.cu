// sgb_sf.cu -- separable-footprint (SF-TR) projector pair for 2D parallel and fan beams, and
// _tau(rg, x, y) of src/geom/tau.jl:7-60.
//
// No counterpart in the reference, which plans this system model (footprint_size in
// src/sys2/footprint.jl:19-36 sizes its footprints, and _tau is documented as the "footprint
// center and support", tau.jl:57-60) but does not contain it.  The model is the SF-TR method of
// Y. Long, J. A. Fessler and J. M. Balter (IEEE Trans. Med. Imag. 29(11):1839-1850, 2010) in its
// 2D (transaxial) form:
//   * bin coordinate u = tau + wb, wb = (nb - 1)/2 + offset; detector bin k covers [k - 1/2, k + 1/2];
//   * the footprint of a rectangular pixel is the trapezoid through the projections
//     t0 <= t1 <= t2 <= t3 of its four corners, height 1 on [t1, t2], times h, the pixel's chord
//     along the ray through its centre (|dx dy| / max(|dy ex|, |dx ey|) for the unit ray direction);
//   * element (k, pixel) = h (G(k + 1/2) - G(k - 1/2)), G the trapezoid's running integral, so a
//     sinogram sample is a bin-averaged line integral.  For parallel beams the trapezoid times h is
//     the exact Radon transform of the pixel.
// Pixels whose mask is false are not in the model; bins outside 0..nb-1 are dropped.
//
// GPU form:
//   * footprints are FP32 and relative to the centre's bin coordinate uc.  Each corner's offset from
//     uc has a closed form without cancellation (flat: K (p + tc q) / (D - q); arc: K atan((D p + x q)
//     / (x^2 + D^2 + x p - D q)), with (p, q) the corner's rotated offset, x and D the centre's
//     coordinates across and along the central ray from the source), so the trapezoid keeps FP32
//     relative accuracy where uc is ~1e3 bins;
//   * both kernels evaluate footprints and elements with the same explicitly rounded FP32 operations
//     (__fmaf_rn and friends cannot be contracted differently in the two kernels), and an element that
//     serves several views and pixels at the same one of them (SfItem), so each element has the same
//     bits in both and the back-projector is the transpose of the forward projector up to summation
//     order;
//   * forward: one thread per detector bin and one CTA per (view, chunk of bins).  The CTA sweeps the
//     image lines (rows, or columns when the view's rays cross columns more steeply or the source
//     lies within the rows' range); per line it computes into shared memory the footprints of the
//     pixels the chunk's wedge of rays can reach, and each bin sums the few pixels its own wedge
//     reaches.  Deterministic, no atomics;
//   * back: one thread per pixel, over the views and the bins its footprint covers; small images split the
//     views over a cluster, summed in rank order;
//   * an element costs some 30 instructions, and under the scan's symmetry (scan_slots) a pixel's images
//     have the same elements in the views that see them alike, at the same bins or at those mirrored about
//     the detector's centre.  So the forward kernel sums a view's bins over the image together with the
//     bins of the views that are its images, over the image's images, and the back-projector takes a pixel
//     with its images: each element is evaluated once for two or four.  (Over half a turn of parallel beams
//     the images of a view are half as many as those of a pixel.)  Scans without symmetry have a forward
//     kernel of their own, sf_project_plain_kernel.  Mirrored elements agree to rounding
//     only (wb + K a and wb - K a round differently): both evaluate them at the forward sweep's view.
// Both directions are bound by issue, most of it the elements.  888 x 90 arc, 512^2: forward 437 -> 136 us,
// back 260 -> 115 us with four slots against one element at a time; a pair of calls 683 -> 262 us.
// Plans compute the per-view constants and the boundary-ray table once, in FP64 on the device.
#include <cooperative_groups.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <type_traits>
#include <vector>

#include "sgb_common.cuh"
#include "sgb_host.h"
#include "sgb_kernels.cuh"

namespace sgb {

namespace {

constexpr double kPi = 3.14159265358979323846;
constexpr int kFwdThreads = 128;                  // threads per forward CTA
constexpr int kFwdBpt = 2;                        // adjacent detector bins per forward thread
constexpr int kFwdBins = kFwdThreads * kFwdBpt;   // detector bins per forward CTA
template <int NS>  // footprints per line pass of a forward CTA
constexpr int kFwdCap = NS == 1 ? 384 : 256;
constexpr int kBackTx = 32, kBackTy = 8;
constexpr int kViewChunk = 64;  // views staged in shared memory per back-projector pass
constexpr float kRangeEps = 0.01f;  // pixel-index margin of the candidate ranges (FP32 rounding)

// FP64 geometry of one plan (host and set-up kernels).
struct SfGeo {
    int kind, nb, na, nx, ny;
    double ds, wb, dsd, dso, so, dx, dy, ox, oy;
    double xlo, xhi, ylo, yhi;  // image extent (pixel edges)
};

// Per-view constants, FP32 rounded from FP64.
struct SfView {
    float cb, sb, K, so;         // cos, sin of the view angle; dsd/ds (fan) or 1/ds (parallel); source offset
    float dso, e1x, e1y, e2x;    // corners (+-hx, +-hy) rotated: +-(e1x, e1y) for (+,+), +-(e2x, e2y) for (+,-)
    float e2y, p0, p1, p2;       // parallel beams: the view's footprint offsets from uc (sorted) ...
    float p3, ph, phr01, phr23;  // ... its amplitude and trapezoid constants
    float pc3;
    int rows;                    // forward sweep: 1 = rows (lines of constant y), 0 = columns
    int map;                     // back: the item's pixel
    int pad;
};
static_assert(sizeof(SfView) == 80, "SfView layout");

// Kernel arguments: sizes, wb = (nb - 1)/2 + offset, the pixel's |dx|, |dy|, |dx dy| and half sizes.
struct SfArgs {
    int nb, na, nx, ny;
    int splits;  // forward: the image lines are split over this many CTAs per (view, chunk of bins)
    int gsplit;  // back: CTAs of a cluster that share a tile's items
    int nitem;   // back: items
    int nrep;    // forward: views that are not images of others
    int fslots;  // forward: slots that give other views (half a turn of parallel beams: half of them)
    ScanSlots sym;
    float wb, ax, ay, axy, hx, hy;
};

// A view and its images in the slots: entry j is slot j's view, kSfRev if its bins run the other way,
// kSfDup if an earlier slot has the same view.  The forward projector evaluates a view's elements at the
// first view of its images (its representative), in the slot that the view has there.
constexpr int kSfRev = 1 << 30, kSfDup = 1 << 29, kSfView = kSfDup - 1;

// What the back-projector takes at a time: for the view w that slot j gives a view v, and slot j's image of
// its pixel, the element that the forward projector evaluates: w's representative `rep` sees it at the pixel
// that `map` (as ScanSlots::Slot::map) gives for the thread's.  `rows`: w per slot, kSfRev if the element's
// bins run the other way there; kSfDup where the slot's element lies at another pixel, in another item (an
// item per view but for views that are their own images: two).
struct SfItem {
    int4 rows;
    int rep, map;
};

// One pixel's footprint in one view, relative to uc: the bin coordinate of the centre (parallel beams: less
// wb, so that a half turn of the pixel negates it exactly).
struct SfRec {
    float uc, d0, d1, d2, d3, hr01, hr23, c3, h;
};

__device__ __forceinline__ float atan_small(float z) {
    // Taylor series of atan to z^5 for |z| < 0.02 (relative error below 1e-11; a pixel corner's angle
    // from its centre seen from the source is ~1e-3), else atanf.
    const float z2 = __fmul_rn(z, z);
    if (z2 < 4e-4f) return __fmul_rn(z, __fmaf_rn(z2, __fmaf_rn(z2, 1.0f / 5.0f, -1.0f / 3.0f), 1.0f));
    return atanf(z);
}

// Sorted offsets and the trapezoid constants: G(b) = hr01 a^2 + m + c3 - hr23 z^2 with
// a = clamp(b, d0, d1) - d0, m = clamp(b, d1, d2) - d1, z = d3 - clamp(b, d2, d3).
__host__ __device__ __forceinline__ void sf_finish(SfRec &r, float o0, float o1, float o2, float o3) {
    const float a = fminf(o0, o1), b = fmaxf(o0, o1), c = fminf(o2, o3), d = fmaxf(o2, o3);
    const float m1 = fmaxf(a, c), m2 = fminf(b, d);
    r.d0 = fminf(a, c);
    r.d3 = fmaxf(b, d);
    r.d1 = fminf(m1, m2);
    r.d2 = fmaxf(m1, m2);
#ifdef __CUDA_ARCH__
    const float w01 = __fsub_rn(r.d1, r.d0), w23 = __fsub_rn(r.d3, r.d2);
    r.hr01 = w01 > 1e-20f ? __fdividef(0.5f, w01) : 0.f;
    r.hr23 = w23 > 1e-20f ? __fdividef(0.5f, w23) : 0.f;
    r.c3 = __fmul_rn(0.5f, w23);
#else
    const float w01 = r.d1 - r.d0, w23 = r.d3 - r.d2;
    r.hr01 = w01 > 1e-20f ? 0.5f / w01 : 0.f;
    r.hr23 = w23 > 1e-20f ? 0.5f / w23 : 0.f;
    r.c3 = 0.5f * w23;
#endif
}

// The trapezoid's running integral from its centre or its start.  Parallel beams: symmetric (d0 = -d3,
// d1 = -d2), and evaluated as the odd function that it is, so that a pixel and its half turn have the same
// elements at mirrored bins, in every bit.
template <int GEO>
__device__ __forceinline__ float sf_cdf(float b, const SfRec &r) {
    if (GEO == 0) {
        const float a = __fsub_rn(fminf(fmaxf(b, r.d0), r.d1), r.d0);
        const float z = __fsub_rn(r.d3, fminf(fmaxf(b, r.d2), r.d3));
        const float p = __fmul_rn(__fmul_rn(r.hr01, a), a), q = __fmul_rn(__fmul_rn(r.hr23, z), z);
        return __fadd_rn(fminf(fmaxf(b, r.d1), r.d2), __fsub_rn(p, q));
    }
    const float a = __fsub_rn(fminf(fmaxf(b, r.d0), r.d1), r.d0);
    const float m = __fsub_rn(fminf(fmaxf(b, r.d1), r.d2), r.d1);
    const float z = __fsub_rn(r.d3, fminf(fmaxf(b, r.d2), r.d3));
    return __fadd_rn(__fmaf_rn(__fmul_rn(r.hr01, a), a, m), __fmaf_rn(-__fmul_rn(r.hr23, z), z, r.c3));
}

// The lower boundary of bin k, from where uc counts (exact where wb is a multiple of 1/4).
template <int GEO>
__device__ __forceinline__ float sf_bound(int k, const SfArgs &A) {
    const float b = (float)k - 0.5f;
    return GEO == 0 ? __fsub_rn(b, A.wb) : b;
}

// Footprint of the pixel centred at (xc, yc).  GEO: 0 parallel, 1 arc, 2 flat.
template <int GEO>
__device__ __forceinline__ SfRec sf_pixel(const SfView &V, const SfArgs &A, float xc, float yc) {
    SfRec r;
    if (GEO == 0) {
        r.uc = __fmul_rn(__fmaf_rn(xc, V.cb, __fmul_rn(yc, V.sb)), V.K);
        r.d0 = V.p0;
        r.d1 = V.p1;
        r.d2 = V.p2;
        r.d3 = V.p3;
        r.hr01 = V.phr01;
        r.hr23 = V.phr23;
        r.c3 = V.pc3;
        r.h = V.ph;
        return r;
    }
    const float x = __fsub_rn(__fmaf_rn(xc, V.cb, __fmul_rn(yc, V.sb)), V.so);    // xb - source offset
    const float D = __fsub_rn(V.dso, __fmaf_rn(-xc, V.sb, __fmul_rn(yc, V.cb)));  // dso - yb
    const float tc = __fdividef(x, D);
    const float r2 = __fmaf_rn(x, x, __fmul_rn(D, D));
    float o0, o1, o2, o3;
    if (GEO == 1) {
        r.uc = __fmaf_rn(V.K, atanf(tc), A.wb);
        const float c1 = __fmaf_rn(D, V.e1x, __fmul_rn(x, V.e1y)), s1 = __fmaf_rn(x, V.e1x, -__fmul_rn(D, V.e1y));
        const float c2 = __fmaf_rn(D, V.e2x, __fmul_rn(x, V.e2y)), s2 = __fmaf_rn(x, V.e2x, -__fmul_rn(D, V.e2y));
        o0 = __fmul_rn(V.K, atan_small(__fdividef(c1, __fadd_rn(r2, s1))));
        o1 = __fmul_rn(V.K, atan_small(__fdividef(-c1, __fsub_rn(r2, s1))));
        o2 = __fmul_rn(V.K, atan_small(__fdividef(c2, __fadd_rn(r2, s2))));
        o3 = __fmul_rn(V.K, atan_small(__fdividef(-c2, __fsub_rn(r2, s2))));
    } else {
        r.uc = __fmaf_rn(V.K, tc, A.wb);
        const float n1 = __fmaf_rn(tc, V.e1y, V.e1x), n2 = __fmaf_rn(tc, V.e2y, V.e2x);
        o0 = __fmul_rn(V.K, __fdividef(n1, __fsub_rn(D, V.e1y)));
        o1 = __fmul_rn(V.K, __fdividef(-n1, __fadd_rn(D, V.e1y)));
        o2 = __fmul_rn(V.K, __fdividef(n2, __fsub_rn(D, V.e2y)));
        o3 = __fmul_rn(V.K, __fdividef(-n2, __fadd_rn(D, V.e2y)));
    }
    sf_finish(r, o0, o1, o2, o3);
    // chord along the ray from the source: direction (x cb + D sb, x sb - D cb), length sqrt(r2)
    const float ex = __fmaf_rn(x, V.cb, __fmul_rn(D, V.sb)), ey = __fmaf_rn(x, V.sb, -__fmul_rn(D, V.cb));
    const float m = fmaxf(fabsf(__fmul_rn(A.ay, ex)), fabsf(__fmul_rn(A.ax, ey)));
    r.h = __fdividef(A.axy, __fmul_rn(m, rsqrtf(r2)));
    return r;
}

// Pixel-index range [ia, ib] (clamped to 0..n-1) of a line whose pixels can meet the wedge between
// two boundary rays: the rays' crossings f = alpha + beta L (in pixel-index units along the line) at
// the line's edges L0 and L1 bound the wedge inside the line (the source lies outside the line's
// range, so the crossings move linearly).  A NaN boundary gives the whole line.
__device__ __forceinline__ void sf_range(float2 lo, float2 hi, float L0, float L1, int n, int &ia, int &ib) {
    if (isnan(lo.x) || isnan(hi.x)) {
        ia = 0;
        ib = n - 1;
        return;
    }
    const float f0 = __fmaf_rn(lo.y, L0, lo.x), f1 = __fmaf_rn(lo.y, L1, lo.x);
    const float f2 = __fmaf_rn(hi.y, L0, hi.x), f3 = __fmaf_rn(hi.y, L1, hi.x);
    const float fl = fminf(fminf(f0, f1), fminf(f2, f3)) + (0.5f - kRangeEps);
    const float fh = fmaxf(fmaxf(f0, f1), fmaxf(f2, f3)) + (0.5f + kRangeEps);
    ia = max(0, (int)floorf(fminf(fmaxf(fl, -1.f), (float)n)));
    ib = min(n - 1, (int)floorf(fminf(fmaxf(fh, -1.f), (float)n)));
}

// ------------------------------------------------------------------- set-up (FP64)
__device__ SfView sf_view_at(const SfGeo &G, double b) {
    const double cb = cos(b), sb = sin(b);
    const double hx = 0.5 * fabs(G.dx), hy = 0.5 * fabs(G.dy);
    SfView V{};
    V.cb = (float)cb;
    V.sb = (float)sb;
    V.K = (float)(G.kind == SGB_PAR ? 1.0 / G.ds : G.dsd / G.ds);
    V.so = (float)G.so;
    V.dso = (float)G.dso;
    V.e1x = (float)(hx * cb + hy * sb);
    V.e1y = (float)(-hx * sb + hy * cb);
    V.e2x = (float)(hx * cb - hy * sb);
    V.e2y = (float)(-hx * sb - hy * cb);
    const bool pref_rows = fabs(cb) >= fabs(sb);
    if (G.kind == SGB_PAR) {
        V.rows = pref_rows;
        SfRec r{};
        const float o1 = (float)((hx * cb + hy * sb) / G.ds), o2 = (float)((hx * cb - hy * sb) / G.ds);
        sf_finish(r, o1, -o1, o2, -o2);
        V.p0 = r.d0;
        V.p1 = r.d1;
        V.p2 = r.d2;
        V.p3 = r.d3;
        V.phr01 = r.hr01;
        V.phr23 = r.hr23;
        V.pc3 = r.c3;
        const double ax = fabs(G.dx), ay = fabs(G.dy);
        V.ph = (float)(ax * ay / fmax(ay * fabs(sb), ax * fabs(cb)));  // ray direction (-sin, cos)
    } else {
        // the sweep's lines must not contain the source: rows need ys outside the image's y range
        const double xs = G.so * cb - G.dso * sb, ys = G.so * sb + G.dso * cb;
        const bool rows_ok = ys < G.ylo || ys > G.yhi, cols_ok = xs < G.xlo || xs > G.xhi;
        V.rows = pref_rows ? (rows_ok || !cols_ok) : !(cols_ok || !rows_ok);
    }
    return V;
}

// The constants of `nview` views, and of the back-projector's items (their view and map).
__global__ void sf_setup_views(SfGeo G, const double *betas, int nview, SfView *views, int nitem, const int2 *items,
                               SfView *item_views) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nview) views[i] = sf_view_at(G, betas[i]);
    if (i >= nitem) return;
    SfView V = sf_view_at(G, betas[items[i].x]);
    V.map = items[i].y;
    item_views[i] = V;
}

// Boundary rays: for boundary j (u = j - 1/2, j = 0..nb) the along-coordinate of its crossing with
// the line at line-coordinate L is A + B L (rows: x at y = L; columns: y at x = L); the table holds it
// in pixel-index units, alpha + beta L with alpha = A / d + c0 and beta = B / d for the along axis's
// pixel size d and centre index c0.  A fan ray that
// does not point toward the lines (the source lies on one side of all of them), or is within 1e-6 of
// parallel to them, is stored as NaN: a wedge bounded by such a ray may contain the direction
// parallel to the lines, where crossings run off to infinity, so its range is the whole line.  Ray
// angles are monotone in j and a detector spans less than 180 degrees, so a wedge whose two bounding
// rays both point toward the lines contains only such rays and its crossings bound it exactly.
__global__ void sf_setup_rays(SfGeo G, const double *betas, const SfView *views, float2 *rays) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int nbd = G.nb + 1;
    if (i >= (long long)G.na * nbd) return;
    const int v = (int)(i / nbd), j = (int)(i % nbd);
    const double b = betas[v], cb = cos(b), sb = sin(b);
    const double tau = (j - 0.5) - G.wb;  // sample units from the detector centre
    const bool rows = views[v].rows != 0;
    double A, B;
    if (G.kind == SGB_PAR) {
        const double s = tau * G.ds;  // x cb + y sb = s
        const double num = rows ? -sb : -cb, den = rows ? cb : sb;
        B = num / den;
        A = s / den;
    } else {
        const double gam = G.kind == SGB_ARC ? tau * G.ds / G.dsd : atan(tau * G.ds / G.dsd);
        const double dxr = sin(b + gam), dyr = -cos(b + gam);  // ray direction from the source
        const double xs = G.so * cb - G.dso * sb, ys = G.so * sb + G.dso * cb;
        B = rows ? dxr / dyr : dyr / dxr;
        A = rows ? xs - B * ys : ys - B * xs;
        const double toward = rows ? (ys > G.yhi ? -dyr : dyr) : (xs > G.xhi ? -dxr : dxr);
        if (!(toward > 1e-6)) B = HUGE_VAL;
    }
    const double d = rows ? G.dx : G.dy, c0 = rows ? (G.nx - 1) / 2.0 + G.ox : (G.ny - 1) / 2.0 + G.oy;
    float2 out;
    if (!(fabs(B) <= 1e6)) out = make_float2(nanf(""), nanf(""));
    else out = make_float2((float)(A / d + c0), (float)(B / d));
    rays[i] = out;
}

// ------------------------------------------------------------------- forward
// The model's image (mask applied) and its transpose: a pass reads consecutive pixels of a line, which
// lie along x or along y.
__global__ void sf_image_kernel(const float *__restrict__ image, const uint8_t *__restrict__ mask, int nx, int ny,
                                float *__restrict__ out, float *__restrict__ outt) {
    __shared__ float tile[32][33];
    const int x = blockIdx.x * 32 + threadIdx.x, y0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int y = y0 + r;
        if (x >= nx || y >= ny) continue;
        const size_t n = x + (size_t)nx * y;
        const float v = mask && !mask[n] ? 0.f : image[n];
        out[n] = v;
        tile[r][threadIdx.x] = v;
    }
    __syncthreads();
    const int y = y0 + threadIdx.x;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int c = blockIdx.x * 32 + r;
        if (c < nx && y < ny) outt[y + (size_t)ny * c] = tile[threadIdx.x][r];
    }
}

// The record of a staged pixel (parallel beams: the view's own but for uc).
template <int GEO>
__device__ __forceinline__ SfRec sf_staged(const SfView &V, float4 a0, const float4 *a1) {
    SfRec r;
    r.uc = a0.x;
    if (GEO == 0) {
        r.d0 = V.p0;
        r.d1 = V.p1;
        r.d2 = V.p2;
        r.d3 = V.p3;
        r.hr01 = V.phr01;
        r.hr23 = V.phr23;
        r.c3 = V.pc3;
    } else {
        r.d0 = a0.y;
        r.d1 = a0.z;
        r.d2 = a0.w;
        r.d3 = a1->x;
        r.hr01 = a1->y;
        r.hr23 = a1->z;
        r.c3 = a1->w;
    }
    return r;
}

// One view at a time, for scans without symmetry: a line's pixels are staged and summed, one barrier between, and
// the CTAs of an SM hide each other's loads.  With one sum per element and bin, fetching a line ahead as the kernel
// below does costs more than it hides (arc, 257 x 257, 384 bins x 181 views: 235 us, a line ahead 256).
template <int GEO>
__global__ void __launch_bounds__(kFwdThreads) sf_project_plain_kernel(SfArgs A, const SfView *__restrict__ views,
                                                                       const float2 *__restrict__ rays,
                                                                       const float *__restrict__ xcs,
                                                                       const float *__restrict__ ycs,
                                                                       const float *__restrict__ image,
                                                                       const float *__restrict__ imaget,
                                                                       float *__restrict__ sino) {
    constexpr int CAP = kFwdCap<1>;
    __shared__ float4 s0[2][CAP];                // uc, d0, d1, d2
    __shared__ float4 s1[GEO != 0 ? 2 : 1][CAP];  // d3, hr01, hr23, c3 (fan beams)
    __shared__ float2 s2[2][CAP];                // h, pixel value
    const int v = blockIdx.y, tid = threadIdx.x;
    const int k0 = blockIdx.x * kFwdBins, kend = min(k0 + kFwdBins, A.nb);
    const int ka = k0 + kFwdBpt * tid, kb = min(ka + kFwdBpt, A.nb);  // this thread's bins [ka, kb)
    const SfView V = views[v];
    const bool rows = V.rows != 0;
    const int nal = rows ? A.nx : A.ny, nln = rows ? A.ny : A.nx;
    const float *lcs = rows ? ycs : xcs, *src = rows ? image : imaget;
    const float hl = rows ? A.hy : A.hx;
    const float2 *R = rays + (size_t)v * (A.nb + 1);
    const float2 cl = R[k0], ch = R[kend];
    const bool active = ka < A.nb;
    const float2 bl = R[min(ka, A.nb)], bh = R[max(kb, 0)];
    const float e0 = sf_bound<GEO>(ka, A), e1 = sf_bound<GEO>(ka + 1, A), e2 = sf_bound<GEO>(ka + 2, A);
    const int per = (nln + A.splits - 1) / A.splits, jb = blockIdx.z * per, je = min(nln, jb + per);
    float acc0 = 0.f, acc1 = 0.f;
    int buf = 0;
    for (int j = jb; j < je; j++) {
        const float lc = lcs[j], L0 = lc - hl, L1 = lc + hl;
        int ia, ib;
        sf_range(cl, ch, L0, L1, nal, ia, ib);
        if (ia > ib) continue;  // same for the whole CTA
        int qa = 0, qb = -1;
        if (active) sf_range(bl, bh, L0, L1, nal, qa, qb);
        for (int p0 = ia; p0 <= ib; p0 += CAP) {
            const int p1 = min(ib, p0 + CAP - 1);
            for (int t = tid; t <= p1 - p0; t += kFwdThreads) {
                const int i = p0 + t;
                const float val = __ldg(src + (size_t)nal * j + i);
                const SfRec r = sf_pixel<GEO>(V, A, __ldg(xcs + (rows ? i : j)), __ldg(ycs + (rows ? j : i)));
                s0[buf][t] = make_float4(r.uc, r.d0, r.d1, r.d2);
                if (GEO != 0) s1[buf][t] = make_float4(r.d3, r.hr01, r.hr23, r.c3);
                s2[buf][t] = make_float2(r.h, val);
            }
            __syncthreads();
            const int ta = max(qa, p0), tb = min(qb, p1);
            for (int i = ta; i <= tb; i++) {
                const int t = i - p0;
                const float2 a2 = s2[buf][t];
                const SfRec r = sf_staged<GEO>(V, s0[buf][t], GEO != 0 ? &s1[buf][t] : nullptr);
                const float g0 = sf_cdf<GEO>(__fsub_rn(e0, r.uc), r), g1 = sf_cdf<GEO>(__fsub_rn(e1, r.uc), r);
                const float g2 = sf_cdf<GEO>(__fsub_rn(e2, r.uc), r);
                acc0 = __fmaf_rn(__fmul_rn(a2.x, __fsub_rn(g1, g0)), a2.y, acc0);
                acc1 = __fmaf_rn(__fmul_rn(a2.x, __fsub_rn(g2, g1)), a2.y, acc1);
            }
            buf ^= 1;
        }
    }
    // splits > 1: partial sums, added in split order by sf_sum_splits
    float *row = sino + (size_t)A.nb * (v + (size_t)A.na * blockIdx.z);
    if (active) row[ka] = acc0;
    if (ka + 1 < A.nb) row[ka + 1] = acc1;
}

template <int GEO, int NS>
__global__ void __launch_bounds__(kFwdThreads) sf_project_kernel(SfArgs A, const SfView *__restrict__ views,
                                                                 const float2 *__restrict__ rays,
                                                                 const float *__restrict__ xcs,
                                                                 const float *__restrict__ ycs,
                                                                 const float *__restrict__ image,
                                                                 const float *__restrict__ imaget,
                                                                 const int4 *__restrict__ images,
                                                                 float *__restrict__ sino) {
    constexpr int CAP = kFwdCap<NS>;
    __shared__ float4 s0[2][CAP];                // uc, d0, d1, d2
    __shared__ float4 s1[GEO != 0 ? 2 : 1][CAP];  // d3, hr01, hr23, c3 (fan beams)
    __shared__ float s2[2][CAP];                 // h
    __shared__ float s3[2][NS][CAP];             // the pixel's value, and its images'
    const int4 im = images[blockIdx.y];
    const int iv[4] = {im.x, im.y, im.z, im.w};
    const int v = iv[0], tid = threadIdx.x;
    const int k0 = blockIdx.x * kFwdBins, kend = min(k0 + kFwdBins, A.nb);
    const int ka = k0 + kFwdBpt * tid, kb = min(ka + kFwdBpt, A.nb);  // this thread's bins [ka, kb)
    const SfView V = views[v];
    const bool rows = V.rows != 0;
    const int nal = rows ? A.nx : A.ny, nln = rows ? A.ny : A.nx;
    const float *lcs = rows ? ycs : xcs;
    const float hl = rows ? A.hy : A.hx;
    const float2 *R = rays + (size_t)v * (A.nb + 1);
    const float2 cl = R[k0], ch = R[kend];
    const bool active = ka < A.nb;
    const float2 bl = R[min(ka, A.nb)], bh = R[max(kb, 0)];
    // boundaries of bins ka and ka + 1 (as the back-projector forms them)
    const float e0 = sf_bound<GEO>(ka, A), e1 = sf_bound<GEO>(ka + 1, A), e2 = sf_bound<GEO>(ka + 2, A);
    const int per = (nln + A.splits - 1) / A.splits, jb = blockIdx.z * per, je = min(nln, jb + per);
    float acc0[NS] = {}, acc1[NS] = {};
    // A pass is at most CAP pixels of a line: [p0, p1] of line j, whose wedge ends at ib.  The next
    // pass's values are requested and its footprints computed while the current one is summed: one
    // barrier per pass, and the loads' latency lies behind the sums.
    struct Pass {
        int j, ib, p0, p1, qa, qb;
    };
    auto lines = [&](Pass &q) {  // the first line from q.j on with pixels
        for (; q.j < je; q.j++) {
            const float lc = lcs[q.j], L0 = lc - hl, L1 = lc + hl;
            sf_range(cl, ch, L0, L1, nal, q.p0, q.ib);
            if (q.p0 > q.ib) continue;  // same for the whole CTA
            q.p1 = min(q.ib, q.p0 + CAP - 1);
            q.qa = 0;
            q.qb = -1;
            if (active) sf_range(bl, bh, L0, L1, nal, q.qa, q.qb);
            return;
        }
    };
    auto advance = [&](Pass q) {
        if (q.p1 < q.ib) {
            q.p0 = q.p1 + 1;
            q.p1 = min(q.ib, q.p0 + CAP - 1);
            return q;
        }
        q.j++;
        lines(q);
        return q;
    };
    constexpr int NT = (CAP + kFwdThreads - 1) / kFwdThreads;  // a thread's pixels of a pass
    float vals[NT][NS];
    // slot s's values along line j: src[s] + ls[s] j + is[s] i, consecutive in memory
    const float *src[NS];
    int ls[NS], is[NS];
#pragma unroll
    for (int s = 0; s < NS; s++) {
        const int f = A.sym.slot[s].map;
        const bool along_x = rows != ((f & 4) != 0);
        is[s] = f & (along_x ? 1 : 2) ? -1 : 1;
        const int pitch = along_x ? A.nx : A.ny, nl = along_x ? A.ny : A.nx;
        const bool back = f & (along_x ? 2 : 1);
        ls[s] = back ? -pitch : pitch;
        src[s] = (along_x ? image : imaget) + (is[s] < 0 ? pitch - 1 : 0) + (back ? (size_t)pitch * (nl - 1) : 0);
    }
    auto request = [&](const Pass &q) {
#pragma unroll
        for (int u = 0; u < NT; u++) {
            const int i = q.p0 + tid + u * kFwdThreads;
            if (q.j >= je || i > q.p1) continue;
#pragma unroll
            for (int s = 0; s < NS; s++) vals[u][s] = __ldg(src[s] + (ptrdiff_t)ls[s] * q.j + is[s] * i);
        }
    };
    auto fill = [&](const Pass &q, int buf) {
#pragma unroll
        for (int u = 0; u < NT; u++) {
            const int t = tid + u * kFwdThreads, i = q.p0 + t;
            if (q.j >= je || i > q.p1) continue;
            const int px = rows ? i : q.j, py = rows ? q.j : i;
            const SfRec r = sf_pixel<GEO>(V, A, __ldg(xcs + px), __ldg(ycs + py));
            s0[buf][t] = make_float4(r.uc, r.d0, r.d1, r.d2);
            if (GEO != 0) s1[buf][t] = make_float4(r.d3, r.hr01, r.hr23, r.c3);
            s2[buf][t] = r.h;
#pragma unroll
            for (int s = 0; s < NS; s++) s3[buf][s][t] = vals[u][s];
        }
    };
    Pass cur{jb, 0, 0, 0, 0, -1};
    lines(cur);
    request(cur);
    fill(cur, 0);
    for (int buf = 0; cur.j < je; buf ^= 1) {
        const Pass nxt = advance(cur);
        __syncthreads();
        request(nxt);
        const int ta = max(cur.qa, cur.p0), tb = min(cur.qb, cur.p1);
        for (int i = ta; i <= tb; i++) {
            const int t = i - cur.p0;
            const float h = s2[buf][t];
            const SfRec r = sf_staged<GEO>(V, s0[buf][t], GEO != 0 ? &s1[buf][t] : nullptr);
            const float g0 = sf_cdf<GEO>(__fsub_rn(e0, r.uc), r), g1 = sf_cdf<GEO>(__fsub_rn(e1, r.uc), r);
            const float g2 = sf_cdf<GEO>(__fsub_rn(e2, r.uc), r);
            const float w0 = __fmul_rn(h, __fsub_rn(g1, g0)), w1 = __fmul_rn(h, __fsub_rn(g2, g1));
#pragma unroll
            for (int s = 0; s < NS; s++) {
                const float val = s3[buf][s][t];
                acc0[s] = __fmaf_rn(w0, val, acc0[s]);
                acc1[s] = __fmaf_rn(w1, val, acc1[s]);
            }
        }
        fill(nxt, buf ^ 1);
        cur = nxt;
    }
    // splits > 1: partial sums, added in split order by sf_sum_splits
#pragma unroll
    for (int s = 0; s < NS; s++) {
        if (iv[s] & kSfDup) continue;
        const int ka1 = ka + 1, vs = iv[s] & kSfView;
        const bool rev = iv[s] & kSfRev;
        float *row = sino + (size_t)A.nb * (vs + (size_t)A.na * blockIdx.z);
        if (active) row[rev ? A.nb - 1 - ka : ka] = acc0[s];
        if (ka1 < A.nb) row[rev ? A.nb - 1 - ka1 : ka1] = acc1[s];
    }
}

__global__ void sf_sum_splits(const float *__restrict__ part, int splits, long long n, float *__restrict__ sino) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = part[i];
    for (int z = 1; z < splits; z++) s = __fadd_rn(s, part[i + n * z]);
    sino[i] = s;
}

// ------------------------------------------------------------------- back
template <int GEO, int NS>
__global__ void __launch_bounds__(kBackTx *kBackTy) sf_back_kernel(SfArgs A, const SfView *__restrict__ views,
                                                                   const float *__restrict__ xcs,
                                                                   const float *__restrict__ ycs,
                                                                   const float *__restrict__ sino,
                                                                   const uint8_t *__restrict__ mask,
                                                                   const int4 *__restrict__ rows,
                                                                   const float *__restrict__ zeros,
                                                                   float *__restrict__ image) {
    __shared__ SfView sv[kViewChunk];
    __shared__ __align__(16) const float *sp[kViewChunk][NS];  // bin 0 of the slots' rows, and the way their bins run
    __shared__ __align__(16) int ss[kViewChunk][NS];
    __shared__ float part[NS][kBackTx * kBackTy];
    const int tid = threadIdx.x + kBackTx * threadIdx.y, rank = blockIdx.z;
    const int px = blockIdx.x * kBackTx + threadIdx.x, py = blockIdx.y * kBackTy + threadIdx.y;
    size_t n[NS];
    bool own[NS], on = false;  // slot s's pixel is this thread's; one of them is in the model
#pragma unroll
    for (int s = 0; s < NS; s++) {
        own[s] = slot_pixel(A.sym, A.nx, A.ny, s, px, py, &n[s]);
        on |= own[s] && (!mask || mask[n[s]]);
    }
    const int cx = min(px, A.nx - 1), cy = min(py, A.ny - 1);
    float xc = xcs[cx], yc = ycs[cy];
    int map = 0;  // of (xc, yc)
    const int va = (int)((long long)A.nitem * rank / A.gsplit), vb = (int)((long long)A.nitem * (rank + 1) / A.gsplit);
    float acc[NS] = {};
    for (int v0 = va; v0 < vb; v0 += kViewChunk) {
        const int nv = min(kViewChunk, vb - v0);
        __syncthreads();
        const int *src = reinterpret_cast<const int *>(views + v0);
        int *dst = reinterpret_cast<int *>(sv);
        for (int t = tid; t < nv * (int)(sizeof(SfView) / 4); t += kBackTx * kBackTy) dst[t] = __ldg(src + t);
        static_assert(kViewChunk * NS <= kBackTx * kBackTy, "a thread stages one slot of one item");
        if (tid < nv * NS) {
            const int e = __ldg(reinterpret_cast<const int *>(rows + v0 + tid / NS) + tid % NS);
            sp[tid / NS][tid % NS] = e & kSfDup ? zeros : sino + (size_t)A.nb * (e & kSfView) + (e & kSfRev ? A.nb - 1 : 0);
            ss[tid / NS][tid % NS] = e & kSfRev ? -1 : 1;
        }
        __syncthreads();
        if (!on) continue;
        for (int vv = 0; vv < nv; vv++) {
            if (NS > 1 && sv[vv].map != map) {  // a few times per call: the items' maps come in runs
                map = sv[vv].map;
                int qx = map & 4 ? cy : cx, qy = map & 4 ? cx : cy;
                if (map & 1) qx = A.nx - 1 - qx;
                if (map & 2) qy = A.ny - 1 - qy;
                xc = __ldg(xcs + qx);
                yc = __ldg(ycs + qy);
            }
            const SfRec r = sf_pixel<GEO>(sv[vv], A, xc, yc);
            const float uc = GEO == 0 ? __fadd_rn(r.uc, A.wb) : r.uc;
            const float lo = __fadd_rn(uc, r.d0) - 0.5f, hi = __fadd_rn(uc, r.d3) + 0.5f;
            const int kf = max(0, (int)ceilf(fminf(fmaxf(lo, -1.f), (float)A.nb)));
            const int kl = min(A.nb - 1, (int)floorf(fminf(fmaxf(hi, -1.f), (float)A.nb)));
            if (kf > kl) continue;
            const float *row[NS];
            int step[NS];
#pragma unroll
            for (int s = 0; s < NS; s++) {
                step[s] = NS == 1 ? 1 : ss[vv][s];
                row[s] = sp[vv][s] + step[s] * kf;
            }
            float gprev = sf_cdf<GEO>(__fsub_rn(sf_bound<GEO>(kf, A), r.uc), r);
            for (int k = kf; k <= kl; k++) {
                const float g = sf_cdf<GEO>(__fsub_rn(sf_bound<GEO>(k + 1, A), r.uc), r);
                const float w = __fmul_rn(r.h, __fsub_rn(g, gprev));
#pragma unroll
                for (int s = 0; s < NS; s++) {
                    acc[s] = __fmaf_rn(w, __ldg(row[s]), acc[s]);
                    row[s] += step[s];
                }
                gprev = g;
            }
        }
    }
    if (A.gsplit == 1) {
#pragma unroll
        for (int s = 0; s < NS; s++)
            if (own[s]) image[n[s]] = !mask || mask[n[s]] ? acc[s] : 0.f;
        return;
    }
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
#pragma unroll
    for (int s = 0; s < NS; s++) part[s][tid] = acc[s];
    cl.sync();
    // each rank finishes its share of the slots' pixels, adding the ranks in order
#pragma unroll
    for (int s = 0; s < NS; s++) {
        if ((tid / 32 + s) % A.gsplit != rank || !own[s]) continue;
        float v = 0.f;
        for (int q = 0; q < A.gsplit; q++) v += cl.map_shared_rank(&part[s][tid], q)[0];
        image[n[s]] = !mask || mask[n[s]] ? v : 0.f;
    }
    cl.sync();  // peers' shared memory stays alive until every rank has read it
}

template <int GEO, int NS>
int sf_launch_back(const SfArgs &A, const SfView *views, const float *xcs, const float *ycs, const float *sino,
                   const uint8_t *mask, const int4 *rows, const float *zeros, float *image, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((A.sym.hx + kBackTx - 1) / kBackTx, (A.sym.hy + kBackTy - 1) / kBackTy, A.gsplit);
    cfg.blockDim = dim3(kBackTx, kBackTy);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = A.gsplit;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, sf_back_kernel<GEO, NS>, A, views, xcs, ycs, sino, mask, rows, zeros, image);
    if (e != cudaSuccess) {
        set_error("sf_back_kernel: launch failed: %s", cudaGetErrorString(e));
        return SGB_ERR_CUDA;
    }
    return after_launch("sf_back_kernel");
}

// One slot count of a direction, for the plan's geometry kind.
template <int NS>
int sf_launch_back_kind(int kind, const SfArgs &A, const SfView *views, const float *xcs, const float *ycs,
                        const float *sino, const uint8_t *mask, const int4 *rows, const float *zeros, float *image,
                        cudaStream_t st) {
    if (kind == SGB_PAR) return sf_launch_back<0, NS>(A, views, xcs, ycs, sino, mask, rows, zeros, image, st);
    if (kind == SGB_ARC) return sf_launch_back<1, NS>(A, views, xcs, ycs, sino, mask, rows, zeros, image, st);
    return sf_launch_back<2, NS>(A, views, xcs, ycs, sino, mask, rows, zeros, image, st);
}

template <int NS>
int sf_launch_forward(int kind, const SfArgs &A, const SfView *views, const float2 *rays, const float *xcs,
                      const float *ycs, const float *src, const float *srct, const int4 *reps, float *dst,
                      cudaStream_t st) {
    const dim3 grid((A.nb + kFwdBins - 1) / kFwdBins, A.nrep, A.splits);
    auto go = [&](auto geo) {
        constexpr int GEO = decltype(geo)::value;
        if constexpr (NS == 1)
            sf_project_plain_kernel<GEO><<<grid, kFwdThreads, 0, st>>>(A, views, rays, xcs, ycs, src, srct, dst);
        else
            sf_project_kernel<GEO, NS><<<grid, kFwdThreads, 0, st>>>(A, views, rays, xcs, ycs, src, srct, reps, dst);
    };
    if (kind == SGB_PAR) go(std::integral_constant<int, 0>{});
    else if (kind == SGB_ARC) go(std::integral_constant<int, 1>{});
    else go(std::integral_constant<int, 2>{});
    return after_launch("sf_project_kernel");
}

}  // namespace

}  // namespace sgb

using namespace sgb;

// One separable-footprint pair: geometry, the per-view constants and the boundary-ray table on the
// device (computed once), and staging buffers for host-pointer calls.
struct sgb_sf_plan {
    SfGeo G{};
    SfArgs A{};
    DevBuf block, din, dout, part;
    // in the block; views, rays, reps and img are the forward projector's, the items and zeros the other's
    const float *axes = nullptr;
    const uint8_t *mask_dev = nullptr;
    const SfView *views = nullptr;
    const float2 *rays = nullptr;
    const int4 *reps = nullptr;  // the representative views' images
    float *img = nullptr;        // the masked image and its transpose
    const SfView *item_views = nullptr;
    const int4 *item_rows = nullptr;
    const float *zeros = nullptr;  // a row
};

namespace {

int sf_geometry(const sgb_sino_geom *rg, const sgb_image_geom *ig, SfGeo *G) {
    SGB_REQUIRE(rg && ig, "sf: null geometry");
    SGB_REQUIRE(rg->kind == SGB_PAR || rg->kind == SGB_ARC || rg->kind == SGB_FLAT, "sf: unknown geometry kind %d",
                rg->kind);
    SGB_REQUIRE(rg->nb > 0 && rg->na > 0 && rg->na <= 65535, "sf: need nb > 0 and 0 < na <= 65535");
    SGB_REQUIRE(rg->d > 0, "sf: detector spacing d must be positive");
    SGB_REQUIRE(ig->ndim == 2 && ig->dims[0] > 0 && ig->dims[1] > 0, "sf: need a 2D ImageGeom with positive dims");
    SGB_REQUIRE(ig->deltas[0] != 0 && ig->deltas[1] != 0, "sf: pixel sizes must be nonzero");
    SfGeo g{};
    g.kind = rg->kind;
    g.nb = rg->nb;
    g.na = rg->na;
    g.nx = ig->dims[0];
    g.ny = ig->dims[1];
    g.ds = rg->d;
    g.wb = (rg->nb - 1) / 2.0 + (double)rg->offset;
    g.dx = ig->deltas[0];
    g.dy = ig->deltas[1];
    g.ox = ig->offsets[0];
    g.oy = ig->offsets[1];
    const double xc0 = (g.nx - 1) / 2.0 + g.ox, yc0 = (g.ny - 1) / 2.0 + g.oy;
    const double x0 = g.dx * (0 - xc0), x1 = g.dx * (g.nx - 1 - xc0), y0 = g.dy * (0 - yc0), y1 = g.dy * (g.ny - 1 - yc0);
    g.xlo = std::min(x0, x1) - 0.5 * std::fabs(g.dx);
    g.xhi = std::max(x0, x1) + 0.5 * std::fabs(g.dx);
    g.ylo = std::min(y0, y1) - 0.5 * std::fabs(g.dy);
    g.yhi = std::max(y0, y1) + 0.5 * std::fabs(g.dy);
    if (g.kind != SGB_PAR) {
        g.dsd = rg->dsd;
        g.dso = rg->dsd - rg->dod;
        g.so = rg->source_offset;
        SGB_REQUIRE(g.dsd > 0 && g.dso > 0, "sf: fan beams need dsd > 0 and dso = dsd - dod > 0");
        // every pixel corner strictly in front of the source in every view
        const double xm = std::fabs(g.dx) * (g.nx / 2.0 + std::fabs(g.ox)), ym = std::fabs(g.dy) * (g.ny / 2.0 + std::fabs(g.oy));
        if (!(std::sqrt(xm * xm + ym * ym) < 0.99 * g.dso)) {
            set_error("sf: the image must lie within 0.99 dso of the rotation centre (pixels behind the source)");
            return SGB_ERR_GEOM;
        }
        if (g.kind == SGB_ARC) {
            const double gmax = std::max(std::fabs(-0.5 - g.wb), std::fabs(g.nb - 0.5 - g.wb)) * g.ds / g.dsd;
            if (!(gmax < kPi / 2 - 0.01)) {
                set_error("sf: the arc detector must span less than +-90 degrees about the central ray");
                return SGB_ERR_GEOM;
            }
        }
    }
    *G = g;
    return SGB_OK;
}

// The pixel whose image in slot b is the thread's pixel's image in slot a, as a map (Slot::map) of the
// thread's: slot a's map, then the inverse of slot b's.
int sf_map_between(int a, int b) {
    auto apply = [](int f, int x, int y, int *u, int *v) {
        *u = f & 4 ? y : x;
        *v = f & 4 ? x : y;
        if (f & 1) *u = -*u;
        if (f & 2) *v = -*v;
    };
    for (int f = 0; f < 8; f++) {  // b after f is a, on a point without symmetry
        int x, y, u, v, p, q;
        apply(f, 1, 2, &x, &y);
        apply(b, x, y, &u, &v);
        apply(a, 1, 2, &p, &q);
        if (u == p && v == q) return f;
    }
    return 0;
}

// The representative views' images, and the back-projector's items.  `half`: a half turn of the pixel gives the
// same elements at mirrored bins (parallel beams, centred detector and image), so that it needs no item.
void sf_items(const ScanSlots &S, int na, bool half, std::vector<int4> &reps, std::vector<SfItem> &items) {
    struct Own {
        int rep, slot;
        bool rev;
    };
    std::vector<Own> own(na, Own{-1, 0, false});
    for (int v = 0; v < na; v++) {
        if (own[v].rep >= 0) continue;
        int e[4] = {v, 0, 0, 0};
        own[v] = {v, 0, false};
        for (int j = 1; j < S.ns; j++) {
            bool rev;
            const int u = slot_view(S, na, j, v, &rev);
            e[j] = u | (rev ? kSfRev : 0);
            if (own[u].rep >= 0) e[j] |= kSfDup;
            else own[u] = {v, j, rev};
        }
        reps.push_back(make_int4(e[0], e[1], e[2], e[3]));
    }
    for (int v = 0; v < na; v++) {
        int row[4], map[4], rep[4];
        for (int j = 0; j < S.ns; j++) {
            bool rev;
            const int w = slot_view(S, na, j, v, &rev);
            row[j] = w | (own[w].rev ? kSfRev : 0);
            rep[j] = own[w].rep;
            // the representative sees slot j's image of the pixel where w's slot takes it from
            map[j] = sf_map_between(S.slot[j].map, S.slot[own[w].slot].map);
            if (half && map[j] & 2) {
                map[j] ^= 3;
                row[j] ^= kSfRev;
            }
        }
        for (int j = 0; j < S.ns; j++) {
            bool first = true;
            for (int i = 0; i < j; i++) first &= rep[i] != rep[j] || map[i] != map[j];
            if (!first) continue;
            int e[4] = {kSfDup, kSfDup, kSfDup, kSfDup};
            for (int i = j; i < S.ns; i++)
                if (rep[i] == rep[j] && map[i] == map[j]) e[i] = row[i];
            items.push_back(SfItem{make_int4(e[0], e[1], e[2], e[3]), rep[j], map[j]});
        }
    }
}

// Line splits of the forward projector: enough CTAs for about two resident waves of four-warp
// CTAs (16 per SM), at most 32 and at least 8 image lines per CTA (4 in a plan without shared elements: 64 x 64
// pixels, 100 bins x 61 views 16.7 and 15.0 us; a one-shot call allocates the partial rows, which costs more).
int sf_default_splits(const SfGeo &G, int nrep, int ns, bool kept) {
    int dev = 0, sms = 152;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaGetLastError();
    const long long ctas = (long long)((G.nb + kFwdBins - 1) / kFwdBins) * nrep;
    const long long want = 2LL * 16 * std::max(sms, 1);
    int s = (int)std::min<long long>(32, std::max<long long>(1, (want + ctas - 1) / ctas));
    const int lines = std::max(G.nx, G.ny), least = ns == 1 && kept ? 4 : 8;
    while (s > 1 && lines / s < least) s--;
    return s;
}

int sf_run(sgb_sf_plan *P, bool forward, const float *in, float *out, int flags, cudaStream_t st) {
    const SfGeo &G = P->G;
    const size_t nimg = (size_t)G.nx * G.ny, nsino = (size_t)G.nb * G.na;
    const size_t nin = forward ? nimg : nsino, nout = forward ? nsino : nimg;
    const void *in_dev;
    SGB_TRY(stage_in(in, nin * sizeof(float), flags, P->din, &in_dev, st));
    float *out_dev = out;
    if (!(flags & SGB_DEVICE_PTRS)) {
        SGB_TRY(P->dout.reserve(nout * sizeof(float)));
        out_dev = P->dout.as<float>();
    }
    const float *xcs = P->axes, *ycs = xcs + G.nx;
    const float *src = static_cast<const float *>(in_dev);
    if (forward) {
        const int splits = P->A.splits;
        static_assert(kFwdBpt == 2, "sf_project_kernel accumulates two bins per thread");
        float *dst = out_dev;
        if (splits > 1) {
            SGB_TRY(P->part.reserve(sizeof(float) * nsino * splits));
            dst = P->part.as<float>();
        }
        sf_image_kernel<<<dim3((G.nx + 31) / 32, (G.ny + 31) / 32), dim3(32, 8), 0, st>>>(
            src, P->mask_dev, G.nx, G.ny, P->img, P->img + nimg);
        SGB_TRY(after_launch("sf_image_kernel"));
        auto go = P->A.fslots == 4 ? sf_launch_forward<4>
                                   : (P->A.fslots == 2 ? sf_launch_forward<2> : sf_launch_forward<1>);
        SGB_TRY(go(G.kind, P->A, P->views, P->rays, xcs, ycs, P->img, P->img + nimg, P->reps, dst, st));
        if (splits > 1) {
            sf_sum_splits<<<(unsigned)((nsino + 255) / 256), 256, 0, st>>>(dst, splits, (long long)nsino, out_dev);
            SGB_TRY(after_launch("sf_sum_splits"));
        }
    } else {
        auto go = P->A.sym.ns == 4 ? sf_launch_back_kind<4>
                                   : (P->A.sym.ns == 2 ? sf_launch_back_kind<2> : sf_launch_back_kind<1>);
        SGB_TRY(go(G.kind, P->A, P->item_views, xcs, ycs, src, P->mask_dev, P->item_rows, P->zeros, out_dev, st));
    }
    if (!(flags & SGB_DEVICE_PTRS))
        SGB_CUDA(cudaMemcpyAsync(out, out_dev, nout * sizeof(float), cudaMemcpyDeviceToHost, st));
    if (flags & SGB_ASYNC) return SGB_OK;
    SGB_CUDA(cudaStreamSynchronize(st));
    return SGB_OK;
}

// What a plan is for.
enum { SF_FORWARD = 1, SF_BACK = 2 };

int sf_plan(const sgb_sino_geom *rg, const sgb_image_geom *ig, int uses, std::unique_ptr<sgb_sf_plan> &out) {
    auto P = std::make_unique<sgb_sf_plan>();
    SGB_TRY(sf_geometry(rg, ig, &P->G));
    SfGeo &G = P->G;
    cudaStream_t st = nullptr;
    SfArgs &A = P->A;
    A.nb = G.nb;
    A.na = G.na;
    A.nx = G.nx;
    A.ny = G.ny;
    A.wb = (float)G.wb;
    A.ax = (float)std::fabs(G.dx);
    A.ay = (float)std::fabs(G.dy);
    A.axy = (float)std::fabs(G.dx * G.dy);
    A.hx = (float)(0.5 * std::fabs(G.dx));
    A.hy = (float)(0.5 * std::fabs(G.dy));
    A.sym = scan_slots(rg->kind, G.na, G.nx, G.ny, 2 * G.wb == G.nb - 1.0, G.so == 0, rg->orbit, rg->orbit_start, ig->deltas,
                       ig->offsets, false);
    std::vector<int4> reps;
    std::vector<SfItem> items;
    const bool centred = 2 * G.wb == G.nb - 1.0;
    sf_items(A.sym, G.na, G.kind == SGB_PAR && centred && G.ox == 0 && G.oy == 0, reps, items);
    A.nrep = (int)reps.size();
    A.fslots = 1;
    for (const int4 &e : reps) {
        if (A.sym.ns == 4 && !(e.z & e.w & kSfDup)) A.fslots = 4;
        else if (A.sym.ns > 1 && !(e.y & kSfDup)) A.fslots = std::max(A.fslots, 2);
    }
    A.nitem = (int)items.size();
    // The tables are one block, its first part one copy; a one-shot call pays for no more than it reads.
    const bool fwd = uses & SF_FORWARD;
    if (!fwd) reps.clear();
    if (!(uses & SF_BACK)) items.clear();
    std::vector<char> host;
    size_t bytes = 0;
    auto place = [&bytes](size_t n) {
        const size_t at = bytes;
        bytes = (bytes + n + 255) / 256 * 256;
        return at;
    };
    auto put = [&](const void *p, size_t n) {
        const size_t at = place(n);
        host.resize(bytes);
        if (n) std::memcpy(host.data() + at, p, n);
        return at;
    };
    const std::vector<double> betas = view_angles(rg->na, rg->orbit, rg->orbit_start);
    const size_t betas_at = put(betas.data(), sizeof(double) * G.na);
    std::vector<float> row(G.nx + G.ny);
    for (int i = 0; i < G.nx; i++) row[i] = (float)(G.dx * (i - ((G.nx - 1) / 2.0 + G.ox)));
    for (int j = 0; j < G.ny; j++) row[G.nx + j] = (float)(G.dy * (j - ((G.ny - 1) / 2.0 + G.oy)));
    const size_t axes_at = put(row.data(), sizeof(float) * row.size());
    const size_t nimg = (size_t)G.nx * G.ny;
    const bool masked = ig->mask && std::memchr(ig->mask, 0, nimg);
    const size_t mask_at = masked ? put(ig->mask, nimg) : 0;
    const size_t reps_at = put(reps.data(), sizeof(int4) * reps.size());
    std::vector<int4> rows;
    std::vector<int2> maps;
    for (const SfItem &it : items) {
        rows.push_back(it.rows);
        maps.push_back(make_int2(it.rep, it.map));
    }
    const size_t rows_at = put(rows.data(), sizeof(int4) * rows.size()), maps_at = put(maps.data(), sizeof(int2) * maps.size());
    row.assign(G.nb, 0.f);
    const size_t zeros_at = put(row.data(), sizeof(float) * G.nb);
    const long long nray = fwd ? (long long)G.na * (G.nb + 1) : 0;
    const size_t views_at = place(sizeof(SfView) * G.na), item_views_at = place(sizeof(SfView) * items.size());
    const size_t rays_at = place(sizeof(float2) * (size_t)nray);
    const size_t img_at = place(fwd ? 2 * sizeof(float) * nimg : 0);  // here: a call may be captured
    SGB_TRY(P->block.reserve(bytes));
    char *base = P->block.as<char>();
    SGB_CUDA(cudaMemcpyAsync(base, host.data(), host.size(), cudaMemcpyHostToDevice, st));
    const double *betas_dev = reinterpret_cast<double *>(base + betas_at);
    SfView *views = reinterpret_cast<SfView *>(base + views_at), *item_views = reinterpret_cast<SfView *>(base + item_views_at);
    float2 *rays = reinterpret_cast<float2 *>(base + rays_at);
    P->axes = reinterpret_cast<float *>(base + axes_at);
    P->mask_dev = masked ? reinterpret_cast<uint8_t *>(base + mask_at) : nullptr;
    P->reps = reinterpret_cast<int4 *>(base + reps_at);
    P->item_rows = reinterpret_cast<int4 *>(base + rows_at);
    P->zeros = reinterpret_cast<float *>(base + zeros_at);
    P->views = views;
    P->item_views = item_views;
    P->rays = rays;
    P->img = reinterpret_cast<float *>(base + img_at);
    A.splits = sf_default_splits(G, A.nrep, A.fslots, uses != SF_FORWARD);
    // back: about four CTAs of 256 pixels per SM, at least 8 views each
    const long long tiles = (long long)((A.sym.hx + kBackTx - 1) / kBackTx) * ((A.sym.hy + kBackTy - 1) / kBackTy);
    A.gsplit = (int)std::max<long long>(1, std::min<long long>({8, G.na / 8, (4LL * std::max(1, num_sms()) + tiles / 2) / tiles}));
    const int nview = fwd ? G.na : 0, nset = std::max(nview, (int)items.size());
    sf_setup_views<<<(nset + 127) / 128, 128, 0, st>>>(G, betas_dev, nview, views, (int)items.size(),
                                                      reinterpret_cast<int2 *>(base + maps_at), item_views);
    SGB_TRY(after_launch("sf_setup_views"));
    if (fwd) {
        sf_setup_rays<<<(unsigned)((nray + 255) / 256), 256, 0, st>>>(G, betas_dev, views, rays);
        SGB_TRY(after_launch("sf_setup_rays"));
    }
    SGB_CUDA(cudaStreamSynchronize(st));
    out = std::move(P);
    return SGB_OK;
}

}  // namespace

extern "C" {

int sgb_sf_plan_create(const sgb_sino_geom *rg, const sgb_image_geom *ig, sgb_sf_plan **out) {
    SGB_REQUIRE(out, "sf_plan_create: null argument");
    *out = nullptr;
    std::unique_ptr<sgb_sf_plan> P;
    SGB_TRY(sf_plan(rg, ig, SF_FORWARD | SF_BACK, P));
    *out = P.release();
    return SGB_OK;
}

int sgb_sf_plan_project(sgb_sf_plan *P, const float *image, float *sino, int flags, void *stream) {
    SGB_REQUIRE(P && image && sino, "sf_plan_project: null argument");
    return sf_run(P, true, image, sino, flags, static_cast<cudaStream_t>(stream));
}

int sgb_sf_plan_backproject(sgb_sf_plan *P, const float *sino, float *image, int flags, void *stream) {
    SGB_REQUIRE(P && sino && image, "sf_plan_backproject: null argument");
    return sf_run(P, false, sino, image, flags, static_cast<cudaStream_t>(stream));
}

int sgb_sf_plan_set_line_splits(sgb_sf_plan *P, int splits) {
    SGB_REQUIRE(P && splits >= 1 && splits <= 64, "sf_plan_set_line_splits: need 1 <= splits <= 64");
    P->A.splits = splits;
    return SGB_OK;
}

int sgb_sf_plan_get_line_splits(const sgb_sf_plan *P, int *splits) {
    SGB_REQUIRE(P && splits, "sf_plan_get_line_splits: null argument");
    *splits = P->A.splits;
    return SGB_OK;
}

int sgb_sf_plan_destroy(sgb_sf_plan *P) {
    delete P;
    return SGB_OK;
}

// One-shot calls: a plan of one direction for the call; they always wait for `stream` before returning.
int sgb_sf_project(const sgb_sino_geom *rg, const sgb_image_geom *ig, const float *image, float *sino, int flags,
                   void *stream) {
    SGB_REQUIRE(image && sino, "sf_project: null argument");
    std::unique_ptr<sgb_sf_plan> P;
    SGB_TRY(sf_plan(rg, ig, SF_FORWARD, P));
    return sf_run(P.get(), true, image, sino, flags & ~SGB_ASYNC, static_cast<cudaStream_t>(stream));
}

int sgb_sf_backproject(const sgb_sino_geom *rg, const sgb_image_geom *ig, const float *sino, float *image, int flags,
                       void *stream) {
    SGB_REQUIRE(image && sino, "sf_backproject: null argument");
    std::unique_ptr<sgb_sf_plan> P;
    SGB_TRY(sf_plan(rg, ig, SF_BACK, P));
    return sf_run(P.get(), false, sino, image, flags & ~SGB_ASYNC, static_cast<cudaStream_t>(stream));
}

// _tau(rg, x, y), src/geom/tau.jl:7-60 (host, FP64): tau[i + n*v] = projected s/ds of point i in view v.
int sgb_tau_sino(const sgb_sino_geom *rg, const double *x, const double *y, long long n, double *tau) {
    SGB_REQUIRE(rg && tau && (n == 0 || (x && y)), "tau: null argument");
    SGB_REQUIRE(n >= 0 && rg->na >= 0, "tau: negative size");
    SGB_REQUIRE(rg->kind == SGB_PAR || rg->kind == SGB_ARC || rg->kind == SGB_FLAT, "tau: unknown geometry kind %d",
                rg->kind);
    const std::vector<double> betas = view_angles(rg->na, rg->orbit, rg->orbit_start);
    const double ds = rg->d, dso = rg->dsd - rg->dod;
    for (int v = 0; v < rg->na; v++) {
        const double cb = std::cos(betas[v]), sb = std::sin(betas[v]);
        for (long long i = 0; i < n; i++) {
            double t;
            if (rg->kind == SGB_PAR) {
                t = (x[i] * cb + y[i] * sb) / ds;  // tau.jl:8-11
            } else {
                const double xb = x[i] * cb + y[i] * sb - rg->source_offset, yb = -x[i] * sb + y[i] * cb;  // :44-49
                const double tg = xb / (dso - yb);                                                        // :51
                t = rg->kind == SGB_ARC ? rg->dsd / ds * std::atan(tg) : rg->dsd / ds * tg;               // :28-32
            }
            tau[i + n * v] = t;
        }
    }
    return SGB_OK;
}

}  // extern "C"
