// sgb_back2_kernel.cuh -- the 2D back-projection kernels, fbp_back_par! / fbp_back_par_xy
// (src/fbp2/back-par.jl:206-315) and fbp_back_fan! / fbp_back_fan_xy (src/fbp2/back-fan.jl:215-336).
// sgb_back2_<detector>.cu instantiate one detector each, so they compile in parallel.
//
// A CTA of 256 threads owns a tile of 32 x 32 pixels: thread (tx, ty) accumulates the pixels (tx, ty + 8k),
// which share the view's per-column terms and give independent accumulation chains.  Views go in chunks.  For each view the CTA maps the
// tile's four corners to detector bins: the parallel, flat and arc maps are monotone in the
// angle under which the source sees a point, so over a rectangle in front of the source the
// extremes are at its vertices.  That bounds the bins the tile reaches, and the view takes one
// of four forms, the same for the whole CTA:
//   fast     every pixel's taps are valid and inside the staged segment: no per-pixel checks
//   checked  segment staged; per pixel the reference's tap rule
//   global   tile not wholly in front of the source (or a segment longer than is staged):
//            taps read from global memory with the reference's rule
//   none     the tile misses the detector
// The segment (the tile's bins plus a 2-3 bin margin, far beyond the rounding difference
// between a corner and an interior pixel) is copied into shared memory by one warp per view.
// One warp then lists the chunk's views grouped by form (fast, checked, global), and each group
// runs as its own loop over one packed float4 of per-view constants: a pixel accumulates its
// views in that fixed order, which is deterministic.  Small images split the views over a cluster of
// G CTAs (grid z = slice group * G + rank); their partial tiles are summed through distributed shared
// memory in rank order.  Threads whose pixels the mask rules out take no part in the sums.
//
// A pixel's bin, fraction and weight take 15 (parallel) to 30 (arc) instructions and a tap about four,
// so they are computed once for all taps that share them (back2_kernel, template NS, SL):
//   SL  slices of a stack see a pixel alike: one 16-byte load per bin for four of them;
//   NS  so do the images of a pixel under the scan's symmetry, each in its own view ("slots"): the
//       quarter turns of a square image where 90 degrees are a whole number of views, else reflections
//       in x and y (whose bins run the other way: staged reversed), else a half turn (scan_slots).
// Not both: 16 sums per pixel halve the tile, and its segments' copies then cost what the geometry
// saves (arc, 512^2 x 8 slices x 984 views: 798 to 1080 us by the view split; slices alone 744, slots
// alone 929, neither 1908).  One image from 720 views, pixels of 0.6 bins, by itself and with slots: 512^2
// arc 209 and 135 us, flat 130 and 114, 320^2 parallel 50 and 43.  Without anything to share, and for small
// images, a pixel is taken by itself (back2_plain_kernel); back2_choose predicts the fastest.
//
// The stack above is bound by its 16-byte shared loads (75 % of the wavefronts, issue 60 %), four
// wavefronts a tap; single images by issue (70 to 79 %): per pixel and view the geometry, and per tap
// two shared loads, the weighted tap and one addition.
#pragma once
#include <cooperative_groups.h>
#include <algorithm>
#include <type_traits>

#include "sgb_common.cuh"
#include "sgb_kernels.cuh"

namespace sgb {
namespace back2 {

enum { B2_PAR = 0, B2_FLAT = 1, B2_ARC = 2, B2_ARC_EXACT = 3, B2_ARC_NARROW = 4 };
enum { V_FAST = 0, V_CHECKED = 1, V_GLOBAL = 2, V_NONE = 3 };
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23

// 1/d to within 1 ulp (the hardware approximation; denormals flush to zero)
__device__ __forceinline__ float rcp_approx(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return r;
}

// atan(q) = q P(q^2) on |q| <= 1, P minimax in absolute error (1.1e-7 rad in float32);
// coefficients from csrc/fit_atan_poly.py.
__device__ __forceinline__ float atan_poly(float q) {
    const float t = q * q;
    float p = 2.456899965e-03f;
    p = fmaf(p, t, -1.440206543e-02f);
    p = fmaf(p, t, 3.978239372e-02f);
    p = fmaf(p, t, -7.234959304e-02f);
    p = fmaf(p, t, 1.049899608e-01f);
    p = fmaf(p, t, -1.416124254e-01f);
    p = fmaf(p, t, 1.998590827e-01f);
    p = fmaf(p, t, -3.333259821e-01f);
    p = fmaf(p, t, 9.999998808e-01f);
    return p * q;
}

// The same on |q| <= 0.6 with 6 terms (8.0e-8 rad), for detectors within +-31 deg.
__device__ __forceinline__ float atan_poly6(float q) {
    const float t = q * q;
    float p = -3.794763982e-02f;
    p = fmaf(p, t, 9.173785150e-02f);
    p = fmaf(p, t, -1.391045451e-01f);
    p = fmaf(p, t, 1.996324360e-01f);
    p = fmaf(p, t, -3.333176374e-01f);
    p = fmaf(p, t, 9.999998212e-01f);
    return p * q;
}

// per-(column, view) terms: parallel a = x cos + wb; fan a = dso + x sin, b = x cos - so
template <int M>
__device__ __forceinline__ void b2_col(const Back2Args &A, float x, float sb, float cb, float *a, float *b) {
    if (M == B2_PAR) {
        *a = fmaf(x, cb, A.wb);                       // back-par.jl:293
        *b = 0.f;
    } else {
        *a = fmaf(x, sb, A.dso_ds);                   // back-fan.jl:302
        *b = fmaf(x, cb, -A.so_ds);                   // :303
    }
}

// detector bin bb and weight w2 of the pixel row y; `front`: d > 0 (fan); `inside`: false
// only for the arc polynomials when d <= 0 or |r/d| exceeds their range (1, or 0.6 for the
// narrow one), where the true tap is off the detector: the launcher uses them only for
// detectors narrower than +-45 deg (+-31 deg), with a 4-bin margin
template <int M>
__device__ __forceinline__ float b2_pix(const Back2Args &A, float a, float b, float y, float sb, float cb,
                                        float *w2, bool *front, bool *inside) {
    *inside = true;
    if (M == B2_PAR) {
        *w2 = 1.f;
        *front = true;
        return fmaf(y, sb, a);
    }
    const float d = fmaf(-y, cb, a);
    const float r = fmaf(y, sb, b);
    *front = d > 0.f;
    if (M == B2_FLAT) {                               // :309-311
        const float mag = A.dsd_ds * rcp_approx(d);
        *w2 = mag * mag;
        return fmaf(mag, r, A.wb);
    }
    *w2 = (A.dsd_ds * A.dsd_ds) * rcp_approx(fmaf(d, d, r * r));  // :305-307
    if (M == B2_ARC_EXACT) return fmaf(A.dsd_ds, atan2f(r, d), A.wb);
    // q = r / d with the reciprocal refined by one Newton-Raphson step
    float rd = rcp_approx(d);
    rd = fmaf(rd, fmaf(-d, rd, 1.f), rd);
    const float q = r * rd;
    if (M == B2_ARC_NARROW) {
        *inside = *front && fabsf(q) <= 0.6f;
        return fmaf(A.dsd_ds, atan_poly6(q), A.wb);
    }
    *inside = *front && fabsf(q) <= 1.f;
    return fmaf(A.dsd_ds, atan_poly(q), A.wb);
}

// Weighted taps are formed first and then added, one rounding at the sum's size for a tap or for the taps of
// two views: t = wa near + wb far, then x += t.  (Two multiply-adds into the sum are fewer instructions, but
// their two roundings at its size make its error 10 to 40 % larger.)
struct B2Pair {
    float x, y;
};
__device__ __forceinline__ B2Pair b2_mul2(float w, float x, float y) {
    B2Pair t;
    asm("{\n\t.reg .b64 v, w;\n\tmov.b64 v, {%2, %3};\n\tmov.b64 w, {%4, %4};\n\tmul.rn.f32x2 v, w, v;\n\t"
        "mov.b64 {%0, %1}, v;\n\t}"
        : "=f"(t.x), "=f"(t.y)
        : "f"(x), "f"(y), "f"(w));
    return t;
}
__device__ __forceinline__ void b2_fma2(B2Pair &t, float w, float x, float y) {
    asm("{\n\t.reg .b64 t, v, w;\n\tmov.b64 t, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tmov.b64 w, {%4, %4};\n\t"
        "fma.rn.f32x2 t, w, v, t;\n\tmov.b64 {%0, %1}, t;\n\t}"
        : "+f"(t.x), "+f"(t.y)
        : "f"(x), "f"(y), "f"(w));
}
__device__ __forceinline__ void b2_add2(float &x, float &y, B2Pair t) {
    asm("{\n\t.reg .b64 s, t;\n\tmov.b64 s, {%0, %1};\n\tmov.b64 t, {%2, %3};\n\tadd.rn.f32x2 s, s, t;\n\t"
        "mov.b64 {%0, %1}, s;\n\t}"
        : "+f"(x), "+f"(y)
        : "f"(t.x), "f"(t.y));
}
__device__ __forceinline__ float lds_f32(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
// the taps of V views (1 or 2): of the NS slots, SB bytes apart, or of the SL slices of one
template <int NS, int SL, int V>
__device__ __forceinline__ void b2_taps(const uint32_t (&a)[V], uint32_t SB, const float (&wa)[V], const float (&wb)[V],
                                        float (&acc)[NS][SL]) {
    if constexpr (SL == 1) {
        static_assert(NS % 2 == 0, "slots in pairs");
#pragma unroll
        for (int j = 0; j < NS; j += 2) {
            B2Pair t;
#pragma unroll
            for (int v = 0; v < V; v++) {
                const uint32_t b = a[v] + (uint32_t)j * SB, c = b + SB;
                const float n0 = lds_f32(b), f0 = lds_f32(b + 4u), n1 = lds_f32(c), f1 = lds_f32(c + 4u);
                if (v == 0) t = b2_mul2(wa[v], n0, n1);
                else b2_fma2(t, wa[v], n0, n1);
                b2_fma2(t, wb[v], f0, f1);
            }
            b2_add2(acc[j][0], acc[j + 1][0], t);
        }
    } else {
        static_assert(NS == 1 && SL == 4, "four slices");
        B2Pair t[2];
#pragma unroll
        for (int v = 0; v < V; v++) {
            float n[4], f[4];
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(n[0]), "=f"(n[1]), "=f"(n[2]), "=f"(n[3]) : "r"(a[v]));
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]) : "r"(a[v] + 16u));
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (v == 0) t[h] = b2_mul2(wa[v], n[2 * h], n[2 * h + 1]);
                else b2_fma2(t[h], wa[v], n[2 * h], n[2 * h + 1]);
                b2_fma2(t[h], wb[v], f[2 * h], f[2 * h + 1]);
            }
        }
        b2_add2(acc[0][0], acc[0][1], t[0]);
        b2_add2(acc[0][2], acc[0][3], t[1]);
    }
}

// A chunk's views (v0 .. v0 + nvc - 1 of at most VC): the bins that the tile's pixels (of an nx x ny domain, from
// ix0, iy00) reach in each, at most wmax of them staged at seg + v pitch, and the view's form.
template <int M, int SL>
__device__ __forceinline__ void b2_forms(const Back2Args &A, int nx, int ny, int ix0, int iy00, int v0, int nvc, int VC,
                                         int wmax, uint32_t seg, uint32_t pitch, float4 *par, int *los, int *lens,
                                         int *forms) {
    constexpr uint32_t VB = 4 * SL;  // bytes per staged bin
    if ((int)threadIdx.x >= 4 * VC) return;
    // lane group of 4 = one view's four corners
    const int v = threadIdx.x >> 2, cr = threadIdx.x & 3;
    const float2 sc = v < nvc ? A.trig[v0 + v] : make_float2(0.f, 1.f);
    const float cx = A.xds[cr & 1 ? min(nx, ix0 + kB2X) - 1 : ix0];
    const float cy = A.yds[cr & 2 ? min(ny, iy00 + kB2Y * kB2P) - 1 : iy00];
    float a, b, w;
    bool fr, in;
    b2_col<M>(A, cx, sc.x, sc.y, &a, &b);
    const float bb = b2_pix<M>(A, a, b, cy, sc.x, sc.y, &w, &fr, &in);
    float bmin = bb, bmax = bb;
    int good = fr && in && bb > -1e6f && bb < 1e6f;
    const unsigned quad = VC % 8 == 0 ? 0xffffffffu : 0xfu << (threadIdx.x & 28);  // whole warps, or not
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
        bmin = fminf(bmin, __shfl_xor_sync(quad, bmin, o));
        bmax = fmaxf(bmax, __shfl_xor_sync(quad, bmax, o));
        good &= __shfl_xor_sync(quad, good, o);
    }
    if (cr || v >= nvc) return;
    int form = V_GLOBAL, lo = 0, len = 0;
    if (good) {
        lo = max(0, (int)floorf(bmin) - 3);
        const int hi = min(A.nb - 1, (int)floorf(bmax) + 2);
        if (hi < lo) {
            form = V_NONE;
        } else if (hi - lo + 1 <= wmax) {
            len = hi - lo + 1;
            form = (bmin >= 1.5f && bmax < (float)A.nb - 0.5f) ? V_FAST : V_CHECKED;
        }
    }
    // fast: bits(m) = floor(bb) + 0x4B400000 and tap floor(bb) - 1 is segment entry
    // floor(bb) - 1 - lo, so its shared address is kb + VB bits(m);
    // checked: j = bits(m) - jbias is that entry, valid for j < jlim;
    // global: the view's index
    uint32_t c0 = (uint32_t)(v0 + v), c1 = 0u;
    if (form == V_FAST) {
        c0 = seg + (uint32_t)v * pitch - VB * (uint32_t)(lo + 1) - VB * 0x4B400000u;
    } else if (form == V_CHECKED) {
        c0 = 0x4B400001u + (uint32_t)lo;
        c1 = (uint32_t)max(len - 1, 0);
    }
    par[v] = make_float4(sc.x, sc.y, __uint_as_float(c0), __uint_as_float(c1));
    los[v] = lo;
    lens[v] = len;
    forms[v] = form;
}

// A chunk's views listed by form: fast up to end[0], checked to end[1], global to end[2] (none dropped); one warp.
__device__ __forceinline__ void b2_list(const int *forms, int nvc, int lane, int *list, int *end) {
    const int f = lane < nvc ? forms[lane] : V_NONE;
    const unsigned lt = (1u << lane) - 1u;
    const unsigned mf = __ballot_sync(0xffffffffu, f == V_FAST);
    const unsigned mc = __ballot_sync(0xffffffffu, f == V_CHECKED);
    const unsigned mg = __ballot_sync(0xffffffffu, f == V_GLOBAL);
    const int nf = __popc(mf), nc = __popc(mc);
    if (f == V_FAST) list[__popc(mf & lt)] = lane;
    else if (f == V_CHECKED) list[nf + __popc(mc & lt)] = lane;
    else if (f == V_GLOBAL) list[nf + nc + __popc(mg & lt)] = lane;
    if (lane == 0) {
        end[0] = nf;
        end[1] = nf + nc;
        end[2] = nf + nc + __popc(mg);
    }
}

__device__ __forceinline__ void b2_copy4(uint32_t dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void b2_copy16(uint32_t dst, const float4 *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// One pixel at a time.  A tile's segments are copied between two barriers, and CTAs hide each other's
// copies: at one tap per pixel and view the geometry is most of the work, and staging a chunk ahead, as the
// kernel below does, costs more than it hides (512 x 512, 721 views, flat: 132 us, staged ahead 151; 64 x 64
// parallel 15.6 and 18.9).  Warps take 32 x 1 pixels.
template <int M>
__global__ void __launch_bounds__(kB2X *kB2Y, kB2PlainCtas) back2_plain_kernel(const __grid_constant__ Back2Args A, int G) {
    __shared__ float seg_s[kB2V][kB2W];
    __shared__ float4 par_s[kB2V];  // per view: sin, cos, form constants (bits), segment bound (bits)
    __shared__ int lo_s[kB2V], len_s[kB2V], form_s[kB2V];
    __shared__ int list_s[kB2V], end_s[3];
    __shared__ float part_s[kB2P][kB2X * kB2Y];
    constexpr int P = kB2P, T = kB2Y * P;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ix0 = blockIdx.x * kB2X, iy00 = blockIdx.y * T;
    const int ix = ix0 + lane, iy0 = iy00 + warp;
    const int g = (int)(blockIdx.z % (unsigned)G), sl = (int)(blockIdx.z / (unsigned)G);
    const int per = (A.nv + G - 1) / G;
    const int va = min(A.nv, g * per), vb = min(A.nv, va + per);
    bool active = ix < A.nx && iy0 < A.ny;
    if (A.mask && active) {  // one of the thread's pixels is wanted
        active = false;
#pragma unroll
        for (int k = 0; k < P; k++)
            if (iy0 + k * kB2Y < A.ny) active |= A.mask[ix + (size_t)A.nx * (iy0 + k * kB2Y)] != 0;
    }
    // rows past the image repeat its last one: their taps stay inside the tile's segments
    const float x = ix < A.nx ? A.xds[ix] : 0.f;
    float y[P], acc[P];
#pragma unroll
    for (int k = 0; k < P; k++) {
        y[k] = A.yds[min(iy0 + k * kB2Y, A.ny - 1)];
        acc[k] = 0.f;
    }
    const float *__restrict__ sino = A.sino + (size_t)sl * A.nb * A.na;
    const unsigned nbm1 = (unsigned)(A.nb - 1);
    const long long vstride = (long long)A.ia_skip * A.nb;
    for (int v0 = va; v0 < vb; v0 += kB2V) {
        const int nvc = min(kB2V, vb - v0);
        __syncthreads();  // the previous chunk is consumed
        b2_forms<M, 1>(A, A.nx, A.ny, ix0, iy00, v0, nvc, kB2V, kB2W, (uint32_t)__cvta_generic_to_shared(&seg_s[0][0]),
                       kB2W * 4u, par_s, lo_s, len_s, form_s);
        __syncthreads();
        if (warp == 0) b2_list(form_s, nvc, lane, list_s, end_s);
        for (int v = warp; v < nvc; v += kB2X * kB2Y / 32) {
            if (form_s[v] > V_CHECKED) continue;
            const float *__restrict__ src = sino + (v0 + v) * vstride + lo_s[v];
            const int len = len_s[v];
            for (int j = lane; j < len; j += 32) seg_s[v][j] = __ldg(src + j);
        }
        __syncthreads();
        if (!active) continue;
        const int e0 = end_s[0], e1 = end_s[1], e2 = end_s[2];
        for (int i = 0; i < e0; i++) {  // fast
            const float4 p = par_s[list_s[i]];
            float a, b;
            b2_col<M>(A, x, p.x, p.y, &a, &b);
            const uint32_t kb = __float_as_uint(p.z);
#pragma unroll
            for (int k = 0; k < P; k++) {
                float w2;
                bool fr, in;
                const float bb = b2_pix<M>(A, a, b, y[k], p.x, p.y, &w2, &fr, &in);
                const float m = __fadd_rd(bb, kMagic);
                const uint32_t ad = kb + 4u * __float_as_uint(m);
                const float s0 = lds_f32(ad), s1 = lds_f32(ad + 4u);
                acc[k] = fmaf(fmaf(bb - (m - kMagic), s1 - s0, s0), w2, acc[k]);  // back-fan.jl:330
            }
        }
        for (int i = e0; i < e1; i++) {  // checked
            const int vi = list_s[i];
            const float4 p = par_s[vi];
            float a, b;
            b2_col<M>(A, x, p.x, p.y, &a, &b);
            const uint32_t jbias = __float_as_uint(p.z), jlim = __float_as_uint(p.w);
            const uint32_t seg = (uint32_t)__cvta_generic_to_shared(&seg_s[vi][0]);
#pragma unroll
            for (int k = 0; k < P; k++) {
                float w2;
                bool fr, in;
                const float bb = b2_pix<M>(A, a, b, y[k], p.x, p.y, &w2, &fr, &in);
                const float m = __fadd_rd(bb, kMagic);
                const uint32_t j = __float_as_uint(m) - jbias;  // as in the kernel below
                const bool ok = j < jlim && in;
                const uint32_t ad = seg + 4u * (ok ? j : 0u);
                const float s0 = lds_f32(ad), s1 = lds_f32(ad + 4u);
                const float val = fmaf(bb - (m - kMagic), s1 - s0, s0);
                acc[k] = fmaf(ok ? val : 0.f, w2, acc[k]);
            }
        }
        for (int i = e1; i < e2; i++) {  // global
            const float4 p = par_s[list_s[i]];
            float a, b;
            b2_col<M>(A, x, p.x, p.y, &a, &b);
            const float *__restrict__ row = sino + (long long)__float_as_uint(p.z) * vstride;
#pragma unroll
            for (int k = 0; k < P; k++) {
                float w2;
                bool fr, in;
                const float bb = b2_pix<M>(A, a, b, y[k], p.x, p.y, &w2, &fr, &in);
                const float m = __fadd_rd(bb, kMagic);
                const uint32_t il1 = __float_as_uint(m) - 0x4B400001u;  // floor(bb) - 1
                if (in && il1 < nbm1) {
                    const float s0 = __ldg(row + il1), s1 = __ldg(row + il1 + 1);
                    acc[k] = fmaf(fmaf(bb - (m - kMagic), s1 - s0, s0), w2, acc[k]);
                }
            }
        }
    }
    auto store = [&](int k, float v) {
        const int iy = iy0 + k * kB2Y;
        if (ix >= A.nx || iy >= A.ny) return;
        const size_t idx = ix + (size_t)A.nx * iy;
        A.image[(size_t)sl * A.nx * A.ny + idx] = (A.mask && !A.mask[idx]) ? 0.f : v;
    };
    if (G == 1) {
#pragma unroll
        for (int k = 0; k < P; k++) store(k, acc[k]);
        return;
    }
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
#pragma unroll
    for (int k = 0; k < P; k++) part_s[k][tid] = acc[k];
    cl.sync();
    // rank g finishes the tile rows k * 8 + warp that are = g mod G, summing ranks 0..G-1 in order
#pragma unroll
    for (int k = 0; k < P; k++) {
        if ((k * kB2Y + warp) % G != g) continue;
        float v = 0.f;
        for (int q = 0; q < G; q++) v += *cl.map_shared_rank(&part_s[k][tid], q);
        store(k, v);
    }
    cl.sync();  // peers' shared memory stays alive until every rank has read it
}

template <int M, int NS, int SL>
__global__ void __launch_bounds__(kB2X *kB2Y, kB2Ctas)
    back2_kernel(const __grid_constant__ Back2Args A, int G) {
    constexpr int VB = 4 * SL;                // bytes per staged bin
    const int W = A.w, VC = A.vc;                       // bins per segment, views per chunk
    const uint32_t SB = (uint32_t)(W * VB), BB = (uint32_t)(VC * NS) * SB;  // bytes per segment and per buffer
    constexpr int NA = NS * SL;               // accumulators per pixel
    constexpr int P = kB2P, T = kB2Y * P;  // passes and rows of a tile
    static_assert(P * NA * kB2X * kB2Y * 4 <= kB2Seg, "the ranks' partial tiles reuse the segments");
    extern __shared__ __align__(16) unsigned char seg_s[];  // [2][VC][NS][W] staged bins
    __shared__ float4 par_s[2][kB2V];  // per view: sin, cos, form constants (bits), segment bound (bits)
    __shared__ int lo_s[2][kB2V], len_s[2][kB2V], form_s[2][kB2V];
    __shared__ int list_s[2][kB2V], end_s[2][3];
    // a warp takes 8 x 4 pixels: their taps share more bins, and bank conflicts fall, than along 32 x 1
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tx = (warp & 3) * 8 + (lane & 7), ty = (warp >> 2) * 4 + (lane >> 3);
    const int ix0 = blockIdx.x * kB2X, iy00 = blockIdx.y * T;
    const int ix = ix0 + tx, iy0 = iy00 + ty;
    const int g = (int)(blockIdx.z % (unsigned)G), sl0 = (int)(blockIdx.z / (unsigned)G) * SL;
    const int per = (A.nv + G - 1) / G;
    const int va = min(A.nv, g * per), vb = min(A.nv, va + per);
    bool active = false;  // one of the thread's pixels is wanted
#pragma unroll
    for (int k = 0; k < P; k++)
#pragma unroll
        for (int j = 0; j < NS; j++) {
            size_t idx;
            if (slot_pixel(A.sym, A.nx, A.ny, j, ix, iy0 + k * kB2Y, &idx)) active |= !A.mask || A.mask[idx];
        }
    // rows past the domain repeat its last one: their taps stay inside the tile's segments
    const float x = A.xds[min(ix, A.sym.hx - 1)];
    float y[P], acc[P][NS][SL];
#pragma unroll
    for (int k = 0; k < P; k++) {
        y[k] = A.yds[min(iy0 + k * kB2Y, A.sym.hy - 1)];
#pragma unroll
        for (int j = 0; j < NS; j++)
#pragma unroll
            for (int s = 0; s < SL; s++) acc[k][j][s] = 0.f;
    }
    // one slice's sinogram, or four slices' interleaved
    const size_t nsino = (size_t)A.nb * A.na;
    const float *__restrict__ sino = A.sino + nsino * sl0;
    const float4 *__restrict__ four = reinterpret_cast<const float4 *>(A.sino4) + nsino * (sl0 / 4);
    const unsigned nbm1 = (unsigned)(A.nb - 1);
    const float fnb = (float)A.nb;
    const long long vstride = (long long)A.ia_skip * A.nb;
    const uint32_t seg0 = (uint32_t)__cvta_generic_to_shared(seg_s);
    for (int i = tid; i < 2 * VC * NS * (2 * VB / 4); i += kB2X * kB2Y)  // the zeros that dropped taps read
        reinterpret_cast<float *>(seg_s + (i / (2 * VB / 4)) * SB + (W - 2) * VB)[i % (2 * VB / 4)] = 0.f;
    const int nchunk = (vb - va + VC - 1) / VC;
    __syncthreads();
    // Chunk c + 1's forms and copies go before chunk c's sums, so that the copies' latency overlaps them.
    for (int c = -1; c < nchunk; c++) {
        const int cn = c + 1, bn = cn & 1, vn = va + cn * VC, nvn = min(VC, vb - vn);
        if (c > 0) __syncthreads();  // chunk c - 1, whose buffer this takes, is consumed
        if (cn < nchunk)
            b2_forms<M, SL>(A, A.sym.hx, A.sym.hy, ix0, iy00, vn, nvn, VC, W - 2, seg0 + bn * BB, NS * SB, par_s[bn],
                            lo_s[bn], len_s[bn], form_s[bn]);
        __syncthreads();
        if (cn < nchunk) {
            if (warp == 0) b2_list(form_s[bn], nvn, lane, list_s[bn], end_s[bn]);
            for (int i = warp; i < nvn * NS; i += kB2X * kB2Y / 32) {
                const int v = i / NS, j = i % NS;
                if (form_s[bn][v] > V_CHECKED) continue;
                bool rev = false;
                const int row = NS == 1 ? vn + v : slot_view(A.sym, A.na, j, vn + v, &rev);
                const int lo = lo_s[bn][v], len = len_s[bn][v];
                // entry e holds bin lo + e, counted from the other end when the slot runs the other way
                const long long o = row * vstride + (rev ? A.nb - 1 - lo : lo);
                const int step = rev ? -1 : 1;
                const uint32_t dst = seg0 + bn * BB + (uint32_t)i * SB;
                for (int e = lane; e < len; e += 32) {
                    if constexpr (SL == 4) b2_copy16(dst + (uint32_t)(e * 16), four + o + step * e);
                    else b2_copy4(dst + (uint32_t)(e * 4), sino + o + step * e);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");  // chunk c has landed
        if (c < 0) {
            if (!__syncthreads_or(active)) break;  // the mask rules the whole tile out
            continue;
        }
        __syncthreads();
        const int bf = c & 1;
        if (!active) continue;
        const int e0 = end_s[bf][0], e1 = end_s[bf][1], e2 = end_s[bf][2];
        auto fast = [&](auto views, int i) {  // the views i .. of the list
            constexpr int V = decltype(views)::value;
            float4 p[V];
            float a[V], b[V];
#pragma unroll
            for (int v = 0; v < V; v++) {
                p[v] = par_s[bf][list_s[bf][i + v]];
                b2_col<M>(A, x, p[v].x, p[v].y, &a[v], &b[v]);
            }
#pragma unroll
            for (int k = 0; k < P; k++) {
                uint32_t ad[V];
                float wa[V], wb[V];
#pragma unroll
                for (int v = 0; v < V; v++) {
                    float w2;
                    bool fr, in;
                    const float bb = b2_pix<M>(A, a[v], b[v], y[k], p[v].x, p[v].y, &w2, &fr, &in);
                    const float m = __fadd_rd(bb, kMagic), f = bb - (m - kMagic);
                    ad[v] = __float_as_uint(p[v].z) + (uint32_t)VB * __float_as_uint(m);
                    wb[v] = w2 * f;
                    wa[v] = w2 - wb[v];  // back-fan.jl:330
                }
                b2_taps<NS, SL, V>(ad, SB, wa, wb, acc[k]);
            }
        };
        int i0 = 0;
        for (; i0 + 1 < e0; i0 += 2) fast(std::integral_constant<int, 2>{}, i0);
        if (i0 < e0) fast(std::integral_constant<int, 1>{}, i0);
        bool ends = false;  // a pixel lies exactly on the detector's first or last bin
        for (int i = e0; i < e1; i++) {  // checked
            const int vi = list_s[bf][i];
            const float4 p = par_s[bf][vi];
            float a, b;
            b2_col<M>(A, x, p.x, p.y, &a, &b);
            const uint32_t jbias = __float_as_uint(p.z), jlim = __float_as_uint(p.w);
            const uint32_t seg = seg0 + bf * BB + (uint32_t)vi * NS * SB;
#pragma unroll
            for (int k = 0; k < P; k++) {
                float w2;
                bool fr, in;
                const float bb = b2_pix<M>(A, a, b, y[k], p.x, p.y, &w2, &fr, &in);
                // floor(bb) from the bits of the round-down add bb + 1.5 * 2^23 (|bb| < 2^22).
                // Every bb outside [1, nb) -- also |bb| >= 2^22, inf and NaN -- maps outside the
                // segment, so j < jlim is the reference's tap rule (back-par.jl:307,
                // back-fan.jl:328) for this tile.
                const float m = __fadd_rd(bb, kMagic);
                const uint32_t e = __float_as_uint(m) - jbias;
                const bool ok = e < jlim && in && (NS == 1 || bb != 1.f);
                if (NS > 1) ends |= bb == 1.f || bb == fnb;
                const float wb = ok ? w2 * (bb - (m - kMagic)) : 0.f, wa = ok ? w2 - wb : 0.f;
                const uint32_t ad[1] = {seg + (uint32_t)VB * (ok ? e : (uint32_t)(W - 2))};
                b2_taps<NS, SL, 1>(ad, SB, {wa}, {wb}, acc[k]);
            }
        }
        for (int i = e1; i < e2; i++) {  // global
            const float4 p = par_s[bf][list_s[bf][i]];
            float a, b;
            b2_col<M>(A, x, p.x, p.y, &a, &b);
            const int v = (int)__float_as_uint(p.z);
#pragma unroll
            for (int k = 0; k < P; k++) {
                float w2;
                bool fr, in;
                const float bb = b2_pix<M>(A, a, b, y[k], p.x, p.y, &w2, &fr, &in);
                const float m = __fadd_rd(bb, kMagic);
                const uint32_t il1 = __float_as_uint(m) - 0x4B400001u;  // floor(bb) - 1
                if (NS > 1) ends |= bb == 1.f || bb == fnb;
                if (in && il1 < nbm1 && (NS == 1 || bb != 1.f)) {
                    const float wb = w2 * (bb - (m - kMagic)), wa = w2 - wb;
#pragma unroll
                    for (int j = 0; j < NS; j++) {
                        bool rev = false;
                        const int row = NS == 1 ? v : slot_view(A.sym, A.na, j, v, &rev);
                        const long long o = row * vstride + (rev ? nbm1 - il1 : il1);
                        const int step = rev ? -1 : 1;
                        if constexpr (SL == 4) {
                            const float4 n = __ldg(four + o), f = __ldg(four + o + step);
                            const float nv[4] = {n.x, n.y, n.z, n.w}, fv[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                            for (int s = 0; s < SL; s++)
                                acc[k][j][s] = __fadd_rn(acc[k][j][s], fmaf(wb, fv[s], __fmul_rn(wa, nv[s])));
                        } else {
                            acc[k][j][0] = __fadd_rn(acc[k][j][0], fmaf(wb, __ldg(sino + o + step), __fmul_rn(wa, __ldg(sino + o))));
                        }
                    }
                }
            }
        }
        // Pixels exactly on the detector's first or last bin, bb = 1 or nb.  The reference takes 1 <= bb < nb
        // (back-par.jl:307, back-fan.jl:328); a slot whose bins run the other way sees nb + 1 - bb.  So a slot
        // that sees its own bin 1 takes it, and one that sees bin nb takes nothing.  Parallel views along an
        // axis put whole pixel columns there.  A pass of its own: per slot in the loops above it cost a third.
        if (NS > 1 && ends)
#pragma unroll 1
            for (int i = e0; i < e2; i++) {
                const int vi = list_s[bf][i];
                const float4 p = par_s[bf][vi];
                float a, b;
                b2_col<M>(A, x, p.x, p.y, &a, &b);
#pragma unroll
                for (int k = 0; k < P; k++) {
                    float w2;
                    bool fr, in;
                    const float bb = b2_pix<M>(A, a, b, y[k], p.x, p.y, &w2, &fr, &in);
                    if (!in || A.nb < 2 || !(bb == 1.f || bb == fnb)) continue;
#pragma unroll
                    for (int j = 0; j < NS; j++) {
                        bool rev;
                        const float *row = sino + slot_view(A.sym, A.na, j, va + c * VC + vi, &rev) * vstride;
                        if (rev != (bb == fnb)) continue;
                        const float n = __ldg(row), f = __ldg(row + 1);
                        acc[k][j][0] = __fadd_rn(acc[k][j][0], __fmul_rn(w2, fmaf(0.f, f - n, n)));
                    }
                }
            }
    }
    auto store = [&](int k, int j, int s, float v) {
        size_t idx;
        if (sl0 + s >= A.nslices || !slot_pixel(A.sym, A.nx, A.ny, j, ix, iy0 + k * kB2Y, &idx)) return;
        A.image[(size_t)(sl0 + s) * A.nx * A.ny + idx] = (A.mask && !A.mask[idx]) ? 0.f : v;
    };
    if (G == 1) {
#pragma unroll
        for (int k = 0; k < P; k++)
#pragma unroll
            for (int j = 0; j < NS; j++)
#pragma unroll
                for (int s = 0; s < SL; s++) store(k, j, s, acc[k][j][s]);
        return;
    }
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    float *part = reinterpret_cast<float *>(seg_s);  // [P * NA][threads]
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int k = 0; k < P; k++)
#pragma unroll
        for (int j = 0; j < NS; j++)
#pragma unroll
            for (int s = 0; s < SL; s++) part[((k * NS + j) * SL + s) * (kB2X * kB2Y) + tid] = acc[k][j][s];
    cl.sync();
    // rank g finishes every G-th sum, adding ranks 0..G-1 in order
    for (int i = g; i < P * NA; i += G) {
        float v = 0.f;
        for (int q = 0; q < G; q++) v += cl.map_shared_rank(part, q)[i * (kB2X * kB2Y) + tid];
        store(i / NA, i / SL % NS, i % SL, v);
    }
    cl.sync();  // peers' shared memory stays alive until every rank has read it
}

template <typename K>
int launch_kernel(K k, const Back2Args &A, int hx, int hy, int groups, int smem, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(floor_div_up(hx, kB2X), floor_div_up(hy, kB2Y * kB2P), groups * A.split);
    cfg.blockDim = dim3(kB2X * kB2Y);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = A.split;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k, A, A.split);
    if (e != cudaSuccess) {
        set_error("back2_kernel: launch failed: %s", cudaGetErrorString(e));
        return SGB_ERR_CUDA;
    }
    return after_launch("back2_kernel");
}

template <int M, int NS, int SL>
int launch_slots(Back2Args A, cudaStream_t st) {
    constexpr int seg = kB2Seg;
    auto k = back2_kernel<M, NS, SL>;
    SGB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, seg));
    A.vc = std::min(kB2V, seg / 2 / (NS * A.w * 4 * SL));
    return launch_kernel(k, A, A.sym.hx, A.sym.hy, floor_div_up(A.nslices, SL), seg, st);
}

template <int M>
int launch(const Back2Args &A, cudaStream_t st) {
    if (A.sl == 4) return launch_slots<M, 1, 4>(A, st);
    if (A.sym.ns == 4) return launch_slots<M, 4, 1>(A, st);
    if (A.sym.ns == 2) return launch_slots<M, 2, 1>(A, st);
    return launch_kernel(back2_plain_kernel<M>, A, A.nx, A.ny, A.nslices, 0, st);
}

}  // namespace back2
}  // namespace sgb
