// sgb_back2_kernel.cuh -- the 2D back-projection kernel template, fbp_back_par! / fbp_back_par_xy
// (src/fbp2/back-par.jl:206-315) and fbp_back_fan! / fbp_back_fan_xy (src/fbp2/back-fan.jl:215-336).
// sgb_back2_<detector>.cu instantiate one detector each, so they compile in parallel.
//
// A CTA of 256 threads owns a tile of 32 x 32 pixels: thread (tx, ty) accumulates the pixels (tx, ty + 8k), which share the view's per-column terms and give
// independent accumulation chains.  Views go in chunks.  For each view the CTA maps the
// tile's four corners to detector bins: the parallel, flat and arc maps are monotone in the
// angle under which the source sees a point, so over a rectangle in front of the source the
// extremes are at its vertices.  That bounds the bins the tile reaches, and the view takes one
// of four forms, the same for the whole CTA:
//   fast     every pixel's taps are valid and inside the staged segment: no per-pixel checks
//   checked  segment staged; per pixel the reference's tap rule, a dropped tap reading zeros
//   global   tile not wholly in front of the source (or a segment longer than 254 bins):
//            taps read from global memory with the reference's rule
//   none     the tile misses the detector
// The segment (the tile's bins plus a 2-3 bin margin, far beyond the rounding difference
// between a corner and an interior pixel) is copied into shared memory by one warp per view.
// One warp then lists the chunk's views grouped by form (fast, checked, global), and each group
// runs as its own loop over one packed float4 of per-view constants: a pixel accumulates its
// views in that fixed order, which is deterministic.  Small images split the views over a cluster of
// G CTAs (grid z = slice group * G + rank); their partial tiles are summed through distributed shared
// memory in rank order.  Tiles that the mask rules out are skipped.
//
// A pixel's bin, fraction and weight take 15 (parallel) to 30 (arc) instructions and a tap about four,
// so they are computed once for all taps that share them (template NS, SL):
//   SL  slices of a stack see a pixel alike: one 16-byte load per bin for four of them;
//   NS  so do the images of a pixel under the scan's symmetry, each in its own view ("slots"): the
//       quarter turns of a square image where 90 degrees are a whole number of views, else reflections
//       in x and y (whose bins run the other way: staged reversed), else a half turn (scan_slots).
// Not both: 16 sums per pixel halve the tile, and its segments' copies then cost what the geometry
// saves (arc, 512^2 x 8 slices x 984 views: 798 to 1080 us by the view split; slices alone 744, slots
// alone 929, neither 1908).  Slots alone: 320^2 x 673 parallel views 49 us against 50 to 66, 531 x 140
// x 1130 arc views 95 against 132.
//
// The stack above is bound by its 16-byte shared loads (75 % of the wavefronts, issue 60 %), four
// wavefronts a tap; single images by issue (70 to 79 %): per pixel and view the geometry, and per tap
// one shared load and two multiply-adds.
#pragma once
#include <cooperative_groups.h>
#include <algorithm>

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

// acc[s] += wa near[s] + wb far[s] for the SL slices of one tap at shared address a, one rounding at the sum's
// size.  (Two multiply-adds into the sum are fewer instructions, but their two roundings at its size make its
// error 10 to 40 % larger.)
__device__ __forceinline__ void b2_add2(float &x0, float &x1, float wa, float wb, float n0, float n1, float f0, float f1) {
    asm("{\n\t.reg .b64 x, n, f, a, b;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 a, {%2, %2};\n\tmov.b64 b, {%3, %3};\n\t"
        "mov.b64 n, {%4, %5};\n\tmov.b64 f, {%6, %7};\n\tmul.rn.f32x2 n, a, n;\n\tfma.rn.f32x2 n, b, f, n;\n\t"
        "add.rn.f32x2 x, x, n;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "+f"(x0), "+f"(x1)
        : "f"(wa), "f"(wb), "f"(n0), "f"(n1), "f"(f0), "f"(f1));
}
template <int SL>
__device__ __forceinline__ void b2_tap(uint32_t a, float wa, float wb, float (&acc)[SL]) {
    if constexpr (SL == 1) {
        float n, f;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(n) : "r"(a));
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"(a + 4u));
        acc[0] = __fadd_rn(acc[0], fmaf(wb, f, __fmul_rn(wa, n)));
    } else {
        static_assert(SL == 4, "one or four slices");
        float n[4], f[4];
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(n[0]), "=f"(n[1]), "=f"(n[2]), "=f"(n[3]) : "r"(a));
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]) : "r"(a + 16u));
        b2_add2(acc[0], acc[1], wa, wb, n[0], n[1], f[0], f[1]);
        b2_add2(acc[2], acc[3], wa, wb, n[2], n[3], f[2], f[3]);
    }
}

// Taps at the detector's ends.  The reference takes 1 <= bb < nb (back-par.jl:307, back-fan.jl:328); a slot
// whose bins run the other way sees nb + 1 - bb, and so takes 1 < bb <= nb.  At bb == 1 (`first`) only the
// slots that run along take the tap; at bb == nb (`last`) only the reversed ones, with the weight on bin nb,
// the far one of the two before it.  Parallel views along an axis put whole pixel columns exactly there.
struct B2End {
    bool first, last;
};
template <int NS>
__device__ __forceinline__ B2End b2_end(float bb, int nb) {
    if constexpr (NS == 1) return {false, false};
    return {bb == 1.f, bb == (float)nb};
}

__device__ __forceinline__ void b2_copy4(uint32_t dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void b2_copy16(uint32_t dst, const float4 *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

template <int M, int NS, int SL>
__global__ void __launch_bounds__(kB2X *kB2Y, (kB2Ctas<NS, SL>))
    back2_kernel(const __grid_constant__ Back2Args A, int G) {
    constexpr int VB = 4 * SL;                // bytes per staged bin
    const int W = A.w, VC = A.vc;                       // bins per segment, views per chunk
    const uint32_t SB = (uint32_t)(W * VB), BB = (uint32_t)(VC * NS) * SB;  // bytes per segment and per buffer
    constexpr int NA = NS * SL;               // accumulators per pixel
    constexpr int P = kB2P, T = kB2Y * P;  // passes and rows of a tile
    static_assert(P * NA * kB2X * kB2Y * 4 <= kB2Seg<NS, SL>, "the ranks' partial tiles reuse the segments");
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
        if (cn < nchunk && tid < 4 * VC) {  // lane group of 4 = one view's four corners
            const int v = tid >> 2, cr = tid & 3;
            const float2 sc = v < nvn ? A.trig[vn + v] : make_float2(0.f, 1.f);
            const float cx = A.xds[cr & 1 ? min(A.sym.hx, ix0 + kB2X) - 1 : ix0];
            const float cy = A.yds[cr & 2 ? min(A.sym.hy, iy00 + T) - 1 : iy00];
            float a, b, w;
            bool fr, in;
            b2_col<M>(A, cx, sc.x, sc.y, &a, &b);
            const float bb = b2_pix<M>(A, a, b, cy, sc.x, sc.y, &w, &fr, &in);
            float bmin = bb, bmax = bb;
            int good = fr && in && bb > -1e6f && bb < 1e6f;
            const unsigned quad = 0xfu << (lane & 28);
#pragma unroll
            for (int o = 1; o <= 2; o <<= 1) {
                bmin = fminf(bmin, __shfl_xor_sync(quad, bmin, o));
                bmax = fmaxf(bmax, __shfl_xor_sync(quad, bmax, o));
                good &= __shfl_xor_sync(quad, good, o);
            }
            if (cr == 0 && v < nvn) {
                int form = V_GLOBAL, lo = 0, len = 0;
                if (good) {
                    lo = max(0, (int)floorf(bmin) - 3);
                    const int hi = min(A.nb - 1, (int)floorf(bmax) + 2);
                    if (hi < lo) {
                        form = V_NONE;
                    } else if (hi - lo + 1 <= W - 2) {
                        len = hi - lo + 1;
                        form = (bmin >= 1.5f && bmax < (float)A.nb - 0.5f) ? V_FAST : V_CHECKED;
                    }
                }
                // fast: bits(m) = floor(bb) + 0x4B400000 and tap floor(bb) - 1 is segment entry
                // floor(bb) - 1 - lo, so its shared address is kb + VB bits(m);
                // checked: j = bits(m) - jbias is that entry, valid for j < jlim;
                // global: the view's index
                const uint32_t seg = seg0 + bn * BB + (uint32_t)v * NS * SB;
                uint32_t c0 = (uint32_t)(vn + v), c1 = 0u;
                if (form == V_FAST) {
                    c0 = seg - (uint32_t)VB * (uint32_t)(lo + 1) - (uint32_t)VB * 0x4B400000u;
                } else if (form == V_CHECKED) {
                    c0 = 0x4B400001u + (uint32_t)lo;
                    c1 = (uint32_t)max(len - 1, 0);
                }
                par_s[bn][v] = make_float4(sc.x, sc.y, __uint_as_float(c0), __uint_as_float(c1));
                lo_s[bn][v] = lo;
                len_s[bn][v] = len;
                form_s[bn][v] = form;
            }
        }
        __syncthreads();
        if (cn < nchunk) {
            if (warp == 0) {  // the chunk's views listed by form: fast, checked, global (none dropped)
                const int f = lane < nvn ? form_s[bn][lane] : V_NONE;
                const unsigned lt = (1u << lane) - 1u;
                const unsigned mf = __ballot_sync(0xffffffffu, f == V_FAST);
                const unsigned mc = __ballot_sync(0xffffffffu, f == V_CHECKED);
                const unsigned mg = __ballot_sync(0xffffffffu, f == V_GLOBAL);
                const int nf = __popc(mf), nc = __popc(mc);
                if (f == V_FAST) list_s[bn][__popc(mf & lt)] = lane;
                else if (f == V_CHECKED) list_s[bn][nf + __popc(mc & lt)] = lane;
                else if (f == V_GLOBAL) list_s[bn][nf + nc + __popc(mg & lt)] = lane;
                if (lane == 0) {
                    end_s[bn][0] = nf;
                    end_s[bn][1] = nf + nc;
                    end_s[bn][2] = nf + nc + __popc(mg);
                }
            }
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
        for (int i = 0; i < e0; i++) {  // fast
            const float4 p = par_s[bf][list_s[bf][i]];
            float a, b;
            b2_col<M>(A, x, p.x, p.y, &a, &b);
            const uint32_t kb = __float_as_uint(p.z);
#pragma unroll
            for (int k = 0; k < P; k++) {
                float w2;
                bool fr, in;
                const float bb = b2_pix<M>(A, a, b, y[k], p.x, p.y, &w2, &fr, &in);
                const float m = __fadd_rd(bb, kMagic), f = bb - (m - kMagic);
                const uint32_t ad = kb + (uint32_t)VB * __float_as_uint(m);
                const float wb = w2 * f, wa = w2 - wb;  // back-fan.jl:330
#pragma unroll
                for (int j = 0; j < NS; j++) b2_tap<SL>(ad + (uint32_t)j * SB, wa, wb, acc[k][j]);
            }
        }
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
                const B2End end = b2_end<NS>(bb, A.nb);
                const uint32_t e = __float_as_uint(m) - jbias - end.last;
                const bool ok = e < jlim && in;
                const float f = end.last ? 1.f : bb - (m - kMagic);
                const float wb = ok ? w2 * f : 0.f, wa = ok ? w2 - wb : 0.f;
                const uint32_t ad = seg + (uint32_t)VB * (ok ? e : (uint32_t)(W - 2));
                if (NS > 1 && (end.first || end.last)) {
#pragma unroll
                    for (int j = 0; j < NS; j++) {
                        bool rev;
                        slot_view(A.sym, A.na, j, va + c * VC + vi, &rev);
                        if (rev == end.last) b2_tap<SL>(ad + (uint32_t)j * SB, wa, wb, acc[k][j]);
                    }
                    continue;
                }
#pragma unroll
                for (int j = 0; j < NS; j++) b2_tap<SL>(ad + (uint32_t)j * SB, wa, wb, acc[k][j]);
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
                const B2End end = b2_end<NS>(bb, A.nb);
                const uint32_t il1 = __float_as_uint(m) - 0x4B400001u - end.last;  // floor(bb) - 1
                if (in && il1 < nbm1) {
                    const float wb = w2 * (end.last ? 1.f : bb - (m - kMagic)), wa = w2 - wb;
#pragma unroll
                    for (int j = 0; j < NS; j++) {
                        bool rev = false;
                        const int row = NS == 1 ? v : slot_view(A.sym, A.na, j, v, &rev);
                        if (NS > 1 && (rev ? end.first : end.last)) continue;
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

template <int M, int NS, int SL>
int launch_slots(Back2Args A, cudaStream_t st) {
    const int G = A.split;
    const int groups = floor_div_up(A.nslices, SL);
    constexpr int seg = kB2Seg<NS, SL>;
    auto k = back2_kernel<M, NS, SL>;
    SGB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, seg));
    A.vc = std::min(kB2V, seg / 2 / (NS * A.w * 4 * SL));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(floor_div_up(A.sym.hx, kB2X), floor_div_up(A.sym.hy, kB2Y * kB2P), groups * G);
    cfg.blockDim = dim3(kB2X * kB2Y);
    cfg.dynamicSmemBytes = seg;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = G;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k, A, G);
    if (e != cudaSuccess) {
        set_error("back2_kernel: launch failed: %s", cudaGetErrorString(e));
        return SGB_ERR_CUDA;
    }
    return after_launch("back2_kernel");
}

template <int M>
int launch(const Back2Args &A, cudaStream_t st) {
    if (A.sl == 4) return launch_slots<M, 1, 4>(A, st);
    return A.sym.ns == 4 ? launch_slots<M, 4, 1>(A, st) : (A.sym.ns == 2 ? launch_slots<M, 2, 1>(A, st) : launch_slots<M, 1, 1>(A, st));
}

}  // namespace back2
}  // namespace sgb
