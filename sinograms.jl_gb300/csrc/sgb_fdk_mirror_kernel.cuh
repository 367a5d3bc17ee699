// sgb_fdk_mirror_kernel.cuh -- TMA-staged FDK back-projection of scans with mirror symmetry.
//
// Same arithmetic and edge rule as cbct_back_fan_voxel (src/fbp3/cbct-back.jl:150-213) and the same
// detector boxes by TMA in an mbarrier ring as fdk_tma_kernel; what changes is which voxels a thread takes.  Reflecting a voxel column and the source angle together,
//   X: (x, y) -> (-x, y), beta -> -beta        s -> -s, same t and weight
//   Y: (x, y) -> (x, -y), beta -> 180 - beta   s -> -s, same t and weight
//   XY: (x, y) -> (-x, -y), beta -> beta + 180 same s, t and weight
//   Z: z -> -z, same view                      t -> -t, same s and weight,
// maps an orbit of whole turns onto itself whenever the reflected angles are views of the scan
// (X: any number of views that start at 0; Y and XY: an even number), and Z any orbit.  A thread
// therefore takes a column of the fundamental domain for every view v, together with its images
// ("slots") in their views: the detector row, its fraction and the interpolation weights, which
// take about half of the unmirrored kernel's instructions, are computed once per voxel and serve
// all slots; per slot there is left one address, one 8-byte load and two (FP32) or three (FP16) FMAs.
//
// FP16 quads (F16 form) use X, Y and XY only, and only on an FP32 voxel grid that is exactly
// symmetric: their t-weights are rounded on a grid anchored at every zbase-th voxel, which a reflection
// in z would move, and their s-fractions to 2^-11, where a column's last FP32 bit can decide.
//
// Bound by the shared loads: an 8-byte tap per lane takes two wavefronts, 4.9e12 updates/s for the
// chip, and next by issue.  512 x 512 x 64 voxels from 180 views: F16 0.97 ms, 8.8 thread instructions
// an update, 73 % of the issue slots, 69 % of the wavefronts (unmirrored 1.15 ms, 10.8); FP32 pairs
// 1.13 ms, 65 % (unmirrored 1.66 ms, 15.0).  Whole steps of 512 x 512 x 256 from 720 views: F16 18.2 to
// 15.5 ms, FP32 24.6 to 18.5.
#pragma once
#include <cooperative_groups.h>
#include <cuda.h>

#include "sgb_fdk_mirror.cuh"
#include "sgb_fdk_tma_dev.cuh"

namespace sgb {
namespace fdkdev {

// Per stage: the view's trig and, for the two detector columns s and -s that the slots see (the
// second only with reflections), what turns a tap's index into a box address.
struct __align__(16) MirStage {
    uint32_t bias[2], span[2];  // bits of floor(bs) - bias <= span: tap well inside the detector, and staged
    float flo, fhi;             // a run with flo <= t < fhi needs no row checks
    uint32_t off[2];            // box address of (row 0, first valid column), without the slot's box
    uint32_t zoff;              // ZM: from a slot's address of row 0 to its image's
    int t0;                     // first staged row (0-based)
    int s0[2];                  // first staged columns
    float2 sc;
};

// What every view of a tile needs of its z-run, kept out of the registers.
struct __align__(16) MirRun {
    float z, zlo, zhi;       // first voxel, and the ends in ascending order
    int iz;                  // index of the first voxel
    float zb[2], koff[2];    // quads: anchor below each 16 voxels, and their offset from it
};

constexpr uint32_t kFloorBits = 0x4B400000u;  // bits(__fadd_rd(v, 1.5 * 2^23)) = floor(v) + kFloorBits

// acc += a * b for two voxels at once (FFMA2: half the issue slots of two FFMAs).
__device__ __forceinline__ void fma2(float &x0, float &x1, float a0, float a1, float b0, float b1) {
    asm("{\n\t.reg .b64 x, a, b;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "fma.rn.f32x2 x, a, b, x;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "+f"(x0), "+f"(x1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

// Floors (as bits) and interpolation weights of two detector rows: m = floor bits, wb = w2 frac,
// wa = w2 - wb.
__device__ __forceinline__ void rows2(float b0, float b1, float w2, uint32_t &m0, uint32_t &m1, float &wa0, float &wa1,
                                      float &wb0, float &wb1) {
    asm("{\n\t.reg .b64 b, m, f, w, c, d;\n\tmov.b64 b, {%6, %7};\n\tmov.b64 w, {%8, %8};\n\t"
        "mov.b64 c, {%9, %9};\n\tadd.rm.f32x2 m, b, c;\n\tsub.rn.f32x2 f, m, c;\n\tsub.rn.f32x2 f, b, f;\n\t"
        "mul.rn.f32x2 f, w, f;\n\tsub.rn.f32x2 d, w, f;\n\tmov.b64 {%0, %1}, m;\n\tmov.b64 {%2, %3}, d;\n\t"
        "mov.b64 {%4, %5}, f;\n\t}"
        : "=r"(m0), "=r"(m1), "=f"(wa0), "=f"(wa1), "=f"(wb0), "=f"(wb1)
        : "f"(b0), "f"(b1), "f"(w2), "f"(12582912.0f));
}

// x or y range of a tile's slot: indices i0 .. i0 + n - 1, mirrored in an axis of `size` voxels.
__device__ __forceinline__ void mir_range(int i0, int n, int size, bool flip, float c0, float d, float *lo, float *hi) {
    const int a = flip ? size - 1 - i0 : i0, b = flip ? size - i0 - n : i0 + n - 1;
    const float u = c0 + a * d, v = c0 + b * d;
    *lo = fminf(u, v);
    *hi = fmaxf(u, v);
}

// Slot j's view for view v of the scan.
__device__ __forceinline__ int mir_slot_view(const FdkMirrorArgs &M, int j, int v) {
    const int u = M.vsgn[j] * v + M.voff[j];  // in (-nviews, 2 nviews)
    return u < 0 ? u + M.nviews : (u >= M.nviews ? u - M.nviews : u);
}

// Voxel extents of slot j of tile (bx, by, bz).
struct MirExtent {
    float xlo, xhi, ylo, yhi, zlo, zhi;
};
__device__ __forceinline__ MirExtent mir_extent(const FdkMirrorArgs &M, int j, int bx, int by, int bz) {
    const FdkTmaArgs &A = M.A;
    MirExtent e;
    mir_range(bx * kTX, kTX, A.nx, M.flip[j] & MIR_X, A.x0, A.dx, &e.xlo, &e.xhi);
    mir_range(by * kTY, kTY, A.ny, M.flip[j] & MIR_Y, A.y0, A.dy, &e.ylo, &e.yhi);
    int iz = M.iz0 + bz * M.kz;
    if (!A.quad && iz + M.kz > A.nz && A.nz >= M.kz) iz = A.nz - M.kz;  // as the kernel's runs
    mir_range(iz, M.kz, A.nz, false, A.z0, A.dz, &e.zlo, &e.zhi);
    return e;
}

// Detector coordinate's factors (bs = fma(c, p, ws)), magnification and weight of a column.
template <bool ARC>
__device__ __forceinline__ void mir_column(const FdkTmaArgs &A, float x, float y, float2 sc, float *c, float *p,
                                           float *mag, float *w2) {
    const float xb = fmaf(x, sc.y, y * sc.x);                 // cbct-back.jl:174
    const float yb = A.dso_ds - fmaf(-x, sc.x, y * sc.y);     // :175
    *mag = __fdividef(A.dsd_ds, yb);
    if (ARC) {
        *c = A.dsd_ds;
        *p = atan2f(xb, yb);
        *w2 = __fdividef(A.dsd_ds * A.dsd_ds, fmaf(xb, xb, yb * yb));
    } else {
        *c = *mag;
        *p = xb;
        *w2 = *mag * *mag;
    }
}

// The slots of a (column, view) whose taps may leave the detector or the box, by the reference's rule; a
// dropped tap reads a safe sample with weight 0.  t is anchored at every zbase-th voxel, as in the
// unmirrored kernel.  On a voxel grid that is exactly symmetric in FP32 (EX) the slots' columns have the
// same bits, so one tap position serves all; otherwise each slot takes its own column, so that rounding
// drops the same taps as there.
template <typename TP, bool ARC, int NV, bool ZM, int KZ, bool EX>
__device__ __forceinline__ void mir_checked(const FdkMirrorArgs &M, int iz, const MirStage &S, uint32_t box,
                                            float (&acc)[NV * (ZM ? 2 : 1)][KZ]) {
    constexpr int NZ = ZM ? 2 : 1, NG = EX ? 1 : NV;  // groups of slots with a column of their own
    const FdkTmaArgs &A = M.A;
    const uint32_t rb = (uint32_t)A.W * 8u;
    const int ix = blockIdx.x * kTX + threadIdx.x % kTX, iy = blockIdx.y * kTY + threadIdx.x / kTX;
#pragma unroll
    for (int g = 0; g < NG; g++) {
        const int gf = NV == 4 ? g : M.flip[g];
        const float x = A.x0 + (gf & MIR_X ? A.nx - 1 - ix : ix) * A.dx;
        const float y = A.y0 + (gf & MIR_Y ? A.ny - 1 - iy : iy) * A.dy;
        const float2 sc = make_float2(gf & MIR_X ? -S.sc.x : S.sc.x, gf & MIR_Y ? -S.sc.y : S.sc.y);
        float c, p, mag, w2;
        mir_column<ARC>(A, x, y, sc, &c, &p, &mag, &w2);
        const float magt = mag * A.inv_dtds, dbt = magt * A.dz;
        float fs[NV];
        uint32_t kb[NV];  // box address of the tap's column in the slot's first row
        float wj[NV];     // w2, or 0 when the s tap drops
#pragma unroll
        for (int j = 0; j < NV; j++) {
            if (!EX && j != g) continue;
            const int flip = NV == 4 ? j : M.flip[j];
            const bool neg = EX && (flip == MIR_X || flip == MIR_Y);
            const float bs = fmaf(c, neg ? -p : p, A.ws), fis = floorf(bs);
            int col = (int)fis - 1 - S.s0[NV == 4 && j >= 2 ? 3 - j : j];
            bool ok = fis >= 1.f && fis < (float)A.ns;  // :197 (s part)
            if (ok && (col < 0 || col > A.W - 2)) {
                atomicOr(A.err, 1);
                ok = false;
            }
            wj[j] = ok ? w2 : 0.f;
            fs[j] = ok ? bs - fis : 0.f;
            kb[j] = box + (uint32_t)(j * NZ * A.box_bytes + (ok ? col : 0) * 8);
        }
#pragma unroll
        for (int zi = 0; zi < NZ; zi++) {
            const int t0 = zi ? M.m2 - S.t0 - A.H - 1 : S.t0;  // the box's first row (0-based)
            const int lo = max(1, t0 + 1), hi = min(A.nt - 1, t0 + A.H - 1);
            if (hi < lo) continue;
            const unsigned span = (unsigned)(hi - lo);
#pragma unroll
            for (int k = 0; k < KZ; k++) {
                const int z = zi ? A.nz - 1 - iz - k : iz + k, zb = z & ~(M.zbase - 1);
                const float kf = (float)(z - zb), b0 = fmaf(magt, A.z0 + zb * A.dz, A.wt);
                const float bt = fmaf(kf, dbt, b0);  // :189,192
                const float fit = floorf(bt);
                const int it = (int)fit;
                const bool ok = (unsigned)(it - lo) <= span;  // :197 (t part)
                if (!ok && it >= 1 && it < A.nt && (unsigned)z < (unsigned)A.nz) atomicOr(A.err, 1);  // not staged
                const uint32_t r = (uint32_t)(((ok ? it : lo) - t0 - 1) * (int)rb + zi * A.box_bytes);
                const float ft = ok ? (kQuad<TP> ? (fmaf(kf, dbt, b0 + kQMagic) - kQMagic) - fit : bt - fit) : 0.f;
#pragma unroll
                for (int j = 0; j < NV; j++) {
                    if (!EX && j != g) continue;
                    float &s = acc[j * NZ + zi][k];
                    const float wk = ok ? wj[j] : 0.f;
                    if constexpr (kQuad<TP>) {
                        unsigned short w2h;
                        uint32_t fsh;
                        asm("cvt.rn.f16.f32 %0, %1;" : "=h"(w2h) : "f"(wk));
                        asm("cvt.rn.f16x2.f32 %0, %1, %1;" : "=r"(fsh) : "f"(fs[j]));
                        quad_tap<false>(lds_quad(kb[j] + r), fsh, pack_f16x2(ft, 0.f), w2h, s);
                    } else {
                        const float a0 = srow<TP>(kb[j] + r, fs[j]), a1 = srow<TP>(kb[j] + r + rb, fs[j]);
                        s = fmaf(wk, fmaf(ft, a1 - a0, a0), s);  // :205-208
                    }
                }
            }
        }
    }
}

// All slots of one (column, view): acc[slot][k] += the tap of voxel k.  Slot s = j (ZM: 2 j and
// 2 j + 1 for z and -z).
template <typename TP, bool ARC, int NV, bool ZM, int KZ, bool EX>
__device__ __forceinline__ void mir_view(const FdkMirrorArgs &M, float x, float y, const MirRun &R, const MirStage &S,
                                         uint32_t box, float (&acc)[NV * (ZM ? 2 : 1)][KZ]) {
    constexpr int NZ = ZM ? 2 : 1, NS = NV * NZ, NU = NV < 2 ? 1 : 2;
    const FdkTmaArgs &A = M.A;
    const uint32_t rb = (uint32_t)A.W * 8u;  // bytes per box row
    const uint32_t bb = (uint32_t)A.box_bytes;
    float c, p, mag, w2;
    mir_column<ARC>(A, x, y, S.sc, &c, &p, &mag, &w2);
    float fs[NV];
    uint32_t kb[NS];  // box address of (row 0, the tap's column); ZM: of the mirrored row
    bool all = true, maybe = false;
    auto column = [&](int j, float bs, uint32_t b) {
        const float m = __fadd_rd(bs, 12582912.0f);
        const uint32_t bits = __float_as_uint(m);
        const uint32_t col = bits - S.bias[j];
        all &= col <= S.span[j];
        maybe |= bits - kFloorBits <= (uint32_t)A.ns;  // 0 <= floor(bs) <= ns: taps, and a sample more
        fs[j] = bs - (m - 12582912.0f);
        kb[j * NZ] = b + S.off[j] + col * 8u;
    };
#pragma unroll
    for (int j = 0; j < NU; j++) {
        const bool neg = NV == 4 ? j == 1 : j && M.flip[1] != (MIR_X | MIR_Y);
        column(j, fmaf(c, neg ? -p : p, A.ws), box + (uint32_t)(j * NZ) * bb);
    }
    if constexpr (NV == 4) {
#pragma unroll
        for (int j = 2; j < 4; j++) {
            fs[j] = fs[3 - j];
            kb[j] = kb[3 - j] + (uint32_t)(2 * j - 3) * bb;
        }
    }
    if (!maybe) return;
    if (ZM)
#pragma unroll
        for (int j = 0; j < NV; j++) kb[j * NZ + NZ - 1] = kb[j * NZ] + S.zoff;
    const float magt = mag * A.inv_dtds;
    const float dbt = magt * A.dz;
    const float bt0 = fmaf(magt, R.z, A.wt);  // :189,192
    const float bmin = fmaf(magt, R.zlo, A.wt), bmax = fmaf(magt, R.zhi, A.wt);
    if (!(all && bmin >= S.flo && bmax < S.fhi)) {
        mir_checked<TP, ARC, NV, ZM, KZ, EX>(M, R.iz, S, box, acc);
        return;
    }

    if constexpr (kQuad<TP>) {
        static_assert(!ZM, "quads do not reflect in z");
        uint32_t fsh[NV];
        unsigned short w2h;
#pragma unroll
        for (int j = 0; j < NV; j++) asm("cvt.rn.f16x2.f32 %0, %1, %1;" : "=r"(fsh[j]) : "f"(fs[j]));
        asm("cvt.rn.f16.f32 %0, %1;" : "=h"(w2h) : "f"(w2));
        constexpr int SUB = KZ < 16 ? KZ : 16;  // divides every zbase
#pragma unroll
        for (int j = 0; j < NV; j++) kb[j] -= kQRowBias * rb;
#pragma unroll
        for (int h = 0; h < KZ / SUB; h++) {
            // the t grid is anchored at the zbase-th voxel below
            const float koff = R.koff[h], b0 = fmaf(magt, R.zb[h], A.wt) + kQMagic;
#pragma unroll
            for (int k = 0; k < SUB; k += 2) {
                const uint32_t m0 = __float_as_uint(fmaf(koff + (float)k, dbt, b0));
                const uint32_t m1 = __float_as_uint(fmaf(koff + (float)(k + 1), dbt, b0));
                const uint32_t r0 = (m0 >> 10) * rb, r1 = (m1 >> 10) * rb;
                const uint32_t ft2 = quad_ft2(m0, m1);
#pragma unroll
                for (int j = 0; j < NV; j++) {
                    const uint2 q0 = lds_quad(kb[j] + r0), q1 = lds_quad(kb[j] + r1);
                    quad_tap<false>(q0, fsh[j], ft2, w2h, acc[j][h * SUB + k]);
                    quad_tap<true>(q1, fsh[j], ft2, w2h, acc[j][h * SUB + k + 1]);
                }
            }
        }
    } else {
        // the row at offset r of slot s and the row after it (away from the mirror for -z)
        auto near_at = [&](int s, uint32_t r) { return ZM && (s & 1) ? kb[s] - r : kb[s] + r; };
        auto step = [&](int s, uint32_t a) { return ZM && (s & 1) ? a - rb : a + rb; };
#pragma unroll
        for (int s = 0; s < NS; s++) kb[s] = near_at(s, (0u - kFloorBits) * rb);
        const unsigned active = __activemask();
        if (__all_sync(active, dbt >= 0.f && dbt < (NS == 2 ? 1.5f : 0.999f))) {
            // streaming: a voxel on its predecessor's detector row, or on the next, loads its far row only
            float nv[NS], fv[NS];
            uint32_t prev = __float_as_uint(__fadd_rd(bt0, 12582912.0f));
#pragma unroll
            for (int s = 0; s < NS; s++) {
                nv[s] = 0.f;
                fv[s] = srow<TP>(near_at(s, prev * rb), fs[s / NZ]);  // :205
                kb[s] = step(s, kb[s]);
            }
            prev -= 1;  // the first voxel advances onto its own row
            auto run = [&](auto skips) {
#pragma unroll
                for (int k = 0; k < KZ; k += 2) {
                    uint32_t m0, m1;
                    float wa0, wa1, wb0, wb1, n0[NS], n1[NS], f0[NS], f1[NS];
                    rows2(fmaf((float)k, dbt, bt0), fmaf((float)(k + 1), dbt, bt0), w2, m0, m1, wa0, wa1, wb0, wb1);
                    const uint32_t d0 = m0 - prev, d1 = m1 - m0;
                    prev = m1;
                    m0 *= rb;
                    m1 *= rb;
#pragma unroll
                    for (int s = 0; s < NS; s++) {
                        n0[s] = d0 ? fv[s] : nv[s];                       // the old far row once passed
                        f0[s] = srow<TP>(near_at(s, m0), fs[s / NZ]);  // :206
                        n1[s] = d1 ? f0[s] : n0[s];
                        f1[s] = srow<TP>(near_at(s, m1), fs[s / NZ]);
                    }
                    if (skips.value) {  // a voxel two or more rows on loads its near row too
                        if (d0 > 1)
#pragma unroll
                            for (int s = 0; s < NS; s++) {
                                n0[s] = srow<TP>(ZM && (s & 1) ? near_at(s, m0) + rb : near_at(s, m0) - rb, fs[s / NZ]);
                                n1[s] = d1 ? n1[s] : n0[s];
                            }
                        if (d1 > 1)
#pragma unroll
                            for (int s = 0; s < NS; s++)
                                n1[s] = srow<TP>(ZM && (s & 1) ? near_at(s, m1) + rb : near_at(s, m1) - rb, fs[s / NZ]);
                    }
#pragma unroll
                    for (int s = 0; s < NS; s++) {
                        fma2(acc[s][k], acc[s][k + 1], wa0, wa1, n0[s], n1[s]);  // :208
                        fma2(acc[s][k], acc[s][k + 1], wb0, wb1, f0[s], f1[s]);
                        nv[s] = n1[s];
                        fv[s] = f1[s];
                    }
                }
            };
            if constexpr (NS == 2) {  // (four slots leave no registers for it)
                if (__all_sync(active, dbt < 0.999f)) run(std::false_type{});
                else run(std::true_type{});
            } else {
                run(std::false_type{});
            }
        } else {
#pragma unroll
            for (int k = 0; k < KZ; k += 2) {
                uint32_t m0, m1;
                float wa0, wa1, wb0, wb1;
                rows2(fmaf((float)k, dbt, bt0), fmaf((float)(k + 1), dbt, bt0), w2, m0, m1, wa0, wa1, wb0, wb1);
#pragma unroll
                for (int s = 0; s < NS; s++) {
                    const uint32_t a0 = near_at(s, m0 * rb), a1 = near_at(s, m1 * rb);
                    fma2(acc[s][k], acc[s][k + 1], wa0, wa1, srow<TP>(a0, fs[s / NZ]), srow<TP>(a1, fs[s / NZ]));
                    fma2(acc[s][k], acc[s][k + 1], wb0, wb1, srow<TP>(step(s, a0), fs[s / NZ]),
                         srow<TP>(step(s, a1), fs[s / NZ]));
                }
            }
        }
    }
}

// Fills a stage with the boxes of view v0 + g (one warp; lane j < NV holds slot j's view and its
// trig).  The slots share the boxes' first row, and X and Y, or the column and XY, their first
// column: equal up to rounding, which the margin covers.
template <typename TP, bool ARC, int NV, int NZ>
__device__ __forceinline__ void mir_fill(const FdkMirrorArgs &M, const CUtensorMap *map, unsigned char *dst,
                                         MirStage &S, const MirExtent *ext, uint64_t *full, float2 sc, int view,
                                         int lane) {
    constexpr int NS = NV * NZ;
    const FdkTmaArgs &A = M.A;
    int s0 = 0, t0 = 0;
    if (lane < NV) {
        const MirExtent e = ext[lane];
        int w, h;
        tile_box<ARC>(A, sc.x, sc.y, e.xlo, e.xhi, e.ylo, e.yhi, e.zlo, e.zhi, &s0, &t0, &w, &h);
    }
    t0 = __shfl_sync(0xffffffffu, t0, 0);
    const int j = lane / NZ, z = lane % NZ;
    if (lane < (NV < 2 ? 1 : 2)) {
        // the detector's first and last taps are left to the checked form: rounding decides whether they drop
        const int first = max(s0, 1), last = min(A.ns - 3, s0 + A.W - 2);
        S.s0[lane] = s0;
        S.bias[lane] = last < first ? 0xffffffffu : kFloorBits + 1u + (uint32_t)first;
        S.span[lane] = last < first ? 0u : (uint32_t)(last - first);
        S.off[lane] = (uint32_t)((first - s0) * 8) - (uint32_t)((t0 + 1) * A.W * 8);
    }
    s0 = __shfl_sync(0xffffffffu, s0, NV == 4 && j >= 2 ? (3 - j) & 31 : j);
    view = __shfl_sync(0xffffffffu, view, j);
    if (lane == 0) {
        // rows whose taps are valid and staged in every slot (ZM: row i and its image m2 - i - 1).
        // Slack: quads round t to 2^-10; FP32 runs round their ends' t, and at a detector row exactly z
        // and -z drop other taps
        constexpr float kSlack = kQuad<TP> ? 1.0f : 0.01f;
        int lo = max(1, t0 + 1), hi = min(A.nt - 1, t0 + A.H - 1);
        if (NZ == 2) {
            lo = max(lo, M.m2 - A.nt);
            hi = min(hi, M.m2 - 2);
        }
        S.sc = sc;
        S.flo = (float)lo + kSlack;
        S.fhi = (float)(hi + 1) - kSlack;
        S.t0 = t0;
        S.zoff = (uint32_t)A.box_bytes + (uint32_t)((2 * t0 + A.H + 1) * A.W * 8);
    }
    // lane 1's columns too have to be in the stage before lane 0's arrival, which publishes it: shuffles
    // order no memory
    __syncwarp();
    if (lane == 0) mbar_arrive_expect_tx(full, (uint32_t)(NS * A.W * A.H * 8));
    __syncwarp();
    if (lane < NS)
        tma_load_3d(dst + (size_t)lane * A.box_bytes, map, s0 * 2, z ? M.m2 - t0 - A.H - 1 : t0, view, full);
}

// 256 threads, 64 accumulators each and two CTAs per SM leave 128 registers: 64 for the loads in flight.
// A ninth, producing warp would round that down to 96 and the kernel would wait on shared-memory latency
// (measured on 512 x 512 x 64 voxels from 180 views: issue 53% with it).  So the warps take turns to
// refill: at view g one of them refills the stage of view g - 2, which every warp but one that lags
// a whole view behind has left (waiting for view g - 1 instead would chain each refill to the warp
// that the refill before has delayed).
template <typename TP, bool ARC, int NV, bool ZM, int KZ, bool EX>
__global__ void __launch_bounds__(kConsumers, 2)
    fdk_mirror_kernel(const __grid_constant__ FdkMirrorArgs M, const __grid_constant__ CUtensorMap map) {
    constexpr int NZ = ZM ? 2 : 1, NS = NV * NZ, NW = kConsumers / 32;
    extern __shared__ __align__(128) unsigned char smraw[];
    unsigned char *sm = smraw + ((128 - (smem_u32(smraw) & 127)) & 127);
    const FdkTmaArgs &A = M.A;
    const int nstage = A.nstage;  // 3 .. NW
    // a cluster of M.split CTAs shares a tile: each takes a range of the views
    const int rank = (int)(blockIdx.z % (unsigned)M.split), bz = (int)(blockIdx.z / (unsigned)M.split);
    const int va = A.v0 + (int)((long long)A.nv * rank / M.split);
    const int nv = A.v0 + (int)((long long)A.nv * (rank + 1) / M.split) - va;
    const uint32_t stage_bytes = (uint32_t)(NS * A.box_bytes);
    MirStage *meta = reinterpret_cast<MirStage *>(sm + (size_t)nstage * stage_bytes);
    uint64_t *full = reinterpret_cast<uint64_t *>(meta + nstage);
    uint64_t *empty = full + nstage;
    MirRun *run = reinterpret_cast<MirRun *>(empty + nstage);  // 2 nstage barriers: 16-byte aligned
    MirExtent *ext = reinterpret_cast<MirExtent *>(run + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < nstage; s++) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, NW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // the last tile of FP32 runs starts early rather than reach past the volume, whose rows may leave the
    // detector (quads keep to the t grid's anchors); it stores only its own voxels
    int iz = M.iz0 + bz * KZ, k_first = 0;
    if (!kQuad<TP> && iz + KZ > A.nz && A.nz >= KZ) {
        k_first = iz + KZ - A.nz;
        iz -= k_first;
    }
    if (tid == 0) {
        const float z0 = A.z0 + iz * A.dz, z1 = A.z0 + (iz + KZ - 1) * A.dz;
        run->z = z0;
        run->zlo = fminf(z0, z1);
        run->zhi = fmaxf(z0, z1);
        run->iz = iz;
        for (int h = 0; h < 2; h++) {
            const int i = iz + 16 * h, zb = i & ~(M.zbase - 1);
            run->zb[h] = A.z0 + zb * A.dz;
            run->koff[h] = (float)(i - zb);
        }
    }
    if (tid < NV) ext[tid] = mir_extent(M, tid, blockIdx.x, blockIdx.y, bz);
    __syncthreads();
    // warps 0 .. nstage - 1 fetch the first views; then at view g = 2 + h - nstage warp h % 8 fetches
    // view h.  Lane j < NV holds slot j's view and trig of the warp's next fetch.
    float2 sc = make_float2(0.f, 1.f);
    int view = 0, next = warp;
    auto look_up = [&]() {
        if (lane < NV && next < nv) {
            view = mir_slot_view(M, lane, va + next);
            sc = A.trig[view];
        }
    };
    auto fetch = [&](int stage) {
        mir_fill<TP, ARC, NV, NZ>(M, &map, sm + (size_t)stage * stage_bytes, meta[stage], ext, full + stage, sc, view, lane);
        next += NW;
        look_up();
    };
    look_up();
    if (warp < nstage && warp < nv) fetch(warp);

    const int ix = blockIdx.x * kTX + tid % kTX, iy = blockIdx.y * kTY + tid / kTX;
    const bool in = ix < M.hx && iy < M.hy;
    const float x = A.x0 + ix * A.dx, y = A.y0 + iy * A.dy;
    float acc[NS][KZ];
#pragma unroll
    for (int s = 0; s < NS; s++)
#pragma unroll
        for (int k = 0; k < KZ; k++) acc[s][k] = 0.f;
    int st = 0;
    unsigned phase = 0;
    bool ok = true;
    const uint32_t base = smem_u32(sm);
    for (int g = 0; g < nv; g++) {
        if (next == g - 2 + nstage && next < nv) {
            const int sp = st >= 2 ? st - 2 : st - 2 + nstage;
            ok = mbar_wait(empty + sp, st >= 2 ? phase : phase ^ 1);
            if (!__all_sync(0xffffffffu, ok)) break;
            fetch(sp);
        }
        ok = mbar_wait(full + st, phase);
        if (!__all_sync(0xffffffffu, ok)) break;
        if (in) mir_view<TP, ARC, NV, ZM, KZ, EX>(M, x, y, *run, meta[st], base + (uint32_t)st * stage_bytes, acc);
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + st);
        if (++st == nstage) {
            st = 0;
            phase ^= 1;
        }
    }
    if (!__all_sync(0xffffffffu, ok)) {  // a wait ran out: drain (bounded) this warp's copies and report
        if (lane == 0) {
            atomicOr(A.err, 2);
            const int mine = next - NW;  // its last fetch
            if (mine >= 0 && !mbar_wait(full + mine % nstage, (mine / nstage) & 1)) atomicOr(A.err, 4);
        }
    }

    float u = 1.f;
    if constexpr (kQuad<TP>) u = *A.qscale;  // undo the quads' power-of-two scale (exact)
    // voxel k of slot s.  A column on the mirror of a halved axis is its own image (slot 0, or slot X or
    // Y of the other axis, has it already), and so is the central plane.
    auto store = [&](int s, int k, float v) {
        const int j = s / NZ, flip = NV == 4 ? j : M.flip[j];
        const int jx = flip & MIR_X ? A.nx - 1 - ix : ix, jy = flip & MIR_Y ? A.ny - 1 - iy : iy;
        const int kk = s % NZ ? A.nz - 1 - iz - k : iz + k;
        if (k < k_first || iz + k >= A.nz || (s % NZ && kk == iz + k)) return;
        if ((flip & MIR_X && M.hx < A.nx && jx == ix) || (flip & MIR_Y && M.hy < A.ny && jy == iy)) return;
        const long long idx = jx + (long long)A.nx * (jy + (long long)A.ny * kk);
        if (kQuad<TP>) v *= u;
        if (A.accum) v += A.image[idx];
        if (A.mask && !A.mask[idx]) v = 0.f;  // :133
        A.image[idx] = v;
    };
    if (M.split == 1) {
        if (!in) return;
#pragma unroll
        for (int s = 0; s < NS; s++)
#pragma unroll
            for (int k = 0; k < KZ; k++) store(s, k, acc[s][k]);
        return;
    }
    // the ranks' partial tiles meet in shared memory, summed in rank order
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    float *part = reinterpret_cast<float *>(sm);  // [NS * KZ][threads] over the ring
    __syncthreads();
#pragma unroll
    for (int s = 0; s < NS; s++)
#pragma unroll
        for (int k = 0; k < KZ; k++) part[(s * KZ + k) * kConsumers + tid] = acc[s][k];
    cl.sync();
    for (int i = rank; i < NS * KZ; i += M.split) {
        float v = 0.f;
        for (int q = 0; q < M.split; q++) v += cl.map_shared_rank(part, q)[i * kConsumers + tid];
        if (in) store(i / KZ, i % KZ, v);
    }
    cl.sync();  // peers' shared memory stays alive until every rank has read it
}

template <typename TP, bool ARC, int NV, bool ZM, int KZ, bool EX>
int launch_mirror_e(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st) {
    const size_t smem = fdk_mirror_smem(M, M.A.nstage);
    auto k = fdk_mirror_kernel<TP, ARC, NV, ZM, KZ, EX>;
    SGB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(floor_div_up(M.hx, kTX), floor_div_up(M.hy, kTY), floor_div_up(M.nzd, KZ) * M.split);
    cfg.blockDim = dim3(kConsumers);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = M.split;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k, M, map);
    if (e != cudaSuccess) {
        set_error("fdk_mirror_kernel: launch failed: %s", cudaGetErrorString(e));
        return SGB_ERR_CUDA;
    }
    return after_launch("fdk_mirror_kernel");
}

template <typename TP, bool ARC, int NV, bool ZM, int KZ>
int launch_mirror_k(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st) {
    if constexpr (!kQuad<TP> && NV > 1)  // quads only come with a symmetric grid; one view slot has no mirror in it
        if (!M.exact) return launch_mirror_e<TP, ARC, NV, ZM, KZ, false>(M, map, st);
    return launch_mirror_e<TP, ARC, NV, ZM, KZ, true>(M, map, st);
}

}  // namespace fdkdev
}  // namespace sgb
