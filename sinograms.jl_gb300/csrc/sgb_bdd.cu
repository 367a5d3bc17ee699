// sgb_bdd.cu -- branchless distance-driven projector pair, src/sys2/bdd_2d.jl.
//
// Per view the reference maps detector boundaries (detm) and pixel boundaries (rowm)
// onto a common axis through the source (map2x / map2y, bdd_2d.jl:249-263), integrates
// one side (integrate1D, :229-241), interpolates the integral at the other side's
// boundaries (linear, Flat extrapolation) and takes |diff|.
//
// The pixel grid of the reference is a set of x boundaries and y row centres
// (:32-35), so for both mapping axes the mapped boundaries of one image "row" are an
// affine function of the pixel index: rowm[c] = r0 + c * delta.  The kernels use that
// closed form instead of a table.  The interpolated prefix integral of a row at a mapped
// point is F(q) = delta * (sum_{c<floor q} val[c] + frac(q) val[floor q]), q = (u-r0)/delta,
// clamped to [0, nPix] (Flat extrapolation).  The forward projector forms the reference's
// |diff| of F at consecutive detector boundaries from the pixels between them directly, or, where
// a bin covers many, from a warp-level prefix scan kept in two-float (hi + lo) arithmetic, so
// nearby prefix values subtract without losing FP32 accuracy.  The back-projector is the
// transpose: a block-wide two-float scan of each view's detector-bin integrals gives the detector
// prefix integral at the knots, and each pixel's
// value is |G(u1) - G(u0)| of that prefix interpolated at the pixel's two mapped boundaries
// (:196-205).  Both are exactly the reference's quantity.  FP64 is kept for the per-view and
// per-row geometry (trig, boundary mapping); the per-sample work is FP32.
//
// With BddArgs.arc the detector boundaries lie on the arc of radius DSD about the source
// (SinoFanArc; an extension with no reference counterpart); everything downstream of the
// mapped boundaries is shared.
//
// Quirks kept: detector y offset -(DSD-DS0) - dSize/2 (:29, flat detector), Flat extrapolation,
// |diff| (the pair is not linear for signed images), the (na, nDet) sinogram layout,
// and in backproject_bdd the aliasing reconImgTmp === reconImg (:139-140), which adds
// the first view's row block once more without the y-axis transpose.
#include <algorithm>

#include "sgb_async.cuh"
#include "sgb_common.cuh"
#include "sgb_kernels.cuh"

namespace sgb {

namespace {

constexpr double kPi = 3.14159265358979323846;
constexpr int kWarps = 8;
constexpr int kThreads = 32 * kWarps;
constexpr int kStageU = 8;  // phantom loads per thread in flight while a row block is staged

__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dev::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dev::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

struct ViewInfo {
    double rtx, rty;
    int axis;  // 1: map onto x (axisCase true), 0: onto y
    int pad;
};

__device__ __forceinline__ double map2x(double x1, double y1, double x2, double y2) {
    return x1 - y1 * (x1 - x2) / (y1 - y2);
}
__device__ __forceinline__ double map2y(double x1, double y1, double x2, double y2) {
    return y1 - x1 * (y1 - y2) / (x1 - x2);
}

__device__ __forceinline__ ViewInfo view_info(double beta, double DS0) {
    ViewInfo vi;
    vi.rtx = -DS0 * sin(beta);  // :45-46
    vi.rty = DS0 * cos(beta);
    vi.axis = !(((beta >= kPi / 4) && (beta <= 3 * kPi / 4)) ||
                ((beta >= 5 * kPi / 4) && (beta <= 7 * kPi / 4)));  // :53-57
    vi.pad = 0;
    return vi;
}

// mapped detector boundary k (0..nDet) for one view, :28-29, 49-50, 60-66.  Arc detector (an
// extension; the reference pair is flat-only): boundary k on the circle of radius DSD about the
// source, at angle (k - nDet/2) dSize / DSD from the central ray, before the view rotation.
__device__ __forceinline__ double det_boundary(const ViewInfo &vi, double beta, int k, int nDet,
                                               double DSD, double DS0, double dSize, int arc) {
    double detX = (-(nDet / 2.0) + k) * dSize;
    double detY = -(DSD - DS0) - dSize / 2;
    if (arc) {
        const double g = (-(nDet / 2.0) + k) * dSize / DSD;
        detX = DSD * sin(g);
        detY = DS0 - DSD * cos(g);
    }
    double sb = sin(beta), cb = cos(beta);
    double rdX = detX * cb - detY * sb, rdY = detX * sb + detY * cb;
    return vi.axis ? map2x(vi.rtx, vi.rty, rdX, rdY) : map2y(vi.rtx, vi.rty, rdX, rdY);
}

// L[n], :71-86, with cos(atan(u)) = 1/sqrt(1+u^2) and sin(acot(v)) = 1/sqrt(1+v^2).
__device__ __forceinline__ double det_scale(const ViewInfo &vi, double d0, double d1, double pSize) {
    double det_mid = (d0 + d1) / 2, detSize = d1 - d0;
    double u = vi.axis ? fabs(vi.rtx - det_mid) / fabs(vi.rty) : fabs(vi.rty - det_mid) / fabs(vi.rtx);
    return fabs(pSize * sqrt(1 + u * u) / detSize);
}

// Affine mapped boundaries of "row" r: rowm[c] = r0 + c * delta, c = 0..nPix.
// x-case: points (B_{c+1}, C_{r+1}); y-case: points (B_{r+1}, C_{nPix+1-c}) with
// B_j = (j-1-nPix/2) pSize and C_i = (nPix/2 + 1/2 - i) pSize (:32-35, 60-68).
__device__ __forceinline__ void row_affine(const ViewInfo &vi, int r, int nPix, double pSize,
                                           double *r0, double *delta) {
    double a, b;
    if (vi.axis) {
        double Y = (nPix / 2.0 + 0.5 - (r + 1)) * pSize;
        a = map2x(vi.rtx, vi.rty, (-(nPix / 2.0)) * pSize, Y);
        b = map2x(vi.rtx, vi.rty, (nPix / 2.0) * pSize, Y);
    } else {
        double X = (-(nPix / 2.0) + r) * pSize;
        a = map2y(vi.rtx, vi.rty, X, (nPix / 2.0 + 0.5 - (nPix + 1)) * pSize);
        b = map2y(vi.rtx, vi.rty, X, (nPix / 2.0 + 0.5 - 1) * pSize);
    }
    *r0 = a;
    *delta = (b - a) / nPix;
}

// Per (view, image row): the affine map of the row's boundaries, as the kernels use it in FP32:
// (r0, delta, 1 / delta, |delta|), each rounded from the FP64 value.  The forward and back
// kernels read this table instead of evaluating the FP64 map per warp: on this GPU FP64 issue is
// narrow, and the map took most of the FP64 pipe's time.
__global__ void bdd_rowmap_kernel(BddArgs G, const ViewInfo *info, float4 *rmap) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)G.na * G.nPix) return;
    const int p = (int)(i / G.nPix), r = (int)(i % G.nPix);
    double r0d, deltad;
    row_affine(info[p], r, G.nPix, G.pSize, &r0d, &deltad);
    rmap[i] = make_float4((float)r0d, (float)deltad, (float)(1.0 / deltad), (float)std::fabs(deltad));
}

// ------------------------------------------------------------ per-view set-up
// forward: info, detm (nDet+1, FP32), L (nDet, FP32).  back: info and the geometry table
// (nDet+1 float4 per view, in ascending knot order: x = knot K[j]; y = the integral of bin j per
// unit sinogram value, L * |ddetm| signed as the reference's prefix, :196, and reversed when
// detm descends, :198-202; z = the same per unit length, the bin's density factor; w of the last
// knot = 1 when detm descends).  Both depend on the geometry only, so plans compute them once;
// bdd_fill_prefix_kernel multiplies in the sinogram per call.
// One CTA per (view, chunk of kSetupChunk bins): the view's constants once, each FP64 boundary
// once into shared memory, then the chunk's outputs from those values (the same FP64 calls).
constexpr int kSetupChunk = kThreads;
__global__ void __launch_bounds__(kThreads) bdd_setup_kernel(BddArgs G, ViewInfo *info, float *detm, float *L,
                                                             float4 *geo) {
    __shared__ ViewInfo vis;
    __shared__ int desc_s;
    __shared__ double bnd[kSetupChunk + 1];
    const int p = blockIdx.x, nDet = G.nDet;
    const int n0 = blockIdx.y * kSetupChunk, n1 = min(nDet, n0 + kSetupChunk), cnt = n1 - n0;
    const double beta = G.angle[p];
    if (threadIdx.x == 0) {
        vis = view_info(beta, G.DS0);
        if (blockIdx.y == 0) info[p] = vis;
        desc_s = geo ? det_boundary(vis, beta, 0, nDet, G.DSD, G.DS0, G.dSize, G.arc) >
                           det_boundary(vis, beta, 1, nDet, G.DSD, G.DS0, G.dSize, G.arc)
                     : 0;
    }
    __syncthreads();
    const ViewInfo vi = vis;
    const bool desc = desc_s != 0;
    // boundaries b0 .. b0 + cnt: those of bins n0 .. n1-1 (reversed for a descending back-projection)
    const int b0 = desc ? nDet - n1 : n0;
    for (int i = threadIdx.x; i <= cnt; i += blockDim.x)
        bnd[i] = det_boundary(vi, beta, b0 + i, nDet, G.DSD, G.DS0, G.dSize, G.arc);
    __syncthreads();
    if (!geo) {
        float *dm = detm + (size_t)p * (nDet + 1);
        for (int k = n0 + threadIdx.x; k <= n1; k += blockDim.x) dm[k] = (float)bnd[k - n0];
        for (int n = n0 + threadIdx.x; n < n1; n += blockDim.x)
            L[(size_t)p * nDet + n] = (float)det_scale(vi, bnd[n - n0], bnd[n + 1 - n0], G.pSize);
        return;
    }
    float4 *T = geo + (size_t)p * (nDet + 1);
    // this chunk writes knots n0 .. n1-1 with their bins, and the last chunk also knot nDet
    for (int j = n0 + threadIdx.x; j < n1 || (j == nDet && n1 == nDet); j += blockDim.x) {
        // ascending knot j is reference boundary desc ? nDet-j : j; ascending bin j covers
        // reference bin n = desc ? nDet-1-j : j
        const int src = desc ? nDet - j : j;
        float cb = 0.f, cd = 0.f;
        if (j < n1) {
            const int n = desc ? nDet - 1 - j : j;
            const double d0 = bnd[n - b0], d1 = bnd[n + 1 - b0];
            const double w = det_scale(vi, d0, d1, G.pSize) * (d1 - d0);
            cb = (float)(desc ? -w : w);  // the bin's integral per unit sinogram value, ascending
            cd = (float)((desc ? -w : w) / std::fabs(d1 - d0));  // and its density
        }
        T[j] = make_float4((float)bnd[src - b0], cb, cd, j == nDet ? (float)desc : 0.f);
    }
}

// Two-float accumulation (Knuth's TwoSum): (hi, lo) += v with the rounding error of the
// high part carried in lo.
__device__ __forceinline__ void two_sum_add(float &hi, float &lo, float v) {
    const float s = hi + v, bb = s - hi;
    lo += (hi - (s - bb)) + (v - bb);
    hi = s;
}

// ------------------------------------------------------------------ forward
// Per view and image row: the row's prefix integral P[c] = sum_{j<c} val[j] (c = 0..nPix, in
// pixel units) is built by a warp-level scan in two-float arithmetic, so that the difference
// of two nearby prefix values keeps FP32 accuracy relative to the pixels between them.  The
// interpolated integral at a mapped detector boundary is F(q) = P[c] + frac(q) val[c],
// c = floor(q), q clamped to [0, nPix] (Flat extrapolation, val[nPix] = 0).  Lane k of the
// warp evaluates boundary k of a group of 32 and takes F at boundary k+1 from its neighbour
// (shuffle): neighbouring lanes read neighbouring pixels (no bank conflicts), each boundary
// is evaluated once, and each bin is |F(k+1) - F(k)| (:98-101).
__global__ void __launch_bounds__(kThreads)
    bdd_project_kernel(BddArgs G, const ViewInfo *info, const float *detm, const float *L, const float4 *rmap,
                       const float *__restrict__ phantom, float *sino, int rows_per_cta) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int nPix = G.nPix, nDet = G.nDet, p = blockIdx.x;
    float2 *pw = reinterpret_cast<float2 *>(smraw);                   // kWarps x (nPix+1): prefix (hi, lo)
    float *vw = reinterpret_cast<float *>(pw + kWarps * (nPix + 1));  // kWarps x (nPix+1): row values
    float *dm = vw + kWarps * (nPix + 1);                              // nDet+1
    float *accw = dm + (nDet + 1);                                     // kWarps x nDet
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    const ViewInfo vi = info[p];
    for (int k = threadIdx.x; k <= nDet; k += kThreads) dm[k] = detm[(size_t)p * (nDet + 1) + k];
    for (int i = threadIdx.x; i < kWarps * nDet; i += kThreads) accw[i] = 0.f;
    float2 *pre = pw + warp * (nPix + 1);
    float *val = vw + warp * (nPix + 1);
    float *acc = accw + warp * nDet;
    const int chunk = ((nPix + 1 + 31) / 32) | 1;  // prefix entries per lane (odd: conflict-free reads)
    const int c_begin = min(nPix + 1, lane * chunk), c_end = min(nPix + 1, c_begin + chunk);
    const int r_begin = blockIdx.y * rows_per_cta, r_end = min(nPix, r_begin + rows_per_cta);
    for (int rb = r_begin; rb < r_end; rb += kWarps) {
        __syncthreads();
        // stage kWarps rows: x-case row r = phantom[r + nPix*c] (eight consecutive r per 32-byte
        // sector); y-case (transposed and reversed, :67) row r = phantom[(nPix-1-c) + nPix*r]
        // (kStageU independent loads in flight per thread before their stores)
        if (vi.axis) {
            const int total = kWarps * nPix;
            for (int i0 = threadIdx.x; i0 < total; i0 += kStageU * kThreads) {
                float v[kStageU];
#pragma unroll
                for (int u = 0; u < kStageU; u++) {
                    const int i = i0 + u * kThreads, r = rb + i % kWarps;
                    v[u] = (i < total && r < r_end) ? __ldg(phantom + r + (size_t)nPix * (i / kWarps)) : 0.f;
                }
#pragma unroll
                for (int u = 0; u < kStageU; u++) {
                    const int i = i0 + u * kThreads;
                    if (i < total) vw[(i % kWarps) * (nPix + 1) + i / kWarps] = v[u];
                }
            }
        } else {
            const int r = rb + warp;
            const float *src = phantom + (size_t)nPix * r + (nPix - 1);
            for (int c0 = lane; c0 < nPix; c0 += kStageU * 32) {
                float v[kStageU];
#pragma unroll
                for (int u = 0; u < kStageU; u++) {
                    const int c = c0 + 32 * u;
                    v[u] = (c < nPix && r < r_end) ? __ldg(src - c) : 0.f;
                }
#pragma unroll
                for (int u = 0; u < kStageU; u++)
                    if (c0 + 32 * u < nPix) val[c0 + 32 * u] = v[u];
            }
        }
        if (threadIdx.x < kWarps) vw[threadIdx.x * (nPix + 1) + nPix] = 0.f;
        __syncthreads();
        const int r = rb + warp;
        if (r >= r_end) continue;  // warp-uniform
        // prefix: lane totals, warp scan of the totals, then the lane's entries
        float th = 0.f, tl = 0.f;
        for (int c = c_begin; c < c_end; c++) two_sum_add(th, tl, val[c]);
        for (int off = 1; off < 32; off <<= 1) {
            const float oh = __shfl_up_sync(full, th, off), ol = __shfl_up_sync(full, tl, off);
            if (lane >= off) {
                two_sum_add(th, tl, oh);
                tl += ol;
            }
        }
        float sh = __shfl_up_sync(full, th, 1), sl = __shfl_up_sync(full, tl, 1);
        if (lane == 0) sh = sl = 0.f;
        for (int c = c_begin; c < c_end; c++) {
            pre[c] = make_float2(sh, sl);
            two_sum_add(sh, sl, val[c]);
        }
        __syncwarp();
        const float4 rmv = rmap[(size_t)p * nPix + r];
        const float r0 = rmv.x, rdelta = rmv.z, adelta = rmv.w;
        const float qmax = (float)nPix;
        // F at mapped detector boundary k (:98, interpolation of the row's prefix integral);
        // floor(q) for 0 <= q <= nPix < 2^22 by the round-down add of 2^23 (no conversions)
        auto F = [&](int k, float &fh, float &fl) {
            const float q = fminf(fmaxf((dm[k] - r0) * rdelta, 0.f), qmax);
            const float m = __fadd_rd(q, 8388608.f);
            const int c = __float_as_int(m) - 0x4B000000;
            const float2 e = pre[c];
            fh = e.x;
            fl = fmaf(q - (m - 8388608.f), val[c], e.y);
        };
        // bin k0 + lane: |F(k+1) - F(k)| * |delta| (:98-101), F(k+1) from the next lane
        float ch, cl;
        F(min(lane, nDet), ch, cl);
        for (int k0 = 0; k0 < nDet; k0 += 32) {
            float nh, nl;
            F(min(k0 + 32 + lane, nDet), nh, nl);
            float uh = __shfl_down_sync(full, ch, 1), ul = __shfl_down_sync(full, cl, 1);
            const float h0 = __shfl_sync(full, nh, 0), l0 = __shfl_sync(full, nl, 0);
            if (lane == 31) {
                uh = h0;
                ul = l0;
            }
            if (k0 + lane < nDet) acc[k0 + lane] += fabsf((uh - ch) + (ul - cl)) * adelta;
            ch = nh;
            cl = nl;
        }
        __syncwarp();
    }
    __syncthreads();
    for (int n = threadIdx.x; n < nDet; n += kThreads) {
        float s = 0.f;
        for (int w = 0; w < kWarps; w++) s += accw[w * nDet + n];
        atomicAdd(sino + p + (size_t)G.na * n, s * L[(size_t)p * nDet + n]);  // :104
    }
}

// The same projection with the bins, not the rows, split over the warps: each warp scans the
// prefix of one of the CTA's kWarps staged rows, then walks its own range of at most NG
// 32-bin groups across all kWarps rows, so its bin sums stay in registers.  Shared memory is
// the staged rows and their prefixes only (no per-warp bin accumulators), which lets four CTAs
// share an SM instead of two.  Each warp evaluates F once more per row than its groups (the
// boundary past its last bin), and the rows of a bin are summed in ascending order.
struct RowMap {
    float r0, rdelta, adelta, pad;
};
static_assert(kWarps % 4 == 0, "the row maps follow the staged rows at a 16-byte boundary");

template <int NG>
__global__ void __launch_bounds__(kThreads, 4)
    bdd_project_bins_kernel(BddArgs G, const ViewInfo *info, const float *detm, const float *L, const float4 *rmap,
                            const float *__restrict__ phantom, float *sino, int rows_per_cta) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int nPix = G.nPix, nDet = G.nDet, p = blockIdx.x;
    float2 *pw = reinterpret_cast<float2 *>(smraw);                   // kWarps x (nPix+1): prefix (hi, lo)
    float *vw = reinterpret_cast<float *>(pw + kWarps * (nPix + 1));  // kWarps x (nPix+1): row values
    RowMap *rm = reinterpret_cast<RowMap *>(vw + kWarps * (nPix + 1));  // kWarps (16-byte aligned: kWarps % 4 == 0)
    float *dm = reinterpret_cast<float *>(rm + kWarps);              // nDet+1
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    const ViewInfo vi = info[p];
    for (int k = threadIdx.x; k <= nDet; k += kThreads) dm[k] = detm[(size_t)p * (nDet + 1) + k];
    const int ngroups = (nDet + 31) / 32;
    const int g0 = warp * ngroups / kWarps, g1 = (warp + 1) * ngroups / kWarps;  // g1 - g0 <= NG (host check)
    float acc[NG];
#pragma unroll
    for (int i = 0; i < NG; i++) acc[i] = 0.f;
    float2 *pre = pw + warp * (nPix + 1);
    float *val = vw + warp * (nPix + 1);
    const int chunk = ((nPix + 1 + 31) / 32) | 1;  // prefix entries per lane (odd: conflict-free reads)
    const int c_begin = min(nPix + 1, lane * chunk), c_end = min(nPix + 1, c_begin + chunk);
    const int r_begin = blockIdx.y * rows_per_cta, r_end = min(nPix, r_begin + rows_per_cta);
    const float qmax = (float)nPix;
    for (int rb = r_begin; rb < r_end; rb += kWarps) {
        __syncthreads();
        // stage kWarps rows (as bdd_project_kernel)
        if (vi.axis) {
            const int total = kWarps * nPix;
            for (int i0 = threadIdx.x; i0 < total; i0 += kStageU * kThreads) {
                float v[kStageU];
#pragma unroll
                for (int u = 0; u < kStageU; u++) {
                    const int i = i0 + u * kThreads, r = rb + i % kWarps;
                    v[u] = (i < total && r < r_end) ? __ldg(phantom + r + (size_t)nPix * (i / kWarps)) : 0.f;
                }
#pragma unroll
                for (int u = 0; u < kStageU; u++) {
                    const int i = i0 + u * kThreads;
                    if (i < total) vw[(i % kWarps) * (nPix + 1) + i / kWarps] = v[u];
                }
            }
        } else {
            const int r = rb + warp;
            const float *src = phantom + (size_t)nPix * r + (nPix - 1);
            for (int c0 = lane; c0 < nPix; c0 += kStageU * 32) {
                float v[kStageU];
#pragma unroll
                for (int u = 0; u < kStageU; u++) {
                    const int c = c0 + 32 * u;
                    v[u] = (c < nPix && r < r_end) ? __ldg(src - c) : 0.f;
                }
#pragma unroll
                for (int u = 0; u < kStageU; u++)
                    if (c0 + 32 * u < nPix) val[c0 + 32 * u] = v[u];
            }
        }
        if (threadIdx.x < kWarps) vw[threadIdx.x * (nPix + 1) + nPix] = 0.f;
        __syncthreads();
        // this warp's row: two-float prefix (as bdd_project_kernel) and its boundary map
        {
            float th = 0.f, tl = 0.f;
            for (int c = c_begin; c < c_end; c++) two_sum_add(th, tl, val[c]);
            for (int off = 1; off < 32; off <<= 1) {
                const float oh = __shfl_up_sync(full, th, off), ol = __shfl_up_sync(full, tl, off);
                if (lane >= off) {
                    two_sum_add(th, tl, oh);
                    tl += ol;
                }
            }
            float sh = __shfl_up_sync(full, th, 1), sl = __shfl_up_sync(full, tl, 1);
            if (lane == 0) sh = sl = 0.f;
            for (int c = c_begin; c < c_end; c++) {
                pre[c] = make_float2(sh, sl);
                two_sum_add(sh, sl, val[c]);
            }
            if (lane == 0) {
                const float4 rmv = rmap[(size_t)p * nPix + min(rb + warp, nPix - 1)];
                rm[warp] = RowMap{rmv.x, rmv.z, rmv.w, 0.f};
            }
        }
        __syncthreads();
        // this warp's bins over the staged rows, in ascending row order
        const int nrows = min(kWarps, r_end - rb);
        for (int j = 0; j < nrows; j++) {
            const RowMap m = rm[j];
            const float2 *pj = pw + j * (nPix + 1);
            const float *vj = vw + j * (nPix + 1);
            auto F = [&](int k, float &fh, float &fl) {  // :98, as bdd_project_kernel
                const float q = fminf(fmaxf((dm[k] - m.r0) * m.rdelta, 0.f), qmax);
                const float mq = __fadd_rd(q, 8388608.f);
                const int c = __float_as_int(mq) - 0x4B000000;
                const float2 e = pj[c];
                fh = e.x;
                fl = fmaf(q - (mq - 8388608.f), vj[c], e.y);
            };
            float ch, cl;
            F(min(g0 * 32 + lane, nDet), ch, cl);
#pragma unroll
            for (int i = 0; i < NG; i++) {
                if (g0 + i < g1) {  // warp-uniform
                    const int k0 = (g0 + i) * 32;
                    float nh, nl;
                    F(min(k0 + 32 + lane, nDet), nh, nl);
                    float uh = __shfl_down_sync(full, ch, 1), ul = __shfl_down_sync(full, cl, 1);
                    const float h0 = __shfl_sync(full, nh, 0), l0 = __shfl_sync(full, nl, 0);
                    if (lane == 31) {
                        uh = h0;
                        ul = l0;
                    }
                    acc[i] += fabsf((uh - ch) + (ul - cl)) * m.adelta;  // :98-101
                    ch = nh;
                    cl = nl;
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NG; i++) {
        const int n = (g0 + i) * 32 + lane;
        if (g0 + i < g1 && n < nDet) atomicAdd(sino + p + (size_t)G.na * n, acc[i] * L[(size_t)p * nDet + n]);  // :104
    }
}

// The same projection without prefixes, for bins that cover few pixels.  A bin between mapped
// boundaries q0, q1 (in pixels, c0 = floor(q0) <= c1 = floor(q1)) integrates
// (c1 - q0) val[c0] + (q1 - c1) val[c1] when c1 <= c0 + 1, and when c1 == c0 the same expression
// still gives (q1 - q0) val[c0]: no prefix integral and no difference of large sums.  Bins that
// cover more pixels add the whole ones between in a loop, which a warp enters only when one of its
// bins does.  A lane holds kDirBins consecutive bins of a group of 31 x kDirBins and takes its last
// boundary from the next lane: a boundary is evaluated once but for 1 in 32.
//
// A warp has whole rows, or every wb-th of their groups when there are more than kDirGroups: the
// bins that cover several pixels lie together at one end of a view, and a split of the bins into
// ranges left the other warps waiting for that end's (121 us at 512^2 x 888 x 90 views, this one
// 72).  Its sums stay in registers over the CTA's rows.  The prefix form took 106 us there: it
// spends about as much on each staged row's scan as on its bins.  Bound by issue (64 % of the
// slots; 48 million instructions, of which staging is an eighth).
constexpr int kDirRows = 8;                // rows per stage
constexpr int kDirBins = 4;                // bins per lane and group
constexpr int kDirGroup = 31 * kDirBins;  // bins per group
constexpr int kDirGroups = 4;              // groups per warp

// staged row pitch: 4 mod 32 words, so the transposing stores (8 rows x 4 columns a warp) spread
// over the banks
__host__ __device__ __forceinline__ int direct_pitch(int nPix) { return (nPix + 1 + 27) / 32 * 32 + 4; }

__global__ void __launch_bounds__(kThreads, 4)
    bdd_project_direct_kernel(BddArgs G, const ViewInfo *info, const float *detm, const float *L, const float4 *rmap,
                              const float *__restrict__ phantom, float *sino, int rows_per_cta, int wb) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int nPix = G.nPix, nDet = G.nDet, p = blockIdx.x;
    const int pitch = direct_pitch(nPix);
    float4 *rm = reinterpret_cast<float4 *>(smraw);             // 2 x kDirRows row maps
    float4 *dms = rm + 2 * kDirRows;                             // kDirGroups x wb x 32: the lanes' boundaries
    float *vw = reinterpret_cast<float *>(dms + kDirGroups * wb * 32);  // 2 x kDirRows x pitch values
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    const int axis = info[p].axis;
    const float *dview = detm + (size_t)p * (nDet + 1);
    const int sub = warp / wb, nsub = kWarps / wb;  // rows sub, sub + nsub, ... of a stage
    const int z0 = blockIdx.z * wb * kDirGroups * kDirGroup;
    const int ngroup = min(kDirGroups * wb, (nDet - z0 + kDirGroup - 1) / kDirGroup);  // of this CTA
    for (int i = threadIdx.x; i < ngroup * 32; i += kThreads) {
        const int k = z0 + (i / 32) * kDirGroup + (i % 32) * kDirBins;
        dms[i] = make_float4(dview[min(k, nDet)], dview[min(k + 1, nDet)], dview[min(k + 2, nDet)],
                             dview[min(k + 3, nDet)]);
    }
    float acc[kDirGroups][kDirBins];
#pragma unroll
    for (int g = 0; g < kDirGroups; g++)
#pragma unroll
        for (int i = 0; i < kDirBins; i++) acc[g][i] = 0.f;
    if (threadIdx.x < 2 * kDirRows) vw[threadIdx.x * pitch + nPix] = 0.f;  // q = nPix reads it
    const int r_begin = blockIdx.y * rows_per_cta, r_end = min(nPix, r_begin + rows_per_cta);
    // x-case row r = phantom[r + nPix*c] (eight consecutive r per 32-byte sector); y-case
    // (transposed and reversed, :67) row r = phantom[(nPix-1-c) + nPix*r]
    auto stage = [&](int rb, int s) {
        const int nr = min(kDirRows, r_end - rb);
        float *dst = vw + s * kDirRows * pitch;
        if (axis) {
            const int j = threadIdx.x % kDirRows;
            if (j < nr) {
                const float *src = phantom + rb + j;
                for (int c = threadIdx.x / kDirRows; c < nPix; c += kThreads / kDirRows)
                    cp_async4(dst + j * pitch + c, src + (size_t)nPix * c);
            }
        } else if (warp < nr) {
            const float *src = phantom + (size_t)nPix * (rb + warp) + (nPix - 1);
            for (int c = lane; c < nPix; c += 32) cp_async4(dst + warp * pitch + c, src - c);
        }
        if (threadIdx.x < nr) cp_async16(rm + s * kDirRows + threadIdx.x, rmap + (size_t)p * nPix + rb + threadIdx.x);
        cp_async_commit();
    };
    const float qmax = (float)nPix;
    stage(r_begin, 0);
    int s = 0;
    for (int rb = r_begin; rb < r_end; rb += kDirRows, s ^= 1) {
        if (rb + kDirRows < r_end) {
            stage(rb + kDirRows, s ^ 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const int nrows = min(kDirRows, r_end - rb);
        for (int j = sub; j < nrows; j += nsub) {
            const float4 m = rm[s * kDirRows + j];  // (r0, delta, 1 / delta, |delta|)
            const float *vj = vw + (s * kDirRows + j) * pitch;
#pragma unroll
            for (int g = 0; g < kDirGroups; g++) {
                const int gi = g * wb + warp % wb;
                if (gi >= ngroup) break;  // uniform
                const float4 d4 = dms[gi * 32 + lane];
                const float dm[kDirBins] = {d4.x, d4.y, d4.z, d4.w};
                float q[kDirBins + 1], c[kDirBins + 1], v[kDirBins + 1];
#pragma unroll
                for (int i = 0; i <= kDirBins; i++) {
                    if (i < kDirBins) q[i] = fminf(fmaxf((dm[i] - m.x) * m.z, 0.f), qmax);
                    else q[i] = __shfl_down_sync(full, q[0], 1);
                    // floor(q) for 0 <= q <= nPix < 2^22 by the round-down add of 2^23
                    const float t = __fadd_rd(q[i], 8388608.f);
                    c[i] = t - 8388608.f;
                    if (i < kDirBins) v[i] = vj[__float_as_int(t) - 0x4B000000];
                    else v[i] = __shfl_down_sync(full, v[0], 1);
                }
                float a[kDirBins], wide = 0.f;
#pragma unroll
                for (int i = 0; i < kDirBins; i++) {
                    const float e = fmaxf(c[i], c[i + 1]);
                    wide = fmaxf(wide, fabsf(c[i + 1] - c[i]));
                    a[i] = fmaf(e - q[i], v[i], (q[i + 1] - e) * v[i + 1]);
                }
                if (wide > 1.5f && lane < 31) {  // (lane 31 has one boundary only)
                    // whole pixels between the boundaries' own, which the sum above has as the lower
                    // one's value
#pragma unroll
                    for (int i = 0; i < kDirBins; i++) {
                        const bool up = q[i] <= q[i + 1];
                        const float vb = up ? v[i] : v[i + 1];
                        const int hi = (int)fmaxf(c[i], c[i + 1]);
                        float t = 0.f;
                        for (int k = (int)fminf(c[i], c[i + 1]) + 1; k < hi; k++) t += vj[k] - vb;
                        a[i] += up ? t : -t;
                    }
                }
#pragma unroll
                for (int i = 0; i < kDirBins; i++) acc[g][i] = fmaf(fabsf(a[i]), m.w, acc[g][i]);  // :98-101
            }
        }
        __syncthreads();
    }
    // the row subsets' sums, in order (the staged rows are done with)
    float *red = vw;  // nsub x (ngroup x kDirGroup)
    const int nb = ngroup * kDirGroup;
#pragma unroll
    for (int g = 0; g < kDirGroups; g++) {
        const int gi = g * wb + warp % wb;
        if (gi >= ngroup || lane == 31) break;
#pragma unroll
        for (int i = 0; i < kDirBins; i++) red[sub * nb + gi * kDirGroup + lane * kDirBins + i] = acc[g][i];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb && z0 + i < nDet; i += kThreads) {
        float t = 0.f;
        for (int w = 0; w < nsub; w++) t += red[w * nb + i];
        atomicAdd(sino + p + (size_t)G.na * (z0 + i), t * L[(size_t)p * nDet + z0 + i]);  // :104
    }
}

// ------------------------------------------------------------------ backward
// The back-projector's table of one view, one contiguous block: the guess table (kCells + 1 pairs:
// the fractional knot index at the start of each of kCells equal cells of the mapped axis, and its
// rise over the cell), the knots K (ascending), the density of each bin, and the two-float prefix
// at the knots.  The first two depend on the geometry only and are written at set-up.
constexpr int kCells = 256;
constexpr int kGuessFloats = 2 * (kCells + 2);  // a multiple of 4 floats
__host__ __device__ __forceinline__ int back_knots(int nDet) { return (nDet + 1 + 3) / 4 * 4; }
__host__ __device__ __forceinline__ int back_view_floats(int nDet) { return kGuessFloats + 4 * back_knots(nDet); }

// Guess table of one view: entry i = (x_i, x_{i+1} - x_i), x_i the fractional knot index at
// kfirst + i (klast - kfirst) / kCells.
__device__ __forceinline__ float knot_index(const float4 *geo, int nDet, float u) {
    int lo = 0, hi = nDet;  // K[lo] <= u < K[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (geo[mid].x <= u) lo = mid; else hi = mid;
    }
    const float w = geo[lo + 1].x - geo[lo].x;
    return (float)lo + fminf(fmaxf((u - geo[lo].x) / w, 0.f), 1.f);
}
__global__ void __launch_bounds__(kThreads) bdd_guess_kernel(BddArgs G, const float4 *__restrict__ geo, float *tab) {
    const int p = blockIdx.x, nDet = G.nDet;
    const float4 *Gv = geo + (size_t)p * (nDet + 1);
    float *T = tab + (size_t)p * back_view_floats(nDet);
    const float k0 = Gv[0].x, h = (Gv[nDet].x - k0) / kCells;
    for (int i = threadIdx.x; i <= kCells; i += kThreads) {
        const float a = knot_index(Gv, nDet, fmaf((float)i, h, k0)), b = knot_index(Gv, nDet, fmaf((float)(i + 1), h, k0));
        reinterpret_cast<float2 *>(T)[i] = make_float2(a, i < kCells ? b - a : 0.f);
    }
    for (int j = threadIdx.x; j <= nDet; j += kThreads) T[kGuessFloats + j] = Gv[j].x;
}

// The back-projector's per-call table: one CTA per view forms each bin's integral B[j] =
// sino * (geometry factor) and density, in ascending knot order, and the two-float prefix of B
// over the knots (integrate1D, :229-241, of the weighted sinogram, :196), by a block-wide scan:
// each thread sums a contiguous run of bins, the runs' totals are scanned within each warp by
// shuffles and across the warps through shared memory, in order.  Knot nDet has density 0 and the
// total.
__global__ void __launch_bounds__(kThreads) bdd_fill_prefix_kernel(BddArgs G, const float *__restrict__ sino,
                                                                  const float4 *__restrict__ geo, float *tab) {
    __shared__ float2 wtot[kWarps];
    const int p = blockIdx.x, nDet = G.nDet;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const float4 *Gv = geo + (size_t)p * (nDet + 1);
    float *dens = tab + (size_t)p * back_view_floats(nDet) + kGuessFloats + back_knots(nDet);
    float2 *pre = reinterpret_cast<float2 *>(dens + back_knots(nDet));
    const bool desc = Gv[nDet].w != 0.f;
    const int chunk = (nDet + kThreads - 1) / kThreads;
    const int j_begin = min(nDet, tid * chunk), j_end = min(nDet, j_begin + chunk);
    // B[j] of ascending bin j (reference bin desc ? nDet-1-j : j)
    float th = 0.f, tl = 0.f;
    for (int j = j_begin; j < j_end; j++)
        two_sum_add(th, tl, sino[p + (size_t)G.na * (desc ? nDet - 1 - j : j)] * Gv[j].y);
    const unsigned full = 0xffffffffu;
    for (int off = 1; off < 32; off <<= 1) {  // inclusive scan of the runs within the warp
        const float oh = __shfl_up_sync(full, th, off), ol = __shfl_up_sync(full, tl, off);
        if (lane >= off) {
            two_sum_add(th, tl, oh);
            tl += ol;
        }
    }
    if (lane == 31) wtot[warp] = make_float2(th, tl);
    __syncthreads();
    float sh = 0.f, sl = 0.f;  // this run's start: the earlier warps, then the earlier lanes
    for (int w = 0; w < warp; w++) {
        two_sum_add(sh, sl, wtot[w].x);
        sl += wtot[w].y;
    }
    float eh = __shfl_up_sync(full, th, 1), el = __shfl_up_sync(full, tl, 1);
    if (lane == 0) eh = el = 0.f;
    two_sum_add(sh, sl, eh);
    sl += el;
    for (int j = j_begin; j < j_end; j++) {
        const float s = sino[p + (size_t)G.na * (desc ? nDet - 1 - j : j)];
        const float4 g = Gv[j];
        dens[j] = s * g.z;
        pre[j] = make_float2(sh, sl);
        two_sum_add(sh, sl, s * g.y);
    }
    if (j_begin < nDet && j_end == nDet) {
        dens[nDet] = 0.f;
        pre[nDet] = make_float2(sh, sl);
    }
}

// Per image row and view: pixel c takes |G(u_{c+1}) - G(u_c)| (:205) at its mapped boundaries
// u_c = r0 + c delta, clamped to the knots (Flat extrapolation, :199-201), G the detector prefix
// integral linearly interpolated (:198-203); the two-float prefix keeps that difference accurate
// to FP32 relative to the pixel's own integral.
//
// A warp has one image row and up to kBackGroups groups of 31 pixels of it; lane c of a group
// holds boundary c and takes the next lane's G.  The boundary's knot interval comes from the
// view's guess table, put right against the knots themselves (rarely by more than nothing: the
// table's linear steps are off by ~0.01 knots at 888 bins).  Neighbouring lanes read neighbouring
// knots, and the pixel sums stay in registers over the CTA's views.  The views that map onto x are
// taken first, then those that map onto y, which add to the transposed row (:210-212).
//
// Bound by issue (65 % of the slots) and shared loads (63 % of the wavefronts).  512^2 x 888 x 90
// views: 70 us; a lane walking the knots along its own run of 16 pixels took 121, its knot reads
// four to a bank and each waiting for the one before.
constexpr int kBackGroups = 9, kBackBatch = 3;  // groups per warp, and of them at a time
__global__ void __launch_bounds__(kThreads, 5)
    bdd_back_kernel(BddArgs G, const ViewInfo *info, const float *tab, const float4 *rmap, float *image,
                    int views_per_cta, int nchunk, int gpc, int nstage) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int nPix = G.nPix, vf = back_view_floats(G.nDet);
    const unsigned nDet = G.nDet;
    float *sm = reinterpret_cast<float *>(smraw);  // nstage x vf
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    const int unit = blockIdx.x * kWarps + warp, r = unit / nchunk;
    const int c0 = (unit % nchunk) * gpc * 31 + lane;
    const float cf = (float)c0;
    const int v_begin = blockIdx.y * views_per_cta, v_end = min(G.na, v_begin + views_per_cta);
    auto stage = [&](int p, int s) {
        const float4 *src = reinterpret_cast<const float4 *>(tab + (size_t)p * vf);
        float4 *dst = reinterpret_cast<float4 *>(sm + s * vf);
        for (int i = threadIdx.x; i < vf / 4; i += kThreads) cp_async16(dst + i, src + i);
        cp_async_commit();
    };
    float acc[kBackGroups];
#pragma unroll
    for (int i = 0; i < kBackGroups; i++) acc[i] = 0.f;
    for (int pass = 1; pass >= 0; pass--) {
        // next view at or after p that this pass takes; view 0 also adds its untransposed row
        // (aliasing of :139-140)
        auto next = [&](int p) {
            while (p < v_end && info[p].axis != pass && !(pass && p == 0)) p++;
            return p;
        };
        int p = next(v_begin), s = 0;
        if (p >= v_end) continue;  // uniform
        stage(p, 0);
        while (p < v_end) {
            const int pn = next(p + 1);
            if (nstage == 2 && pn < v_end) {
                stage(pn, s ^ 1);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncthreads();
            if (r < nPix) {
                const float2 *guess = reinterpret_cast<const float2 *>(sm + s * vf);
                const float *K = sm + s * vf + kGuessFloats, *dens = K + back_knots(nDet);
                const float2 *pre = reinterpret_cast<const float2 *>(dens + back_knots(nDet));
                const float4 rmv = rmap[(size_t)p * nPix + r];
                const float r0 = rmv.x, delta = rmv.y;
                const float kfirst = K[0], klast = K[nDet];
                const float scale = klast > kfirst ? (float)kCells / (klast - kfirst) : 0.f;
                const float wt = (pass && p == 0 && info[0].axis) ? 2.f : 1.f;
#pragma unroll
                for (int ib = 0; ib < kBackGroups; ib += kBackBatch) {
                    if (ib >= gpc) break;  // uniform
                    // floors by the round-down add of 2^23; the unsigned minima keep any index in
                    // its table
                    float u[kBackBatch], ka[kBackBatch], kb[kBackBatch];
                    unsigned j[kBackBatch];
                    bool off = false;
#pragma unroll
                    for (int i = 0; i < kBackBatch; i++) {
                        u[i] = fminf(fmaxf(fmaf(cf + 31.f * (ib + i), delta, r0), kfirst), klast);
                        const float x = (u[i] - kfirst) * scale, t = __fadd_rd(x, 8388608.f);
                        const float2 e = guess[min(__float_as_uint(t) - 0x4B000000u, (unsigned)kCells)];
                        const float y = fmaf(x - (t - 8388608.f), e.y, e.x);
                        j[i] = min(__float_as_uint(__fadd_rd(y, 8388608.f)) - 0x4B000000u, nDet - 1);
                        ka[i] = K[j[i]];
                        kb[i] = K[j[i] + 1];
                        off |= kb[i] <= u[i] || ka[i] > u[i];
                    }
                    if (off) {  // the largest j < nDet with K[j] <= u
#pragma unroll
                        for (int i = 0; i < kBackBatch; i++) {
                            while (kb[i] <= u[i] && j[i] < nDet - 1) {
                                j[i]++;
                                ka[i] = kb[i];
                                kb[i] = K[j[i] + 1];
                            }
                            while (ka[i] > u[i] && j[i] > 0) {
                                j[i]--;
                                ka[i] = K[j[i]];
                            }
                        }
                    }
#pragma unroll
                    for (int i = 0; i < kBackBatch; i++) {
                        const float2 g = pre[j[i]];
                        const float gh = g.x, gl = fmaf(u[i] - ka[i], dens[j[i]], g.y);
                        const float hh = __shfl_down_sync(full, gh, 1), hl = __shfl_down_sync(full, gl, 1);
                        acc[ib + i] = fmaf(fabsf((hh - gh) + (hl - gl)), wt, acc[ib + i]);  // :205
                    }
                }
            }
            __syncthreads();
            if (nstage == 2) s ^= 1;
            else if (pn < v_end) stage(pn, 0);
            p = pn;
        }
#pragma unroll
        for (int i = 0; i < kBackGroups; i++) {
            const int c = c0 + 31 * i;
            if (i < gpc && lane < 31 && r < nPix && c < nPix && acc[i] != 0.f)
                atomicAdd(pass ? image + r + (size_t)nPix * c                       // :210
                               : image + (nPix - 1 - c) + (size_t)nPix * r, acc[i]);  // :212, reverse(., 2)'
            acc[i] = 0.f;
        }
    }
}

size_t info_bytes(int na) { return ((size_t)na * sizeof(ViewInfo) + 255) & ~(size_t)255; }

size_t project_smem(const BddArgs &G) {
    return (sizeof(float2) + sizeof(float)) * (size_t)kWarps * (G.nPix + 1) +
           sizeof(float) * ((size_t)(G.nDet + 1) + (size_t)kWarps * G.nDet);
}
size_t project_bins_smem(const BddArgs &G) {
    return (sizeof(float2) + sizeof(float)) * (size_t)kWarps * (G.nPix + 1) + sizeof(RowMap) * kWarps +
           sizeof(float) * (size_t)(G.nDet + 1);
}
size_t project_direct_smem(const BddArgs &G, int wb) {
    const size_t rows = 2 * kDirRows * (size_t)direct_pitch(G.nPix), sums = (size_t)kWarps * kDirGroups * kDirGroup;
    return sizeof(float4) * (2 * kDirRows + 32 * (size_t)kDirGroups * wb) + sizeof(float) * std::max(rows, sums);
}
// The sizes this pair takes: the tables of one view with eight rows of both images, as the limit
// has always been stated.
bool back_fits(const BddArgs &G) {
    return 16 * (size_t)((G.nDet + 1 + 7) / 8 * 8) + 8 * (size_t)kWarps * (G.nPix + G.nPix / 16 + 1) <= 220 * 1024;
}
// A mapped bin's width in pixels at the image centre; up to kDirectStep the direct kernel projects.
// us a projection, prefix and direct, 512^2 from 90 views: bins of 0.6 pixels 143 and 107, 1.0 110 and 113,
// 1.2 101 and 96, 2.0 89 and 78, 4.0 78 and 62; from 360 views 538 and 303, 411 and 335, 380 and 305, 335 and
// 249, 290 and 194.  Wider bins keep the prefix form: its differences stay good to FP32 however many pixels
// lie in a bin.
constexpr double kDirectStep = 6.0;
double central_step(const BddArgs &G) { return G.dSize * G.DS0 / (G.DSD * G.pSize); }

// Blocks per SM that `smem` bytes a block leave room for, at most `cap` (what the registers allow).
int resident(size_t smem, int cap) { return std::max(1, std::min(cap, (int)(228 * 1024 / (smem + 1024)))); }

// The split of n items over base x split CTAs, `res` of them at a time on an SM, with the least
// time.  An SM issues at a fixed rate, so a wave takes as long as the items of its CTAs on one SM,
// each CTA with one item more (its first stage and its atomic adds), and a last wave that is less
// than 0.7 full no less than that: fewer warps leave issue slots idle.  Returns the items per CTA.
int split_items(int n, long long base, int res) {
    const long long sms = std::max(1, num_sms()), wave = sms * res;
    int best = n;
    double tb = 1e300;
    for (int s = 1; s <= n;) {
        const int per = (n + s - 1) / s;
        s = per > 1 ? (n + per - 2) / (per - 1) : n + 1;  // the next s with another per
        const long long ctas = base * ((n + per - 1) / per), rest = ctas % wave;
        const double last = rest ? std::max(0.7 * res, (double)((rest + sms - 1) / sms)) : 0.0;
        const double t = ((double)(ctas / wave) * res + last) * (per + 1);
        if (t < tb) {
            tb = t;
            best = per;
        }
        if (ctas > 16 * wave) break;
    }
    return best;
}

}  // namespace

// Scratch layouts.  Forward: view records | detm (na x (nDet+1)) | L (na x nDet) | row maps
// (na x nPix float4).  Back: view records | per-view tables (guess, knots, densities, prefix) |
// geometry table (na x (nDet+1) float4) | row maps.
size_t proj_rowmap_offset(const BddArgs &G) {
    return (info_bytes(G.na) + sizeof(float) * ((size_t)G.na * (G.nDet + 1) + (size_t)G.na * G.nDet) + 15) / 16 * 16;
}
size_t back_geo_offset(const BddArgs &G) {
    return info_bytes(G.na) + sizeof(float) * (size_t)G.na * back_view_floats(G.nDet);
}
size_t back_rowmap_offset(const BddArgs &G) {
    return back_geo_offset(G) + sizeof(float4) * (size_t)G.na * (G.nDet + 1);
}

size_t bdd_project_scratch(const BddArgs &G) {
    return proj_rowmap_offset(G) + sizeof(float4) * (size_t)G.na * G.nPix;
}

size_t bdd_back_scratch(const BddArgs &G) {
    return back_rowmap_offset(G) + sizeof(float4) * (size_t)G.na * G.nPix;
}

int launch_bdd_project_setup(const BddArgs &G, void *scratch, cudaStream_t st) {
    if (project_smem(G) > 220 * 1024) {
        set_error("project_bdd: nPix=%d nDet=%d exceed the shared-memory tile", G.nPix, G.nDet);
        return SGB_ERR_ARG;
    }
    ViewInfo *info = static_cast<ViewInfo *>(scratch);
    float *detm = reinterpret_cast<float *>(static_cast<char *>(scratch) + info_bytes(G.na));
    float *L = detm + (size_t)G.na * (G.nDet + 1);
    bdd_setup_kernel<<<dim3(G.na, (G.nDet + kSetupChunk - 1) / kSetupChunk), kThreads, 0, st>>>(G, info, detm, L,
                                                                                             nullptr);
    SGB_TRY(after_launch("bdd_setup_kernel"));
    float4 *rmap = reinterpret_cast<float4 *>(static_cast<char *>(scratch) + proj_rowmap_offset(G));
    const long long nr = (long long)G.na * G.nPix;
    bdd_rowmap_kernel<<<(unsigned)((nr + kThreads - 1) / kThreads), kThreads, 0, st>>>(G, info, rmap);
    return after_launch("bdd_rowmap_kernel");
}

int launch_bdd_project(const BddArgs &G, const float *phantom, float *sino, void *scratch,
                       cudaStream_t st) {
    SGB_TRY(launch_bdd_project_setup(G, scratch, st));
    return launch_bdd_project_main(G, phantom, sino, scratch, st);
}

int launch_bdd_project_main(const BddArgs &G, const float *phantom, float *sino, const void *scratch,
                            cudaStream_t st) {
    const size_t smem = project_smem(G);
    if (smem > 220 * 1024) {
        set_error("project_bdd: nPix=%d nDet=%d exceed the shared-memory tile", G.nPix, G.nDet);
        return SGB_ERR_ARG;
    }
    const ViewInfo *info = static_cast<const ViewInfo *>(scratch);
    const float *detm = reinterpret_cast<const float *>(static_cast<const char *>(scratch) + info_bytes(G.na));
    const float *L = detm + (size_t)G.na * (G.nDet + 1);
    const float4 *rmap = reinterpret_cast<const float4 *>(static_cast<const char *>(scratch) + proj_rowmap_offset(G));
    SGB_CUDA(cudaMemsetAsync(sino, 0, sizeof(float) * (size_t)G.na * G.nDet, st));
    if (central_step(G) <= kDirectStep) {
        int wb = 1;  // warps that share a row's groups
        while (wb < kWarps && wb * kDirGroups * kDirGroup < G.nDet) wb *= 2;
        const int z = (G.nDet + wb * kDirGroups * kDirGroup - 1) / (wb * kDirGroups * kDirGroup);
        const size_t sd = project_direct_smem(G, wb);
        const int blocks = split_items((G.nPix + kDirRows - 1) / kDirRows, (long long)G.na * z, resident(sd, 4));
        const int rpc = blocks * kDirRows;
        SGB_CUDA(cudaFuncSetAttribute(bdd_project_direct_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sd));
        bdd_project_direct_kernel<<<dim3(G.na, (G.nPix + rpc - 1) / rpc, z), kThreads, sd, st>>>(
            G, info, detm, L, rmap, phantom, sino, rpc, wb);
        return after_launch("bdd_project_direct_kernel");
    }
    // rows split over CTAs so that each SM holds ~8 of them (views x row blocks)
    const int target = 8 * std::max(1, num_sms());
    int rsplit = std::max(1, std::min((G.nPix + kWarps - 1) / kWarps, (target + G.na - 1) / G.na));
    int rows = (G.nPix + rsplit - 1) / rsplit;
    rows = (rows + kWarps - 1) / kWarps * kWarps;
    rsplit = (G.nPix + rows - 1) / rows;
    // bins split over the warps (sums in registers) while each warp's range fits NG groups of 32
    const int ngroups = (G.nDet + 31) / 32;
    if (ngroups <= kWarps * 8) {
        const size_t sb = project_bins_smem(G);
        if (ngroups <= kWarps * 4) {
            SGB_CUDA(cudaFuncSetAttribute(bdd_project_bins_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sb));
            bdd_project_bins_kernel<4><<<dim3(G.na, rsplit), kThreads, sb, st>>>(G, info, detm, L, rmap, phantom, sino,
                                                                                 rows);
        } else {
            SGB_CUDA(cudaFuncSetAttribute(bdd_project_bins_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sb));
            bdd_project_bins_kernel<8><<<dim3(G.na, rsplit), kThreads, sb, st>>>(G, info, detm, L, rmap, phantom, sino,
                                                                                 rows);
        }
        return after_launch("bdd_project_bins_kernel");
    }
    SGB_CUDA(cudaFuncSetAttribute(bdd_project_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    bdd_project_kernel<<<dim3(G.na, rsplit), kThreads, smem, st>>>(G, info, detm, L, rmap, phantom, sino, rows);
    return after_launch("bdd_project_kernel");
}

int launch_bdd_back_setup(const BddArgs &G, void *scratch, cudaStream_t st) {
    if (!back_fits(G)) {
        set_error("backproject_bdd: nPix=%d nDet=%d exceed the shared-memory tile", G.nPix, G.nDet);
        return SGB_ERR_ARG;
    }
    ViewInfo *info = static_cast<ViewInfo *>(scratch);
    float *tab = reinterpret_cast<float *>(static_cast<char *>(scratch) + info_bytes(G.na));
    float4 *geo = reinterpret_cast<float4 *>(static_cast<char *>(scratch) + back_geo_offset(G));
    bdd_setup_kernel<<<dim3(G.na, (G.nDet + kSetupChunk - 1) / kSetupChunk), kThreads, 0, st>>>(G, info, nullptr, nullptr,
                                                                                             geo);
    SGB_TRY(after_launch("bdd_setup_kernel"));
    bdd_guess_kernel<<<G.na, kThreads, 0, st>>>(G, geo, tab);
    SGB_TRY(after_launch("bdd_guess_kernel"));
    float4 *rmap = reinterpret_cast<float4 *>(static_cast<char *>(scratch) + back_rowmap_offset(G));
    const long long nr = (long long)G.na * G.nPix;
    bdd_rowmap_kernel<<<(unsigned)((nr + kThreads - 1) / kThreads), kThreads, 0, st>>>(G, info, rmap);
    return after_launch("bdd_rowmap_kernel");
}

int launch_bdd_back_main(const BddArgs &G, const float *sino, float *image, void *scratch, cudaStream_t st) {
    if (!back_fits(G)) {
        set_error("backproject_bdd: nPix=%d nDet=%d exceed the shared-memory tile", G.nPix, G.nDet);
        return SGB_ERR_ARG;
    }
    const ViewInfo *info = static_cast<const ViewInfo *>(scratch);
    float *tab = reinterpret_cast<float *>(static_cast<char *>(scratch) + info_bytes(G.na));
    const float4 *geo = reinterpret_cast<const float4 *>(static_cast<const char *>(scratch) + back_geo_offset(G));
    const float4 *rmap = reinterpret_cast<const float4 *>(static_cast<const char *>(scratch) + back_rowmap_offset(G));
    SGB_CUDA(cudaMemsetAsync(image, 0, sizeof(float) * (size_t)G.nPix * G.nPix, st));
    bdd_fill_prefix_kernel<<<G.na, kThreads, 0, st>>>(G, sino, geo, tab);
    SGB_TRY(after_launch("bdd_fill_prefix_kernel"));
    // a warp per (row, chunk of at most kBackGroups groups of 31 pixels)
    const int ngroups = (G.nPix + 30) / 31, nchunk = (ngroups + kBackGroups - 1) / kBackGroups;
    const int gpc = (ngroups + nchunk - 1) / nchunk;
    const long long gx = ((long long)G.nPix * nchunk + kWarps - 1) / kWarps;
    const size_t vbytes = sizeof(float) * (size_t)back_view_floats(G.nDet);
    const int nstage = 2 * vbytes <= 220 * 1024 ? 2 : 1;
    const size_t smem = nstage * vbytes;
    const int vpc = split_items(G.na, gx, resident(smem, 5));
    SGB_CUDA(cudaFuncSetAttribute(bdd_back_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    bdd_back_kernel<<<dim3((unsigned)gx, (G.na + vpc - 1) / vpc), kThreads, smem, st>>>(G, info, tab, rmap, image, vpc,
                                                                                        nchunk, gpc, nstage);
    return after_launch("bdd_back_kernel");
}

int launch_bdd_back(const BddArgs &G, const float *sino, float *image, void *scratch, cudaStream_t st) {
    SGB_TRY(launch_bdd_back_setup(G, scratch, st));
    return launch_bdd_back_main(G, sino, image, scratch, st);
}

}  // namespace sgb
