// sgb_fdk_mirror.cu -- host side of the mirrored FDK back-projector: which reflections a scan has,
// the boxes' device pre-pass, and the dispatch (kernel in sgb_fdk_mirror_kernel.cuh).
#include <algorithm>
#include <cmath>

#include "sgb_fdk_mirror_kernel.cuh"
#include "sgb_kernels.cuh"

namespace sgb {

namespace {

using namespace fdkdev;

template <bool ARC>
__global__ void mirror_extent_kernel(FdkMirrorArgs M, int ntx, int nty, int ntz, int *ext) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long ntile = (long long)ntx * nty * ntz;
    if (i >= ntile * M.nviews) return;
    const int v = (int)(i / ntile), t = (int)(i % ntile);
    int wmax = 0, hmax = 0;
    for (int j = 0; j < M.nvs; j++) {
        const MirExtent e = mir_extent(M, j, t % ntx, (t / ntx) % nty, t / (ntx * nty));
        const float2 sc = M.A.trig[mir_slot_view(M, j, v)];
        int s0, t0, w, h;
        tile_box<ARC>(M.A, sc.x, sc.y, e.xlo, e.xhi, e.ylo, e.yhi, e.zlo, e.zhi, &s0, &t0, &w, &h);
        wmax = max(wmax, w);
        hmax = max(hmax, h);
    }
    atomicMax(ext + 0, wmax);
    atomicMax(ext + 1, hmax);
}

// x when it is an integer up to the rounding of the angles it comes from
bool whole(double x, int n, int *out) {
    const double r = std::nearbyint(x);
    if (!(std::fabs(x - r) < 1e-9 * std::max(1.0, std::fabs(x)))) return false;
    const double m = std::fmod(r, (double)n);
    *out = (int)(m < 0 ? m + n : m);
    return true;
}

bool symmetric_grid(float c0, float d, int n) {
    for (int i = 0; i < n; i++)
        if (std::fmaf((float)i, d, c0) != -std::fmaf((float)(n - 1 - i), d, c0)) return false;
    return true;
}

}  // namespace

void fdk_mirror_slots(FdkMirrorArgs &M, const FdkTmaArgs &A, double orbit, double orbit_start, const double *offsets,
                      double offset_t) {
    M = FdkMirrorArgs{};
    M.A = A;
    M.nvs = 1;
    M.nviews = A.na;
    M.vsgn[0] = 1;
    M.hx = A.nx;
    M.hy = A.ny;
    M.nzd = A.nz;
    if (A.elem_bytes != 8 || A.zsrc || A.ia_skip != 1) return;
    M.exact = symmetric_grid(A.x0, A.dx, A.nx) && symmetric_grid(A.y0, A.dy, A.ny);
    if (A.quad && !M.exact) return;
    const double turns = std::fabs(orbit) / 360.0, step = orbit / A.na;
    int vx = 0, vy = 0, vxy = 0;
    bool x = false, y = false, xy = false;
    if (turns >= 1 && turns == std::floor(turns)) {  // whole turns: the views repeat every 360 degrees
        x = offsets[0] == 0 && whole(-2 * orbit_start / step, A.na, &vx);
        y = offsets[1] == 0 && whole((180 - 2 * orbit_start) / step, A.na, &vy);
        xy = offsets[0] == 0 && offsets[1] == 0 && whole(180 / step, A.na, &vxy);
    }
    auto slot = [&](int j, int flip) {
        M.flip[j] = flip;
        M.vsgn[j] = flip == (MIR_X | MIR_Y) ? 1 : -1;
        M.voff[j] = flip == MIR_X ? vx : (flip == MIR_Y ? vy : vxy);
    };
    if (x && y && xy) {
        M.nvs = 4;
        for (int j = 1; j < 4; j++) slot(j, j);
    } else if (x || y || xy) {
        M.nvs = 2;
        slot(1, x ? MIR_X : (y ? MIR_Y : MIR_X | MIR_Y));
    }
    int f = 0;
    for (int j = 0; j < M.nvs; j++) f |= M.flip[j];
    // XY alone needs one axis halved
    if (f & MIR_X && !(M.nvs == 2 && f & MIR_Y)) M.hx = (A.nx + 1) / 2;
    if (f & MIR_Y) M.hy = (A.ny + 1) / 2;
    // FP32 only (see the kernel); four view slots already share as much as pays
    M.zm = !A.quad && M.nvs < 4 && offsets[2] == 0 && 2 * offset_t == std::floor(2 * offset_t);
    if (M.zm) {
        M.iz0 = A.nz / 2;
        M.nzd = A.nz - M.iz0;
        M.m2 = A.nt + 1 + (int)(2 * offset_t);
    }
    M.zbase = A.quad ? A.zu : 16;
}

size_t fdk_mirror_smem(const FdkMirrorArgs &M, int nstage) {
    const int ns = M.nvs * (M.zm ? 2 : 1);
    const size_t ring = (size_t)nstage * ((size_t)ns * M.A.box_bytes + sizeof(MirStage) + 2 * sizeof(uint64_t)) +
                        sizeof(MirRun) + M.nvs * sizeof(MirExtent);
    const size_t part = M.split > 1 ? sizeof(float) * ns * M.kz * kConsumers : 0;  // the ranks' partial tiles
    return 128 + std::max(ring, part);
}

namespace {

// Predicted times in us.  A CTA takes for a view its columns' geometry (`column`, arcs `arc` more), `voxel`
// and per slot `tap` (`tapz` with slots at -z) for each voxel of a run, and `byte` for each byte of its boxes.
// Taps take up to `two` times as much more where voxels lie several detector rows apart, so that each loads
// rows of its own, and runs that pass the detector's edge go `edge` times slower.  A second CTA on an SM takes
// `shared` of the first's time, a few rounds of CTAs even out less than many, a split takes its reduction.
// Fitted to 3500 launches of 290 FP32 and 1200 of 141 F16 scans (48 to 400 columns a side, 1 to 256 slices, 40
// to 700 views, voxels 0.1 to 9 detector rows apart, volumes inside the detector and past it): of the two
// kernels and the mirrored one's runs and splits (powers of two: clusters of others fill the chip worse) the
// fastest prediction took 4 % more than the fastest launch in the geometric mean, and on 15 scans 4 to 19 %
// more than the unmirrored kernel; the mirrored kernel wherever its boxes fit had taken up to 3.5 times as much.
struct FdkCost {
    double column, arc, voxel, tap, tapz, two, step2, step4, width, slope, byte, shared, uneven, edge, view, sum, rank,
        fixed;
};
constexpr FdkCost kMirrorPair = {0.118, 0.0638, 0.00927, 0.00615, 0.00617, 1.54, 0.125, 0.0227, 0.575, 0.0123,
                                 8.63e-6, 0.557, 0.0332, 1.93, 0.029, 4.99, 0.151, 10.7};
constexpr FdkCost kMirrorQuad = {0.106, 0.0663, 0.0144, 0.0102, 0.0243, 0.453, 0.392, 3.19, 1e-3, 0,
                                 7.86e-6, 0.503, 0.0646, 0.545, 0.01, 5.33, 0, 8.52};
constexpr FdkCost kPlainPair = {0.0858, 0.122, 0.0145, 0.00734, 0, 0.34, 0.784, 0.784, 1.4e-3, 0.0789,
                                1e-5, 0.388, 0.0414, 0.111, 0, 0, 0, 9.65};
constexpr FdkCost kPlainQuad = {0.135, 0.103, 0.00558, 0.00943, 0, 0.0961, 0, 0, 1e9, 0.0078,
                                1.3e-5, 0.378, 0, 0.101, 0, 0, 0, 10.7};

// Share of the (column, view) pairs of runs of kz voxels from iz0 that pass the detector's first or last row, from
// a coarse sample of columns and angles.
double edge_share(const FdkTmaArgs &A, int iz0, int kz, bool whole_runs) {
    const double limit = (A.nt - 1) / 2.0 - 0.02;
    double toward[8];
    for (int a = 0; a < 8; a++) toward[a] = std::cos((a + 0.5) * 0.39269908169872414);  // pi / 8
    long long out = 0, all = 0;
    for (int b = 0; iz0 + b * kz < A.nz; b++) {
        int iz = iz0 + b * kz;
        if (whole_runs && iz + kz > A.nz && A.nz >= kz) iz = A.nz - kz;
        const double z = std::max(std::fabs(A.z0 + iz * A.dz), std::fabs(A.z0 + (iz + kz - 1) * A.dz)) * A.inv_dtds;
        for (int i = 0; i < 36; i++) {
            const double x = A.x0 + A.dx * (A.nx * (i % 6 + 0.5) / 6 - 0.5), y = A.y0 + A.dy * (A.ny * (i / 6 + 0.5) / 6 - 0.5);
            const double r = std::hypot(x, y);
            for (int a = 0; a < 8; a++, all++) out += z * A.dsd_ds > limit * (A.dso_ds - r * toward[a]);
        }
    }
    return all ? (double)out / (double)all : 0;
}

// A CTA's time per view (slots: voxels per (x, y, z) of the run) and a launch's.
double cta_view(const FdkCost &c, const FdkTmaArgs &A, int kz, int slots, int nvs, bool zm, double edge) {
    const double step = std::fabs(A.dz) * A.inv_dtds * A.dsd_ds / A.dso_ds, over = step - (slots == 2 ? c.step2 : c.step4);
    const double two = 1 + c.two / (1 + std::exp(-std::max(-30.0, std::min(30.0, over / c.width)))) + c.slope * std::max(0.0, over);
    return (c.column + (A.is_arc ? c.arc * std::sqrt((double)nvs) : 0) + kz * c.voxel + kz * slots * (zm ? c.tapz : c.tap) * two +
            (double)slots * A.box_bytes * c.byte) *
           (1 + edge * c.edge);
}
double launch_us(const FdkCost &c, double view, int nv, int split, long long ctas, int per) {
    const long long sms = std::max(1, num_sms()), busiest = (ctas * split + sms - 1) / sms, rounds = (busiest + per - 1) / per;
    const double t = busiest <= per ? view * (per == 2 ? 1 + c.shared * (busiest - 1) : (double)busiest)
                                    : view * (1 + c.shared * (per - 1)) * busiest / per * (1 + c.uneven / rounds);
    return (floor_div_up(nv, split) + c.view * rounds) * t + (split > 1 ? c.sum * rounds + c.rank * split : 0) + c.fixed;
}

}  // namespace

double fdk_tma_predict(const FdkTmaArgs &A) {
    const FdkCost &c = A.quad ? kPlainQuad : kPlainPair;
    const double view = cta_view(c, A, A.zu, 1, 1, false, edge_share(A, 0, A.zu, true));
    return launch_us(c, view, A.nv, 1, (long long)floor_div_up(A.nx, kTX) * floor_div_up(A.ny, kTY) * floor_div_up(A.nz, A.zu), 2);
}

int fdk_mirror_prepare(FdkMirrorArgs &M, int *ext_dev, cudaStream_t st, double limit_us, bool *fits) {
    *fits = false;
    const int ns = M.nvs * (M.zm ? 2 : 1);
    if (ns == 1) return SGB_OK;
    const int tx = floor_div_up(M.hx, kTX), ty = floor_div_up(M.hy, kTY);
    const FdkCost &c = M.A.quad ? kMirrorQuad : kMirrorPair;
    FdkMirrorArgs best{};
    double best_us = limit_us;
    for (int half = 0; half < 2; half++) {
        FdkMirrorArgs T = M;
        FdkTmaArgs &A = T.A;
        A.align = 2;  // 16 bytes
        A.vps = 1;
        T.kz = half ? 32 / ns : 64 / ns;
        T.split = 1;
        const int ntz = floor_div_up(T.nzd, T.kz);
        const long long ctas = (long long)tx * ty * ntz;
        auto fits_grid = [&](int g) { return A.nv >= 8 * g && ctas * g <= (1 << 30) && ntz * g <= 65535; };
        const double edge = edge_share(A, M.iz0, T.kz, !A.quad);
        // Whatever the boxes are, a launch is predicted to take longer than without any: the pre-pass, some 12 us,
        // is spared where none can be the fastest (16 x 16 x 4 voxels, 30 views: a plan 380 and 330 us).
        A.box_bytes = 0;
        const double least = cta_view(c, A, T.kz, ns, M.nvs, M.zm, edge);
        double bound = limit_us;
        for (int g = 1; g <= 8 && fits_grid(g); g *= 2)
            for (int per = 1; per <= 2; per++) bound = std::min(bound, launch_us(c, least, A.nv, g, ctas, per));
        if (bound >= best_us) continue;
        SGB_CUDA(cudaMemsetAsync(ext_dev, 0, 2 * sizeof(int), st));
        const long long n = (long long)tx * ty * ntz * T.nviews;
        const unsigned blocks = (unsigned)((n + 255) / 256);
        if (A.is_arc) mirror_extent_kernel<true><<<blocks, 256, 0, st>>>(T, tx, ty, ntz, ext_dev);
        else mirror_extent_kernel<false><<<blocks, 256, 0, st>>>(T, tx, ty, ntz, ext_dev);
        SGB_TRY(after_launch("mirror_extent_kernel"));
        int ext[2];
        SGB_CUDA(cudaMemcpyAsync(ext, ext_dev, sizeof ext, cudaMemcpyDeviceToHost, st));
        SGB_CUDA(cudaStreamSynchronize(st));
        A.W = (ext[0] + 1) / 2 * 2;
        A.H = ext[1];
        if (A.W > 128 || A.H <= 1 || A.H > 256) continue;
        A.box_bytes = (int)(((size_t)A.W * A.H * 8 + 127) / 128 * 128);
        A.nstage = fdk_mirror_smem(T, 4) <= 112 * 1024 ? 4 : 3;
        if (fdk_mirror_smem(T, A.nstage) > 226 * 1024) continue;
        const double view = cta_view(c, A, T.kz, ns, M.nvs, M.zm, edge);
        for (int g = 1; g <= 8 && fits_grid(g); g *= 2) {
            T.split = g;
            const size_t smem = fdk_mirror_smem(T, A.nstage);
            if (smem > 226 * 1024) break;
            const double us = launch_us(c, view, A.nv, g, ctas, smem <= 112 * 1024 ? 2 : 1);
            if (us < best_us) {
                best_us = us;
                best = T;
                *fits = true;
            }
        }
    }
    if (*fits) M = best;
    return SGB_OK;
}

int launch_fdk_mirror(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st) {
    const int passes = std::max(1, std::min(M.A.passes, M.A.nv));
    for (int p = 0; p < passes; p++) {
        FdkMirrorArgs T = M;
        T.A.v0 = M.A.v0 + (int)((long long)M.A.nv * p / passes);
        T.A.nv = (int)((long long)M.A.nv * (p + 1) / passes) - (T.A.v0 - M.A.v0);
        T.A.accum = M.A.accum || p > 0;
        SGB_TRY(M.A.quad ? (M.A.is_arc ? launch_fdk_mirror_quad_arc(T, map, st) : launch_fdk_mirror_quad_flat(T, map, st))
                         : (M.A.is_arc ? launch_fdk_mirror_pair_arc(T, map, st) : launch_fdk_mirror_pair_flat(T, map, st)));
    }
    return SGB_OK;
}

}  // namespace sgb
