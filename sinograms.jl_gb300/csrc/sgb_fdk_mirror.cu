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

int fdk_mirror_prepare(FdkMirrorArgs &M, int *ext_dev, cudaStream_t st, bool *fits) {
    *fits = false;
    const int ns = M.nvs * (M.zm ? 2 : 1);
    if (ns == 1) return SGB_OK;
    const int tx = floor_div_up(M.hx, kTX), ty = floor_div_up(M.hy, kTY), sms = std::max(1, num_sms());
    // Run length and view split by the time they predict: the busiest SM's CTAs, each so many us per
    // view.  Fitted to 22 volumes from 51 x 166 x 221 to 512 x 512 x 256: 64 accumulators per thread take
    // 1.54 us for a CTA alone on its SM and 1.74 us for two (32 accumulators: 1.19 and 1.39), and where
    // voxels lie 1.5 detector rows or more apart, so that each loads two rows, 2.2 and 2.8 (1.4 and 1.7).
    // A split costs its reduction, about 4 us, and 1.5% per rank.  The choice came within 10% of the
    // fastest of all runs and splits on 18 of them, and within 25% on the others.
    FdkMirrorArgs best{};
    double best_us = 1e30;
    for (int half = 0; half < 2; half++) {
        FdkMirrorArgs T = M;
        FdkTmaArgs &A = T.A;
        A.align = 2;  // 16 bytes
        A.vps = 1;
        T.kz = half ? 32 / ns : 64 / ns;
        T.split = 1;
        const int ntz = floor_div_up(T.nzd, T.kz);
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
        const int per = fdk_mirror_smem(T, A.nstage) <= 112 * 1024 ? 2 : 1;  // CTAs that fit an SM
        const bool coarse = std::fabs(A.dz) * A.inv_dtds * A.dsd_ds / A.dso_ds >= 1.5f;
        const double alone = coarse ? (half ? 1.4 : 2.2) : (half ? 1.19 : 1.54);
        const double more = coarse ? (half ? 0.3 : 0.6) : 0.20;
        const long long ctas = (long long)tx * ty * ntz;
        for (int g = 1; g <= 8; g++) {
            if (A.nv < 8 * g || ctas * g > (1 << 30) || ntz * g > 65535) break;
            const long long busiest = (ctas * g + sms - 1) / sms;
            const double view = busiest <= per ? alone + more * (busiest - 1) : (alone + more * (per - 1)) * busiest / per;
            const double us = (double)((A.nv + g - 1) / g) * view * (1 + 0.015 * (g - 1)) + (g > 1 ? 4 : 0);
            if (us < best_us) {
                best_us = us;
                best = T;
                best.split = g;
            }
        }
    }
    if (best_us > 1e29) return SGB_OK;
    M = best;
    *fits = true;
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
