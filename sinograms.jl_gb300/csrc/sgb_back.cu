// sgb_back.cu -- voxel/pixel-driven back-projectors.
//
// FDK: cbct_back_fan! / cbct_back_fan_voxel (src/fbp3/cbct-back.jl:95-213).
// 2D:  dispatch over detectors and symmetries (kernel in sgb_back2_kernel.cuh).
//
// Per-view sin/cos come from FP64 angles (view_trig_kernel) and sit in shared memory.
// A thread owns one (x, y) column and kZ consecutive voxels along z: the column's
// per-view geometry (magnification, detector s, weight) is computed once and reused
// for all kZ voxels, which only differ in the detector row coordinate t.
// Interpolation is manual bilinear with the reference's edge rule: the whole tap is
// dropped unless 1 <= floor(bs) < ns and 1 <= floor(bt) < nt (cbct-back.jl:197).
#include "sgb_common.cuh"
#include "sgb_kernels.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace sgb {

namespace {

__global__ void view_trig_kernel(const double *__restrict__ betas, int nv, int ia_skip,
                                 float2 *__restrict__ trig) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    double s, c;
    sincos(betas[(long long)v * ia_skip], &s, &c);
    trig[v] = make_float2((float)s, (float)c);
}

constexpr int kBX = 32, kBY = 4;  // FDK CTA: 32 x 4 columns
constexpr int kVChunk = 1024;     // views staged in shared memory per pass

// GEO: 0 CtFanFlat, 1 CtFanArc, 2 CtPar (3D parallel beam: s' = x_beta, t' = z, unit weight)
template <typename TP, int GEO, int kZ>
__global__ void __launch_bounds__(kBX *kBY) fdk_back_kernel(FdkArgs A) {
    __shared__ float2 trig_s[kVChunk];
    __shared__ float zs_s[kVChunk];  // source z / ds per view (0 for a circular orbit)
    const int ix = blockIdx.x * kBX + threadIdx.x;
    const int iy = blockIdx.y * kBY + threadIdx.y;
    const int iz0 = blockIdx.z * kZ;
    const bool active = ix < A.nx && iy < A.ny;
    const TP *__restrict__ proj = static_cast<const TP *>(A.proj);

    const float x = active ? A.xds[ix] : 0.f;
    const float y = active ? A.yds[iy] : 0.f;
    float z[kZ], acc[kZ];
#pragma unroll
    for (int k = 0; k < kZ; k++) {
        z[k] = (iz0 + k < A.nz) ? A.zds[iz0 + k] : 0.f;
        acc[k] = 0.f;
    }
    const int ns = A.ns, nt = A.nt;
    const float fns = (float)ns, fnt = (float)nt;
    const int pitch = A.pitch;
    const long long view_stride = (long long)pitch * nt;
    const int tid = threadIdx.y * kBX + threadIdx.x;

    for (int v0 = 0; v0 < A.nv; v0 += kVChunk) {
        const int nvc = min(kVChunk, A.nv - v0);
        __syncthreads();
        for (int i = tid; i < nvc; i += kBX * kBY) {
            trig_s[i] = A.trig[v0 + i];
            zs_s[i] = A.zsrc ? A.zsrc[v0 + i] : 0.f;
        }
        __syncthreads();
        if (!active) continue;
        for (int vi = 0; vi < nvc; vi++) {
            const float2 sc = trig_s[vi];
            const float zs = zs_s[vi];
            const float sb = sc.x, cb = sc.y;
            const float xb = fmaf(x, cb, y * sb);                    // cbct-back.jl:174
            float mag, sp, w2;
            if (GEO == 2) {  // parallel beam: the fan map with the source at infinity (back-par.jl:293)
                mag = 1.f;
                sp = xb;
                w2 = 1.f;
            } else {
                const float yb = A.dso_ds - fmaf(-x, sb, y * cb);    // :175
                if (GEO == 1) {                                      // :177-181
                    sp = A.dsd_ds * atan2f(xb, yb);
                    mag = __fdividef(A.dsd_ds, yb);
                    w2 = __fdividef(A.dsd_ds * A.dsd_ds, fmaf(xb, xb, yb * yb));
                } else {                                             // :183-185
                    mag = __fdividef(A.dsd_ds, yb);
                    sp = mag * xb;
                    w2 = mag * mag;
                }
            }
            const float bs = sp + A.ws;                              // :191
            const float fis = floorf(bs);
            if (!(fis >= 1.f && fis < fns)) continue;                // :197 (s part)
            const float fs = bs - fis;
            const float magt = mag * A.inv_dtds;
            const TP *base = proj + (long long)(v0 + vi) * A.ia_skip * view_stride + ((int)fis - 1);
#pragma unroll
            for (int k = 0; k < kZ; k++) {
                const float bt = fmaf(magt, z[k] - zs, A.wt);        // :188-192
                const float fit = floorf(bt);
                if (fit >= 1.f && fit < fnt) {                       // :197 (t part)
                    const float ft = bt - fit;
                    const TP *p = base + (long long)((int)fit - 1) * pitch;
                    const float p00 = ld_proj(p), p10 = ld_proj(p + 1);
                    const float p01 = ld_proj(p + pitch), p11 = ld_proj(p + pitch + 1);
                    const float a0 = fmaf(fs, p10 - p00, p00);       // :205
                    const float a1 = fmaf(fs, p11 - p01, p01);       // :206
                    acc[k] = fmaf(w2, fmaf(ft, a1 - a0, a0), acc[k]); // :208
                }
            }
        }
    }
    if (!active) return;
#pragma unroll
    for (int k = 0; k < kZ; k++) {
        const int iz = iz0 + k;
        if (iz >= A.nz) break;
        const long long idx = ix + (long long)A.nx * (iy + (long long)A.ny * iz);
        float v = acc[k];
        if (A.mask && !A.mask[idx]) v = 0.f;  // :133
        A.image[idx] = v;
    }
}

template <typename TP, int GEO>
int launch_fdk_z(const FdkArgs &A, cudaStream_t st) {
    constexpr int kZ = 8;
    dim3 block(kBX, kBY);
    dim3 grid(floor_div_up(A.nx, kBX), floor_div_up(A.ny, kBY), floor_div_up(A.nz, kZ));
    fdk_back_kernel<TP, GEO, kZ><<<grid, block, 0, st>>>(A);
    return after_launch("fdk_back_kernel");
}

__global__ void interleave4_kernel(const float *__restrict__ in, float4 *__restrict__ out, long long n, int nslices) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int s = blockIdx.y * 4;
    const float *p = in + i + n * s;
    out[i + n * blockIdx.y] = make_float4(__ldg(p), s + 1 < nslices ? __ldg(p + n) : 0.f,
                                          s + 2 < nslices ? __ldg(p + 2 * n) : 0.f, s + 3 < nslices ? __ldg(p + 3 * n) : 0.f);
}

}  // namespace

int launch_interleave4(const float *in, float *out, long long n, int nslices, cudaStream_t st) {
    const dim3 grid((unsigned)((n + 255) / 256), floor_div_up(nslices, 4));
    interleave4_kernel<<<grid, 256, 0, st>>>(in, reinterpret_cast<float4 *>(out), n, nslices);
    return after_launch("interleave4_kernel");
}

int launch_view_trig(const double *betas_dev, int na, int ia_skip, float2 *trig, cudaStream_t st) {
    int nv = (na + ia_skip - 1) / ia_skip;
    view_trig_kernel<<<floor_div_up(nv, 128), 128, 0, st>>>(betas_dev, nv, ia_skip, trig);
    return after_launch("view_trig_kernel");
}

int launch_fdk_back(const FdkArgs &A, cudaStream_t st) {
    if (A.nx <= 0 || A.ny <= 0 || A.nz <= 0) return SGB_OK;
    const int geo = A.is_par ? 2 : (A.is_arc ? 1 : 0);
    if (A.bf16)
        return geo == 2 ? launch_fdk_z<__nv_bfloat16, 2>(A, st)
                        : (geo == 1 ? launch_fdk_z<__nv_bfloat16, 1>(A, st) : launch_fdk_z<__nv_bfloat16, 0>(A, st));
    return geo == 2 ? launch_fdk_z<float, 2>(A, st)
                    : (geo == 1 ? launch_fdk_z<float, 1>(A, st) : launch_fdk_z<float, 0>(A, st));
}

// Staged bins per segment: what a 32 x 32 tile of dx x dy pixels (in bins) with pixels within `reach` (in bins)
// of the centre spans at most, with the kernel's margins; tiles that span more read global memory.
void back2_window(Back2Args &A, double dx, double dy, double reach) {
    const double corner = std::hypot(dx * A.nx, dy * A.ny) / 2, r = std::min(corner, reach + 32 * std::hypot(dx, dy));
    const double mag = A.mode == SGB_PAR ? 1.0 : A.dsd_ds / std::max(1e-3, A.dso_ds - r);
    const double span = 1.05 * mag * 31 * std::hypot(dx, dy) + 10;
    A.w = span < 256 ? ((int)span + 7) / 8 * 8 : 256;
}

float back2_wanted(const uint8_t *mask, int nx, int ny, double dx, double dy, double ox, double oy, double *reach) {
    const int tx = floor_div_up(nx, kB2X), ty = floor_div_up(ny, kB2Y * kB2P);
    std::vector<char> in((size_t)tx * ty, 0);
    double far = 0;
    for (int y = 0; y < ny; y++) {
        const uint8_t *row = mask + (size_t)nx * y;
        int first = 0, last = nx - 1;  // the row's ends, the farthest of its pixels
        while (first < nx && !row[first]) first++;
        if (first == nx) continue;
        while (!row[last]) last--;
        const double v = dy * (y - ((ny - 1) / 2.0 + oy));
        for (int x : {first, last}) {
            const double u = dx * (x - ((nx - 1) / 2.0 + ox));
            far = std::max(far, u * u + v * v);
        }
        char *tiles = in.data() + (size_t)tx * (y / (kB2Y * kB2P));
        for (int t = first / kB2X; t <= last / kB2X; t++)
            for (int x = std::max(first, t * kB2X); !tiles[t] && x <= last && x < (t + 1) * kB2X; x++) tiles[t] = row[x] != 0;
    }
    *reach = std::sqrt(far);
    size_t n = 0;
    for (char c : in) n += c;
    return (float)n / (float)in.size();
}

// Which pixels and views share geometry: needs the grid centred (offsets 0) on the axes that a slot
// mirrors, and for slots whose bins run the other way a centred detector.
ScanSlots scan_slots(int kind, int na, int nx, int ny, bool centred, bool source_centred, double orbit,
                     double orbit_start, const double *deltas, const double *offsets, bool prefer_turn) {
    ScanSlots S{};
    S.ns = 1;
    S.hx = nx;
    S.hy = ny;
    S.slot[0].sgn = 1;
    const double step = orbit / na, turns = std::fabs(orbit) / 360.0;
    const bool whole = turns >= 1 && turns == std::floor(turns), half = kind == SGB_PAR && std::fabs(orbit) == 180.0;
    if (!(whole || half)) return S;
    S.half = half;
    const int period = half ? 2 * na : na;
    auto views = [&](double angle, int *off) {  // `angle` as a whole number of views
        const double q = angle / step, r = std::nearbyint(q);
        if (!(std::fabs(q - r) < 1e-9 * std::max(1.0, std::fabs(q)))) return false;
        const double m = std::fmod(r, (double)period);
        *off = (int)(m < 0 ? m + period : m);
        return true;
    };
    const bool cx = offsets[0] == 0, cy = offsets[1] == 0, square = nx == ny && std::fabs(deltas[0]) == std::fabs(deltas[1]);
    int o90 = 0, o180 = 0, ox = 0, oy = 0;
    const bool turn90 = cx && cy && square && views(90, &o90) && (centred || !half);
    const bool turn180 = cx && cy && views(180, &o180) && (centred || !half);
    const bool mirror = centred && source_centred;
    const bool mx = mirror && cx && views(-2 * orbit_start, &ox), my = mirror && cy && views(180 - 2 * orbit_start, &oy);
    const bool both = mx && my && turn180;
    if (turn90 && (prefer_turn || !both)) {
        S.ns = 4;
        S.turn = 1;
        S.hx = S.hy = (nx + 1) / 2;
        const bool same = (deltas[0] > 0) == (deltas[1] > 0);  // (x, y) -> (-y, x) in pixel indices
        for (int j = 1; j < 4; j++)
            S.slot[j] = {j == 2 ? 3 : 4 + ((j == 1) == same ? 1 : 2), 1, (int)((long long)j * o90 % period), 0};
    } else if (both) {
        S.ns = 4;
        S.hx = (nx + 1) / 2;
        S.hy = (ny + 1) / 2;
        S.slot[1] = {1, -1, ox, 1};
        S.slot[2] = {2, -1, oy, 1};
        S.slot[3] = {3, 1, o180, 0};
    } else if (turn180) {
        S.ns = 2;
        S.hy = (ny + 1) / 2;
        S.slot[1] = {3, 1, o180, 0};
    } else if (mx) {
        S.ns = 2;
        S.hx = (nx + 1) / 2;
        S.slot[1] = {1, -1, ox, 1};
    } else if (my) {
        S.ns = 2;
        S.hy = (ny + 1) / 2;
        S.slot[1] = {2, -1, oy, 1};
    }
    return S;
}

void back2_choose(Back2Args &A, bool fours) {
    // Predicted time in us.  A view of a tile costs each thread its pixels' geometry and taps and the staging
    // (`scale` us per instruction); CTAs of an SM share its issue slots, one alone taking `alone` times its
    // share, and a few rounds of them even out less than many.  The pixel-by-pixel kernel waits out each
    // chunk's copies, the other overlaps them but no chunk takes less.  Summing a split and interleaving slices
    // take the rest.  Fitted to 5000 launches of 300 scans (48 to 640 pixels a side, 45 to 1200 views, 1 to 16
    // slices, every form and split): the choice takes 3 % more than the fastest launch of its scan in the
    // geometric mean.  Every pixel by itself with views split by SMs alone took 20 % more than the choice; on
    // 17 scans, most of 7 to 15 us, 3 to 10 % less.
    struct Cost {
        double par, flat, arc, tap, base, seg, scale, alone, uneven, chunk, split, rank, sum;
    };
    static const Cost plain = {3.95, 8.24, 18.4, 2.93, 6.72, 70.9, 0.0013, 2.73, 0.145, 0.81, 1.11, 0.059, 0.702},
                      slots = {0.094, 0.474, 4.99, 2.53, 14.1, 31.4, 0.00203, 2.71, 0.211, 2.93, 1.66, 0.108, 0.36},
                      slices = {7.96, 1.83, 7.46, 2.19, 8.73, 38, 0.00206, 2.68, 0.161, 5.3, 2.17, 0.72, 0.25};
    const int sms = std::max(1, num_sms());
    Back2Args best = A;
    double best_us = 1e30;
    for (int form : {B2_FORM_SLOTS, B2_FORM_PLAIN, B2_FORM_FOURS}) {
        const int ns = form == B2_FORM_SLOTS ? A.sym.ns : 1, sl = form == B2_FORM_FOURS ? 4 : 1, n = ns * sl;
        if (A.want_form != B2_FORM_AUTO && form != A.want_form && !(A.want_form == B2_FORM_FOURS && !fours)) continue;
        if (sl == 4 && (!fours || (A.nslices == 1 && A.want_form != B2_FORM_FOURS))) continue;
        const Cost &c = n == 1 ? plain : (sl == 4 ? slices : slots);
        const int ctas = n == 1 ? kB2PlainCtas : kB2Ctas;
        const int hx = ns > 1 ? A.sym.hx : A.nx, hy = ns > 1 ? A.sym.hy : A.ny;
        const long long groups = floor_div_up(A.nslices, sl);
        const double all = (double)floor_div_up(hx, kB2X) * floor_div_up(hy, kB2Y * kB2P) * groups;
        const long long tiles = std::max(1LL, (long long)std::ceil(all * A.wanted));
        const double geometry = A.mode == SGB_PAR ? c.par : (A.mode == SGB_FLAT ? c.flat : c.arc);
        const double view = c.scale * (kB2P * (geometry + ns * c.tap) + c.base + n * A.w / c.seg);
        for (int g = 1; g <= 8 && groups * g <= 65535; g++) {
            if (A.want_split ? g != A.want_split
                             // eight views a rank at least; and the tiles alone may fill the chip
                             : g > 1 && (A.nv < 8 * g || tiles >= 2LL * ctas * sms)) continue;
            const long long busiest = (tiles * g + sms - 1) / sms;
            const double waves = (double)(busiest / ctas), rest = (double)(busiest % ctas), rounds = waves + (rest > 0);
            const double share = (waves * std::max(c.alone, (double)ctas) + (rest ? std::max(c.alone, rest) : 0)) *
                                 (1 + c.uneven / rounds);
            const int views = floor_div_up(A.nv, g);
            const int vc = n == 1 ? kB2V : std::max(1, std::min(kB2V, kB2Seg / 2 / (n * A.w * 4)));
            double us = 0;
            if (n == 1) {
                us = views * view * share + floor_div_up(views, vc) * c.chunk * rounds;
            } else {
                const int full = views / vc, left = views % vc;
                us = full * std::max(vc * view * share, c.chunk * rounds) +
                     (left ? std::max(left * view * share, c.chunk * rounds) : 0);
            }
            if (g > 1) us += c.split + c.rank * g + c.sum * n * (double)(tiles * g) / sms;
            if (sl == 4) us += 8 + 1.2e-5 * A.nb * (double)A.na * A.nslices;
            if (us < best_us) {
                best_us = us;
                best.sym.ns = ns;
                best.sl = sl;
                best.split = g;
                best.sym.hx = hx;
                best.sym.hy = hy;
                best.sym.turn = ns > 1 ? A.sym.turn : 0;
            }
        }
    }
    A = best;
}

int launch_back2(const Back2Args &A, cudaStream_t st) {
    if (A.nx <= 0 || A.ny <= 0 || A.nslices <= 0) return SGB_OK;
    SGB_REQUIRE(A.nslices <= 65535, "fbp back-projection: too many slices");
    switch (A.mode) {
    case SGB_PAR: return launch_back2_par(A, st);
    case SGB_ARC: {
        // the angle polynomials cover |r/d| <= 0.6 (6 terms) and <= 1 (9 terms): detectors whose
        // taps stay inside +-atan(0.6) or +-45 deg (with a 4-bin margin) use them, wider ones atan2f
        const double half = (std::max(std::fabs(1.0 - A.wb), std::fabs((double)A.nb - A.wb)) + 4.0) / A.dsd_ds;
        if (half < 0.5404195002705842) return launch_back2_arc_narrow(A, st);
        return half < 0.7853981633974483 ? launch_back2_arc(A, st) : launch_back2_arc_exact(A, st);
    }
    default: return launch_back2_flat(A, st);
    }
}

}  // namespace sgb
