// sgb_fdk_mirror.cuh -- launch interface of the mirrored FDK back-projector (internal; the method
// is described in sgb_fdk_mirror_kernel.cuh).
#pragma once
#include "sgb_fdk_tma.cuh"

namespace sgb {

// Reflections of a view slot: the voxel column's x and/or y changes sign.
enum { MIR_X = 1, MIR_Y = 2 };

struct FdkMirrorArgs {
    FdkTmaArgs A;    // the scan; W, H, box_bytes and nstage of the mirrored boxes
    int nvs;         // view slots (1, 2 or 4): columns of one thread, each with the view that sees it alike
    int zm;          // 1: each slot also takes the voxels at -z
    int kz;          // voxels along z per slot and thread
    int split;       // CTAs of a cluster that share a tile's views
    int hx, hy;      // columns of the fundamental domain
    int iz0, nzd;    // its first z index and its z extent
    int nviews;      // views of the scan
    int zbase;       // FP16 quads: voxels between the anchors of the 2^-10 t grid (sgb_fdk_tma_dev.cuh)
    int exact;       // the FP32 voxel grid is exactly symmetric
    int m2;          // zm: detector row i and row m2 - i see z and -z
    int flip[4], vsgn[4], voff[4];  // slot j: reflection, and its view (vsgn v + voff) mod nviews
};

// Slots of a scan's symmetry (nvs and zm; 1 and 0 when it has none that the storage form can use).
void fdk_mirror_slots(FdkMirrorArgs &M, const FdkTmaArgs &A, double orbit, double orbit_start, const double *offsets,
                      double offset_t);
// Predicted time in us of the unmirrored kernel, prepared with its run length and box.
double fdk_tma_predict(const FdkTmaArgs &A);
// Run length, view split, box (device pre-pass) and ring; false when the mirrored boxes do not fit shared memory
// or no launch is predicted to take less than limit_us.
int fdk_mirror_prepare(FdkMirrorArgs &M, int *ext_dev, cudaStream_t st, double limit_us, bool *fits);
int launch_fdk_mirror(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st);
size_t fdk_mirror_smem(const FdkMirrorArgs &M, int nstage);
// one storage form and detector each (sgb_fdk_mirror_<form>_<detector>.cu)
int launch_fdk_mirror_pair_flat(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st);
int launch_fdk_mirror_pair_arc(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st);
int launch_fdk_mirror_quad_flat(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st);
int launch_fdk_mirror_quad_arc(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st);

}  // namespace sgb
