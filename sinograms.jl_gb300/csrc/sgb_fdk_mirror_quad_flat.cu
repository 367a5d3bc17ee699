// sgb_fdk_mirror_quad_flat.cu -- mirrored FDK back-projection of FP16 quads (F16 form), flat detector.
#include "sgb_fdk_mirror_kernel.cuh"

namespace sgb {

int launch_fdk_mirror_quad_flat(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st) {
    using namespace fdkdev;
    if (M.nvs == 4) return M.kz == 16 ? launch_mirror_k<Quad16, false, 4, false, 16>(M, map, st) : launch_mirror_k<Quad16, false, 4, false, 8>(M, map, st);
    return M.kz == 32 ? launch_mirror_k<Quad16, false, 2, false, 32>(M, map, st) : launch_mirror_k<Quad16, false, 2, false, 16>(M, map, st);
}

}  // namespace sgb
