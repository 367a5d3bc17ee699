// sgb_fdk_mirror_pair.cuh -- the mirrored FDK back-projector's FP32 pair instantiations (one detector
// per translation unit).
#pragma once
#include "sgb_fdk_mirror_kernel.cuh"

namespace sgb {
namespace fdkdev {

template <bool ARC>
int launch_mirror_pair(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st) {
    if (M.nvs == 4) return M.kz == 16 ? launch_mirror_k<float2, ARC, 4, false, 16>(M, map, st) : launch_mirror_k<float2, ARC, 4, false, 8>(M, map, st);
    if (M.nvs == 2 && M.zm) return M.kz == 16 ? launch_mirror_k<float2, ARC, 2, true, 16>(M, map, st) : launch_mirror_k<float2, ARC, 2, true, 8>(M, map, st);
    if (M.nvs == 2) return M.kz == 32 ? launch_mirror_k<float2, ARC, 2, false, 32>(M, map, st) : launch_mirror_k<float2, ARC, 2, false, 16>(M, map, st);
    return M.kz == 32 ? launch_mirror_k<float2, ARC, 1, true, 32>(M, map, st) : launch_mirror_k<float2, ARC, 1, true, 16>(M, map, st);
}

}  // namespace fdkdev
}  // namespace sgb
