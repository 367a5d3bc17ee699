// sgb_fdk_mirror_pair_flat.cu -- mirrored FDK back-projection of FP32 pairs, flat detector.
#include "sgb_fdk_mirror_pair.cuh"

namespace sgb {

int launch_fdk_mirror_pair_flat(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st) {
    return fdkdev::launch_mirror_pair<false>(M, map, st);
}

}  // namespace sgb
