// sgb_fdk_mirror_pair_arc.cu -- mirrored FDK back-projection of FP32 pairs, arc detector.
#include "sgb_fdk_mirror_pair.cuh"

namespace sgb {

int launch_fdk_mirror_pair_arc(const FdkMirrorArgs &M, const CUtensorMap &map, cudaStream_t st) {
    return fdkdev::launch_mirror_pair<true>(M, map, st);
}

}  // namespace sgb
