// sgb_back2_arc.cu -- 2D back-projection, arc detector within +-45 degrees.
#include "sgb_back2_kernel.cuh"

namespace sgb {

int launch_back2_arc(const Back2Args &A, cudaStream_t st) { return back2::launch<back2::B2_ARC>(A, st); }

}  // namespace sgb
