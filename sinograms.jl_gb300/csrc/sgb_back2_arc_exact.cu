// sgb_back2_arc_exact.cu -- 2D back-projection, arc detector wider than +-45 degrees.
#include "sgb_back2_kernel.cuh"

namespace sgb {

int launch_back2_arc_exact(const Back2Args &A, cudaStream_t st) { return back2::launch<back2::B2_ARC_EXACT>(A, st); }

}  // namespace sgb
